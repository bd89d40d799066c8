// tdse_adjoint.cu -- gradient of a band-limited harmonic yield with respect to the driving
// field: the adjoint of the FP64 Crank-Nicolson-Numerov propagation (the differentiable form).
//
// Forward model of one instance (tdse_step.cuh; reference 1DTDSE/sources/prop.c:115-347):
//   psi_{k+1} = Phi_k U psi_k,   U = 2 A^{-1} M2 - I,   Phi_k = diag(e^{i F_k dt x_j}),
//   s_{k+1}   = -sum_j |psi_{k+1,j}|^2 gv_j + F_k          (sourceterm, gv = -V')
//   L         = dt^2/(2 pi) sum_{q in Q} |D_q|^2,  D_q = sum_{n<S} s_n e^{-2 pi i q n / S}
// With lambda = dL/dRe psi + i dL/dIm psi and a_n = dL/ds_n:
//   lambda_S = 0 (s_S is not a spectrum sample),
//   dL/dF_k  = a_{k+1} - dt sum_j x_j Im(conj(lambda_{k+1,j}) psi_{k+1,j})
//   lambda_k = U^H Phi_k^H lambda_{k+1} - 2 a_k gv .* psi_k,   U^H mu = 2 M2 (A^H)^{-1} mu - mu,
// A^H solved with its own factorisation (build_grids_kernel, adj_tab) by the same
// partitioned solve.  The forward pass stores psi every K steps (ckpt_*); going backwards,
// each segment is recomputed forwards from its checkpoint into a per-CTA history, then
// swept backwards.  Cost: about three forward passes.  Batches that leave SMs idle spread each
// instance over a thread-block cluster (adjoint_cluster_kernel).
#include <cuda_runtime.h>

#include "../../include/mma_tdse.h"
#include "common.cuh"
#include "launch.cuh"
#include "tdse_cluster.cuh"
#include "tdse_solver.cuh"
#include "tdse_step.cuh"

namespace mma {
namespace adj {

constexpr double kTwoPi = 6.283185307179586476925286766559;

// ---------------------------------------------------------------------------- loss gradient
// One CTA per instance: D_q over the band by direct sums (angle 2 pi (q n mod S)/S, exact
// integer reduction), L, then a_n = 2 c2 Re(sum_q D_q e^{+2 pi i q n / S}).
__global__ void __launch_bounds__(kThreads) loss_grad_kernel(const mma_tdse_instance* insts, const double* outputs,
                                                             const double* tmax, double dt, double w_lo,
                                                             double w_hi, double* loss, double* a,
                                                             const int64_t* a_off)
{
    extern __shared__ double2 Dq[];  // band coefficients
    __shared__ double red[kWarps];
    const mma_tdse_instance I = insts[blockIdx.x];
    const int64_t S = I.n_steps;
    const double* s = outputs + I.out_off + 2 * (S + 1);
    const double tm = tmax[blockIdx.x];
    int64_t q_lo = (int64_t)ceil(w_lo * tm / kTwoPi), q_hi = (int64_t)floor(w_hi * tm / kTwoPi);
    if (q_lo < 1) q_lo = 1;
    if (q_hi > S / 2) q_hi = S / 2;
    const int64_t nq = q_hi >= q_lo ? q_hi - q_lo + 1 : 0;
    const double c2 = dt * dt / kTwoPi;
    double part = 0.0;
    for (int64_t iq = threadIdx.x; iq < nq; iq += blockDim.x) {
        const int64_t q = q_lo + iq;
        double re = 0.0, im = 0.0;
        for (int64_t n = 0; n < S; n++) {
            double sn, cs;
            sincospi(2.0 * (double)((q * n) % S) / (double)S, &sn, &cs);
            re = fma(s[n], cs, re);
            im = fma(-s[n], sn, im);
        }
        Dq[iq] = make_double2(re, im);
        part += c2 * (re * re + im * im);
    }
    double v[1] = {part};
    block_sum<1>(v, red);
    if (threadIdx.x == 0) loss[blockIdx.x] = v[0];
    double* ai = a + a_off[blockIdx.x];
    for (int64_t n = threadIdx.x; n <= S; n += blockDim.x) {
        double acc = 0.0;
        if (n < S)
            for (int64_t iq = 0; iq < nq; iq++) {
                const int64_t q = q_lo + iq;
                double sn, cs;
                sincospi(2.0 * (double)((q * n) % S) / (double)S, &sn, &cs);
                acc = fma(Dq[iq].x, cs, fma(-Dq[iq].y, sn, acc));
            }
        ai[n] = 2.0 * c2 * acc;
    }
}

// ---------------------------------------------------------------------------- adjoint sweep
struct Args {
    const mma_tdse_instance* insts;
    int n_inst;
    const mma_tdse_grid* grids;
    const double* fields;
    const double* ckpts;
    const double* a;
    const int64_t* a_off;
    double* grad;
    const int64_t* grad_off;
    int* counter;
    cd* scratch;  // per CTA: yl [max_L], history [(max_K + 1) max_L]
    int64_t max_L, max_K;
};

__global__ void __launch_bounds__(kThreads, 1) adjoint_fp64_kernel(Args P)
{
    extern __shared__ double2 smem_dyn[];
    cd* lam = reinterpret_cast<cd*>(smem_dyn);  // lambda, chunk-interleaved, [L]
    __shared__ cd sc[2 * kWarps], sb[2 * kWarps];
    __shared__ double red[kWarps];
    __shared__ int64_t s_inst, s_gate;
    const int t = threadIdx.x;
    cd* yl = P.scratch + (int64_t)blockIdx.x * (P.max_K + 2) * P.max_L;
    cd* hist = yl + P.max_L;

    for (;;) {
        if (t == 0) s_inst = atomicAdd(P.counter, 1);
        __syncthreads();
        const int64_t inst = s_inst;
        if (inst >= P.n_inst) break;
        const mma_tdse_instance I = P.insts[inst];
        const mma_tdse_grid G = P.grids[I.grid];
        const int64_t n = G.n, m = G.m, L = m * kThreads, S = I.n_steps, K = I.ckpt_every;
        const cd* ctab = reinterpret_cast<const cd*>(G.cn_tab);
        const cd* atab = reinterpret_cast<const cd*>(G.adj_tab);
        const cd *GVX = ctab + CN_GVX * L;
        const cd *aib = atab + CN_IB6 * L, *ah = atab + CN_H * L, *aF = atab + CN_F * L, *ag = atab + CN_G * L,
                 *aG = atab + CN_GG * L;
        const double* f = P.fields + I.field_off;
        const double* ai = P.a + P.a_off[inst];
        double* gi = P.grad + P.grad_off[inst];
        const double dt = G.dt, dx = G.dx;
        if (L > P.max_L || K > P.max_K) {  // wider than the launch was sized for: a NaN gradient
            for (int64_t e = t; e < S; e += kThreads) gi[e] = __longlong_as_double(0x7ff8000000000000LL);
            __syncthreads();
            continue;
        }
        if (t == 0) s_gate = gate_index(f, I.n_field, S, I.gate_floor);
        for (int64_t i = 0; i < m; i++) lam[i * kThreads + t] = cd{0.0, 0.0};  // lambda_S = 0
        __syncthreads();
        const int64_t gate = s_gate;
        const int64_t s0 = t * m;
        const double xs = (s0 < n) ? GVX[t].im : 0.0;
        auto field = [&](int64_t k) { return (k <= gate || k >= I.n_field) ? 0.0 : f[k]; };
        const int64_t nseg = (S + K - 1) / K;
        for (int64_t c = nseg - 1; c >= 0; c--) {
            const int64_t k0 = c * K, k1 = (k0 + K < S) ? k0 + K : S;
            // ---- recompute states k0 .. k1 into the history (hist[h] = psi_{k0+h})
            const double* cp = P.ckpts + I.ckpt_off + c * 2 * n;
            for (int64_t i = 0; i < m; i++) {
                const int64_t j = s0 + i;
                hist[i * kThreads + t] = (j < n) ? ld2(cp + 2 * j) : cd{0.0, 0.0};
            }
            __syncthreads();
            for (int64_t k = k0; k < k1; k++) {
                cd* cur = hist + (k - k0) * P.max_L;
                cd* nxt = cur + P.max_L;
                for (int64_t i = 0; i < m; i++) nxt[i * kThreads + t] = cur[i * kThreads + t];
                __syncthreads();
                cn_step_fp64(nxt, yl, ctab, m, L, field(k), dt, dx, xs, sc, sb, [](int64_t, int64_t, const cd&) {});
                __syncthreads();
            }
            // ---- adjoint steps k = k1-1 .. k0
            for (int64_t k = k1 - 1; k >= k0; k--) {
                const cd* pnext = hist + (k + 1 - k0) * P.max_L;
                const cd* pcur = hist + (k - k0) * P.max_L;
                const double Fk = field(k);
                double sn, cs;
                sincos(Fk * dt * xs, &sn, &cs);
                cd ph{cs, sn};
                sincos(Fk * dt * dx, &sn, &cs);
                const cd z{cs, sn};
                // pass A: gradient term, mu = conj(Phi) lambda, forward sweep of A^H z = mu
                double gsum = 0.0;
                cd yprev{0.0, 0.0};
                for (int64_t i = 0; i < m; i++) {
                    const int64_t q = i * kThreads + t;
                    const cd l = lam[q], p = pnext[q];
                    gsum = fma(GVX[q].im, l.re * p.im - l.im * p.re, gsum);  // x Im(conj(l) p)
                    const cd mu{fma(ph.re, l.re, ph.im * l.im), fma(ph.re, l.im, -ph.im * l.re)};
                    ph = cmul(ph, z);
                    lam[q] = mu;
                    const cd y = cfms(ah[q], yprev, cmul(aib[q], mu));
                    yl[q] = y;
                    yprev = y;
                }
                const cd yin = scan_forward<cd>(aF[(m - 1) * kThreads + t], yprev, sc, sb);
                cd unext{0.0, 0.0};
                for (int64_t i = m - 1; i >= 0; i--) {
                    const int64_t q = i * kThreads + t;
                    const cd y = cfma(aF[q], yin, yl[q]);
                    const cd u = cfms(ag[q], unext, y);
                    yl[q] = u;
                    unext = u;
                }
                const cd uin = scan_backward<cd>(aG[t], unext, sc + kWarps, sb + kWarps);
                for (int64_t i = 0; i < m; i++) {
                    const int64_t q = i * kThreads + t;
                    yl[q] = cfma(aG[q], uin, yl[q]);  // z = (A^H)^{-1} mu
                }
                double v[1] = {gsum};
                block_sum<1>(v, red);  // also orders the z writes before the neighbour reads
                if (t == 0) gi[k] = ai[k + 1] - dt * v[0];
                // pass D: lambda_k = 2 M2 z - mu - 2 a_k gv psi_k  (2 M2 z = (z_- + 10 z + z_+)/6)
                const double ak = ai[k];
                cd zm = (t == 0) ? cd{0.0, 0.0} : yl[(m - 1) * kThreads + t - 1];
                cd zc = yl[t];
                for (int64_t i = 0; i < m; i++) {
                    const int64_t q = i * kThreads + t;
                    const cd zn = (i + 1 < m) ? yl[q + kThreads] : ((t + 1 < kThreads) ? yl[t + 1] : cd{0.0, 0.0});
                    const cd mu = lam[q], p = pcur[q];
                    const double w = -2.0 * ak * GVX[q].re;
                    cd l{(zm.re + zn.re + 10.0 * zc.re) / 6.0 - mu.re + w * p.re,
                         (zm.im + zn.im + 10.0 * zc.im) / 6.0 - mu.im + w * p.im};
                    if (s0 + i >= n) l = cd{0.0, 0.0};
                    lam[q] = l;
                    zm = zc;
                    zc = zn;
                }
                __syncthreads();
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------- adjoint sweep, cluster
// The same sweep with an instance spread over a cluster (tdse_cluster.cu has the scheme).  lambda, psi
// and the sweep buffer stay in shared memory with the tables of the phase at hand: the step's while a
// segment is recomputed, those of A^H while it is swept back (reloaded from L2 once per segment).
// An adjoint step needs two cluster barriers: z beside the chunk is known without an exchange, on the
// right as the carry z_in of the backward scan, on the left as y_in - g z_first (y_in the carry of the
// forward scan), so lambda_k = 2 M2 z - mu - 2 a_k gv psi_k follows in the pass that makes z.
// Bound by the FP64 pipe: about 30 + 40 operations per site and step and 200 per thread.
// Per step of one 8001-site instance: 269 us on one CTA, 23 us on a cluster of 16; 64 instances 272 ->
// 114 us (36 clusters of 4).
struct ClusterArgs {
    Args A;
    int m_cap;
    int64_t hist_stride;  // complex entries of one state in a cluster's history
};

constexpr int kGradRing = 8;
static_assert(4 * kGradRing == 32, "one warp sums the collected steps");

__host__ __device__ inline size_t adj_site_bytes() { return 6 * 16; }
__host__ __device__ inline size_t adj_fixed_bytes(int nc)
{
    using namespace clk;
    const size_t nw = (size_t)nc * kW;
    return 16 * (2 * nw + 2 * kW * nw + 2 * kPhSteps * kPh) + 8 * kGradRing * nw;
}

__global__ void __launch_bounds__(clk::kT, 1) adjoint_cluster_kernel(ClusterArgs Q)
{
    using namespace clk;
    typedef Fp64 N;
    const Args& P = Q.A;
    cg::cluster_group cluster = cg::this_cluster();
    const int NC = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), NW = NC * kW;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, g = rank * kW + w;
    extern __shared__ __align__(16) unsigned char smem[];
    const int ML = Q.m_cap * kT;
    cd* const lam = reinterpret_cast<cd*>(smem);
    cd *const psi = lam + ML, *const yv = psi + ML, *const ib = yv + ML, *const hh = ib + ML, *const gg = hh + ML;
    cd *const totF = gg + ML, *const totB = totF + NW, *const wtF = totB + NW, *const wtB = wtF + kW * NW,
              *const phs = wtB + kW * NW;
    double* const ring = reinterpret_cast<double*>(phs + 2 * kPhSteps * kPh);
    Scan<N> scan(cluster, totF, totB, wtF, wtB);
    __shared__ cd edge[2];
    __shared__ int s_inst;
    __shared__ long long s_gate;

    for (;;) {
        cluster.sync();
        if (rank == 0 && t == 0) {
            const int v = atomicAdd(P.counter, 1);
            for (int r = 0; r < NC; r++) *cluster.map_shared_rank(&s_inst, r) = v;
        }
        cluster.sync();
        const int inst = s_inst;
        if (inst >= P.n_inst) break;
        const mma_tdse_instance I = P.insts[inst];
        const mma_tdse_grid G = P.grids[I.grid];
        const int64_t S = I.n_steps, K = I.ckpt_every;
        const int n = (int)G.n, m256 = (int)G.m;
        const int64_t L = G.m * kThreads;
        const cd* ctab = reinterpret_cast<const cd*>(G.cn_tab);
        const cd* atab = reinterpret_cast<const cd*>(G.adj_tab);
        const double* f = P.fields + I.field_off;
        const double* ai = P.a + P.a_off[inst];
        double* gi = P.grad + P.grad_off[inst];
        const double dt = G.dt, dx = G.dx, x0 = G.x[0];
        const int m = (n + NC * kT - 1) / (NC * kT);
        if (L > P.max_L || m > Q.m_cap || K > P.max_K) {  // wider than the launch was sized for
            for (int64_t e = (int64_t)rank * kT + t; e < S; e += NC * kT) gi[e] = __longlong_as_double(0x7ff8000000000000LL);
            continue;
        }
        const int c0 = rank * kT + t, s0 = c0 * m;
        // this cluster's history, [state][site of the chunk][chunk]
        cd* const hist = P.scratch + (int64_t)(blockIdx.x / NC) * (P.max_K + 1) * Q.hist_stride + c0;
        const int64_t row = NC * kT;
        auto hst = [&](int64_t h, int i) { return hist + h * Q.hist_stride + i * row; };
        if (t == 0) {
            s_gate = S;
            // the grid's ends; every other edge comes from its neighbour, perhaps already
            if (rank == 0) edge[0] = N::zero();
            if (rank == NC - 1) edge[1] = N::zero();
        }
        __syncthreads();
        for (int64_t b = 0; b < S; b += kT) {
            const int64_t k = b + t;
            bool hit = false;
            if (k < S) {
                double fa = (k < I.n_field) ? f[k] : 0.0, fb = (k + 1 < I.n_field) ? f[k + 1] : 0.0;
                if (fabs(fa) <= I.gate_floor) fa = 0.0;
                if (fabs(fb) <= I.gate_floor) fb = 0.0;
                hit = fa * fb <= 0.0;
                if (hit) atomicMin(&s_gate, (long long)k);
            }
            if (__syncthreads_or(hit)) break;
        }
        __syncthreads();
        const int64_t gate = s_gate;
        auto applied = [&](int64_t k) { return (k < 0 || k <= gate || k >= I.n_field) ? 0.0 : f[k]; };
        // the tables of the step (tab = cn_tab) or of A^H, and the scans' constants for them; returns g
        // of the site before the chunk.  Contains cluster barriers.
        auto load_tables = [&](const cd* tab) {
            cd cF = N::one(), cB = N::one(), gprev = N::zero();
            for (int i = 0; i < m; i++) {
                const int j = s0 + i, q = i * kT + t;
                cd a = N::zero(), h = a, gq = a;
                if (j < n) {
                    const int64_t e = (int64_t)(j % m256) * kThreads + j / m256;
                    a = tab[CN_IB6 * L + e];
                    h = tab[CN_H * L + e];
                    gq = tab[CN_G * L + e];
                }
                ib[q] = a;
                hh[q] = h;
                gg[q] = gq;
                cF = N::mul(cF, N::neg(h));
                cB = N::mul(cB, N::neg(gq));
            }
            if (s0 > 0 && s0 - 1 < n)
                gprev = tab[CN_G * L + (int64_t)((s0 - 1) % m256) * kThreads + (s0 - 1) / m256];
            scan.setup(cluster, cF, cB);
            return gprev;
        };
        auto send_edges = [&] {
            if (t == 0 && rank > 0) *cluster.map_shared_rank(&edge[1], rank - 1) = psi[0];
            if (t == kT - 1 && rank + 1 < NC) *cluster.map_shared_rank(&edge[0], rank + 1) = psi[(m - 1) * kT + t];
        };
        // phases of the steps k0, k0 + dir, ... into half `b` of the table: e^{i F dt x} at site `site` of
        // the warps' first chunks and the factors between chunks, then e^{-dir' i F dt dx}
        auto phases = [&](int64_t k0, int dir, int site, int half) {
            if (t >= kPhSteps * kPh) return;
            const int a = t % kPh;
            const int64_t k = k0 + dir * (t / kPh);
            const double Fdt = (k < S ? applied(k) : 0.0) * dt, step = (double)m * dx;
            double ang;
            if (a < kPhA) ang = Fdt * (step * (4 * a));
            else if (a < kPhA + kPhB) ang = Fdt * (step * (a - kPhA));
            else if (a < kPh - 1) ang = Fdt * (x0 + dx * (double)((rank * kT + 32 * (a - kPhA - kPhB)) * m + site));
            else ang = -(double)dir * (Fdt * dx);
            double sn, cs;
            sincos(ang, &sn, &cs);
            phs[half * kPhSteps * kPh + t] = cd{cs, sn};
        };
        auto start_phase = [&](const cd* ps) {
            return cmul(cmul(ps[lane >> 2], ps[kPhA + (lane & 3)]), ps[kPhA + kPhB + w]);
        };
        for (int i = 0; i < m; i++) lam[i * kT + t] = N::zero();  // lambda_S = 0
        // rank 0: the gradient of steps k, k - 1, ... (cnt of them) from ring slots slot0, slot0 + 1, ...
        auto flush = [&](int64_t k, int cnt) {
            if (w == 0) {  // four lanes a step; the whole warp shuffles
                const int sl = lane / 4;
                double s = 0.0;
                if (sl < cnt)
                    for (int q = lane % 4; q < NW; q += 4) s += ring[sl * NW + q];
                s += shfl_xor(s, 1);
                s += shfl_xor(s, 2);
                if (sl < cnt && lane % 4 == 0) gi[k - sl] = ai[k - sl + 1] - dt * s;
            }
        };

        const int64_t nseg = (S + K - 1) / K;
        for (int64_t c = nseg - 1; c >= 0; c--) {
            const int64_t k0 = c * K, k1 = (k0 + K < S) ? k0 + K : S;
            // ---- recompute states k0 .. k1 into the history
            const double* cp = P.ckpts + I.ckpt_off + c * 2 * n;
            for (int i = 0; i < m; i++) {
                const int j = s0 + i;
                const cd v = (j < n) ? ld2(cp + 2 * j) : N::zero();
                psi[i * kT + t] = v;
                *hst(0, i) = v;
            }
            send_edges();
            phases(k0, 1, m - 1, 0);
            load_tables(ctab);  // its barriers also publish the edges and the phases
            for (int64_t k = k0; k < k1; k++) {
                const int64_t e = k - k0;
                const int kp = (int)(e % kPhSteps);
                cd pm = (t == 0) ? edge[0] : psi[(m - 1) * kT + t - 1];
                const cd nx = (t == kT - 1) ? edge[1] : psi[t + 1];
                cd pc = psi[t];
                cd b = N::zero();
#pragma unroll 2
                for (int i = 0; i < m; i++) {
                    const int q = i * kT + t;
                    const cd pn = (i + 1 < m) ? psi[q + kT] : nx;
                    const cd r = N::rhs(ib[q], pc, pm, pn);
                    yv[q] = r;
                    b = cfms(hh[q], b, r);
                    pm = pc;
                    pc = pn;
                }
                b = scan.forward_out(cluster, b);
                cluster.barrier_arrive();
                if (kp == kPhSteps - 1) phases(k + 1, 1, m - 1, (int)((e / kPhSteps + 1) % 2));
                cd bx = N::shup(b, 1);
                cluster.barrier_wait();
                cd y = scan.forward_in(bx);
#pragma unroll 2
                for (int i = 0; i < m; i++) {
                    const int q = i * kT + t;
                    y = cfms(hh[q], y, yv[q]);
                    yv[q] = y;
                }
                b = y;
#pragma unroll 2
                for (int i = m - 2; i >= 0; i--) {
                    const int q = i * kT + t;
                    b = cfms(gg[q], b, yv[q]);
                }
                b = scan.backward_out(cluster, b);
                cluster.barrier_arrive();
                bx = N::shdn(b, 1);
                const cd* ps = phs + ((int)(e / kPhSteps % 2) * kPhSteps + kp) * kPh;
                cd ph = start_phase(ps);
                const cd zc = ps[kPh - 1];
                cluster.barrier_wait();
                cd u = scan.backward_in(bx);
#pragma unroll 2
                for (int i = m - 1; i >= 0; i--) {
                    const int q = i * kT + t;
                    u = cfms(gg[q], u, yv[q]);
                    const cd pn = N::update(ph, u, psi[q]);
                    psi[q] = pn;
                    *hst(e + 1, i) = pn;
                    ph = cmul(ph, zc);
                }
                send_edges();
                cluster.sync();
            }
            // ---- adjoint steps k = k1 - 1 .. k0; psi holds state k + 1
            phases(k1 - 1, -1, 0, 0);
            const cd gprev = load_tables(atab);
            for (int64_t k = k1 - 1; k >= k0; k--) {
                const int64_t e = k1 - 1 - k;
                const int kp = (int)(e % kPhSteps);
                const double ak2 = -2.0 * ai[k];
                const cd* ps = phs + ((int)(e / kPhSteps % 2) * kPhSteps + kp) * kPh;
                cd ph = start_phase(ps);
                const cd z = ps[kPh - 1];
                // gradient term, mu = conj(Phi) lambda, forward sweep of A^H z = mu
                double gsum = 0.0;
                cd b = N::zero();
#pragma unroll 2
                for (int i = 0; i < m; i++) {
                    const int q = i * kT + t;
                    const cd l = lam[q], p = psi[q];
                    const double x = x0 + dx * (double)(s0 + i);
                    gsum = fma(x, fma(l.re, p.im, -l.im * p.re), gsum);  // x Im(conj(l) p)
                    const cd mu{fma(ph.re, l.re, ph.im * l.im), fma(ph.re, l.im, -ph.im * l.re)};
                    ph = cmul(ph, z);
                    lam[q] = mu;
                    const cd r = cmul(ib[q], mu);
                    yv[q] = r;
                    b = cfms(hh[q], b, r);
                }
                b = scan.forward_out(cluster, b);
#pragma unroll
                for (int d = 16; d >= 1; d >>= 1) gsum += shfl_xor(gsum, d);
                if (lane == 0) cluster.map_shared_rank(ring, 0)[(int)(e % kGradRing) * NW + g] = gsum;
                cluster.barrier_arrive();
                if (kp == kPhSteps - 1) phases(k - 1, -1, 0, (int)((e / kPhSteps + 1) % 2));
                cd bx = N::shup(b, 1);
                cluster.barrier_wait();
                if (rank == 0 && (e % kGradRing == kGradRing - 1 || k == k0))
                    flush(k + e % kGradRing, (int)(e % kGradRing) + 1);
                const cd yin = scan.forward_in(bx);
                cd y = yin;
#pragma unroll 2
                for (int i = 0; i < m; i++) {
                    const int q = i * kT + t;
                    y = cfms(hh[q], y, yv[q]);
                    yv[q] = y;
                }
                b = y;
#pragma unroll 2
                for (int i = m - 2; i >= 0; i--) {
                    const int q = i * kT + t;
                    b = cfms(gg[q], b, yv[q]);
                }
                b = scan.backward_out(cluster, b);
                cluster.barrier_arrive();
                bx = N::shdn(b, 1);
                // psi_k and -V' of the next site, one iteration ahead of their use
                cd pre_p;
                double pre_v;
                auto prefetch = [&](int i) {
                    const int j = s0 + i < n ? s0 + i : n - 1;
                    pre_p = *hst(k - k0, i);
                    pre_v = ctab[CN_GVX * L + (int64_t)(j % m256) * kThreads + j / m256].re;
                };
                prefetch(m - 1);
                cluster.barrier_wait();
                // z from the exact carry; lambda_k = 2 M2 z - mu - 2 a_k gv psi_k one site behind it
                cd zn = scan.backward_in(bx), zc = cfms(gg[(m - 1) * kT + t], zn, yv[(m - 1) * kT + t]);
#pragma unroll 2
                for (int i = m - 1; i >= 0; i--) {
                    const int q = i * kT + t, j = s0 + i;
                    const cd zm = i > 0 ? cfms(gg[q - kT], zc, yv[q - kT]) : cfms(gprev, zc, yin);
                    const cd p = pre_p, mu = lam[q];
                    const double v = ak2 * pre_v;
                    if (i > 0) prefetch(i - 1);
                    cd l = N::zero();
                    if (j < n) {
                        l = cd{fma(v, p.re, fma(1.0 / 6.0, fma(10.0, zc.re, zm.re + zn.re), -mu.re)),
                               fma(v, p.im, fma(1.0 / 6.0, fma(10.0, zc.im, zm.im + zn.im), -mu.im))};
                    }
                    lam[q] = l;
                    psi[q] = p;  // state k, the next step's psi_{k+1}
                    zn = zc;
                    zc = zm;
                }
            }
            cluster.sync();  // the last step's carries are read before the next tables' constants replace them
        }
    }
}

}  // namespace adj
}  // namespace mma

using namespace mma;

namespace {

// Expected us per step (recompute and adjoint) of the whole batch, fitted to runs (measured / model):
// one CTA 301 sites 41.9 / 41.7, 2001 sites 85.5 / 87.3, 8001 sites 269 / 270; cluster 8001 sites
// NC = 4 55.6 / 54.2, 8 33.4 / 32.6, 16 23.0 / 21.8, 301 sites NC = 4 13.1 / 13.7.
double adj_one_cta_us(int m256, int n_inst, int sms) { return (double)((n_inst + sms - 1) / sms) * (26.5 + 7.6 * m256); }
double adj_cluster_us(int m, int n_inst, int run, int nc, int sms)
{
    const int full = n_inst / run, rest = n_inst % run;
    const double one = 11.0 + 2.7 * m, two = 1.25 * one;  // two CTAs of the launch on an SM: 1.1 to 1.5 measured
    return full * (run * nc > sms ? two : one) + (rest == 0 ? 0.0 : rest * nc > sms ? two : one);
}

cudaLaunchConfig_t adj_config(int nc, int clusters, size_t smem, cudaStream_t st, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(clusters * nc));
    cfg.blockDim = dim3(clk::kT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)nc;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

struct AdjCluster {
    int nc, m, clusters;
    size_t smem;
};

// The cluster size with the least expected time, or false where one CTA per instance is expected to
// finish sooner.  A cluster's history needs (K + 1) states in the caller's scratch.
bool choose_adj_cluster(int max_m, int K, int n_inst, int sms, size_t scratch_bytes, AdjCluster* out)
{
    auto kern = adj::adjoint_cluster_kernel;
    double best = adj_one_cta_us(max_m, n_inst, sms);
    bool found = false;
    for (int nc = clk::kMaxNC; nc >= 1; nc--) {
        const int m = (max_m * kThreads + nc * clk::kT - 1) / (nc * clk::kT);
        const size_t smem = (size_t)m * clk::kT * adj::adj_site_bytes() + adj::adj_fixed_bytes(nc);
        const size_t hist = sizeof(cd) * (size_t)(K + 1) * nc * clk::kT * m;
        if (smem > 226 * 1024 || (nc > 1 && (nc - 1) * m * clk::kT >= max_m * kThreads) || scratch_bytes < hist) continue;
        int run = sms * (smem > 112 * 1024 ? 1 : 2) / nc;  // if every SM could be filled
        if ((size_t)run > scratch_bytes / hist) run = (int)(scratch_bytes / hist);
        if (run > n_inst) run = n_inst;
        if (run < 1 || adj_cluster_us(m, n_inst, run, nc, sms) >= best) continue;
        if (allow_smem(kern) != cudaSuccess ||
            !succeeded(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
            return false;
        cudaLaunchAttribute at{};
        cudaLaunchConfig_t cfg = adj_config(nc, 1, smem, nullptr, &at);
        int active = 0;
        if (!succeeded(cudaOccupancyMaxActiveClusters(&active, kern, &cfg)) || active < 1) continue;
        if (run > active) run = active;
        const double us = adj_cluster_us(m, n_inst, run, nc, sms);
        if (us < best) {
            best = us;
            *out = AdjCluster{nc, m, run, smem};
            found = true;
        }
    }
    return found;
}

}  // namespace

extern "C" int mma_tdse_loss_grad(const mma_tdse_instance* insts, int n_inst, const double* outputs,
                                  const double* tmax, double dt, double w_lo, double w_hi, double* loss, double* a,
                                  const int64_t* a_off, void* stream)
{
    if (n_inst <= 0) return MMA_OK;
    if (!insts || !outputs || !tmax || !loss || !a || !a_off || !(dt > 0.0) || !(w_hi >= w_lo)) return MMA_ERR_ARG;
    // the band holds at most S/2 bins; 12288 bins of shared memory cover S <= 24576
    const size_t smem = sizeof(double2) * 12288;
    cudaFuncSetAttribute(adj::loss_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    adj::loss_grad_kernel<<<n_inst, kThreads, smem, (cudaStream_t)stream>>>(insts, outputs, tmax, dt, w_lo, w_hi,
                                                                           loss, a, a_off);
    return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
}

extern "C" size_t mma_tdse_adjoint_scratch_bytes(int max_m, int max_ckpt_every, int grid_ctas)
{
    if (grid_ctas <= 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        grid_ctas = sms > 0 ? sms : 1;
    }
    const size_t L = (size_t)max_m * kThreads;
    return sizeof(cd) * L * ((size_t)max_ckpt_every + 2) * (size_t)grid_ctas;
}

extern "C" int mma_tdse_adjoint(const mma_tdse_instance* insts, int n_inst, const mma_tdse_grid* grids,
                                const mma_tdse_buffers* bufs, const double* a, const int64_t* a_off, double* grad,
                                const int64_t* grad_off, int max_m, int max_ckpt_every, int grid_ctas, void* stream)
{
    if (n_inst <= 0) return MMA_OK;
    if (!insts || !grids || !bufs || !bufs->fields || !bufs->snapshots || !bufs->counter || !bufs->scratch || !a ||
        !a_off || !grad || !grad_off || max_m < 1 || max_ckpt_every < 1)
        return MMA_ERR_ARG;
    const size_t smem = (size_t)max_m * kThreads * sizeof(cd);
    if (smem > 220 * 1024) return MMA_ERR_TOO_LARGE;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MMA_ERR_NO_DEVICE;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (grid_ctas <= 0) grid_ctas = sms;
    if (grid_ctas > n_inst) grid_ctas = n_inst;
    if (bufs->scratch_bytes < mma_tdse_adjoint_scratch_bytes(max_m, max_ckpt_every, grid_ctas)) return MMA_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(bufs->counter, 0, sizeof(int), st) != cudaSuccess) return MMA_ERR_CUDA;
    adj::Args A{insts, n_inst, grids, bufs->fields, bufs->snapshots, a, a_off, grad, grad_off, bufs->counter,
                reinterpret_cast<cd*>(bufs->scratch), (int64_t)max_m * kThreads, (int64_t)max_ckpt_every};
    // a caller that asks for fewer CTAs than the batch could use keeps the one-CTA kernel and that limit
    const bool limited = grid_ctas < n_inst && grid_ctas < sms;
    AdjCluster ac;
    if (!limited && choose_adj_cluster(max_m, max_ckpt_every, n_inst, sms, bufs->scratch_bytes, &ac)) {
        adj::ClusterArgs Q{A, ac.m, (int64_t)ac.nc * clk::kT * ac.m};
        auto kern = adj::adjoint_cluster_kernel;
        if (allow_smem(kern) != cudaSuccess)
            return MMA_ERR_CUDA;
        cudaLaunchAttribute at{};
        cudaLaunchConfig_t cfg = adj_config(ac.nc, ac.clusters, ac.smem, st, &at);
        return succeeded(cudaLaunchKernelEx(&cfg, kern, Q)) ? MMA_OK : MMA_ERR_CUDA;
    }
    allow_smem(adj::adjoint_fp64_kernel);
    adj::adjoint_fp64_kernel<<<grid_ctas, kThreads, smem, st>>>(A);
    return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
}
