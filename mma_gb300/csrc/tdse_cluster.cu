// tdse_cluster.cu -- the TDSE propagation with one instance spread over a thread-block cluster.
//
// propagate_fp64_kernel and propagate_df64_kernel give an instance one CTA, so a batch smaller than
// the GPU leaves SMs idle and a single call runs on one of 152.  Here a cluster of NC CTAs (1 to 16,
// chosen by the host below) shares one instance: NC x 128 threads each own m contiguous sites, and
// every table, psi and the sweep live in the cluster's shared memory for the whole pulse.
//
// A step is the partitioned solve of tdse_solver.cuh with three differences that keep the work per
// thread small, because at few sites per thread the scans and reductions cost as much as the sites:
//   * the coefficients of the chunk maps Y_t = b_t + c_t Y_{t-1} do not change in time, so every
//     product of them that the scan needs is computed once per instance (registers) and a scan level
//     is one complex multiply-add;
//   * the carry into a warp is sum_k W_k b_{g-1-k} over the earlier warps' totals with constant
//     weights W_k = prod c, cut where |W_k| < 1e-25: with dx = 0.1 and dt = 0.25 the solve decays by
//     0.77 per site and a warp of 4-site chunks needs 2 terms;
//   * each sweep is repeated from its exact carry instead of being corrected with chunk products
//     (F, G of the CN tables): the same operation count, and no tables that depend on the chunking.
// Warp totals travel as remote shared-memory stores to every later (forward) or earlier (backward)
// CTA, each followed by a cluster barrier; a third barrier ends the step with the edge values of psi.
// The observables' warp sums collect in rank 0 for 8 steps and are then summed by all its threads.
//
// Bound by the FP64 pipe of the cluster's SMs (FP64: 40 operations per site and about 100 per thread
// and step, one warp per sub-partition) or by the latency of the scans (float-float); per step, one
// CTA -> cluster: one 8001-site instance 108.8 -> 11.6 us in FP64 and 35.1 -> 5.4 us in float-float
// (NC = 16), 601 sites 24.3 -> 6.7 us (FP64, NC = 8), 24 float-float instances 35.3 -> 8.8 us.
#include <cuda_runtime.h>

#include "launch.cuh"
#include "tdse_cluster.cuh"
#include "tdse_host.cuh"

namespace mma {
namespace clk {

constexpr int kRing = 8, kObs = 5;         // steps of observables collected before they are summed
constexpr int kGroups = 3;                 // thread groups that share those sums (kGroups kRing kObs <= kT)

struct Args {
    const mma_tdse_instance* insts;
    int n_inst;
    const mma_tdse_grid* grids;
    const double* fields;
    double* outputs;
    double* psi_final;
    double* snapshots;
    int* counter;
    int m_cap;      // sites per thread the shared memory was sized for
    int64_t max_L;  // widest grid of the launch (padded sites), as the caller stated it
};

// Dynamic shared memory: per padded site psi, sweep, 1/(6 beta), h, g, (-V', x) [16 bytes each] and
// Re psi0 [8 bytes]; then the warp totals, their weights, the phases and the observables' ring.
__host__ __device__ inline size_t site_bytes() { return 6 * 16 + 8; }
__host__ __device__ inline size_t fixed_bytes(int nc)
{
    const size_t nw = (size_t)nc * kW;
    return 16 * (2 * nw + 2 * kW * nw + 2 * kPhSteps * kPh) + 8 * (kRing * nw * kObs + kGroups * kRing * kObs);
}

template <class N>
__global__ void __launch_bounds__(kT, 1) propagate_cluster_kernel(Args P)
{
    typedef typename N::C C;
    typedef typename N::R R;
    static_assert(sizeof(C) == 16 && sizeof(R) == 8, "shared-memory layout");
    cg::cluster_group cluster = cg::this_cluster();
    const int NC = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), NW = NC * kW;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, g = rank * kW + w;
    extern __shared__ __align__(16) unsigned char smem[];
    const int ML = P.m_cap * kT;
    C* const psi = reinterpret_cast<C*>(smem);
    C *const yv = psi + ML, *const ib = yv + ML, *const hh = ib + ML, *const gg = hh + ML, *const gx = gg + ML;
    C *const totF = gx + ML, *const totB = totF + NW, *const wtF = totB + NW, *const wtB = wtF + kW * NW,
             *const phs = wtB + kW * NW;
    R* const p0 = reinterpret_cast<R*>(phs + 2 * kPhSteps * kPh);
    R* const ring = p0 + ML;
    R* const part = ring + kRing * NW * kObs;
    Scan<N> scan(cluster, totF, totB, wtF, wtB);
    __shared__ C edge[2];
    __shared__ int s_inst;
    __shared__ long long s_gate;
    __shared__ int s_lo, s_hi;
    __shared__ double s_red[kW];

    for (;;) {
        cluster.sync();  // no CTA still reads or writes the previous instance's state
        if (rank == 0 && t == 0) {
            const int v = atomicAdd(P.counter, 1);
            for (int r = 0; r < NC; r++) *cluster.map_shared_rank(&s_inst, r) = v;
        }
        cluster.sync();
        const int inst = s_inst;
        if (inst >= P.n_inst) break;
        const mma_tdse_instance I = P.insts[inst];
        const mma_tdse_grid G = P.grids[I.grid];
        const int64_t S = I.n_steps;
        const int n = (int)G.n, m256 = (int)G.m;
        const int64_t L = G.m * kThreads;
        const double* f = P.fields + I.field_off;
        double* out = P.outputs + I.out_off;
        double *o_t = out, *o_e = out + (S + 1), *o_src = out + 2 * (S + 1), *o_ptot = out + 3 * (S + 1),
               *o_pint = out + 4 * (S + 1), *o_x = out + 5 * (S + 1);
        const double dt = G.dt, dx = G.dx;
        const int m = (n + NC * kT - 1) / (NC * kT);
        if (L > P.max_L || m > P.m_cap) {
            // a grid wider than the launch was sized for: NaN outputs, as in the one-CTA kernel
            for (int64_t e = (int64_t)rank * kT + t; e < 6 * (S + 1); e += NC * kT)
                out[e] = __longlong_as_double(0x7ff8000000000000LL);
            continue;
        }
        const int c0 = rank * kT + t;  // chunk of this thread: sites c0 m .. c0 m + m - 1
        const int s0 = c0 * m;
        // ---- tables of the thread's sites (the grid's tables are interleaved for 256 chunks of m256)
        const C* tab = N::table(G);
        C cF = N::one(), cB = N::one();
        bool im = false;
        for (int i = 0; i < m; i++) {
            const int j = s0 + i, q = i * kT + t;
            C a = N::zero(), h = a, gq = a, x = a, p = a;
            if (j < n) {
                const int64_t e = (int64_t)(j % m256) * kThreads + j / m256;
                a = tab[CN_IB6 * L + e];
                h = tab[CN_H * L + e];
                gq = tab[CN_G * L + e];
                x = tab[CN_GVX * L + e];
                p = tab[CN_PSI0 * L + e];
            }
            ib[q] = a;
            hh[q] = h;
            gg[q] = gq;
            gx[q] = x;
            psi[q] = p;
            p0[q] = N::re(p);
            im |= N::has_im(p);
            cF = N::mul(cF, N::neg(h));
            cB = N::mul(cB, N::neg(gq));
        }
        // ---- zero gate (prop.c:125-134) and population window (tools_algorithmic.c:19-43)
        if (t == 0) {
            s_gate = S;
            s_lo = s_hi = n - 1;
            edge[0] = edge[1] = N::zero();
        }
        const bool psi0_im = __syncthreads_or(im);
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
        // lo: the first i with -x_int <= x[i+1] (0 where the window starts left of the grid); hi: one
        // past the first i with x_int <= x[i+1]; both within the grid
        const double x0 = G.x[0];
        for (int i = t; i + 1 < n; i += kT) {
            const double xn = G.x[i + 1];
            if (-G.x_int <= xn) atomicMin(&s_lo, i);
            if (G.x_int <= xn) atomicMin(&s_hi, i + 1);
            if (-G.x_int <= xn && G.x_int <= xn) break;
        }
        __syncthreads();
        const int lo = (-G.x_int < x0) ? 0 : s_lo, hi = (G.x_int < x0) ? 0 : s_hi;
        const int64_t gate = s_gate;
        const bool warp_win = __any_sync(0xffffffffu, s0 <= hi && s0 + m > lo);
        auto applied = [&](int64_t k) { return (k <= gate || k >= I.n_field || k >= S) ? 0.0 : f[k]; };

        scan.setup(cluster, cF, cB);
        auto send_edges = [&] {
            if (t == 0 && rank > 0) *cluster.map_shared_rank(&edge[1], rank - 1) = psi[0];
            if (t == kT - 1 && rank + 1 < NC) *cluster.map_shared_rank(&edge[0], rank + 1) = psi[(m - 1) * kT + t];
        };
        send_edges();
        if (rank == 0) {  // initial window population (prop.c:87-93)
            double v = 0.0;
            for (int j = lo + t; j <= hi; j += kT)
                v += G.psi0[2 * j] * G.psi0[2 * j] + G.psi0[2 * j + 1] * G.psi0[2 * j + 1];
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) v += shfl_xor(v, d);
            if (lane == 0) s_red[w] = v;
            __syncthreads();
            if (t == 0) {
                o_t[0] = I.tmin;
                o_e[0] = 0.0;
                o_src[0] = 0.0;
                o_ptot[0] = 1.0;
                o_x[0] = 0.0;
                o_pint[0] = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
            }
        }
        double tt = I.tmin;
        // rank 0: the series of steps k0 .. k0 + cnt - 1 from the ring (prop.c:293-347)
        auto flush = [&](int64_t k0, int cnt) {
            const int grp = t / (kRing * kObs), v = t % (kRing * kObs);
            if (grp < kGroups) {
                R s = N::rzero();
                for (int q = grp; q < NW; q += kGroups) s = N::radd(s, ring[((v / kObs) * NW + q) * kObs + v % kObs]);
                part[grp * kRing * kObs + v] = s;
            }
            __syncthreads();
            const int c = t % kObs;
            if (t < cnt * kObs) {
                auto total = [&](int q) {
                    R s = part[q];
#pragma unroll
                    for (int r = 1; r < kGroups; r++) s = N::radd(s, part[r * kRing * kObs + q]);
                    return N::rd(s);
                };
                const int64_t k = k0 + t / kObs;
                const double v0 = total(t);
                if (c == 0) {
                    const double F = applied(k);
                    o_e[k + 1] = F;
                    o_src[k + 1] = -v0 + F;
                } else if (c == 1) {
                    o_x[k + 1] = v0;
                } else if (c == 2) {
                    const double v1 = total(t + 1);
                    o_ptot[k + 1] = v0 * v0 + v1 * v1;
                } else if (c == 4) {
                    o_pint[k + 1] = v0;
                }
            }
            if (t == kT - 1)
                for (int s = 0; s < cnt; s++) {  // t accumulates by repeated addition, as the reference's
                    tt += dt;
                    o_t[k0 + s + 1] = tt;
                }
            __syncthreads();  // part is rewritten by the next flush
        };
        const bool ckpt = I.ckpt_every > 0 && I.ckpt_off >= 0 && P.snapshots;
        auto store_state = [&](double* dst) {  // natural order, 2 doubles per site
            for (int i = 0; i < m; i++)
                if (s0 + i < n) {
                    double re, imv;
                    N::to_d(psi[i * kT + t], re, imv);
                    st2(dst + 2 * (s0 + i), cd{re, imv});
                }
        };
        if (ckpt) store_state(P.snapshots + I.ckpt_off);
        // the phases of kPhSteps steps from k0 on, one angle per thread, into the half of the table that
        // no thread reads: a batch is computed during the last step of the one before, so the barriers
        // of that step separate it from its readers
        auto phases = [&](int64_t k0) {
            if (t >= kPhSteps * kPh) return;
            const int a = t % kPh;
            const double Fdt = applied(k0 + t / kPh) * dt, step = (double)m * dx;
            double ang;
            if (a < kPhA) ang = Fdt * (step * (4 * a));
            else if (a < kPhA + kPhB) ang = Fdt * (step * (a - kPhA));
            else if (a < kPh - 1)  // the last site of the warp's first chunk
                ang = Fdt * (x0 + dx * (double)((rank * kT + 32 * (a - kPhA - kPhB)) * m + m - 1));
            else ang = -(Fdt * dx);
            double sn, cs;
            sincos(ang, &sn, &cs);
            phs[(int)(k0 / kPhSteps % 2) * kPhSteps * kPh + t] = N::from(cs, sn);
        };
        phases(0);
        cluster.sync();  // weights computed from totF / totB, edges in place

        for (int64_t k = 0; k < S; k++) {
            // ---- forward sweep from zero of the right-hand side 2 M2 psi: the chunk's end value
            C pm = (t == 0) ? edge[0] : psi[(m - 1) * kT + t - 1];
            const C nx = (t == kT - 1) ? edge[1] : psi[t + 1];
            C pc = psi[t];
            C b = N::zero();
#pragma unroll 2
            for (int i = 0; i < m; i++) {
                const int q = i * kT + t;
                const C pn = (i + 1 < m) ? psi[q + kT] : nx;
                const C r = N::rhs(ib[q], pc, pm, pn);
                yv[q] = r;
                b = N::fms(hh[q], b, r);
                pm = pc;
                pc = pn;
            }
            b = scan.forward_out(cluster, b);
            cluster.barrier_arrive();
            const int kp = (int)(k % kPhSteps);
            if (kp == kPhSteps - 1) phases(k + 1);
            C bx = N::shup(b, 1);
            cluster.barrier_wait();
            if (rank == 0 && k > 0 && k % kRing == 0) flush(k - kRing, kRing);
            // ---- forward sweep from the exact carry, backward sweep from zero
            C y = scan.forward_in(bx);
#pragma unroll 2
            for (int i = 0; i < m; i++) {
                const int q = i * kT + t;
                y = N::fms(hh[q], y, yv[q]);
                yv[q] = y;
            }
            b = y;
#pragma unroll 2
            for (int i = m - 2; i >= 0; i--) {
                const int q = i * kT + t;
                b = N::fms(gg[q], b, yv[q]);
            }
            b = scan.backward_out(cluster, b);
            cluster.barrier_arrive();
            bx = N::shdn(b, 1);
            const C* ps = phs + ((int)(k / kPhSteps % 2) * kPhSteps + kp) * kPh;
            C ph = N::mul(N::mul(ps[lane >> 2], ps[kPhA + (lane & 3)]), ps[kPhA + kPhB + w]);
            const C zc = ps[kPh - 1];
            cluster.barrier_wait();
            // ---- backward sweep from the exact carry, CN update, phase e^{+i F dt x}, observables
            C u = scan.backward_in(bx);
            typename N::Acc acc;
#pragma unroll 2
            for (int i = m - 1; i >= 0; i--) {
                const int q = i * kT + t, j = s0 + i;
                u = N::fms(gg[q], u, yv[q]);
                const C pn = N::update(ph, u, psi[q]);
                psi[q] = pn;
                ph = N::mul(ph, zc);
                acc.add(pn, gx[q], p0[q], j >= lo && j <= hi);
                if (psi0_im && j < n) {
                    const int64_t e = (int64_t)(j % m256) * kThreads + j / m256;
                    acc.add_im(pn, N::re(N::mul(C(N::from(0.0, -1.0)), tab[CN_PSI0 * L + e])));
                }
            }
            send_edges();
            cluster.barrier_arrive();
            {   // warp sums: four values in six additions (each level halves what a lane carries)
                R v[4];
                acc.get(v);
                const bool h16 = lane & 16, h8 = lane & 8;
                R a = N::radd(h16 ? v[2] : v[0], N::rxor(h16 ? v[0] : v[2], 16));
                R c = N::radd(h16 ? v[3] : v[1], N::rxor(h16 ? v[1] : v[3], 16));
                R s = N::radd(h8 ? c : a, N::rxor(h8 ? a : c, 8));
#pragma unroll
                for (int d = 4; d >= 1; d >>= 1) s = N::radd(s, N::rxor(s, d));
                R win = N::rzero();
                if (warp_win) {
                    win = acc.window();
#pragma unroll
                    for (int d = 16; d >= 1; d >>= 1) win = N::radd(win, N::rxor(win, d));
                }
                R* dst = cluster.map_shared_rank(ring, 0) + ((int)(k % kRing) * NW + g) * kObs;
                if ((lane & 7) == 0) dst[lane >> 3] = s;
                if (lane == 1) dst[4] = win;
            }
            if (ckpt && (k + 1) % I.ckpt_every == 0 && k + 1 < S)
                store_state(P.snapshots + I.ckpt_off + (k + 1) / I.ckpt_every * 2 * (int64_t)n);
            if (I.snap_off >= 0 && P.snapshots) {  // prop.c:248-263
                int64_t slot = -1;
                if (k % I.snap_every == 0 && k / I.snap_every < I.n_snap - 1) slot = k / I.snap_every;
                if (k == S - 1) slot = I.n_snap - 1;
                if (slot >= 0) store_state(P.snapshots + I.snap_off + slot * 2 * (int64_t)n);
            }
            cluster.barrier_wait();
        }
        cluster.sync();  // the last steps' sums are in rank 0's ring
        if (rank == 0) flush((S - 1) / kRing * kRing, (int)(S - (S - 1) / kRing * kRing));
        if (P.psi_final && I.psi_off >= 0) store_state(P.psi_final + I.psi_off);
    }
}

}  // namespace clk
}  // namespace mma

using namespace mma;

namespace {

template <class N>
int launch(const clk::Args& A, int nc, int clusters, size_t smem, cudaStream_t st)
{
    auto k = clk::propagate_cluster_kernel<N>;
    if (allow_smem(k) != cudaSuccess ||
        !succeeded(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
        return MMA_ERR_CUDA;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(clusters * nc));
    cfg.blockDim = dim3(clk::kT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)nc;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return succeeded(cudaLaunchKernelEx(&cfg, k, A)) ? MMA_OK : MMA_ERR_CUDA;
}

template <class N>
int active_clusters(int nc, size_t smem)
{
    auto k = clk::propagate_cluster_kernel<N>;
    if (allow_smem(k) != cudaSuccess ||
        !succeeded(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
        return 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)nc);
    cfg.blockDim = dim3(clk::kT);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)nc;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int c = 0;
    return succeeded(cudaOccupancyMaxActiveClusters(&c, k, &cfg)) ? c : 0;
}

}  // namespace

namespace mma {

// Where the line lies between one CTA and a cluster per instance, and the cluster size: the smallest
// expected time of a step of the whole batch.  The models were fitted to runs of 1 to 304 instances on
// grids of 601 to 8001 sites (us per step, measured / model):
//   one CTA    FP64   601 sites  24.3 / 24.3    8001 sites  108.8 / 108.7   256 x 4001 sites  125 / 124
//              df64   601 sites   7.6 /  7.5    8001 sites   34.1 /  34.1   304 x 8001 sites  54.0 / 54.0
//   cluster    FP64  8001 sites  NC = 4  29.0 / 28.8   8  17.3 / 17.2   16  11.7 / 11.4;  256 x 4001, NC = 2  115 / 115
//              df64  8001 sites  NC = 4  10.1 / 10.1   8   6.9 /  7.2   16   5.6 /  5.7
// A second CTA on an SM costs FP64 its pipe time (16.1 us a wave measured at m = 4, 17.4 modelled) and
// the float-float form, bound by latency, about two thirds of the first.
namespace {
double one_cta_us(int m256, int precision, int n_inst, int sms)
{
    if (precision != 2) return (double)((n_inst + sms - 1) / sms) * (15.6 + 2.91 * m256);
    const double one = 4.8 + 0.915 * m256, two = 7.8 + 1.445 * m256;
    const int full = n_inst / (2 * sms), rest = n_inst % (2 * sms);
    return full * two + (rest == 0 ? 0.0 : rest <= sms ? one : two);
}
double cluster_us(int m, int precision, int waves, int per_sm)
{
    if (precision != 2) return waves * (4.0 + 0.35 * m + per_sm * (1.6 + 1.1 * m));
    return waves * (4.2 + 0.37 * m) * (1.0 + 0.65 * (per_sm - 1));
}
}  // namespace

bool choose_cluster(int max_m, int precision, int n_inst, int sms, ClusterPlan* plan)
{
    double best = one_cta_us(max_m, precision, n_inst, sms);
    bool found = false, tried[clk::kMaxNC + 1] = {};
    for (;;) {
        // the most promising size not looked at yet, if every SM could be filled: the number of
        // clusters that are really resident depends on the GPU's partition and is asked for it alone
        int pick = 0;
        double promise = best;
        ClusterPlan cand{};
        for (int nc = 1; nc <= clk::kMaxNC; nc++) {
            if (tried[nc]) continue;
            const int m = (max_m * kThreads + nc * clk::kT - 1) / (nc * clk::kT);
            const size_t smem = (size_t)m * clk::kT * clk::site_bytes() + clk::fixed_bytes(nc);
            if (smem > 226 * 1024 || (nc > 1 && (nc - 1) * m * clk::kT >= max_m * kThreads)) continue;
            const int fit = sms * (smem > 112 * 1024 ? 1 : 2) / nc;
            const int run = fit < n_inst ? fit : n_inst;
            const double us = run < 1 ? best : cluster_us(m, precision, (n_inst + run - 1) / run, (run * nc + sms - 1) / sms);
            if (us < promise) {
                promise = us;
                pick = nc;
                cand = ClusterPlan{nc, m, smem, 0};
            }
        }
        if (!pick) return found;
        tried[pick] = true;
        cand.active = precision == 2 ? active_clusters<clk::Df64>(pick, cand.smem) : active_clusters<clk::Fp64>(pick, cand.smem);
        if (cand.active < 1) continue;
        const int run = cand.active < n_inst ? cand.active : n_inst;
        const double us = cluster_us(cand.m, precision, (n_inst + run - 1) / run, (run * pick + sms - 1) / sms);
        if (us < best) {
            best = us;
            *plan = cand;
            found = true;
        }
    }
}

int launch_cluster(const ClusterPlan& p, const mma_tdse_instance* insts, int n_inst, const mma_tdse_grid* grids,
                   const mma_tdse_buffers* bufs, int max_m, int precision, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(bufs->counter, 0, sizeof(int), st) != cudaSuccess) return MMA_ERR_CUDA;
    clk::Args A{insts, n_inst, grids, bufs->fields, bufs->outputs, bufs->psi_final, bufs->snapshots, bufs->counter,
                p.m, (int64_t)max_m * kThreads};
    const int clusters = p.active < n_inst ? p.active : n_inst;
    return precision == 2 ? launch<clk::Df64>(A, p.nc, clusters, p.smem, st)
                          : launch<clk::Fp64>(A, p.nc, clusters, p.smem, st);
}

}  // namespace mma
