// tdse_df64.cu -- float-float ("df64") form of the TDSE propagation: the FP64 Crank-Nicolson-
// Numerov step (prop.c:115-347, the same tables and partitioned solve as propagate_fp64_kernel)
// carried out in double-word FP32 arithmetic.
//
// On this GPU FP32 runs at about 62x the FP64 rate, so a double-word operation of 6-25 FP32
// instructions still outruns one FP64 operation.  A value is a pair (hi, lo) of floats with
// |lo| <= ulp(hi)/2, about 48 significant bits; every operation below is built from two
// error-free transformations:
//   * TwoSum (Knuth): s + e = a + b exactly, s = fl(a + b);
//   * TwoProduct with an FMA: p + e = a b exactly, p = fl(a b), e = fma(a, b, -p);
// with the accurate double-word addition of Joldes, Muller and Popescu ("Tight and rigorous
// error bounds for basic building blocks of double-word arithmetic", ACM TOMS 2017, Alg. 6):
// relative error about 3 u^2 (u = 2^-24).  Products and sums of products fold their low-order
// terms with FMAs before one final renormalisation.
//
// The complex values of the site loops run as packed FP32x2 pairs, (re.hi, im.hi) and (re.lo,
// im.lo): real and imaginary parts take the same operations, so one FP32x2 instruction does two.
// Against the same arithmetic written per component: 27% fewer instructions, the same bits,
// 2.5% faster (the kernel is then bound by the latency of the sweeps' dependency chains).
//
// Layout as in the FP64 kernel: site j = t m + i at q = i T + t; the tables are the FP64 tables
// split once per grid into float4 (re.hi, im.hi, re.lo, im.lo) (mma_tdse_build_df_tables).  psi
// and the sweep buffer live in the caller's scratch (L2-resident, 16 bytes per site each) rather than in shared
// memory, so that two 256-thread CTAs fit on an SM: the double-word operations are long
// dependency chains and 16 warps hide them better than 8 (measured 27% faster on config 1).
// Each pass reads its operands through a small cp.async ring in shared memory, two sites ahead,
// which hides the L2 latency without registers (30% faster at one CTA per SM, 9% at two).
// No warp carries serial FP64 work into the scan barriers (a 32-lane FP64 instruction holds a
// sub-partition's FP64 unit for about 64 cycles): the phase factors come from FP64 sincos spread over the
// threads for some twenty steps at a time, and the observables' warp sums stay double-word until lanes
// of warp 0 convert them.
//
// Bound by the double-word chains' latency and the CTA barriers between the passes (304 instances, 884 steps:
// FMA pipe 60% busy, issue 54%, an eighth of the warps' time at barriers).  Per step of 304 instances of 8001 sites (two CTAs
// an SM): 58.9 us before the operand ring was aligned, the chunks kept their own frames (below), the
// correction and the backward sweep became one sum and a real psi0 took half a projection; 54.0 us now
// with 11% fewer instructions.  The whole benchmark map, 4 cycles: 667 -> 609 ms.
#include <cuda_runtime.h>

#include "../../include/mma_tdse.h"
#include "common.cuh"
#include "df64.cuh"
#include "launch.cuh"
#include "tdse_step.cuh"

namespace mma {
namespace dfk {

// 16-byte global -> shared copy (L2 only), grouped per iteration; a thread reads back only what it
// copied itself, so completing its own groups (cp.async.wait_group) is the only wait
__device__ __forceinline__ void cp16(float4* dst_smem, const float4* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// exclusive CTA scans of the affine maps Y_t = b_t + c_t Y_{t-1} (forward) and
// U_t = b_t + c_t U_{t+1} (backward), as scan_forward / scan_backward (tdse_solver.cuh)
__device__ pk scan_fwd(pk c, pk b, pk* sc, pk* sb)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const pk cp = pshup(c, d), bp = pshup(b, d);
        if (lane >= d) {
            b = cfma_p(c, bp, b);
            c = cmul_p(c, cp);
        }
    }
    if (lane == 31) {
        sc[w] = c;
        sb[w] = b;
    }
    __syncthreads();
    pk yw{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    for (int q = 0; q < w; q++) yw = cfma_p(sc[q], yw, sb[q]);
    const pk cp = pshup(c, 1), bp = pshup(b, 1);
    return lane == 0 ? yw : cfma_p(cp, yw, bp);
}

__device__ pk scan_bwd(pk c, pk b, pk* sc, pk* sb)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const pk cp = pshdn(c, d), bp = pshdn(b, d);
        if (lane + d < 32) {
            b = cfma_p(c, bp, b);
            c = cmul_p(c, cp);
        }
    }
    if (lane == 0) {
        sc[w] = c;
        sb[w] = b;
    }
    __syncthreads();
    pk uw{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    for (int q = kWarps - 1; q > w; q--) uw = cfma_p(sc[q], uw, sb[q]);
    const pk cp = pshdn(c, 1), bp = pshdn(b, 1);
    return lane == 31 ? uw : cfma_p(cp, uw, bp);
}

// The step's observables from the per-warp double-word partial sums (lane c < 5 sums column c
// over the warps), in FP64 from there: sourceterm -<V'> + F, <x>, |<psi0|psi>|^2 and the window
// population (prop.c:266-300, tools_algorithmic.c:19-43).  Called by one warp.
__device__ __forceinline__ void observables_out(const df* redf, int lane, int64_t k, double F_prev, double* o_src,
                                                double* o_x, double* o_ptot, double* o_pint)
{
    df s{0.f, 0.f};
    if (lane < 5)
#pragma unroll
        for (int q = 0; q < kWarps; q++) s = add(s, redf[q * 5 + lane]);
    const double v = to_d(s);
    const double v3 = __shfl_down_sync(0xffffffffu, v, 1);  // lane 2 gets the imaginary projection
    if (lane == 0) o_src[k] = -v + F_prev;
    if (lane == 1) o_x[k] = v;
    if (lane == 2) o_ptot[k] = v * v + v3 * v3;
    if (lane == 4) o_pint[k] = v;
}

struct Args {
    const mma_tdse_instance* insts;
    int n_inst;
    const mma_tdse_grid* grids;
    const double* fields;
    double* outputs;
    double* psi_final;
    double* snapshots;
    int* counter;
    float4* scratch;  // per CTA: yl [L], then psi [L]
    int64_t max_L;
};

// The phase e^{i F dt x} of a step splits into a part that is constant over a thread's chunk and one
// that is the same for every thread: x = x_{s0(t)} + i dx.  The first is never applied: thread t keeps
// psi in its own frame, psi = B_t psi~ with B_t = e^{i A x_{s0}}, A = dt (sum of the fields so far).  The
// solve commutes with a constant, so inside a chunk nothing changes, and between neighbours only the one
// factor R = B_{t+1}/B_t = e^{i A m dx} enters: the halo values, the scans' coefficients and their
// carries.  Per site that saves the phase's recurrence (one of about ten double-word products), per
// thread the products of its start phase; <psi0|psi> is summed over the lanes and warps with powers of R.
// Factors per step: R before the step, R^1, 2, 4, 8, 16 and R^{32 w} after it, then z^i = e^{i F dt i dx}
// for the chunk's sites (in two levels, i = 32 a + b, where a chunk has more than kFlat sites).
constexpr int kRb = 0, kRp = 1, kRw = 6, kZ = kRw + kWarps;
constexpr int kFlat = 512, kFactors = 1024;  // factors of as many steps as fit are computed at a time
__host__ __device__ inline int z_entries(int m) { return m <= kFlat ? m : 32 + (m + 31) / 32; }
__host__ __device__ inline int factor_entries(int m) { return kZ + z_entries(m) > kFactors ? kZ + z_entries(m) : kFactors; }
constexpr int kMaxSteps = kFactors / (kZ + 1);
// Operand ring: each pass copies the operands of site i + kDepth - 1 into shared memory while it
// computes site i (kSlots float4 per site at most, pass 3), so the L2 latency of psi, the sweep
// buffer and the tables is hidden without holding registers.
constexpr int kDepth = 3, kSlots = 5;
constexpr int kRingBytes = kDepth * kSlots * kThreads * 16;  // 61,440 bytes per CTA
inline size_t smem_bytes(int max_m) { return kRingBytes + 16 * (size_t)factor_entries(max_m); }

template <bool FLAT>
__global__ void __launch_bounds__(kThreads, 2) propagate_df64_kernel(Args P)
{
    // [kDepth][kSlots][kThreads], then the factors of the steps.  The alignment matters: with the ring off a
    // 64-byte boundary every 64-byte half of a warp's copy is fetched twice (L2 reads 0.78 -> 1.54 G sectors)
    extern __shared__ __align__(128) float4 ring[];
    pk* const fac = reinterpret_cast<pk*>(ring + kDepth * kSlots * kThreads);
    __shared__ pk sc[2 * kWarps], sb[2 * kWarps];
    __shared__ double red[kWarps];
    __shared__ df redf[kWarps * 5];  // per warp: -<V'>, <x>, <psi0|psi> (re, im), window population
    __shared__ double s_A[kMaxSteps + 1];  // A before the current block of steps and after each of them
    __shared__ int64_t s_inst, s_gate, s_lo, s_hi;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    float4* yl = P.scratch + blockIdx.x * P.max_L;
    float4* psi = P.scratch + (gridDim.x + blockIdx.x) * P.max_L;

    for (;;) {
        if (t == 0) s_inst = atomicAdd(P.counter, 1);
        __syncthreads();
        const int64_t inst = s_inst;
        if (inst >= P.n_inst) break;
        const mma_tdse_instance I = P.insts[inst];
        const mma_tdse_grid G = P.grids[I.grid];
        const int64_t n = G.n, m = G.m, L = m * kThreads, S = I.n_steps;
        const float4* tab = reinterpret_cast<const float4*>(G.df_tab);
        const float4 *IB = tab + CN_IB6 * L, *HH = tab + CN_H * L, *FF = tab + CN_F * L, *GG_ = tab + CN_G * L,
                     *GP = tab + CN_GG * L, *P0 = tab + CN_PSI0 * L, *GVX = tab + CN_GVX * L;
        const double* f = P.fields + I.field_off;
        double* out = P.outputs + I.out_off;
        double *o_t = out, *o_e = out + (S + 1), *o_src = out + 2 * (S + 1), *o_ptot = out + 3 * (S + 1),
               *o_pint = out + 4 * (S + 1), *o_x = out + 5 * (S + 1);
        const double dt = G.dt, dx = G.dx;
        if (L > P.max_L) {
            // a grid wider than the launch was sized for would overrun this CTA's buffers and the factors in
            // shared memory: NaN outputs, as in the FP64 kernel
            for (int64_t e = t; e < 6 * (S + 1); e += kThreads) out[e] = __longlong_as_double(0x7ff8000000000000LL);
            __syncthreads();
            continue;
        }
        if (t == 0) {
            s_gate = gate_index(f, I.n_field, S, I.gate_floor);
            const int64_t num_r = n - 1;  // PopInt window (tools_algorithmic.c:19-43)
            int64_t lo = -1, hi;
            if (!(-G.x_int < G.x[0])) {
                int64_t i = 0;
                while (i < num_r && !(-G.x_int <= G.x[i + 1])) i++;
                lo = i;
            }
            if (G.x_int < G.x[0]) {
                hi = 0;
            } else {
                int64_t i = 0;
                while (i < num_r && !(G.x_int <= G.x[i + 1])) i++;
                hi = (i < num_r) ? i + 1 : num_r + 1;
            }
            s_lo = lo < 0 ? 0 : lo;
            s_hi = hi > num_r ? num_r : hi;
        }
        bool im = false;
        for (int64_t i = 0; i < m; i++) {
            const float4 v = P0[i * kThreads + t];
            psi[i * kThreads + t] = v;
            im |= v.y != 0.f;
        }
        const bool psi0_im = __syncthreads_or(im);
        const int64_t lo = s_lo, hi = s_hi, gate = s_gate;
        const int64_t s0 = t * m;
        {   // initial window population (prop.c:87-93), FP64 from the FP64 ground state
            double v[1] = {0.0};
            for (int64_t j = t; j < n; j += kThreads)
                if (j >= lo && j <= hi) v[0] += G.psi0[2 * j] * G.psi0[2 * j] + G.psi0[2 * j + 1] * G.psi0[2 * j + 1];
            block_sum<1>(v, red);
            if (t == 0) {
                o_t[0] = I.tmin;
                o_e[0] = 0.0;
                o_src[0] = 0.0;
                o_ptot[0] = 1.0;
                o_pint[0] = v[0];
                o_x[0] = 0.0;
            }
        }
        double tt = I.tmin, Fprev = 0.0;
        const double xs = s0 < n ? G.x[s0] : 0.0;
        auto applied = [&](int64_t k) { return (k <= gate || k >= I.n_field || k >= S) ? 0.0 : f[k]; };
        auto store_psi = [&](double* dst, double A) {  // psi = B_t psi~, natural order
            double sn, cs;
            sincos(A * xs, &sn, &cs);
            for (int64_t i = 0; i < m; i++)
                if (s0 + i < n) {
                    const pk v = pld(psi + i * kThreads + t);
                    const double re = (double)v.h.x + (double)v.l.x, im = (double)v.h.y + (double)v.l.y;
                    dst[2 * (s0 + i)] = re * cs - im * sn;
                    dst[2 * (s0 + i) + 1] = re * sn + im * cs;
                }
        };
        const int mi = (int)m;  // sites per thread: 32-bit indices in the site loops
        const int per = kZ + (FLAT ? mi : z_entries(kFlat < mi ? mi : kFlat + 1)), nb = kFactors / per > 1 ? kFactors / per : 1;
        int kb = nb;  // steps of the current block done
        if (t == 0) s_A[0] = 0.0;
        for (int64_t k = 0; k < S; k++) {
            const double Fk = applied(k);
            if (w == 0) {
                if (k > 0) observables_out(redf, lane, k, Fprev, o_src, o_x, o_ptot, o_pint);
                if (lane == 0) {
                    tt += dt;
                    o_t[k + 1] = tt;
                    o_e[k + 1] = Fk;
                }
            }
            Fprev = Fk;
            // the factors of the next block of steps in FP64, spread evenly over the threads (a 32-lane
            // FP64 instruction holds a sub-partition's FP64 unit for about 64 cycles)
            if (kb == nb) {
                if (k > 0 && t == 0) s_A[0] = s_A[nb];
                __syncthreads();
                if (t >= 1 && t <= nb) {
                    double A = s_A[0];
                    for (int j = 0; j < t; j++) A += dt * applied(k + j);
                    s_A[t] = A;
                }
                __syncthreads();
                for (int e = t; e < nb * per; e += kThreads) {
                    const int st = e / per, q = e % per;
                    const double step = (double)m * dx;
                    double ang;
                    if (q == kRb) ang = s_A[st] * step;
                    else if (q < kRw) ang = s_A[st + 1] * (step * (1 << (q - kRp)));
                    else if (q < kZ) ang = s_A[st + 1] * (step * (32 * (q - kRw)));
                    else {
                        const int i = q - kZ;
                        ang = applied(k + st) * dt * (dx * (double)(FLAT || i < 32 ? i : 32 * (i - 32)));
                    }
                    double sn, cs;
                    sincos(ang, &sn, &cs);
                    const df c2 = from_d(cs), s2 = from_d(sn);
                    fac[e] = pk{make_float2(c2.hi, s2.hi), make_float2(c2.lo, s2.lo)};
                }
                __syncthreads();
                kb = 0;
            }
            const pk* const fk = fac + kb * per;
            kb++;
            const pk Rb = fk[kRb], Rbc{make_float2(Rb.h.x, -Rb.h.y), make_float2(Rb.l.x, -Rb.l.y)};
            // ---- pass 1: local forward sweep of the right-hand side 2 M2 psi
            const pk zero{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            float4* const my = ring + t;
            constexpr int kStage = kSlots * kThreads;
            // site i's operands: psi of site i + 1 (the next thread's first site after the last),
            // H and 1/(2 beta)
            auto issue1 = [&](int i, float4* r) {
                const int q = i * kThreads + t;
                cp16(r, (i + 1 < mi) ? psi + q + kThreads : psi + (t + 1 < kThreads ? t + 1 : t));
                cp16(r + kThreads, HH + q);
                cp16(r + 2 * kThreads, IB + q);
            };
#pragma unroll
            for (int d = 0; d < kDepth - 1; d++) {
                if (d < mi) issue1(d, my + d * kStage);
                cp_commit();
            }
            pk pm = (t == 0) ? zero : cmul_p(Rbc, pld(psi + (m - 1) * kThreads + t - 1));
            pk pc = pld(psi + t);
            pk yprev = zero;
            int su = 0;  // ring stage of the current site; the stage before it is refilled
            auto site1 = [&](int i, bool last) {
                float4* const r = my + su * kStage;
                if (i + kDepth - 1 < mi) issue1(i + kDepth - 1, my + (su == 0 ? kDepth - 1 : su - 1) * kStage);
                cp_commit();
                cp_wait<kDepth - 1>();
                pk pn = !last || t + 1 < kThreads ? pld(r) : zero;
                if (last) pn = cmul_p(Rb, pn);  // the next thread's first site, in this thread's frame
                const pk r2 = ten_sum_p(pc, pm, pn);
                yprev = cfms_p(pld(r + kThreads), yprev, cmul_pu(pld(r + 2 * kThreads), r2));
                pst(yl + i * kThreads + t, yprev);
                pm = pc;
                pc = pn;
                su = su + 1 == kDepth ? 0 : su + 1;
            };
#pragma unroll 2
            for (int i = 0; i + 1 < mi; i++) site1(i, false);
            site1(mi - 1, true);
            const pk yin = cmul_p(Rbc, scan_fwd(cmul_p(Rbc, pld(FF + (m - 1) * kThreads + t)), yprev, sc, sb));
            // ---- pass 2: forward correction, local backward sweep
            auto issue2 = [&](int i, float4* r) {  // F, y and G of site i
                const int q = i * kThreads + t;
                cp16(r, FF + q);
                cp16(r + kThreads, yl + q);
                cp16(r + 2 * kThreads, GG_ + q);
            };
#pragma unroll
            for (int d = 0; d < kDepth - 1; d++) {
                if (d < mi) issue2(mi - 1 - d, my + d * kStage);
                cp_commit();
            }
            pk unext = zero;
            su = 0;
#pragma unroll 2
            for (int j = 0; j < mi; j++) {  // site i = mi - 1 - j
                float4* const r = my + su * kStage;
                if (j + kDepth - 1 < mi) issue2(mi - kDepth - j, my + (su == 0 ? kDepth - 1 : su - 1) * kStage);
                cp_commit();
                cp_wait<kDepth - 1>();
                unext = correct_sweep_p(pld(r), yin, pld(r + kThreads), pld(r + 2 * kThreads), unext);
                pst(yl + (mi - 1 - j) * kThreads + t, unext);
                su = su + 1 == kDepth ? 0 : su + 1;
            }
            const pk uin = cmul_p(Rb, scan_bwd(cmul_p(Rb, pld(GP + t)), unext, sc + kWarps, sb + kWarps));
            // ---- pass 3: backward correction, CN update, phase e^{+i F dt x}, observables
            const pk* const zk = fk + kZ;
            // lanes (-<V'>, <x>) and the projection (re, im) on psi0
            pk acc01 = zero, acc23 = zero;
            df acc[5];
            auto issue3 = [&](int i, float4* r) {  // G, u, psi, (-V', x) and psi0 of site i
                const int q = i * kThreads + t;
                cp16(r, GP + q);
                cp16(r + kThreads, yl + q);
                cp16(r + 2 * kThreads, psi + q);
                cp16(r + 3 * kThreads, GVX + q);
                cp16(r + 4 * kThreads, P0 + q);
            };
#pragma unroll
            for (int d = 0; d < kDepth - 1; d++) {
                if (d < mi) issue3(d, my + d * kStage);
                cp_commit();
            }
            su = 0;
#pragma unroll 2
            for (int i = 0; i < mi; i++) {
                float4* const r = my + su * kStage;
                if (i + kDepth - 1 < mi) issue3(i + kDepth - 1, my + (su == 0 ? kDepth - 1 : su - 1) * kStage);
                cp_commit();
                cp_wait<kDepth - 1>();
                su = su + 1 == kDepth ? 0 : su + 1;
                const int q = i * kThreads + t;
                const pk gp = pld(r), yv = pld(r + kThreads), po = pld(r + 2 * kThreads);
                // u - psi with u = G u_in + y, the CN update before the phase
                const pk d = cn_update_p(gp, uin, yv, po);
                pk z;
                if constexpr (FLAT) z = zk[i]; else z = cmul_p(zk[32 + (i >> 5)], zk[i & 31]);
                const pk pn = cmul_p(z, d);
                pst(psi + q, pn);
                const df n2 = norm2_u(pn);
                const pk gx = pld(r + 3 * kThreads), p0 = pld(r + 4 * kThreads);
                acc_mul_p(acc01, n2.hi, n2.lo, gx);
                if (psi0_im) acc_proj_p(acc23, pn, p0);
                else acc_mul_p(acc23, p0.h.x, p0.l.x, pn);
            }
            acc01 = renorm2(acc01.h, acc01.l);
            acc23 = renorm2(acc23.h, acc23.l);
            acc[0] = df{acc01.h.x, acc01.l.x};
            acc[1] = df{acc01.h.y, acc01.l.y};
            // <psi0|psi> = sum_t B_t p_t: over the lanes with R^1, 2, 4, 8, 16, then over the warps (R^{32 w};
            // the common B_0 does not change its modulus).  The complex projection is its conjugate.
            if (psi0_im) acc23 = pk{make_float2(acc23.h.x, -acc23.h.y), make_float2(acc23.l.x, -acc23.l.y)};
#pragma unroll
            for (int l = 0; l < 5; l++) acc23 = cfma_p(fk[kRp + l], pshdn(acc23, 1 << l), acc23);
            acc23 = cmul_p(fk[kRw + w], acc23);
            acc[2] = df{acc23.h.x, acc23.l.x};
            acc[3] = df{acc23.h.y, acc23.l.y};
            acc[4] = df{0.f, 0.f};  // the few sites of the population window in this chunk
            for (int64_t j = (lo > s0 ? lo : s0); j <= hi && j < s0 + m; j++) {
                const df n = norm2_u(pld(psi + (j - s0) * kThreads + t));
                acc[4] = add(acc[4], renorm(n.hi, n.lo));
            }
            // warp sums in double-word arithmetic; across warps at the next step (observables_out)
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1)
#pragma unroll
                for (int c = 0; c < 5; c++)
                    if (c < 2 || c > 3) acc[c] = add(acc[c], shfl_xor_df(acc[c], d));
            if (lane == 0)
#pragma unroll
                for (int c = 0; c < 5; c++) redf[w * 5 + c] = acc[c];
            if (I.snap_off >= 0 && P.snapshots) {  // prop.c:248-263
                int64_t slot = -1;
                if (k % I.snap_every == 0 && k / I.snap_every < I.n_snap - 1) slot = k / I.snap_every;
                if (k == S - 1) slot = I.n_snap - 1;
                if (slot >= 0) {
                    store_psi(P.snapshots + I.snap_off + slot * 2 * n, s_A[kb]);
                }
            }
            __syncthreads();
        }
        if (w == 0) observables_out(redf, lane, S, Fprev, o_src, o_x, o_ptot, o_pint);
        if (P.psi_final && I.psi_off >= 0) {
            store_psi(P.psi_final + I.psi_off, s_A[kb]);
        }
        __syncthreads();
    }
}

// the FP64 CN tables of a grid split into (hi, lo) float pairs, slot by slot in the same layout
__global__ void __launch_bounds__(kThreads) build_df_kernel(const mma_tdse_grid* grids)
{
    const mma_tdse_grid G = grids[blockIdx.x];
    const int64_t L = G.m * kThreads, cnt = (int64_t)CN_SLOTS * L;  // complex entries
    const cd* src = reinterpret_cast<const cd*>(G.cn_tab);
    float4* dst = reinterpret_cast<float4*>(G.df_tab);
    for (int64_t q = threadIdx.x; q < cnt; q += blockDim.x) {
        const cd v = src[q];
        const df re = from_d(v.re), im = from_d(v.im);
        dst[q] = make_float4(re.hi, im.hi, re.lo, im.lo);  // the packed layout (re.hi, im.hi, re.lo, im.lo)
    }
}

}  // namespace dfk
}  // namespace mma

using namespace mma;

extern "C" int mma_tdse_build_df_tables(const mma_tdse_grid* grids_dev, const mma_tdse_grid* grids_host, int n_grids,
                                        void* stream)
{
    if (n_grids <= 0 || !grids_dev || !grids_host) return MMA_ERR_ARG;
    for (int g = 0; g < n_grids; g++)
        if (!grids_host[g].df_tab || !grids_host[g].cn_tab) return MMA_ERR_ARG;
    dfk::build_df_kernel<<<n_grids, kThreads, 0, (cudaStream_t)stream>>>(grids_dev);
    return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
}

// CTAs of the float-float form resident at once (two per SM), and the scratch they need:
// per CTA the sweep buffer and psi, 16 bytes per site each.
static bool df64_smem_attr()
{
    return allow_smem(dfk::propagate_df64_kernel<true>) == cudaSuccess &&
           allow_smem(dfk::propagate_df64_kernel<false>) == cudaSuccess;
}

extern "C" int mma_tdse_df64_default_ctas()
{
    int dev = 0, sms = 0, per_sm = 0;
    const size_t smem = dfk::smem_bytes(1);  // up to some thousand sites per thread take no more
    if (cudaGetDevice(&dev) != cudaSuccess || !df64_smem_attr()) return 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dfk::propagate_df64_kernel<true>, kThreads, smem);
    return sms * (per_sm > 0 ? per_sm : 1);
}

extern "C" size_t mma_tdse_df64_scratch_bytes(int max_m, int grid_ctas)
{
    return (size_t)max_m * kThreads * 16 * 2 * (size_t)grid_ctas;
}

// Launch of the float-float form (called by mma_tdse_propagate_ex for precision 2).
extern "C" int mma_tdse_propagate_df64_impl(const mma_tdse_instance* insts, int n_inst, const mma_tdse_grid* grids,
                                            const mma_tdse_buffers* bufs, int max_m, int grid_ctas, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(bufs->counter, 0, sizeof(int), st) != cudaSuccess) return MMA_ERR_CUDA;
    dfk::Args A{insts, n_inst, grids, bufs->fields, bufs->outputs, bufs->psi_final, bufs->snapshots, bufs->counter,
                reinterpret_cast<float4*>(bufs->scratch), (int64_t)max_m * kThreads};
    const size_t smem = dfk::smem_bytes(max_m);
    if (!df64_smem_attr()) return MMA_ERR_CUDA;
    auto kern = max_m <= dfk::kFlat ? dfk::propagate_df64_kernel<true> : dfk::propagate_df64_kernel<false>;
    kern<<<grid_ctas, kThreads, smem, st>>>(A);
    return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
}
