// hankel_plain.cu -- far-field (Hankel) kernels of the FP64 form.
//
// Reference: Hankel/Hankel_transform.py:452-519 (HankelTransform), :523-686 (Hankel_long).
// Per plane k and frequency w (k_w = w/c, D_k = distance - z_k):
//   A_k[w, r]   = pre_k(w) e^{-i k_w r^2/(2 D_k)} r S_k[w, r] wr_r      (wr = r trapezoid weights)
//   P_k[w, rho] = sum_r A_k[w, r] J0(k_w r rho / D_k)
//   FF[rho, w]  = sum_k tau_k P_k[w, rho]                               (tau = z trapezoid weights)
//
// Everything is FP64 and bound by the FP64 pipe (1.25 TFLOP/s), so the work is operations:
//   * J0 (and J1) come from Taylor sums of 12 terms about nodes 1/4 apart (|d| <= 1/8, truncation
//     (1/8)^11/11! = 3e-18 in J1), whose coefficients follow from J0 and J1 at the node by Bessel's
//     equation x y'' + y' + x y = 0.  The table (112 bytes a node) is made once per call.  11 FMAs
//     a J0 against about 147 FP64 operations a term with CUDA's j0 (measured).  The far field is within
//     1.3e-16 of its largest value of extended-precision sums (64 planes x 512 r, arguments up to 330), where
//     sums with CUDA's j0, itself up to 1.1e-13 off there, were within 1.1e-15.  Arguments beyond the
//     table's nodes take j0.
//   * Where at most two planes are wanted for themselves, FF contracts z first through the
//     multiplication theorem J0(lambda y) = sum_m (1 - lambda^2)^m / m! G_m(y), G_m = (y/2)^m J_m(y),
//     lambda = d_ref/D_k: B_m[w, r] = sum_k tau_k (1 - lambda_k^2)^m / m! A_k, then
//     FF = sum_{r, m} G_m(k r rho/d_ref) B_m[w, r], with G_{m+1} = m G_m - (y/2)^2 G_{m-1}.  The number
//     of terms is taken per radius so that the dropped tail, x^M/M! e^x with x = max|1 - lambda^2| y/2,
//     is below 1e-17.  The recurrence's rounding grows as the upward recurrence of J_m does, but
//     enters scaled by (1 - lambda^2)^m, so it stays below that of J0 itself.
// 64 omega x 64 planes x 512 r x 128 rho with two planes: 155 ms (one j0 a term, one CTA per
// frequency) -> 1.5 ms for the call; stage 1 0.31 ms, stage 2 1.10 ms, tables 0.06 ms.  Every plane of
// 32 omega: 155 -> 5.7 ms (direct sum).
#include <cuda_runtime.h>

#include <cmath>

#include "../../include/mma_hankel.h"
#include "../../include/mma_tdse.h"
#include "hankel_common.cuh"
#include "launch.cuh"

namespace mma {
namespace hk {
namespace plain {

constexpr int kT = 256, kWarpsP = kT / 32;
constexpr int kMaxRho = 2048;  // limit of the entry point
constexpr int kCoef = 12, kRow = 14;  // Taylor coefficients of a node, its centre, padding (16-byte rows)
constexpr int kNodes = 16384;         // table limit: arguments up to 4096
constexpr int kTerms = 32;            // series terms at most
constexpr int kSel = 2;               // planes the series form evaluates beside FF
constexpr int kPlanes = 16, kRad = 64;  // stage 1: planes per pass, radii per CTA
// the largest x that M terms serve, x^M/M! e^x <= 1e-17 (rounded down)
__constant__ double kCut[kTerms + 1] = {
    0, 1e-17, 4.47213e-09, 3.91486e-06, 0.000124462, 0.00103692, 0.00439107, 0.0125767, 0.0281295, 0.0532467, 0.0895544, 0.138072, 0.199288, 0.273265, 0.359759, 0.458314, 0.568344, 0.689189, 0.820157, 0.960555, 1.1097, 1.26697, 1.43173, 1.60342, 1.78152, 1.96553, 2.15501, 2.34954, 2.54876, 2.75231, 2.95987, 3.17116, 3.38592};

struct Plan {
    double d_ref, sigma, k_max, r_max, rho_max, d_min, u_max;
    double selw[kSel][kTerms];     // (1 - lambda^2)^m / m! of the selected planes
    int nodes, series;
};

__device__ __forceinline__ int terms_for(double x)
{
    int M = 2;
    while (M < kTerms && !(x <= kCut[M])) M += 2;
    return M;
}

__device__ double block_max(double v, double* red)
{
    for (int d = 16; d >= 1; d >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, d));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (int q = 1; q < kWarpsP; q++) v = fmax(v, red[q]);
    return v;
}

// One CTA: extents of the grids, the reference distance, the plane weights w[k][m] = tau_k v_k^m / m!
// (v = 1 - lambda^2), u[k] = 1/(2 D_k) - 1/(2 d_ref), and whether the series serves this call.
__global__ void __launch_bounds__(kT) plan_kernel(mma_hankel_problem P, const double* og, const double* rg,
                                                  const double* zg, const double* rho, const int64_t* slot, int n_planes,
                                                  Plan* out, double* w, double* u)
{
    __shared__ double red[kWarpsP];
    const int t = threadIdx.x;
    double km = 0.0, rm = 0.0, hm = 0.0, dn = 0.0, dx = 0.0, bad = 0.0;  // dn: largest 1/|D|
    for (int64_t i = t; i < P.n_omega; i += kT) km = fmax(km, fabs(og[i]));
    for (int64_t i = t; i < P.n_r; i += kT) rm = fmax(rm, fabs(rg[i]));
    for (int64_t i = t; i < P.n_rho; i += kT) hm = fmax(hm, fabs(rho[i]));
    for (int64_t i = t; i < P.n_z; i += kT) {
        const double D = P.distance - zg[i];
        if (!(D > 0.0)) bad = 1.0;
        dn = fmax(dn, 1.0 / fabs(D));
        dx = fmax(dx, fabs(D));
    }
    km = block_max(km, red) / kC;
    rm = block_max(rm, red);
    hm = block_max(hm, red);
    dn = block_max(dn, red);
    dx = block_max(dx, red);
    bad = block_max(bad, red);
    const double d_min = 1.0 / dn, d_ref = sqrt(2.0 / (dn * dn + 1.0 / (dx * dx)));
    double sg = 0.0, um = 0.0;
    for (int64_t i = t; i < P.n_z; i += kT) {
        const double D = P.distance - zg[i], tau = trap_w(zg, i, P.n_z);
        // 1 - lambda^2 and the phase's offset without cancellation
        const double v = (D - d_ref) * (D + d_ref) / (D * D), ui = (d_ref - D) / (2.0 * D * d_ref);
        sg = fmax(sg, fabs(v));
        um = fmax(um, fabs(ui));
        u[i] = ui;
        double c = tau;
#pragma unroll
        for (int m = 0; m < kTerms; m++) {
            w[i * kTerms + m] = c;
            c *= v * (1.0 / (m + 1));
        }
        if (slot && slot[i] >= 0 && slot[i] < kSel) {
            c = 1.0;
#pragma unroll
            for (int m = 0; m < kTerms; m++) {
                out->selw[slot[i]][m] = c;
                c *= v * (1.0 / (m + 1));
            }
        }
    }
    sg = block_max(sg, red);
    um = block_max(um, red);
    if (t == 0) {
        const double y = km * rm * hm / d_min;  // the largest argument of any plane
        out->d_ref = d_ref;
        out->sigma = sg;
        out->k_max = km;
        out->r_max = rm;
        out->rho_max = hm;
        out->d_min = d_min;
        out->u_max = um;
        const double want = 4.0 * y + 2.0;
        out->nodes = want < (double)kNodes ? (int)want : kNodes;
        // the series: operations per (omega, r) of both stages against the direct sum's
        const double x = 0.5 * sg * km * rm * hm / d_ref;
        const double M = terms_for(x);
        const double two = 80.0 * P.n_z + 2.0 * M * P.n_z + (30.0 + 6.0 * M) * P.n_rho, one = 17.0 * (double)P.n_z * P.n_rho;
        // distances whose squares leave the range of doubles (infinity too) have no reference distance
        const bool range = dn < 1e150 && dx < 1e150;
        out->series = n_planes <= kSel && bad == 0.0 && range && x <= kCut[kTerms] && want < (double)kNodes && two < one;
    }
}

// J0 and J1 at a node to rounding (CUDA's j1 is up to 4.4e-13 off on [25, 330], which a Taylor sum would
// carry into every value about the node): below 25 Miller's backward recurrence normalised by
// J0 + 2 (J2 + J4 + ...) = 1 (Abramowitz & Stegun 9.12), above it Hankel's asymptotic series
// (9.2.5-9.2.10), whose smallest term there is e^{-2x} = 2e-22.
__device__ void bessel01(double x, double& J0, double& J1)
{
    if (x < 25.0) {
        double p = 1e-250, pn = 0.0, even = 0.0;  // p ~ J_n, pn ~ J_{n+1}, from n = 72: J_72(25) = 5e-24
        const double ix = 2.0 / x;
        for (int n = 72; n > 0; n--) {
            if ((n & 1) == 0) even += p;
            const double q = fma(n * ix, p, -pn);
            pn = p;
            p = q;
        }
        const double s = 1.0 / fma(2.0, even, p);
        J0 = p * s;
        J1 = pn * s;
        return;
    }
    double sn, cs, P[2], Q[2];
    sincos(x, &sn, &cs);
#pragma unroll
    for (int nu = 0; nu < 2; nu++) {
        double t = 1.0;
        P[nu] = 1.0;
        Q[nu] = 0.0;
        for (int k = 0; k < 40 && fabs(t) > 1e-18; k++) {
            t *= (4.0 * nu - (2.0 * k + 1.0) * (2.0 * k + 1.0)) / ((k + 1) * 8.0 * x);
            // terms k + 1 = 1, 2, 3, 4, ...: Q, -P, -Q, P, ...
            const int r = (k + 1) & 3;
            if (r == 1) Q[nu] += t;
            else if (r == 2) P[nu] -= t;
            else if (r == 3) Q[nu] -= t;
            else P[nu] += t;
        }
    }
    const double f = rsqrt(3.14159265358979323846 * x);
    J0 = f * (P[0] * (cs + sn) - Q[0] * (sn - cs));
    J1 = f * (P[1] * (sn - cs) + Q[1] * (sn + cs));
}

// Taylor coefficients of J0 about node i/4: c_0 = J0, c_1 = -J1 and Bessel's equation; about 0 the
// power series.
__global__ void node_kernel(const Plan* plan, double* tab)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= plan->nodes) return;
    double* row = tab + (size_t)i * kRow;
    const double x = 0.25 * i;
    double c[kCoef];
    if (i == 0) {
        double v = 1.0;
        for (int n = 0; n < kCoef; n += 2) {
            c[n] = v;
            c[n + 1] = 0.0;
            v *= -0.25 / ((n / 2 + 1) * (n / 2 + 1));
        }
    } else {
        double J1;
        bessel01(x, c[0], J1);
        c[1] = -J1;
#pragma unroll
        for (int n = 0; n + 2 < kCoef; n++)
            c[n + 2] = -((n + 1) * (n + 1) * c[n + 1] + x * c[n] + (n > 0 ? c[n - 1] : 0.0)) / ((n + 2) * (n + 1) * x);
    }
#pragma unroll
    for (int n = 0; n < kCoef; n++) row[n] = c[n];
    row[kCoef] = x;
    row[kCoef + 1] = 0.0;
}

// e^{-i d}: the Taylor sums serve |d| <= 1/16 (next terms d^10/10!, d^11/11! below 3e-19)
__device__ __forceinline__ double2 phase_of(double d, bool small_)
{
    double sn, cs;
    if (small_) {
        const double q = d * d;
        sn = d * fma(q, fma(q, fma(q, fma(q, 1.0 / 362880.0, -1.0 / 5040.0), 1.0 / 120.0), -1.0 / 6.0), 1.0);
        cs = fma(q, fma(q, fma(q, fma(q, 1.0 / 40320.0, -1.0 / 720.0), 1.0 / 24.0), -0.5), 1.0);
    } else {
        sincos(d, &sn, &cs);
    }
    return make_double2(cs, -sn);
}
__device__ __forceinline__ double2 cm(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// ------------------------------------------------------------------------ series, stage 1
// B_m[w, r] = sum_k tau_k v_k^m / m! A_k[w, r]: a CTA takes 64 radii of one frequency.  Per pass of 16
// planes its threads form the A_k once into shared memory, then thread (r, group of 8 terms)
// accumulates; groups beyond the terms that the tile's largest argument needs do nothing.
__global__ void __launch_bounds__(kT) series_contract(mma_hankel_problem P, const Plan* plan, const double* og,
                                                      const double* rg, const double* zg, const void* src,
                                                      const double2* pre, const int64_t* slot, const double* w,
                                                      const double* u, int64_t o0, int64_t tiles, double2* B,
                                                      double2* asel)
{
    if (!plan->series) return;
    __shared__ double2 A[kPlanes][kRad];
    __shared__ double wk[kPlanes][kTerms];
    __shared__ double s_r[2];
    const int t = threadIdx.x, ri = t % kRad, mg = t / kRad;
    const int64_t ol = blockIdx.x / tiles, o = o0 + ol, r = blockIdx.x % tiles * kRad + ri;
    const bool in = r < P.n_r;
    const double k = og[o] / kC, rr = in ? rg[r] : 0.0, rw = in ? rr * trap_w(rg, r, P.n_r) : 0.0;
    const double kr2 = k * (rr * rr);
    double rmax = fabs(rr);
    for (int d = 16; d >= 1; d >>= 1) rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, d));
    if (t < kRad && (t & 31) == 0) s_r[t >> 5] = rmax;
    __syncthreads();
    rmax = fmax(s_r[0], s_r[1]);
    const int M = terms_for(0.5 * plan->sigma * fabs(k) * rmax * plan->rho_max / plan->d_ref);
    const bool small_ = fabs(k) * rmax * rmax * plan->u_max <= 0.0625;
    const double2 ref = P.near_field ? phase_of(kr2 / (2.0 * plan->d_ref), false) : make_double2(1.0, 0.0);
    double2 acc[8];
#pragma unroll
    for (int q = 0; q < 8; q++) acc[q] = make_double2(0.0, 0.0);
    for (int64_t k0 = 0; k0 < P.n_z; k0 += kPlanes) {
        const int np = (int)(P.n_z - k0 < kPlanes ? P.n_z - k0 : kPlanes);
        for (int kk = mg; kk < np; kk += kT / kRad) {
            double2 a = make_double2(0.0, 0.0);
            if (in) {
                const int64_t kz = k0 + kk;
                a = load_src_d(src, kz * P.plane_stride + o * P.omega_stride + r, P.source_c128);
                a = cm(a, pre_at(P, pre, kz, o, r));
                if (P.near_field) a = cm(a, phase_of(kr2 * u[kz], small_));
                a = make_double2(a.x * rw, a.y * rw);
                if (slot && slot[kz] >= 0 && slot[kz] < kSel) asel[(ol * kSel + slot[kz]) * P.n_r + r] = cm(a, ref);
            }
            A[kk][ri] = a;
        }
        for (int e = t; e < np * kTerms; e += kT) wk[e / kTerms][e % kTerms] = w[k0 * kTerms + e];
        __syncthreads();
        if (mg * 8 < M) {
            for (int kk = 0; kk < np; kk++) {
                const double2 a = A[kk][ri];
                const double* c = wk[kk] + mg * 8;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    acc[q].x = fma(c[q], a.x, acc[q].x);
                    acc[q].y = fma(c[q], a.y, acc[q].y);
                }
            }
        }
        __syncthreads();
    }
    if (in) {
        double2* b = B + (ol * P.n_r + r) * kTerms + mg * 8;
#pragma unroll
        for (int q = 0; q < 8; q++) b[q] = cm(acc[q], ref);
    }
}

// ------------------------------------------------------------------------ series, stage 2
// FF[rho, w] and the selected planes: a CTA takes RT screen radii of one frequency; its eight warps
// (and, for RT < 32, the 32/RT groups of lanes in each) share the medium's radii, 32 at a time through
// shared memory.  The launch takes the RT with the least work on the busiest SM.
template <int NS, int RT>
__global__ void __launch_bounds__(kT) series_sum(mma_hankel_problem P, const Plan* plan, const double* og,
                                                 const double* rg, const double* rho, const double2* B,
                                                 const double2* asel, const double* tab, int64_t o0, int64_t tiles,
                                                 int n_planes, double2* ff, double2* planes)
{
    if (!plan->series) return;
    constexpr int kSub = 32 / RT, kPar = kWarpsP * kSub;  // radii in flight
    __shared__ double2 Bs[32][kTerms + 1];  // a row more than the terms: the groups' rows in other banks
    __shared__ double2 As[NS > 0 ? NS : 1][32];
    __shared__ double pw[kTerms][2];
    __shared__ double rs[32];
    __shared__ double2 red[kWarpsP][32];
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const int64_t ol = blockIdx.x / tiles, o = o0 + ol, j = blockIdx.x % tiles * RT + lane % RT;
    const double k = fabs(og[o] / kC), rj = j < P.n_rho ? fabs(rho[j]) : 0.0;
    const double yk = k * rj / plan->d_ref;
    double ymax = yk;
    for (int d = 16; d >= 1; d >>= 1) ymax = fmax(ymax, __shfl_xor_sync(0xffffffffu, ymax, d));
    const int last = plan->nodes - 1;
    const double half_sigma = 0.5 * plan->sigma;
    for (int e = t; e < kTerms * 2; e += kT) pw[e / 2][e % 2] = e % 2 < n_planes ? plan->selw[e % 2][e / 2] : 0.0;
    double2 f = make_double2(0.0, 0.0), pl[NS > 0 ? NS : 1];
    for (int s = 0; s < NS; s++) pl[s] = f;
    for (int64_t r0 = 0; r0 < P.n_r; r0 += 32) {
        const int nr = (int)(P.n_r - r0 < 32 ? P.n_r - r0 : 32);
        __syncthreads();
        for (int e = t; e < nr * kTerms; e += kT) Bs[e / kTerms][e % kTerms] = B[(ol * P.n_r + r0) * kTerms + e];
        for (int e = nr * kTerms + t; e < 32 * kTerms; e += kT) Bs[e / kTerms][e % kTerms] = make_double2(0.0, 0.0);
        if constexpr (NS > 0)
            for (int e = t; e < NS * 32; e += kT)
                As[e / 32][e % 32] = e / 32 < n_planes && e % 32 < nr ? asel[(ol * kSel + e / 32) * P.n_r + r0 + e % 32]
                                                                      : make_double2(0.0, 0.0);
        if (t < 32) rs[t] = t < nr ? fabs(rg[r0 + t]) : 0.0;
        __syncthreads();
        for (int i0 = wp * kSub; i0 < nr; i0 += kPar) {
            const int i = i0 + lane / RT;
            double rtop = rs[i0];
#pragma unroll
            for (int s = 1; s < kSub; s++) rtop = fmax(rtop, rs[i0 + s]);
            const int M = terms_for(half_sigma * rtop * ymax);  // the same for the whole warp
            const double y = yk * rs[i];
            int nd = (int)fma(4.0f, (float)y, 0.5f);
            nd = nd < last ? nd : last;
            const double* c = tab + (size_t)nd * kRow;
            const double d = y - c[kCoef];
            double g0 = c[kCoef - 1], dj = 0.0;  // J0 and its derivative -J1 by one Horner sweep
#pragma unroll
            for (int n = kCoef - 2; n >= 0; n--) {
                dj = fma(dj, d, g0);
                g0 = fma(g0, d, c[n]);
            }
            const double h = 0.5 * y, q = h * h;
            double g1 = -h * dj;
            const double2* b = Bs[i];
            f.x = fma(g0, b[0].x, f.x);
            f.y = fma(g0, b[0].y, f.y);
            f.x = fma(g1, b[1].x, f.x);
            f.y = fma(g1, b[1].y, f.y);
            double js[NS > 0 ? NS : 1];
#pragma unroll
            for (int s = 0; s < NS; s++) js[s] = fma(pw[1][s], g1, pw[0][s] * g0);
            double mm = 1.0;  // m of G_{m+1} = m G_m - (y/2)^2 G_{m-1}
            for (int m = 2; m < M; m += 2) {
                g0 = fma(-q, g0, mm * g1);
                g1 = fma(-q, g1, (mm + 1.0) * g0);
                mm += 2.0;
                f.x = fma(g0, b[m].x, f.x);
                f.y = fma(g0, b[m].y, f.y);
                f.x = fma(g1, b[m + 1].x, f.x);
                f.y = fma(g1, b[m + 1].y, f.y);
#pragma unroll
                for (int s = 0; s < NS; s++) js[s] = fma(pw[m + 1][s], g1, fma(pw[m][s], g0, js[s]));
            }
#pragma unroll
            for (int s = 0; s < NS; s++) {
                pl[s].x = fma(js[s], As[s][i].x, pl[s].x);
                pl[s].y = fma(js[s], As[s][i].y, pl[s].y);
            }
        }
    }
    auto total = [&](double2 v) {  // over the lane groups and the warps, in a fixed order
#pragma unroll
        for (int d = RT; d < 32; d <<= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
        }
        __syncthreads();
        red[wp][lane] = v;
        __syncthreads();
        double2 s = red[0][lane];
        for (int q = 1; q < kWarpsP; q++) s = make_double2(s.x + red[q][lane].x, s.y + red[q][lane].y);
        return s;
    };
    f = total(f);
    const bool out = wp == 0 && lane < RT && j < P.n_rho;
    if (out) ff[j * P.n_omega + o] = f;
#pragma unroll
    for (int s = 0; s < NS; s++) {
        const double2 v = total(pl[s]);
        if (out && s < n_planes) planes[(s * P.n_rho + j) * P.n_omega + o] = v;
    }
}

// ------------------------------------------------------------------------ direct sum
// One J0 per (w, k, rho, r): a CTA takes 32 screen radii (lanes) of one frequency, its eight warps
// share the medium's radii.  Per plane the CTA builds A_k[r] in shared memory; the nodes that its
// arguments reach sit behind it where they fit (`room` doubles), else they are read through L1.
__global__ void __launch_bounds__(kT) direct_kernel(mma_hankel_problem P, const Plan* plan, const double* og,
                                                    const double* rg, const double* zg, const double* rho,
                                                    const void* src, const double2* pre, const double* tab,
                                                    int64_t tiles, int64_t room, double2* ff, const int64_t* slot,
                                                    double2* planes)
{
    if (plan->series) return;
    extern __shared__ double2 A[];  // n_r, then the nodes
    __shared__ double2 red[kWarpsP][32];
    double* const near_ = reinterpret_cast<double*>(A + P.n_r);
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5;
    const int64_t Nr = P.n_r, o = blockIdx.x / tiles, j = blockIdx.x % tiles * 32 + lane;
    const double k = og[o] / kC, rj = j < P.n_rho ? rho[j] : 0.0;
    double hmax = fabs(rj);
    for (int d = 16; d >= 1; d >>= 1) hmax = fmax(hmax, __shfl_xor_sync(0xffffffffu, hmax, d));
    const double want = 4.0 * (fabs(k) * plan->r_max * hmax / plan->d_min) + 2.0;
    const int nodes = want < (double)plan->nodes ? (int)want : plan->nodes;  // nodes this CTA reaches
    const bool own = (int64_t)nodes * kRow <= room;
    if (own)
        for (int e = t; e < nodes * kRow; e += kT) near_[e] = tab[e];
    auto total = [&](double2 v) {
        __syncthreads();
        red[wp][lane] = v;
        __syncthreads();
        double2 s = red[0][lane];
        for (int q = 1; q < kWarpsP; q++) s = make_double2(s.x + red[q][lane].x, s.y + red[q][lane].y);
        return s;
    };
    double2 acc = make_double2(0.0, 0.0);
    for (int64_t kz = 0; kz < P.n_z; kz++) {
        const double D = P.distance - zg[kz];
        __syncthreads();
        for (int64_t r = t; r < Nr; r += kT) {
            const double rr = rg[r];
            double2 a = cm(load_src_d(src, kz * P.plane_stride + o * P.omega_stride + r, P.source_c128), pre_at(P, pre, kz, o, r));
            if (P.near_field) a = cm(a, phase_of(k * (rr * rr) / (2.0 * D), false));  // Hankel_transform.py:506
            const double w = rr * trap_w(rg, r, Nr);
            A[r] = make_double2(a.x * w, a.y * w);
        }
        __syncthreads();
        const double yk = fabs(k * rj / D);
        double2 p = make_double2(0.0, 0.0);
        auto sum = [&](const double* T) {
#pragma unroll 2
            for (int64_t r = wp; r < Nr; r += kWarpsP) {
                const double y = yk * fabs(rg[r]);
                const int nd = (int)fma(4.0f, (float)y, 0.5f);
                double J;
                if (nd >= 0 && nd < nodes) {
                    const double* c = T + (size_t)nd * kRow;
                    const double d = y - c[kCoef];
                    J = c[kCoef - 1];
#pragma unroll
                    for (int n = kCoef - 2; n >= 0; n--) J = fma(J, d, c[n]);
                } else {
                    J = ::j0(y);
                }
                p.x = fma(A[r].x, J, p.x);
                p.y = fma(A[r].y, J, p.y);
            }
        };
        if (own) sum(near_); else sum(tab);
        const double tau = trap_w(zg, kz, P.n_z);
        acc.x = fma(tau, p.x, acc.x);
        acc.y = fma(tau, p.y, acc.y);
        const int64_t sl = slot ? slot[kz] : -1;
        if (sl >= 0 && planes) {
            p = total(p);
            if (wp == 0 && j < P.n_rho) planes[(sl * P.n_rho + j) * P.n_omega + o] = p;
        }
    }
    acc = total(acc);
    if (wp == 0 && j < P.n_rho) ff[j * P.n_omega + o] = acc;
}

// ------------------------------------------------------------------------ workspace
int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

size_t up(size_t v) { return (v + 255) / 256 * 256; }
// frequencies per pass of the series: B takes 512 bytes per (omega, r), kept to 64 MB
int64_t block_of(const mma_hankel_problem* p)
{
    const int64_t n = ((int64_t)64 << 20) / (p->n_r * kTerms * 16);
    return n < 1 ? 1 : n < p->n_omega ? n : p->n_omega;
}
struct Layout {
    size_t tab, w, u, B, asel, total;
};
Layout layout(const mma_hankel_problem* p)
{
    Layout l;
    const size_t ob = (size_t)block_of(p), nr = (size_t)p->n_r;
    l.tab = up(sizeof(Plan));
    l.w = l.tab + up(sizeof(double) * kNodes * kRow);
    l.u = l.w + up(sizeof(double) * (size_t)p->n_z * kTerms);
    l.B = l.u + up(sizeof(double) * (size_t)p->n_z);
    l.asel = l.B + up(sizeof(double2) * ob * nr * kTerms);
    l.total = l.asel + up(sizeof(double2) * ob * nr * kSel);
    return l;
}

}  // namespace plain
}  // namespace hk
}  // namespace mma

using namespace mma::hk;

extern "C" size_t mma_hankel_plain_scratch_bytes(const mma_hankel_problem* p) { return valid(p) ? plain::layout(p).total : 0; }

extern "C" int mma_hankel_plain_ws(const mma_hankel_problem* p, const double* ogrid, const double* rgrid,
                                   const double* zgrid, const double* rho, const void* source, const double* pre,
                                   double* ff, const int64_t* plane_slot, int n_planes, double* planes, void* scratch,
                                   size_t scratch_bytes, void* stream)
{
    using namespace plain;
    if (!valid(p) || !ogrid || !rgrid || !zgrid || !rho || !source || !ff || !scratch) return MMA_ERR_ARG;
    if (p->n_rho > kMaxRho) return MMA_ERR_TOO_LARGE;
    if ((n_planes > 0) != (plane_slot != nullptr && planes != nullptr)) return MMA_ERR_ARG;
    const size_t a_bytes = sizeof(double2) * (size_t)p->n_r;
    if (a_bytes > 220 * 1024) return MMA_ERR_TOO_LARGE;
    const Layout l = layout(p);
    if (scratch_bytes < l.total) return MMA_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    char* base = static_cast<char*>(scratch);
    Plan* plan = reinterpret_cast<Plan*>(base);
    double *tab = reinterpret_cast<double*>(base + l.tab), *w = reinterpret_cast<double*>(base + l.w),
           *u = reinterpret_cast<double*>(base + l.u);
    double2 *B = reinterpret_cast<double2*>(base + l.B), *asel = reinterpret_cast<double2*>(base + l.asel);
    const double2* pre2 = reinterpret_cast<const double2*>(pre);
    double2 *ff2 = reinterpret_cast<double2*>(ff), *pl2 = reinterpret_cast<double2*>(planes);
    const int64_t* slot = n_planes > 0 ? plane_slot : nullptr;
    plan_kernel<<<1, kT, 0, st>>>(*p, ogrid, rgrid, zgrid, rho, slot, n_planes, plan, w, u);
    node_kernel<<<kNodes / 128, 128, 0, st>>>(plan, tab);
    const int64_t jt = (p->n_rho + 31) / 32, rt = (p->n_r + kRad - 1) / kRad, ob = block_of(p);
    if (n_planes <= kSel)  // the kernels below return at once where the plan decided against the series
        for (int64_t o0 = 0; o0 < p->n_omega; o0 += ob) {
            const int64_t no = p->n_omega - o0 < ob ? p->n_omega - o0 : ob;
            series_contract<<<(unsigned)(no * rt), kT, 0, st>>>(*p, plan, ogrid, rgrid, zgrid, source, pre2, slot, w, u,
                                                                 o0, rt, B, asel);
            // screen radii per CTA: CTAs on the busiest SM times the radii of each (and about 1 more
            // for staging B); 64 omega x 128 rho: 63 with 8 radii, 66 with 32
            const int sms = sm_count();
            int best = 32;
            int64_t cost = INT64_MAX;
            for (int q = 32; q >= 8; q /= 2) {
                const int64_t c = ((p->n_rho + q - 1) / q * no + sms - 1) / sms * (q + 1);
                if (c < cost) {
                    cost = c;
                    best = q;
                }
            }
            auto sum = n_planes > 0 ? (best == 32 ? series_sum<kSel, 32> : best == 16 ? series_sum<kSel, 16> : series_sum<kSel, 8>)
                                    : (best == 32 ? series_sum<0, 32> : best == 16 ? series_sum<0, 16> : series_sum<0, 8>);
            const int64_t nt = (p->n_rho + best - 1) / best;
            sum<<<(unsigned)(no * nt), kT, 0, st>>>(*p, plan, ogrid, rgrid, rho, B, asel, tab, o0, nt, n_planes, ff2, pl2);
        }
    // the nodes of arguments up to about 320 beside A, else what fits
    size_t smem = a_bytes + sizeof(double) * 1300 * kRow;
    if (smem > 220 * 1024) smem = 220 * 1024;
    if (mma::allow_smem(direct_kernel) != cudaSuccess)
        return MMA_ERR_CUDA;
    direct_kernel<<<(unsigned)(p->n_omega * jt), kT, smem, st>>>(*p, plan, ogrid, rgrid, zgrid, rho, source, pre2, tab, jt,
                                                                 (int64_t)((smem - a_bytes) / sizeof(double)), ff2, slot,
                                                                 pl2);
    return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
}

extern "C" int mma_hankel_plain(const mma_hankel_problem* p, const double* ogrid, const double* rgrid,
                                const double* zgrid, const double* rho, const void* source, const double* pre,
                                double* ff, const int64_t* plane_slot, int n_planes, double* planes, void* stream)
{
    if (!valid(p)) return MMA_ERR_ARG;
    const size_t bytes = mma_hankel_plain_scratch_bytes(p);
    void* ws = nullptr;
    if (!mma::succeeded(cudaMallocAsync(&ws, bytes, (cudaStream_t)stream))) return MMA_ERR_CUDA;
    const int rc = mma_hankel_plain_ws(p, ogrid, rgrid, zgrid, rho, source, pre, ff, plane_slot, n_planes, planes, ws,
                                       bytes, stream);
    return mma::succeeded(cudaFreeAsync(ws, (cudaStream_t)stream)) ? rc : MMA_ERR_CUDA;
}
