// tdse_analysis.cu -- analysis kernels of the TDSE library, batched on the GPU:
//   * the photoelectron spectrum by the resolvent window method (1DTDSE/sources/tools.c:206-316,
//     window_analysis): for every energy E_i two complex Numerov-tridiagonal solves,
//       (M2 (E_i - dE - i dE - V) - K) u1 = M2 psi,   (M2 (E_i + dE + i dE - V) - K) u2 = M2 u1,
//       PES_i = dx dE^4 sum_j |u2_j|^2,
//     by two threads per energy that eliminate from both ends, or a warp per energy (tridiag.c:26-70,
//     251-274), in FP64 and with the elimination factors interleaved so that a warp's loads coalesce;
//   * the Gabor transform (tools_fftw3.c:158-213, GaborTransform): for every window centre
//     t_w = t_min + w (t_max - t_min)/N_G the signal times exp(-((t_j - t_w)/a)^2), a real DFT
//     (this library's own, dft.cu, batched over windows and signals) and dt/sqrt(2 pi) |DFT_k| for
//     k < N_freq.
// The arithmetic follows the reference's expressions and their order (FP64).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdlib>
#include <cstring>

#include "../../include/mma_tdse.h"
#include "common.cuh"
#include "dft.cuh"
#include "launch.cuh"

namespace mma {
namespace an {

constexpr double kPi = 3.14159265358979323846;

// Both kernels below share the row arithmetic.  Row j of (M2 (Es -/+ i dE - V) - K) couples u_{j-1},
// u_j, u_{j+1} by w_{j-1}, b_j, w_{j+1} (tools.c:257-275):
//   w_j = (Es - V_j)/12 + 0.5/dx^2 -/+ i dE/12,  b_j = 10 (Es - V_j)/12 - 1/dx^2 -/+ i 10 dE/12,
// and the elimination in either direction is gamma_j = w_j / beta_p, beta_j = b_j - w_p gamma_j,
// y_j = (r_j - w_p y_p)/beta_j with p the row before, then u_p = y_p - gamma_j u_j backwards
// (tridiag.c:26-70), with one reciprocal of |beta|^2 per row.
struct PesArgs {
    int64_t n;  // rows = num_r + 1
    double dx, dE, Estep, E_start;
    int num_E, e0, count;  // energies e0 .. e0 + count - 1 of num_E
    const double* V12;     // V / 12
    const cd* rhs0;        // M2 psi
    double* pes;           // [num_E]
};

// The rows of one energy and window (sg = -1: first, +1: second).  Energy and potential are combined
// before the 1/dx^2 terms, as in the reference: with Es/12 + 0.5/dx^2 formed once, its rounding is the
// same in every row, an energy shift that the 1/dE of the window amplifies (7 times the error).
struct Rows {
    double e12, e10, diag, off, wi, bi;
    __device__ Rows(const PesArgs& A, int ie, double sg)
    {
        const double Es = (A.E_start + A.Estep * ie) + sg * A.dE, s = sg < 0 ? -1.0 : 1.0;
        e12 = Es / 12.;
        e10 = 10 * Es / 12.;
        diag = 1. / (A.dx * A.dx);
        off = -0.5 / (A.dx * A.dx);
        wi = s * (A.dE / 12);
        bi = s * (10 * A.dE / 12);
    }
    __device__ cd w(double v12) const { return cd{(e12 - v12) - off, wi}; }
    __device__ cd b(double v12) const { return cd{fma(-10.0, v12, e10) - diag, bi}; }
};

__device__ __forceinline__ cd cinv(cd b)
{
    const double s = 1.0 / fma(b.re, b.re, b.im * b.im);
    return cd{b.re * s, -b.im * s};
}
__device__ __forceinline__ cd ldro(const cd* p)  // read-only for the whole launch
{
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return cd{v.x, v.y};
}
// M2 u of a row
__device__ __forceinline__ cd m2(cd m, cd c, cd p)
{
    constexpr double k12 = 1.0 / 12.;
    return cd{fma(10.0, c.re, p.re + m.re) * k12, fma(10.0, c.im, p.im + m.im) * k12};
}

// fn(k, ld(k)) for k = 0 .. cnt - 1, the loads of a block of B one block ahead of their use: a row of a
// substitution is six operations, about 400 cycles of a pipe that one warp feeds, and its loads take
// a thousand (a wave of pairs 15.4 ms without this, 12.4 with)
template <int B, typename Ld, typename Fn>
__device__ __forceinline__ void piped(int64_t cnt, Ld ld, Fn fn)
{
    typedef decltype(ld((int64_t)0)) V;
    V cur[B], nxt[B];
#pragma unroll
    for (int q = 0; q < B; q++)
        if (q < cnt) cur[q] = ld(q);
    for (int64_t k = 0; k < cnt; k += B) {
#pragma unroll
        for (int q = 0; q < B; q++)
            if (k + B + q < cnt) nxt[q] = ld(k + B + q);
#pragma unroll
        for (int q = 0; q < B; q++)
            if (k + q < cnt) fn(k + q, cur[q]);
#pragma unroll
        for (int q = 0; q < B; q++) cur[q] = nxt[q];
    }
}
struct Two {
    cd g, y;
};
struct Three {
    cd g, y, f;
};

// Energy-independent tables: x_k = k dx - xmax with xmax = 0.5 num_r dx (tools.c:231, 246), V(x_k) =
// -1/sqrt(a^2 + x^2) (tools.c:91-95) kept as V/12, and the right-hand side of the first solve, M2 psi =
// (10 psi_j + psi_{j-1} + psi_{j+1})/12 (tridiag.c:261-268), the same for every energy; in natural order
// and, rows beyond the grid zero, with row j = s m + i at [i][s] for the warp kernel (s < 32).
__global__ void pes_tables(int64_t n, int64_t m, int num_r, double dx, double a, const double* psi, double* V12,
                           cd* rhs0, double* V12t, cd* rhs0t)
{
    const double xmax = __dmul_rn(__dmul_rn(0.5, (double)num_r), dx);
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < 32 * m; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t q = k % m * 32 + k / m;
        if (k >= n) {
            V12t[q] = 0.0;
            rhs0t[q] = cd{0.0, 0.0};
            continue;
        }
        const double x = __dsub_rn(__dmul_rn((double)k, dx), xmax);
        const double v = (-1.0 / sqrt(a * a + x * x)) / 12.;
        const cd pc{psi[2 * k], psi[2 * k + 1]};
        const cd pm = k > 0 ? cd{psi[2 * k - 2], psi[2 * k - 1]} : cd{0.0, 0.0};
        const cd pn = k + 1 < n ? cd{psi[2 * k + 2], psi[2 * k + 3]} : cd{0.0, 0.0};
        const cd r{10 * pc.re / 12. + (pn.re + pm.re) / 12., 10 * pc.im / 12. + (pn.im + pm.im) / 12.};
        V12[k] = V12t[q] = v;
        rhs0[k] = rhs0t[q] = r;
    }
}

// ------------------------------------------------------------------------ two threads per energy
// Elimination from both ends towards the middle and substitution outwards again: the operations of one
// Thomas sweep at half its length, on twice the threads.  A CTA takes 64 energies; its four warps (two
// groups of energies, two sides) sit on the SM's four sub-partitions, whose FP64 pipes they fill: a full
// wave is 64 energies an SM.  One thread per energy left two of the four pipes of each SM idle.
struct PesPair {
    PesArgs A;
    cd* gam;  // [n][stride]
    cd* u;    // [n][stride]
    int64_t stride;
};

__device__ __forceinline__ void pes_pair(const PesPair& Q)
{
    const PesArgs& A = Q.A;
    __shared__ cd s_y[2][64], s_g[2][64];
    __shared__ double s_n[64];
    const int w = threadIdx.x >> 5, side = w >> 1, el = (w & 1) * 32 + (threadIdx.x & 31);
    int e = blockIdx.x * 64 + el;
    const bool live = e < A.count;
    if (!live) e = A.count - 1;  // an idle lane repeats the last energy into no output and no buffer
    const int64_t n = A.n, h = n / 2, C = Q.stride;
    const int64_t d = side ? -1 : 1, first = side ? n - 1 : 0, cnt = side ? n - h : h;
    cd* const gam = Q.gam + e;
    cd* const u = Q.u + e;
    cd mine{0.0, 0.0}, other{0.0, 0.0};  // the solution at the last row of this side and of the other
    double nrm = 0.0;
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        const Rows R(A, A.e0 + e, pass ? 1.0 : -1.0);
        cd pm{0.0, 0.0}, pc{0.0, 0.0}, pn{0.0, 0.0};
        if (pass) {
            pc = cnt > 1 ? u[first * C] : mine;
            pn = cnt > 2 ? u[(first + d) * C] : cnt > 1 ? mine : other;
        }
        cd wp{0.0, 0.0}, ibeta{0.0, 0.0}, y{0.0, 0.0};
#pragma unroll 2
        for (int64_t i = 0; i < cnt; i++) {
            const int64_t j = first + d * i;
            const double v = __ldg(A.V12 + j);
            const cd wj = R.w(v);
            cd r;
            if (pass) {
                r = m2(pm, pc, pn);
                pm = pc;
                pc = pn;
                pn = i + 3 < cnt ? u[(j + 2 * d) * C] : i + 3 == cnt ? mine : other;
            } else {
                r = ldro(A.rhs0 + j);
            }
            const cd g = cmul(wj, ibeta);
            ibeta = cinv(cfms(wp, g, R.b(v)));
            y = cmul(cfms(wp, y, r), ibeta);
            wp = wj;
            if (live) {
                gam[j * C] = g;
                u[j * C] = y;
            }
        }
        // the two middle rows: u_a = y_a - g_a u_b, u_b = y_b - g_b u_a
        s_y[side][el] = y;
        s_g[side][el] = cmul(R.w(A.V12[side ? h - 1 : h]), ibeta);
        __syncthreads();
        const cd yo = s_y[1 - side][el], go = s_g[1 - side][el], gm = s_g[side][el];
        const cd det = cfms(gm, go, cd{1.0, 0.0});
        mine = cmul(cfms(gm, yo, y), cinv(det));
        other = cfms(go, mine, yo);
        __syncthreads();
        // substitution outwards; the middle row's value stays in a register (the second pass reads it there)
        cd un = mine;
        nrm = un.re * un.re + un.im * un.im;
        const int64_t top = first + d * (cnt - 2);  // row of k = 0
        piped<4>(
            cnt - 1, [&](int64_t k) { return Two{gam[(top - d * k + d) * C], u[(top - d * k) * C]}; },
            [&](int64_t k, const Two& v) {
                un = cfms(v.g, un, v.y);
                if (live && pass == 0) u[(top - d * k) * C] = un;
                nrm = fma(un.re, un.re, fma(un.im, un.im, nrm));
            });
    }
    if (side) s_n[el] = nrm;
    __syncthreads();
    if (!side && live) A.pes[A.e0 + e] = (nrm + s_n[el]) * A.dx * pow(A.dE, 4.);
}

// ------------------------------------------------------------------------ one warp per energy
// Lane s owns rows s m .. s m + m - 1 and eliminates them from its first row on, carrying the dependence
// f_j on the row before the chunk (u_j = y_j + f_j u_L - gamma_{j+1} u_{j+1}).  A backward pass without
// stores expresses the chunk's first value by u_L and its last value z; the 32 last values then satisfy a
// tridiagonal system across the lanes (parallel cyclic reduction, five levels), and a second backward
// pass gives u.  About 66 FP64 operations a row and solve against 42 of the pair kernel, but 1/32 of its
// chain: few energies, and what full waves of the pair kernel leave over, run here.
struct PesWarp {
    PesArgs A;
    int64_t m;
    cd* buf;  // per warp: gamma, y (then u), f, each [m][32]
};

__device__ __forceinline__ void pes_warp(const PesWarp& Q, int block, int blocks)
{
    const PesArgs& A = Q.A;
    const int lane = threadIdx.x & 31, slot = block * 4 + (threadIdx.x >> 5), slots = blocks * 4;
    const int64_t m = Q.m, n = A.n;
    cd* const gam = Q.buf + (int64_t)slot * 96 * m + lane;
    cd* const yb = gam + 32 * m;
    cd* const fb = yb + 32 * m;
    const int64_t a = lane * m, left = n - a;
    const int64_t cnt = left < 0 ? 0 : left < m ? left : m;  // rows of this lane
    const cd zero{0.0, 0.0};
    auto from = [](cd v, int l) { return cd{shfl_idx(v.re, l), shfl_idx(v.im, l)}; };
    for (int e = slot; e < A.count; e += slots) {
        double nrm = 0.0;
        cd uL = zero, uR = zero;  // solution of the first window beside the chunk
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {
            const Rows R(A, A.e0 + e, pass ? 1.0 : -1.0);
            cd wp = lane > 0 && cnt > 0 ? R.w(A.V12[(m - 1) * 32 + lane - 1]) : zero;  // w of the row before the chunk
            cd ibeta = zero, y = zero, f = cd{1.0, 0.0};
            cd pm = uL, pc = pass ? yb[0] : zero, pn = zero;
            for (int64_t i = 0; i < cnt; i++) {
                const double v = __ldg(A.V12 + i * 32 + lane);
                const cd wj = R.w(v);
                cd r;
                if (pass) {
                    pn = i + 1 < cnt ? yb[(i + 1) * 32] : uR;
                    r = m2(pm, pc, pn);
                    pm = pc;
                    pc = pn;
                } else {
                    r = ldro(A.rhs0 + i * 32 + lane);
                }
                const cd g = cmul(wj, ibeta);  // 0 in the chunk's first row: the elimination starts afresh
                const cd beta = i > 0 ? cfms(wp, g, R.b(v)) : R.b(v);
                ibeta = cinv(beta);
                const cd hq = cmul(wp, ibeta);
                y = cfms(hq, y, cmul(r, ibeta));
                f = cfms(hq, f, zero);
                gam[i * 32] = g;
                yb[i * 32] = y;
                fb[i * 32] = f;
                wp = wj;
            }
            // u_first = Y + F u_L + H z
            cd Y = zero, F = zero, H = cd{1.0, 0.0};
            auto row = [&](int64_t k) {
                const int64_t i = cnt - 2 - k;
                return Three{gam[(i + 1) * 32], yb[i * 32], fb[i * 32]};
            };
            piped<2>(cnt - 1, row, [&](int64_t, const Three& v) {
                Y = cfms(v.g, Y, v.y);
                F = cfms(v.g, F, v.f);
                H = cfms(v.g, H, zero);
            });
            // z_s (1 + g F') = (y - g Y') + f z_{s-1} - g H' z_{s+1}, primes: the next lane's chunk
            const bool next = lane < 31 && a + m < n;
            const cd gb = next ? cmul(R.w(A.V12[lane + 1]), ibeta) : zero;
            const cd Yn = from(Y, lane + 1 < 32 ? lane + 1 : 31), Fn = from(F, lane + 1 < 32 ? lane + 1 : 31),
                     Hn = from(H, lane + 1 < 32 ? lane + 1 : 31);
            cd iq = cinv(cfma(gb, Fn, cd{1.0, 0.0}));
            if (cnt == 0) y = f = zero;
            cd Rz = cmul(cfms(gb, Yn, y), iq), Az = lane > 0 ? cmul(f, iq) : zero, Cz = cmul(cfms(gb, Hn, zero), iq);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int lo = lane - d < 0 ? 0 : lane - d, hi = lane + d > 31 ? 31 : lane + d;
                const cd Rm = from(Rz, lo), Am = from(Az, lo), Cm = from(Cz, lo);
                const cd Rp = from(Rz, hi), Ap = from(Az, hi), Cp = from(Cz, hi);
                iq = cinv(cfms(Cz, Ap, cfms(Az, Cm, cd{1.0, 0.0})));
                Rz = cmul(cfma(Cz, Rp, cfma(Az, Rm, Rz)), iq);
                Az = cmul(cmul(Az, Am), iq);
                Cz = cmul(cmul(Cz, Cp), iq);
                if (lane < 2 * d) Az = zero;
                if (lane + 2 * d > 31) Cz = zero;
            }
            const cd z = Rz, zl = from(z, lane > 0 ? lane - 1 : 0);
            const cd vL = lane > 0 ? zl : zero;
            cd u = z;
            if (cnt > 0) {
                nrm = u.re * u.re + u.im * u.im;
                if (pass == 0) yb[(cnt - 1) * 32] = u;
            }
            piped<2>(cnt - 1, row, [&](int64_t k, const Three& v) {
                u = cfms(v.g, u, cfma(v.f, vL, v.y));
                if (pass == 0) yb[(cnt - 2 - k) * 32] = u;
                nrm = fma(u.re, u.re, fma(u.im, u.im, nrm));
            });
            uL = vL;  // and the next lane's first value
            const cd un = from(u, lane + 1 < 32 ? lane + 1 : 31);
            uR = next ? un : zero;
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) nrm += shfl_xor(nrm, d);
        if (lane == 0) A.pes[A.e0 + e] = nrm * A.dx * pow(A.dE, 4.);
    }
}

// A wave of pairs (the first `pairs` CTAs) and the energies beyond it a warp each (the others), which
// share the SMs: the pairs' one warp per pipe leaves a quarter of its cycles free.
__global__ void __launch_bounds__(128) pes_kernel(PesPair Q, int pairs, PesWarp W)
{
    if ((int)blockIdx.x < pairs) pes_pair(Q);
    else pes_warp(W, blockIdx.x - pairs, gridDim.x - pairs);
}

// Gabor windows exp(-(ia (j dt - (t_min + w dt_G)))^2) (tools_fftw3.c:180-196, ia = 1/a), the
// same for every signal: tabulated once per call, [N_G][N]
__global__ void gabor_table(int N, int N_G, double dt, double t_min, double dt_G, double ia, double* win)
{
    const int64_t total = (int64_t)N_G * N;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = q % N, w = q / N;
        const double arg = ia * (((double)j) * dt - (t_min + ((double)w) * dt_G));
        win[q] = exp(-(arg * arg));  // arg * arg: the correctly rounded square, as pow(arg, 2.)
    }
}

// windowed signals in[(s N_G + w) N + j] = win[w][j] signal_s[j]
__global__ void gabor_window(const double* sig, int64_t stride, int n_sig, int N, int N_G, const double* win,
                             double* in)
{
    const int64_t total = (int64_t)n_sig * N_G * N;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = q % N, b = q / N, w = b % N_G, s = b / N_G;
        in[q] = win[w * N + j] * sig[s * stride + j];
    }
}

// |DFT| of the first N_freq bins times dt/sqrt(2 pi) (tools_fftw3.c:203-205)
__global__ void gabor_abs(const double2* out, int64_t Nc, int64_t nb, int N_freq, double norm, double* g)
{
    const int64_t total = nb * N_freq;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = q % N_freq, b = q / N_freq;
        const double2 v = out[b * Nc + k];
        g[q] = norm * sqrt((v.x * v.x + v.y * v.y));
    }
}

int grid_for(int64_t total) { return (int)((total + 255) / 256 < 8192 ? (total + 255) / 256 : 8192); }

}  // namespace an
}  // namespace mma

using namespace mma;


namespace {
// scratch: V/12 [n + 1] | M2 psi [n] | gam [n][chunk] | u [n][chunk]
size_t pes_fixed(size_t n) { return (sizeof(double) * (n + 1) + 255) / 256 * 256 + (sizeof(cd) * n + 255) / 256 * 256; }

int pes_sms()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 152;  // sizes can be asked for without a device
}

// Whether pairs serve `left` energies (or the first wave of them, 64 energies an SM) of n rows sooner than a
// warp each.  Pairs take a chain of n/2 rows twice, however many they are; a warp each has 1/32 of the chain
// but 66 operations a row against 40 and, per energy, two cyclic reductions across its lanes, as much as six
// rows a lane.  us, measured / model: pairs 51 rows 77 / 88, 601 rows 980 / 979, 8001 rows 13000 / 12970;
// warps 51 rows, 3000 energies 188 / 167, 601 rows, 10 energies 112 / 109, 3000 energies 620 / 637, 8001
// rows, 50 energies 1370 / 1340, 3000 energies 7040 / 7040, 5000 energies 11000 / 11030.  (One thread an
// energy took 26 to 34 ms for 8001 rows; 10000 energies take 13.9 ms, a wave of pairs and 272 warps.)
bool pes_by_pairs(int64_t left, int64_t n, int sms)
{
    if (n < 4) return false;
    if (left >= (int64_t)64 * sms) return true;
    const double m = (double)((n + 31) / 32), chain = 8.0 + 5.3 * m;
    const double load = 0.8 * chain + (double)left * (0.035 + 0.0078 * m) * 152.0 / sms;
    return 5.0 + 1.62 * (double)n < (chain > load ? chain : load);
}
}  // namespace

extern "C" size_t mma_tdse_pes_scratch_bytes(int num_r, int chunk)
{
    if (num_r < 1 || chunk < 1) return 0;
    const size_t n = (size_t)num_r + 1, m = (n + 31) / 32;
    // the pairs' two arrays of `chunk` energies, then gamma, y and f of the energies that a warp each
    // takes: those beyond full waves of pairs, as many as run at once (16 warps an SM)
    const int sms = pes_sms();
    const size_t wave = 64 * (size_t)sms, left = (size_t)chunk % wave;
    const size_t rest = left > 0 && !pes_by_pairs((int64_t)left, (int64_t)n, sms) ? left : 0;
    const size_t warps = ((size_t)chunk < wave ? (size_t)chunk : rest) + 3;
    return pes_fixed(n) + 32 * m * 24 + 512 + 2 * sizeof(cd) * n * ((size_t)chunk - rest) +
           48 * 32 * m * ((warps < 16 * (size_t)sms ? warps : 16 * (size_t)sms) / 4 * 4);
}

extern "C" int mma_tdse_pes(const double* psi, int num_r, double dx, double trg_a, int num_E, double dE, double Estep,
                            double E_start, double* pes, void* scratch, size_t scratch_bytes, void* stream)
{
    if (!psi || !pes || !scratch || num_r < 1 || num_E < 1 || !(dx > 0.0)) return MMA_ERR_ARG;
    const int64_t n = (int64_t)num_r + 1, m = (n + 31) / 32;
    const size_t fixed = pes_fixed((size_t)n);
    if (scratch_bytes < fixed + 2 * sizeof(cd) * (size_t)n) return MMA_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    char* sc = static_cast<char*>(scratch);
    double* V12 = reinterpret_cast<double*>(sc);
    cd* rhs0 = reinterpret_cast<cd*>(sc + (sizeof(double) * (size_t)(n + 1) + 255) / 256 * 256);
    // behind the fixed tables: the warp kernel's tables, then either kernel's buffers
    const size_t tabs = ((size_t)(32 * m) * 24 + 255) / 256 * 256, one = sizeof(cd) * 96 * (size_t)m;
    char* rest = sc + fixed;
    size_t room = scratch_bytes - fixed;
    void* own = nullptr;
    if (room < tabs + 4 * one) {  // a workspace of the least size the call takes: a few warps' worth of its own
        room = tabs + 16 * one;
        if (!succeeded(cudaMallocAsync(&own, room, st))) return MMA_ERR_CUDA;
        rest = static_cast<char*>(own);
    }
    cd* rhs0t = reinterpret_cast<cd*>(rest);
    double* V12t = reinterpret_cast<double*>(rhs0t + 32 * m);
    cd* buf = reinterpret_cast<cd*>(rest + tabs);
    room -= tabs;
    an::pes_tables<<<an::grid_for(32 * m), 256, 0, st>>>(n, m, num_r, dx, trg_a, psi, V12, rhs0, V12t, rhs0t);
    const int sms = pes_sms(), wave = 64 * sms;
    an::PesArgs A{n, dx, dE, Estep, E_start, num_E, 0, 0, V12, rhs0, pes};
    for (int done = 0; done < num_E;) {
        const int left = num_E - done;
        int np = pes_by_pairs(left, n, sms) ? (left < wave ? left : wave) : 0;
        // a rest for pairs too joins its wave's launch: the SMs that get a second CTA are done no later than
        // after a second launch (51 rows, 12000 energies: 232 us a call in two launches, 190 in one)
        if (np == wave && left < 2 * (int64_t)wave && pes_by_pairs(left - wave, n, sms) &&
            room >= 2 * sizeof(cd) * (size_t)n * left)
            np = left;
        if (room < 2 * sizeof(cd) * (size_t)n * np) np = 0;
        an::PesPair Q{A, buf, buf + (size_t)n * np, np};
        Q.A.e0 = done;
        Q.A.count = np;
        done += np;
        const size_t used = 2 * sizeof(cd) * (size_t)n * np;
        int nw = num_E - done;
        if (np > 0 && (pes_by_pairs(nw, n, sms) || room < used + 4 * one)) nw = 0;  // the next launch's
        int64_t blocks = (int64_t)((room - used) / (4 * one));
        if (blocks > 4 * sms) blocks = 4 * sms;
        if (blocks > (nw + 3) / 4) blocks = (nw + 3) / 4;
        an::PesWarp W{A, m, buf + 2 * (size_t)n * np};
        W.A.e0 = done;
        W.A.count = nw;
        W.A.V12 = V12t;
        W.A.rhs0 = rhs0t;
        done += nw;
        const int pairs = (np + 63) / 64;
        an::pes_kernel<<<(unsigned)(pairs + blocks), 128, 0, st>>>(Q, pairs, W);
    }
    const bool ok = cudaGetLastError() == cudaSuccess;
    if (own && !succeeded(cudaFreeAsync(own, st))) return MMA_ERR_CUDA;
    return ok ? MMA_OK : MMA_ERR_CUDA;
}

extern "C" size_t mma_gabor_scratch_bytes(int n_sig, int N, int N_G)
{
    if (n_sig < 1 || N < 2 || N_G < 1) return 0;
    const size_t nb = (size_t)n_sig * N_G, Nc = (size_t)N / 2 + 1;
    return (sizeof(double) * nb * N + 255) / 256 * 256 + sizeof(double2) * nb * Nc;
}

extern "C" int mma_gabor(const double* signals, int64_t stride, int n_sig, double dt, int N, int N_freq, int N_G,
                         double t_min, double t_max, double a, double* gabor, void* scratch, size_t scratch_bytes,
                         void* stream)
{
    if (!signals || !gabor || !scratch || n_sig < 1 || N < 2 || N_G < 1 || N_freq < 1 || stride < N) return MMA_ERR_ARG;
    const int64_t Nc = N / 2 + 1;
    if (N_freq > Nc || !(a != 0.0)) return MMA_ERR_ARG;
    if (scratch_bytes < mma_gabor_scratch_bytes(n_sig, N, N_G)) return MMA_ERR_ARG;
    if ((int64_t)n_sig * N_G > 2147483647LL) return MMA_ERR_TOO_LARGE;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t nb = (int64_t)n_sig * N_G;
    double* in = static_cast<double*>(scratch);
    double2* out = reinterpret_cast<double2*>(static_cast<char*>(scratch) + (sizeof(double) * nb * N + 255) / 256 * 256);
    const double ia = 1.0 / a, dt_G = (t_max - t_min) / N_G;
    // the window table sits at the front of the DFT output buffer: it is read before the DFT writes there
    double* win = reinterpret_cast<double*>(out);
    an::gabor_table<<<an::grid_for((int64_t)N_G * N), 256, 0, st>>>(N, N_G, dt, t_min, dt_G, ia, win);
    const mma::dft::Plan* p = nullptr;
    int rc = mma::dft::get_plan(N, st, &p);
    if (rc != MMA_OK) return rc;
    const double norm = dt / sqrt(2. * an::kPi);
    if (mma::dft::windowed(p, signals, stride, n_sig, win, N_G, N_freq, norm, gabor, st))
        return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
    an::gabor_window<<<an::grid_for(nb * N), 256, 0, st>>>(signals, stride, n_sig, N, N_G, win, in);
    rc = mma::dft::r2c(p, in, N, out, Nc, (int)nb, st);
    if (rc != MMA_OK) return rc;
    an::gabor_abs<<<an::grid_for(nb * N_freq), 256, 0, st>>>(out, Nc, nb, N_freq, norm, gabor);
    return cudaGetLastError() == cudaSuccess ? MMA_OK : MMA_ERR_CUDA;
}
