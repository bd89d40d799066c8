// tdse_cluster.cuh -- device parts shared by the kernels that spread a TDSE instance over a
// thread-block cluster (tdse_cluster.cu, tdse_adjoint.cu): the arithmetic of the FP64 and the
// float-float form, and the scans of the partitioned solve across the cluster.
#pragma once

#include <cooperative_groups.h>

#include "../../include/mma_tdse.h"
#include "common.cuh"
#include "df64.cuh"
#include "tdse_step.cuh"

namespace cg = cooperative_groups;

namespace mma {
namespace clk {

constexpr int kT = 128, kW = kT / 32;  // one warp per sub-partition: FP64 issue is the limit, not latency
constexpr int kMaxNC = 16;  // the largest cluster the hardware takes (over 8: opt-in)
constexpr int kPhA = 8, kPhB = 4;  // lane = 4 a + b: e^{i F dt (4 a m dx)}, e^{i F dt (b m dx)}
constexpr int kPh = kPhA + kPhB + kW + 1;  // + the warps' start phases + e^{-i F dt dx}
constexpr int kPhSteps = kT / kPh;         // steps whose phases one pass of the CTA computes
constexpr double kTiny = 1e-25;  // a warp this weakly coupled, 1e-9 of FP64's rounding, is left out of a carry

// ------------------------------------------------------------------ arithmetic of the two forms
struct Fp64 {
    typedef cd C;
    typedef double R;  // a partial sum
    static __device__ const C* table(const mma_tdse_grid& G) { return reinterpret_cast<const C*>(G.cn_tab); }
    static __device__ C zero() { return cd{0.0, 0.0}; }
    static __device__ C one() { return cd{1.0, 0.0}; }
    static __device__ C neg(C a) { return cd{-a.re, -a.im}; }
    static __device__ bool tiny(C a) { return fabs(a.re) + fabs(a.im) < kTiny; }
    static __device__ C mul(C a, C b) { return cmul(a, b); }
    static __device__ C fma(C a, C b, C z) { return cfma(a, b, z); }
    static __device__ C fms(C a, C b, C z) { return cfms(a, b, z); }
    static __device__ C rhs(C ib, C p, C a, C b)
    {
        return cmul(ib, cd{::fma(10.0, p.re, a.re + b.re), ::fma(10.0, p.im, a.im + b.im)});
    }
    static __device__ C update(C ph, C u, C p) { return cmul(ph, u - p); }
    static __device__ C shup(C v, int d) { return cd{shfl_up(v.re, d), shfl_up(v.im, d)}; }
    static __device__ C shdn(C v, int d) { return cd{shfl_down(v.re, d), shfl_down(v.im, d)}; }
    static __device__ C bcast(C v, int l) { return cd{shfl_idx(v.re, l), shfl_idx(v.im, l)}; }
    static __device__ C from(double re, double im) { return cd{re, im}; }
    static __device__ void to_d(C v, double& re, double& im) { re = v.re, im = v.im; }
    static __device__ R re(C v) { return v.re; }
    static __device__ bool has_im(C v) { return v.im != 0.0; }
    static __device__ R rzero() { return 0.0; }
    static __device__ R radd(R a, R b) { return a + b; }
    static __device__ R rxor(R a, int d) { return shfl_xor(a, d); }
    static __device__ double rd(R a) { return a; }
    struct Acc {
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, w = 0.0;
        __device__ void add(C pn, C gx, R p0, bool in)
        {
            const double n2 = ::fma(pn.re, pn.re, pn.im * pn.im);
            a0 = ::fma(n2, gx.re, a0);
            a1 = ::fma(n2, gx.im, a1);
            a2 = ::fma(pn.re, p0, a2);
            a3 = ::fma(pn.im, p0, a3);
            if (in) w += n2;
        }
        // the imaginary part of a complex ground state: <psi0|psi> += conj(i p0i) psi
        __device__ void add_im(C pn, R p0i)
        {
            a2 = ::fma(pn.im, p0i, a2);
            a3 = ::fma(-pn.re, p0i, a3);
        }
        __device__ void get(R (&v)[4]) { v[0] = a0, v[1] = a1, v[2] = a2, v[3] = a3; }
        __device__ R window() { return w; }
    };
};

struct Df64 {
    typedef dfk::pk C;
    typedef dfk::df R;
    static __device__ const C* table(const mma_tdse_grid& G) { return reinterpret_cast<const C*>(G.df_tab); }
    static __device__ C zero() { return C{make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
    static __device__ C one() { return C{make_float2(1.f, 0.f), make_float2(0.f, 0.f)}; }
    static __device__ C neg(C a) { return C{dfk::ng2(a.h), dfk::ng2(a.l)}; }
    static __device__ bool tiny(C a) { return fabsf(a.h.x) + fabsf(a.h.y) < (float)kTiny; }
    static __device__ C mul(C a, C b) { return dfk::cmul_p(a, b); }
    static __device__ C fma(C a, C b, C z) { return dfk::cfma_p(a, b, z); }
    static __device__ C fms(C a, C b, C z) { return dfk::cfms_p(a, b, z); }
    static __device__ C rhs(C ib, C p, C a, C b) { return dfk::cmul_pu(ib, dfk::ten_sum_p(p, a, b)); }
    static __device__ C update(C ph, C u, C p)
    {
        float2 s, t;
        dfk::two_sum2(u.h, dfk::ng2(p.h), s, t);
        return dfk::cmul_p(ph, C{s, dfk::add2(t, dfk::sub2(u.l, p.l))});
    }
    static __device__ C shup(C v, int d) { return dfk::pshup(v, d); }
    static __device__ C shdn(C v, int d) { return dfk::pshdn(v, d); }
    static __device__ C bcast(C v, int l)
    {
        return C{make_float2(__shfl_sync(0xffffffffu, v.h.x, l), __shfl_sync(0xffffffffu, v.h.y, l)),
                 make_float2(__shfl_sync(0xffffffffu, v.l.x, l), __shfl_sync(0xffffffffu, v.l.y, l))};
    }
    static __device__ C from(double re, double im)
    {
        const dfk::df a = dfk::from_d(re), b = dfk::from_d(im);
        return C{make_float2(a.hi, b.hi), make_float2(a.lo, b.lo)};
    }
    static __device__ void to_d(C v, double& re, double& im)
    {
        re = (double)v.h.x + (double)v.l.x;
        im = (double)v.h.y + (double)v.l.y;
    }
    static __device__ R re(C v) { return R{v.h.x, v.l.x}; }
    static __device__ bool has_im(C v) { return v.h.y != 0.f; }
    static __device__ R rzero() { return R{0.f, 0.f}; }
    static __device__ R radd(R a, R b) { return dfk::add(a, b); }
    static __device__ R rxor(R a, int d) { return dfk::shfl_xor_df(a, d); }
    static __device__ double rd(R a) { return dfk::to_d(a); }
    struct Acc {
        C a01 = zero(), a23 = zero();
        R w = rzero();
        __device__ void add(C pn, C gx, R p0, bool in)
        {
            const R n2 = dfk::norm2_u(pn);
            dfk::acc_mul_p(a01, n2.hi, n2.lo, gx);
            dfk::acc_mul_p(a23, p0.hi, p0.lo, pn);
            if (in) w = dfk::add(w, dfk::renorm(n2.hi, n2.lo));
        }
        __device__ void add_im(C pn, R p0i) { dfk::acc_mul_p(a23, p0i.hi, p0i.lo, C{dfk::mipair(pn.h), dfk::mipair(pn.l)}); }
        __device__ void get(R (&v)[4])
        {
            const C x = dfk::renorm2(a01.h, a01.l), y = dfk::renorm2(a23.h, a23.l);
            v[0] = R{x.h.x, x.l.x}, v[1] = R{x.h.y, x.l.y}, v[2] = R{y.h.x, y.l.x}, v[3] = R{y.h.y, y.l.y};
        }
        __device__ R window() { return w; }
    };
};

// ------------------------------------------------------------------ the scans of a cluster
// The chunk maps' constant products (tdse_cluster.cu states the scheme).  totF / totB: one slot per
// warp of the cluster in every CTA's shared memory; wtF / wtB: this CTA's warps' weights [kW][NW].
template <class N>
struct Scan {
    typedef typename N::C C;
    C f_lv[5], b_lv[5];  // products over 1, 2, 4, 8, 16 chunks up to (from) this thread's
    C f_ex, b_ex;        // products of the warp's chunks before (after) this thread's
    int KF, KB;          // earlier (later) warps whose weight counts
    C *totF, *totB, *wtF, *wtB;
    int NC, NW, rank, lane, w, g;

    __device__ Scan(cg::cluster_group& cl, C* tF, C* tB, C* wF, C* wB)
        : totF(tF), totB(tB), wtF(wF), wtB(wB), NC((int)cl.num_blocks()), NW(NC * kW), rank((int)cl.block_rank()),
          lane(threadIdx.x & 31), w(threadIdx.x >> 5), g(rank * kW + w)
    {
    }

    // cF, cB: the thread's chunk products prod(-h), prod(-g).  Two cluster barriers: the caller's
    // earlier writes are visible after them, and the slots are free for the first step.
    __device__ void setup(cg::cluster_group& cl, C cF, C cB)
    {
#pragma unroll
        for (int l = 0; l < 5; l++) {
            f_lv[l] = cF;
            b_lv[l] = cB;
            const C up = N::shup(cF, 1 << l), dn = N::shdn(cB, 1 << l);
            if (lane >= (1 << l)) cF = N::mul(cF, up);
            if (lane + (1 << l) < 32) cB = N::mul(cB, dn);
        }
        const C wF = N::bcast(cF, 31), wB = N::bcast(cB, 0);
        f_ex = N::shup(cF, 1);
        b_ex = N::shdn(cB, 1);
        if (lane < NC) {
            cl.map_shared_rank(totF, lane)[g] = wF;
            cl.map_shared_rank(totB, lane)[g] = wB;
        }
        cl.sync();
        KF = KB = 0;
        if (lane == 0) {
            C W = N::one();
            for (; KF < g && !N::tiny(W); KF++) {
                wtF[w * NW + KF] = W;
                W = N::mul(W, totF[g - 1 - KF]);
            }
            W = N::one();
            for (; KB < NW - 1 - g && !N::tiny(W); KB++) {
                wtB[w * NW + KB] = W;
                W = N::mul(W, totB[g + 1 + KB]);
            }
        }
        KF = __shfl_sync(0xffffffffu, KF, 0);
        KB = __shfl_sync(0xffffffffu, KB, 0);
        cl.sync();
    }
    // the chunk's end value b -> the value at the chunk before within the warp; the warp's total goes
    // to every CTA that may need it.  A cluster barrier must follow before *_in.
    __device__ C forward_out(cg::cluster_group& cl, C b)
    {
#pragma unroll
        for (int l = 0; l < 5; l++) {
            const C up = N::shup(b, 1 << l);
            if (lane >= (1 << l)) b = N::fma(f_lv[l], up, b);
        }
        const C tot = N::bcast(b, 31);
        if (lane >= rank && lane < NC) cl.map_shared_rank(totF, lane)[g] = tot;
        return b;
    }
    __device__ C backward_out(cg::cluster_group& cl, C b)
    {
#pragma unroll
        for (int l = 0; l < 5; l++) {
            const C dn = N::shdn(b, 1 << l);
            if (lane + (1 << l) < 32) b = N::fma(b_lv[l], dn, b);
        }
        const C tot = N::bcast(b, 0);
        if (lane <= rank) cl.map_shared_rank(totB, lane)[g] = tot;
        return b;
    }
    // the carry into the thread's chunk; bx: the neighbouring lane's *_out value
    __device__ C forward_in(C bx) const
    {
        C yw = N::zero();
        for (int q = 0; q < KF; q++) yw = N::fma(wtF[w * NW + q], totF[g - 1 - q], yw);
        return lane == 0 ? yw : N::fma(f_ex, yw, bx);
    }
    __device__ C backward_in(C bx) const
    {
        C uw = N::zero();
        for (int q = 0; q < KB; q++) uw = N::fma(wtB[w * NW + q], totB[g + 1 + q], uw);
        return lane == 31 ? uw : N::fma(b_ex, uw, bx);
    }
};

}  // namespace clk
}  // namespace mma
