// df64.cuh -- double-word FP32 ("float-float") arithmetic of the TDSE kernels: a value is a pair
// (hi, lo) of floats with |lo| <= ulp(hi)/2, about 48 significant bits, and complex values run as
// packed FP32x2 pairs.  The error-free transformations and the sources of the algorithms are stated
// in tdse_df64.cu.
#pragma once

#include "common.cuh"

namespace mma {
namespace dfk {

struct df {
    float hi, lo;
};

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e)  // |a| >= |b|
{
    s = a + b;
    e = b - (s - a);
}
__device__ __forceinline__ df renorm(float s, float e)
{
    df r;
    fast_two_sum(s, e, r.hi, r.lo);
    return r;
}
// x + y (Joldes, Muller, Popescu 2017, Algorithm 6)
__device__ __forceinline__ df add(df x, df y)
{
    float sh, sl, th, tl;
    two_sum(x.hi, y.hi, sh, sl);
    two_sum(x.lo, y.lo, th, tl);
    sl += th;
    fast_two_sum(sh, sl, sh, sl);
    sl += tl;
    return renorm(sh, sl);
}
__device__ __forceinline__ df from_d(double v)
{
    const float h = (float)v;
    return df{h, (float)(v - (double)h)};
}
__device__ __forceinline__ double to_d(df v) { return (double)v.hi + (double)v.lo; }

// ------------------------------------------------------------------ packed complex double-words
// A complex double-word value as two FP32x2 pairs: h = (re.hi, im.hi), l = (re.lo, im.lo), stored
// as the float4 (re.hi, im.hi, re.lo, im.lo).  Real and imaginary parts go through the same
// sequence of operations, so one packed FP32x2 instruction does the work of two FP32 ones; each
// lane gets exactly the IEEE operations of the component-wise double-word formula stated beside
// the routine, in the same order.  A complex product a b takes a's parts as broadcast pairs and
// b as (b) and i b = (-b.im, b.re), so lane re gets a.re b.re + a.im (-b.im) and lane im
// a.re b.im + a.im b.re.
struct pk {
    float2 h, l;
};
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t*>(&a)),
                                                "l"(*reinterpret_cast<uint64_t*>(&b)));
    return *reinterpret_cast<float2*>(&r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 ng2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 bc(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 ipair(float2 a) { return make_float2(-a.y, a.x); }   // i (x + i y)
__device__ __forceinline__ float2 mipair(float2 a) { return make_float2(a.y, -a.x); }  // -i (x + i y)
__device__ __forceinline__ pk pld(const float4* p)
{
    const float4 v = *p;
    return pk{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ void pst(float4* p, pk v) { *p = make_float4(v.h.x, v.h.y, v.l.x, v.l.y); }
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e)
{
    s = add2(a, b);
    const float2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
__device__ __forceinline__ pk renorm2(float2 s, float2 e)
{
    pk r;
    r.h = add2(s, e);
    r.l = sub2(e, sub2(r.h, s));
    return r;
}
// lanes of x1 y1 + x2 y2 (x broadcast operands, y per-lane operands), double-word products exact
// to first order: the leading products p, q and their folded low-order parts ep, eq
struct prods {
    float2 p, q, ep, eq;
};
__device__ __forceinline__ prods products(float2 x1h, float2 x1l, float2 y1h, float2 y1l, float2 x2h, float2 x2l,
                                          float2 y2h, float2 y2l)
{
    prods r;
    r.p = mul2(x1h, y1h);
    r.q = mul2(x2h, y2h);
    r.ep = fma2(x1h, y1h, ng2(r.p));
    r.eq = fma2(x2h, y2h, ng2(r.q));
    r.ep = fma2(x1h, y1l, fma2(x1l, y1h, r.ep));
    r.eq = fma2(x2h, y2l, fma2(x2l, y2h, r.eq));
    return r;
}
// the double-word products of a b: lane re a.re b.re + a.im (-b.im), lane im a.re b.im + a.im b.re
__device__ __forceinline__ prods cprods(pk a, pk b)
{
    return products(bc(a.h.x), bc(a.l.x), b.h, b.l, bc(a.h.y), bc(a.l.y), ipair(b.h), ipair(b.l));
}
__device__ __forceinline__ pk cmul_pu(pk a, pk b)
{
    const prods r = cprods(a, b);
    float2 s1, t1;
    two_sum2(r.p, r.q, s1, t1);
    return pk{s1, add2(t1, add2(r.ep, r.eq))};
}
__device__ __forceinline__ pk cmul_p(pk a, pk b)
{
    const pk u = cmul_pu(a, b);
    return renorm2(u.h, u.l);
}
// a sum of two products plus z per lane: TwoSum of the leading products, TwoSum with z.hi,
// every low-order term folded once, one renormalisation
// z + a b
__device__ __forceinline__ pk dot_add(const prods& r, pk z)
{
    float2 s1, t1, s2, t2;
    two_sum2(r.p, r.q, s1, t1);
    two_sum2(s1, z.h, s2, t2);
    return renorm2(s2, add2(add2(add2(t1, t2), add2(r.ep, r.eq)), z.l));
}
__device__ __forceinline__ pk cfma_p(pk a, pk b, pk z) { return dot_add(cprods(a, b), z); }
// z - a b: lane re (-a.re) b.re + a.im b.im, lane im (-a.re) b.im + a.im (-b.re)
__device__ __forceinline__ pk cfms_p(pk a, pk b, pk z)
{
    return dot_add(products(bc(-a.h.x), bc(-a.l.x), b.h, b.l, bc(a.h.y), bc(a.l.y), mipair(b.h), mipair(b.l)), z);
}
// f y0 + y - g u: the forward correction and the backward sweep of a site in one sum (five leading
// terms by four TwoSums, every low-order term folded once, one renormalisation)
__device__ __forceinline__ pk correct_sweep_p(pk f, pk y0, pk y, pk g, pk u)
{
    const prods a = cprods(f, y0);
    const prods b = products(bc(-g.h.x), bc(-g.l.x), u.h, u.l, bc(g.h.y), bc(g.l.y), mipair(u.h), mipair(u.l));
    float2 s1, t1, s2, t2, s3, t3, s4, t4;
    two_sum2(a.p, a.q, s1, t1);
    two_sum2(s1, y.h, s2, t2);  // off the chain of u
    two_sum2(b.p, b.q, s3, t3);
    two_sum2(s2, s3, s4, t4);
    const float2 la = add2(add2(t1, t2), add2(add2(a.ep, a.eq), y.l));
    return renorm2(s4, add2(add2(add2(t3, t4), add2(b.ep, b.eq)), la));
}
// 10 p + a + b per lane (the Numerov right-hand side), one TwoSum per pair of leading terms,
// unnormalised (feeds a product)
__device__ __forceinline__ pk ten_sum_p(pk p, pk a, pk b)
{
    const float2 x = mul2(bc(10.f), p.h);
    const float2 ex = fma2(bc(10.f), p.l, fma2(bc(10.f), p.h, ng2(x)));
    float2 s1, t1, s2, t2;
    two_sum2(a.h, b.h, s1, t1);
    two_sum2(x, s1, s2, t2);
    return pk{s2, add2(add2(add2(t1, t2), ex), add2(a.l, b.l))};
}
// g u + y - p per lane (the CN update before the phase): the four leading terms by three
// TwoSums, every low-order term folded once, unnormalised (feeds a product)
__device__ __forceinline__ pk cn_update_p(pk g, pk u, pk y, pk p)
{
    const prods r = cprods(g, u);
    float2 s1, t1, s2, t2, s3, t3;
    two_sum2(r.p, r.q, s1, t1);
    two_sum2(y.h, ng2(p.h), s2, t2);
    two_sum2(s1, s2, s3, t3);
    return pk{s3, add2(add2(add2(t1, t2), t3), add2(add2(r.ep, r.eq), add2(y.l, ng2(p.l))))};
}
// Accumulators of a site loop: hi takes each term's leading part by a TwoSum, lo gathers every
// low-order part; renormalised once after the loop (lo stays far below ulp(hi) over a chunk).
// acc += x y per lane with x broadcast
__device__ __forceinline__ void acc_mul_p(pk& acc, float xh, float xl, pk y)
{
    const float2 X = bc(xh);
    const float2 p = mul2(X, y.h);
    float2 ep = fma2(X, y.h, ng2(p));
    ep = fma2(X, y.l, fma2(bc(xl), y.h, ep));
    float2 s, e;
    two_sum2(acc.h, p, s, e);
    acc.h = s;
    acc.l = add2(acc.l, add2(e, ep));
}
// acc += (a.re b.re + a.im b.im, a.re b.im - a.im b.re): the projection of a on b
__device__ __forceinline__ void acc_proj_p(pk& acc, pk a, pk b)
{
    const prods r = products(bc(a.h.x), bc(a.l.x), b.h, b.l, bc(a.h.y), bc(a.l.y), mipair(b.h), mipair(b.l));
    float2 s1, t1, s2, t2;
    two_sum2(r.p, r.q, s1, t1);
    two_sum2(acc.h, s1, s2, t2);
    acc.h = s2;
    acc.l = add2(acc.l, add2(add2(t1, t2), add2(r.ep, r.eq)));
}
// |v|^2, unnormalised: packed double-word squares, then the TwoSum of the two lanes
__device__ __forceinline__ df norm2_u(pk v)
{
    const float2 p = mul2(v.h, v.h);
    float2 ep = fma2(v.h, v.h, ng2(p));
    ep = fma2(v.h, v.l, fma2(v.l, v.h, ep));
    float s1, t1;
    two_sum(p.x, p.y, s1, t1);
    return df{s1, t1 + (ep.x + ep.y)};
}
__device__ __forceinline__ pk pshup(pk v, int d)
{
    return pk{make_float2(__shfl_up_sync(0xffffffffu, v.h.x, d), __shfl_up_sync(0xffffffffu, v.h.y, d)),
              make_float2(__shfl_up_sync(0xffffffffu, v.l.x, d), __shfl_up_sync(0xffffffffu, v.l.y, d))};
}
__device__ __forceinline__ pk pshdn(pk v, int d)
{
    return pk{make_float2(__shfl_down_sync(0xffffffffu, v.h.x, d), __shfl_down_sync(0xffffffffu, v.h.y, d)),
              make_float2(__shfl_down_sync(0xffffffffu, v.l.x, d), __shfl_down_sync(0xffffffffu, v.l.y, d))};
}

__device__ __forceinline__ df shfl_xor_df(df v, int d)
{
    return df{__shfl_xor_sync(0xffffffffu, v.hi, d), __shfl_xor_sync(0xffffffffu, v.lo, d)};
}

}  // namespace dfk
}  // namespace mma
