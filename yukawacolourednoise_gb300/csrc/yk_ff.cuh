// yk_ff.cuh -- float-float (hi + lo) arithmetic of the mixed CG kernels.
#pragma once

#include "yk_common.cuh"

namespace yk {

// ---------------------------------------------------------------------------
// Float-float sums (hi + lo, about 48 significant bits) for the mixed solver:
// GB300 issues FP64 at 1/64 of the FP32 rate, so its reductions run on the
// FP32 pipes.  Knuth's two-sum; no multiplications, so no FMA contraction.
// ---------------------------------------------------------------------------
struct FF {
    float hi, lo;
};

__device__ __forceinline__ FF ff_add(FF a, FF b)
{
    const float s = a.hi + b.hi;
    const float bp = s - a.hi;
    float e = (a.hi - (s - bp)) + (b.hi - bp);
    e += a.lo + b.lo;
    const float hi = s + e;
    return FF{hi, e - (hi - s)};
}

__device__ __forceinline__ FF ff_of(double x)
{
    const float hi = (float)x;
    return FF{hi, (float)(x - (double)hi)};
}

__device__ __forceinline__ FF ff_shfl_xor(FF a, int o)
{
    return FF{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
}

// Float-float products and the reciprocal (Dekker's product with the exact
// FMA error term; one Newton step from the FP32 reciprocal).  The explicitly
// rounded intrinsics keep the compiler from contracting the product that the
// error term subtracts.
__device__ __forceinline__ FF ff_renorm(float p, float e)
{
    const float hi = __fadd_rn(p, e);
    return FF{hi, __fsub_rn(e, __fsub_rn(hi, p))};
}

__device__ __forceinline__ FF ff_mul(FF a, FF b)
{
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return ff_renorm(p, e);
}

__device__ __forceinline__ FF ff_mul_f(FF a, float b)
{
    const float p = __fmul_rn(a.hi, b);
    float e = __fmaf_rn(a.hi, b, -p);
    e = __fmaf_rn(a.lo, b, e);
    return ff_renorm(p, e);
}

__device__ __forceinline__ FF ff_sub(FF a, FF b) { return ff_add(a, FF{-b.hi, -b.lo}); }
__device__ __forceinline__ double dbl_of(FF a) { return (double)a.hi + (double)a.lo; }

// 1 / d: y = rn(1 / d.hi), then y + y (1 - d y) with d y and the correction in
// float-float (relative error about 2^-47)
__device__ __forceinline__ FF ff_rcp(FF d)
{
    const float y = __frcp_rn(d.hi);
    const FF e = ff_sub(FF{1.f, 0.f}, ff_mul_f(d, y));
    return ff_add(FF{y, 0.f}, ff_mul_f(e, y));
}

// float-float times float (Dekker's product through the FMA, then a fast two-sum)
__device__ __forceinline__ FF ff_mul(FF a, float b)
{
    const float p = a.hi * b;
    float err = fmaf(a.hi, b, -p);
    err = fmaf(a.lo, b, err);
    const float s = p + err;
    return FF{s, err - (s - p)};
}

__device__ __forceinline__ FF ff_neg(FF a) { return FF{-a.hi, -a.lo}; }

__device__ __forceinline__ FF ff_sign(FF a, float s) { return FF{s * a.hi, s * a.lo}; }

// The even-odd kernels' reliable updates, round 0 and reconstruction in
// float-float (about 48 significant bits, on the FP32 pipes: GB300 issues
// FP64 at 1/64 of the FP32 rate and these passes were bound by it).  chi_e,
// rhs_e and the odd intermediate keep the FP64 vectors' 32 bytes a compact
// site: four hi words, then four lo words; 1 / A_o keeps its 8 bytes as (hi,
// lo).  Only the kernels read them; chi goes out to the force in FP64.
struct SiteFF {
    FF v[4];
};

__device__ __forceinline__ SiteFF ld_ff(const double* base, int m)
{
    const float4* p = reinterpret_cast<const float4*>(base) + 2 * (size_t)m;
    const float4 h = p[0], l = p[1];
    return SiteFF{{FF{h.x, l.x}, FF{h.y, l.y}, FF{h.z, l.z}, FF{h.w, l.w}}};
}

__device__ __forceinline__ void st_ff(double* base, int m, const SiteFF& s)
{
    float4* p = reinterpret_cast<float4*>(base) + 2 * (size_t)m;
    p[0] = make_float4(s.v[0].hi, s.v[1].hi, s.v[2].hi, s.v[3].hi);
    p[1] = make_float4(s.v[0].lo, s.v[1].lo, s.v[2].lo, s.v[3].lo);
}

__device__ __forceinline__ FF ld_ff1(const double* base, int m)
{
    const float2 v = reinterpret_cast<const float2*>(base)[m];
    return FF{v.x, v.y};
}

__device__ __forceinline__ void st_ff1(double* base, int m, FF v)
{
    reinterpret_cast<float2*>(base)[m] = make_float2(v.hi, v.lo);
}

// FP64 <-> FP32 by the bits, on the integer pipes: a conversion that touches an
// FP64 register issues at the FP64 rate, and in a branch for rare values the
// compiler would run it always and select.  widen: exact.  narrow: of a double
// that is a normal FP32 number or zero.  ff_split: the top 24 bits and the next 24
// of a double, as ff_of within 2^-48.  Below FP32's normal range narrow and
// ff_split give zero, above it infinity; NaN stays NaN.
__device__ __forceinline__ double widen(float f)
{
    const bool sub = !(fabsf(f) >= 0x1p-126f);   // zero, subnormal or NaN
    const unsigned u = __float_as_uint(sub ? f * 0x1p64f : f);
    unsigned e = ((u >> 23) & 0xffu) + (sub ? 896u - 64u : 896u);
    if (((u >> 23) & 0xffu) == 0xffu) e = 0x7ffu;
    if ((u & 0x7fffffffu) == 0u) e = 0u;
    return __hiloint2double((int)((u & 0x80000000u) | (e << 20) | ((u & 0x7fffffu) >> 3)), (int)(u << 29));
}

__device__ __forceinline__ float narrow(double d)
{
    const unsigned h = (unsigned)__double2hiint(d), l = (unsigned)__double2loint(d), e = (h >> 20) & 0x7ffu;
    unsigned v = (((h & 0x7fffffffu) - (896u << 20)) << 3) | (l >> 29);
    if (e < 897u) v = 0u;
    if (e > 1150u) v = e == 0x7ffu && ((h & 0xfffffu) | l) != 0u ? 0x7fffffffu : 0x7f800000u;
    return __uint_as_float((h & 0x80000000u) | v);
}

__device__ __forceinline__ FF ff_split(double d)
{
    const unsigned h = (unsigned)__double2hiint(d), l = (unsigned)__double2loint(d), e = (h >> 20) & 0x7ffu;
    const float hi = narrow(d);
    // the low 29 bits times 2^(e - 1075), the exponent in two steps that stay in range
    const float lo = (float)(int)(l & 0x1fffffffu) * 0x1p-52f * __uint_as_float(((e - 896u) << 23 & 0x7f800000u) | (h & 0x80000000u));
    const FF r = ff_renorm(hi, lo);
    return e - 897u < 254u ? r : FF{hi, 0.f};
}

// a source vector's site as float-float: the Langevin sources are FP32 normals
// (exact in FP32) when generated; other right-hand sides are split
__device__ __forceinline__ SiteFF ff_site_of(const Site<double, 1>& e, bool exact32)
{
    SiteFF s;
#pragma unroll
    for (int i = 0; i < 4; ++i) s.v[i] = exact32 ? FF{narrow(e.v[i]), 0.f} : ff_of(e.v[i]);
    return s;
}

}  // namespace yk
