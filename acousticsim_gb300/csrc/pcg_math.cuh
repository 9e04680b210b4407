// Arithmetic shared by the PCG kernels (device only): every driver and every
// kernel variant forms its row products, its sums and its scalars with these,
// so their results agree bit for bit.
#pragma once
#include "device.cuh"

namespace cloth {

__device__ __forceinline__ float3 operator+(float3 a, float3 b)
{
    return make_float3(a.x + b.x, a.y + b.y, a.z + b.z);
}
__device__ __forceinline__ float3 operator-(float3 a, float3 b)
{
    return make_float3(a.x - b.x, a.y - b.y, a.z - b.z);
}
__device__ __forceinline__ float3 operator*(float s, float3 a)
{
    return make_float3(s * a.x, s * a.y, s * a.z);
}
__device__ __forceinline__ float3 xyz(float4 v) { return make_float3(v.x, v.y, v.z); }
__device__ __forceinline__ float4 f4(float3 v, float w = 0.f)
{
    return make_float4(v.x, v.y, v.z, w);
}
// Row-level products stay in FP32; sums from 32 rows upward are FP64 (GB300's
// FP64 pipe is narrow, so FP64 work is kept per warp, not per row).
__device__ __forceinline__ float fdot(float3 a, float3 b)
{
    return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x));
}
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// sum of squares in component order, as tCudaMatrix::norm (CudaMatrix.h:314-320)
__device__ __forceinline__ float norm3(float3 a)
{
    float s = a.x * a.x;
    s = s + a.y * a.y;
    s = s + a.z * a.z;
    return sqrtf(s);
}
// symmetric 3x3 (00 01 02 11 12 22) times vector
// (explicit fused multiply-adds: device code is built without implicit
// contraction, so every kernel variant rounds the same way)
__device__ __forceinline__ float3 symv(const float *s, float3 v)
{
    return make_float3(fmaf(s[2], v.z, fmaf(s[1], v.y, s[0] * v.x)),
                       fmaf(s[4], v.z, fmaf(s[3], v.y, s[1] * v.x)),
                       fmaf(s[5], v.z, fmaf(s[4], v.y, s[2] * v.x)));
}
// p = z + beta p_old with one rounding per component (the persistent
// kernels' form, so every PCG driver forms the same p)
__device__ __forceinline__ float3 pform(float3 z, float beta, float3 po)
{
    return make_float3(fmaf(beta, po.x, z.x), fmaf(beta, po.y, z.y), fmaf(beta, po.z, z.z));
}
// w x p: the skew part of a block of the dihedral-bending model (an upper
// block is S p + w x p, its transposed lower block S p - w x p)
__device__ __forceinline__ float3 skewv(float4 w, float3 p)
{
    return make_float3(fmaf(w.y, p.z, -(w.z * p.y)), fmaf(w.z, p.x, -(w.x * p.z)),
                       fmaf(w.x, p.y, -(w.y * p.x)));
}
__device__ __forceinline__ void load_sym(const float4 *a0, const float2 *a1,
                                         size_t o, float *s)
{
    float4 u = a0[o];
    float2 w = a1[o];
    s[0] = u.x;
    s[1] = u.y;
    s[2] = u.z;
    s[3] = u.w;
    s[4] = w.x;
    s[5] = w.y;
}

__device__ __forceinline__ bool test_converged(const InstDesc &d,
                                               const InstState &s, double rr)
{
    bool ok = false;
    if (d.rel_tol2 > 0.0 && rr <= d.rel_tol2 * s.bb)
        ok = true;
    if (d.abs_tol2 > 0.0 && rr <= d.abs_tol2)
        ok = true;
    return ok;
}

// round(v * 2^s) as a signed 128-bit integer, returned as H * 2^32 + L with
// 0 <= L < 2^32 (integer operations only).  Exact addition of these limbs
// makes a team sum independent of how the rows are split over blocks.
__device__ __forceinline__ void fx_split(float v, int s, long long &H,
                                         unsigned long long &L)
{
    const unsigned bits = __float_as_uint(v);
    const int e = int((bits >> 23) & 0xffu);
    H = 0;
    L = 0;
    if (e == 0 || e == 255)
        return; // zero, subnormal (below any scale in use) or Inf/NaN (fx_note)
    const unsigned long long m = (bits & 0x7fffffu) | 0x800000u;
    const int sh = e - 150 + s; // |v| = m * 2^(e - 150)
    unsigned long long fh = 0ull, fl = 0ull;
    if (sh >= 104)
    {
        fh = 0x3fffffffffffffffull; // out of range: fx_note flags it
        fl = ~0ull;
    }
    else if (sh >= 64)
        fh = m << (sh - 64);
    else if (sh > 0)
    {
        fl = m << sh;
        fh = m >> (64 - sh);
    }
    else if (sh == 0)
        fl = m;
    else if (sh > -25)
        fl = (m + (1ull << (-sh - 1))) >> (-sh);
    if (bits & 0x80000000u)
    {
        fl = ~fl + 1ull;
        fh = ~fh + (fl == 0ull ? 1ull : 0ull);
    }
    L = fl & 0xffffffffull;
    H = (long long)((fh << 32) | (fl >> 32));
}

// Which sums count, in every driver alike: each 32-row chunk below 2^(kChunkBits + 24)
// units and finite, their exact total within 2^95, and (p.q and r.z, judged at the end
// of the iteration) the total not so far below the sum of the chunks' magnitudes that
// the chunks' FP32 rounding leaves nothing of it, nor (r.z and r.r) one that rises
// from zero.
//
// The limbs hold the total modulo 2^96, so chunks of 2^75 units and more, which are
// rare (a sum's last value has about 2^70), are counted in units of 2^72 too; the
// others' part of 2^19 chunks (16 million rows) stays in range.
constexpr int kChunkBits = 86, kChunkBig = 52, kTopUnit = 72;
__device__ __forceinline__ void fx_note(float v, int s, InstState *st, int bq, int q)
{
    const unsigned bits = __float_as_uint(v);
    const int e = int((bits >> 23) & 0xffu), sh = e - 150 + s;
    if (e == 0 || (sh < kChunkBig && e != 255))
        return;
    if (e == 255 || sh >= kChunkBits)
    {
        atomicOr(&st->acc_bad[bq][q], 1);
        return;
    }
    long long m = (long long)((bits & 0x7fffffu) | 0x800000u);
    if (bits & 0x80000000u)
        m = -m;
    m = sh >= kTopUnit ? m * (1ll << (sh - kTopUnit)) : m >> (kTopUnit - sh);
    atomicAdd(&st->acc_top[bq][q], (unsigned long long)m);
}
// A chunk's magnitude m 2^sh in units of 2^66, at most 2^18; and whether a total, floor(V
// / 2^kCancelUnit), is below 2^-kCancelBits of its chunks' magnitudes: p.q of an
// indefinite system, or r.z where diagonal blocks are, once FP32 (rows of 2^-24, and
// more in their sums) no longer resolves it.  alpha and beta are then noise and the solve
// stalls until max_iters (256x256 with stiff dihedral bending: a residual of 0.4 after
// 20,000 iterations); ended as NaN, a step escalates it to FP64.  Solves that converge
// stay far from it (small negative stiffness: p.q a hundredth of a chunk).
constexpr int kCancelBits = 13, kCancelUnit = 66 - kCancelBits;
__device__ __forceinline__ unsigned fx_mag(unsigned m, int sh)
{
    return min(m >> min(max(66 - sh, 0), 31), 1u << 18);
}
__device__ __forceinline__ unsigned fx_mag(float v, int s)
{
    const unsigned bits = __float_as_uint(v);
    const int e = int((bits >> 23) & 0xffu);
    return e == 0 || e == 255 ? 0u : fx_mag((bits & 0x7fffffu) | 0x800000u, e - 150 + s);
}
__device__ __forceinline__ bool fx_cancels(long long total, unsigned long long mag)
{
    return (unsigned long long)(total ^ (total >> 63)) < mag;
}
__device__ __forceinline__ void fx_clear(InstState *st, int bq)
{
    for (int q = 0; q < 3; q++)
    {
        st->acc[bq][q][0] = 0ull;
        st->acc[bq][q][1] = 0ull;
        st->acc_top[bq][q] = 0ull;
        st->acc_bad[bq][q] = 0;
    }
    st->acc_mag[bq][0] = st->acc_mag[bq][1] = 0ull;
}

// Scale exponent for an estimate of a sum (from the double's exponent bits).
__device__ __forceinline__ int fx_scale(double est)
{
    const long long b = __double_as_longlong(est);
    const int e = int((b >> 52) & 0x7ff);
    if (e == 0 || e == 0x7ff)
        return 100;
    const int s = kFxTop - (e - 1023);
    return max(-900, min(900, s));
}

// 2^e for |e| < 1000, built from the exponent field
__device__ __forceinline__ double pow2(int e)
{
    return __longlong_as_double((long long)(1023 + e) << 52);
}

__device__ __forceinline__ double fx_value(unsigned long long H, unsigned long long L,
                                           int s)
{
    return double((long long)H) * pow2(32 - s) + double(L) * pow2(-s);
}

__device__ __forceinline__ bool fx_cancels(const InstState *st, int bq, int q)
{
    const long long H = (long long)(__ldcg(&st->acc[bq][q][0]) + (__ldcg(&st->acc[bq][q][1]) >> 32));
    return fx_cancels(H >> (kCancelUnit - 32), __ldcg(&st->acc_mag[bq][q]));
}
// A residual that had gone below FP32's range and comes back (a solve without tolerances
// that goes on past its end): rounding noise, which grows without bound.
__device__ __forceinline__ bool fx_from_zero(double last, double now)
{
    return last == 0.0 && now != 0.0;
}
// A sum's total; *bad where it is out of range.
__device__ __forceinline__ double fx_total(const InstState *st, int bq, int q, int s, int *bad)
{
    const unsigned long long L = __ldcg(&st->acc[bq][q][1]);
    const unsigned long long H = __ldcg(&st->acc[bq][q][0]) + (L >> 32);
    const long long top = (long long)__ldcg(&st->acc_top[bq][q]);
    // the total over 2^72, as the limbs have it (24 bits) and as it is
    const long long hi = (long long)H >> (kTopUnit - 32);
    const long long rest = (long long)((unsigned long long)(hi - top) << 40) >> 40;
    if (__ldcg(&st->acc_bad[bq][q]) != 0 || top + rest != hi)
        *bad = 1;
    return fx_value(H, L & 0xffffffffull, s);
}

} // namespace cloth
