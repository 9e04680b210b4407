// Persistent block-Jacobi PCG with the matrix on chip (k_pcg_team).
//
// One cooperative launch runs every PCG iteration of every instance of a
// launch set.  A block owns a contiguous row range of one instance and keeps
// everything it iterates on next to its SM: the rows' 3x3 blocks, local column
// indices and inverse diagonal blocks and p over the block's column range (halo)
// in shared memory (the first blocks of a row in registers), dx, r, z and p of its
// rows in registers.  Per iteration its rows of z are stored to the L2, those of
// its halo read from there, and two team sums exchanged.
//
// What bounds it: with the matrix on chip an iteration is a chain of
// latencies - two team sums (an L2 reduction and its poll, ~1,400 cycles each)
// and the SpMV's walk over ~11 blocks per row.  The design shortens that
// chain:
//   * the sums' words carry their own arrival counts, so the poll that sees
//     the last arrival has the data (no release fence, no second load);
//   * a z row is published with the iteration in its unused fourth word in
//     one 16-byte store, so a reader needs no barrier to know it is new; it
//     polls the rows it needs while the r.z sum is under way;
//   * a control warp folds the chunk sums, talks to the team and forms alpha
//     and beta from integers and FP32 (FP64 division costs ~1,000 cycles on
//     this GPU's narrow FP64 pipe) unless that leaves their rounding open, and the
//     next fixed-point scales from exponents; the FP64 scalars are formed at the end.
// The arithmetic is that of the other PCG drivers, bit for bit.
//
// Measured (one GB300, us per PCG iteration over a whole step, before: the
// kernel that reads the matrix from L2 and forms the scalars in FP64): 16x16
// 13.1 -> 2.2, 64x64 12.2 -> 2.6, 97x61 11.8 -> 3.3, 193x255 12.4 -> 4.0,
// 256x256 12.7 -> 4.2, 512x512 21.5 -> 13.8, 128x128 with dihedral bending
// 14.1 -> 3.8.
#include "internal.h"
#include "pcg_math.cuh"

#include <type_traits>

namespace cloth {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWorkers = kTeamWorkers;
constexpr int kWarps = kWorkers / 32;
constexpr int kLeave = 10;    // stop code: iterations used up, the solve goes on later
constexpr int kHaloAhead = 3; // halo rows per thread polled before beta is known

// ---- named barriers: 1 the workers, 2-6 workers with the control warp
__device__ __forceinline__ void bar_sync(int id, int n)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// ---- z rows with their iteration in w, one 16-byte access each
__device__ __forceinline__ void st_row(float4 *p, float3 v, unsigned tag)
{
    const unsigned long long lo = (unsigned long long)__float_as_uint(v.x) |
                                  (unsigned long long)__float_as_uint(v.y) << 32;
    const unsigned long long hi = (unsigned long long)__float_as_uint(v.z) |
                                  (unsigned long long)tag << 32;
    asm volatile("{ .reg .b128 t; mov.b128 t, {%0, %1}; st.relaxed.gpu.global.b128 [%2], t; }" ::
                     "l"(lo), "l"(hi), "l"(p)
                 : "memory");
}
// The row once its tag is there; sets *err when the bounded wait gives up.
__device__ __forceinline__ float3 poll_row(const float4 *p, unsigned tag, unsigned limit,
                                           volatile int *err)
{
    unsigned long long lo, hi;
    for (unsigned n = 0;;)
    {
        asm volatile(
            "{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
            : "=l"(lo), "=l"(hi)
            : "l"(p)
            : "memory");
        if (unsigned(hi >> 32) == tag)
            break;
        if (++n > limit)
        {
            *err = 1;
            break;
        }
        if (n > 256)
            __nanosleep(32);
    }
    return make_float3(__uint_as_float(unsigned(lo)), __uint_as_float(unsigned(lo >> 32)),
                       __uint_as_float(unsigned(hi)));
}

// ---- a team that is one thread-block cluster exchanges through its blocks'
// shared memory: 16-byte remote stores that count on the receiver's mbarrier
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return unsigned(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned peer_addr(unsigned addr, unsigned rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void peer_store(unsigned addr, unsigned bar, int a, int b, int c, int d)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], "
                 "{%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// Waits for a phase; false when the bounded wait gave up.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, unsigned limit)
{
    for (unsigned n = 0;;)
    {
        unsigned done;
        asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, "
                     "[%1], %2; "
                     "selp.u32 %0, 1, 0, p; }"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (done)
            return true;
        if (++n > limit)
            return false;
        if (n > 4096)
            __nanosleep(32);
    }
}

// ---- team sums.  A sum is the exact total V of fixed-point chunk sums, in
// units of 2^-s, kept as signed 24-bit digits d0 .. d4 (each chunk adds to two
// of them).  V itself has to lie within 2^95 units; its chunks may be up to
// 2^15 times larger and cancel, as those of an indefinite system's p.q do (a
// 20 x 20 cloth of negative stiffness has p.q of a hundredth of a chunk's).
// Four words carry it, one per digit (d4 in d3's): the digit's sum, biased per
// block, with the number of blocks that added to the word in its top byte.  A block
// that saw a chunk out of range (or Inf / NaN) adds kTopBad in place of d4, which no
// others' digits outweigh.  The magnitudes of p.q's and r.z's chunks (fx_mag) go beside
// p.q and r.r and are looked at off the chain: what they say is told at the end of the
// iteration (us per iteration, without them -> with: 16x16 2.62 -> 2.63, 64x64 2.77 ->
// 2.82, 97x61 2.99 -> 3.02, 193x255 3.89 -> 3.96, 512x512 14.31 -> 14.41).
constexpr int kTopBad = 1 << 21;
constexpr int kCountShift = 56;
constexpr unsigned long long kOne = 1ull << kCountShift;
constexpr unsigned long long kBias = 1ull << 47;
constexpr unsigned long long kSumMask = kOne - 1;

// V = hi 2^48 + lo, 0 <= lo < 2^48.
struct Raw
{
    long long hi;
    unsigned long long lo;
    int s;
};
__device__ __forceinline__ Raw raw(double d)
{
    Raw r;
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const int e = int((b >> 52) & 0x7ff);
    long long m = e ? (long long)((b & 0xfffffffffffffull) | 0x10000000000000ull) : 0ll;
    if (b >> 63)
        m = -m;
    r.hi = m >> 48;
    r.lo = (unsigned long long)m & 0xffffffffffffull;
    r.s = e ? 1075 - e : 0;
    return r;
}
// The FP64 value the drivers that sum 64-bit limbs decode.
__device__ __forceinline__ double value(const Raw &r)
{
    return fx_value((unsigned long long)r.hi << 16 | r.lo >> 32, r.lo & 0xffffffffull, r.s);
}

// A 32-row chunk's FP32 sum as digits, one sum per group of 8 lanes (v and its scale
// s are theirs): lane j's part of digit j, lane 5 counting sums out of range, lane 6 the
// magnitude; false where the lane has none.
__device__ __forceinline__ bool chunk_digit(float v, int s, int &x)
{
    const unsigned bits = __float_as_uint(v);
    const int e = int((bits >> 23) & 0xffu), j = threadIdx.x & 7;
    unsigned m = (bits & 0x7fffffu) | 0x800000u;
    int sh = e - 150 + s; // |v| = m 2^sh units
    bool bad = false;
    if (__any_sync(kFull, unsigned(sh) >= unsigned(kChunkBits) || unsigned(e - 1) >= 254u))
    {
        // zero or subnormal (below any scale in use), Inf / NaN, out of range,
        // or digits below the unit
        if (e == 0)
        {
            m = 0u;
            sh = 0;
        }
        bad = e == 255 || sh >= kChunkBits;
        if (sh < 0)
        {
            m = sh > -25 ? (m + (1u << (-sh - 1))) >> -sh : 0u;
            sh = 0;
        }
        sh = min(sh, kChunkBits - 1);
    }
    const int k = (sh * 43) >> 10, off = sh - 24 * k; // sh / 24, sh % 24
    x = j == k ? int((m << off) & 0xffffffu) : int(m >> (24 - off));
    const int sign = int(bits) >> 31;
    x = (x ^ sign) - sign;
    const int mag = int(fx_mag(m, sh)); // (no branch: k_pcg_wide spilled)
    x = j == 6 ? mag : x;
    bool has = unsigned(j - k) < 2u || j == 6;
    if (bad)
    {
        x = 1;
        has = j == 5;
    }
    return has;
}
// Adds the sums to the block's digits dig[0 .. 6] of their quantity.
__device__ __forceinline__ void chunk_add(int *dig, float v, int s, bool on)
{
    int x;
    if (chunk_digit(v, s, x) && on)
        atomicAdd(dig + (threadIdx.x & 7), x);
}
// Adds the digits that groups of 8 lanes gathered (up to 16 chunks a warp) to the
// block's, carried first, so that 15 warps sum them in 32 bits.
__device__ __forceinline__ void digits_add(int *dig, int d, bool on)
{
    const int j = threadIdx.x & 7;
    const int c = j < 4 ? d >> 24 : 0;
    const int below = __shfl_up_sync(kFull, c, 1);
    if (j < 4)
        d &= 0xffffff;
    if (j >= 1 && j <= 4)
        d += below;
    if (on && j < 7 && d != 0)
        atomicAdd(dig + j, d);
}
// The sums of a warp's K chunks (the same in every lane; zero where it has
// none): p.q.
template <int K>
__device__ __forceinline__ void chunks_add(int (*dig)[8], const int *scale, const float (&pq)[K])
{
    const int g = (threadIdx.x & 31) >> 3;
    float v = pq[0];
#pragma unroll
    for (int k = 1; k < K; k++)
        v = g == k ? pq[k] : v;
    chunk_add(dig[0], v, scale[0], g < K);
}
// Both r.z and r.r of a warp's K chunks: the first half-warp holds the first
// one's sums, the second the other's (warp_sum2).
template <int K>
__device__ __forceinline__ void chunks_add2(int (*dig)[8], const int *scale, const float (&v2)[K])
{
    const int g = (threadIdx.x & 31) >> 3, q = 1 + (g >> 1);
    const int s = scale[q];
    // two chunks at a time, one per group of a half-warp
#pragma unroll
    for (int k = 0; k < K; k += 2)
        chunk_add(dig[q], (g & 1) && k + 1 < K ? v2[k + 1 < K ? k + 1 : k] : v2[k], s,
                  !(g & 1) || k + 1 < K);
}
// warp_sum of a in the first half-warp and of b in the second: the same pairs
// are added at every step, so the sums are warp_sum's bit for bit.
__device__ __forceinline__ float warp_sum2(float a, float b)
{
    const bool hi = threadIdx.x & 16;
    float v = (hi ? b : a) + __shfl_xor_sync(kFull, hi ? a : b, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// V from its digits (d4 in d3's higher bits); true when it is out of the 96-bit range.
__device__ __forceinline__ bool combine(long long d0, long long d1, long long d2, long long d3,
                                        int s, Raw &r)
{
    const long long lo = d0 + d1 * (1ll << 24);
    r.hi = d2 + d3 * (1ll << 24) + (lo >> 48);
    r.lo = (unsigned long long)lo & 0xffffffffffffull;
    r.s = s;
    const long long top = d3 + ((d2 + (lo >> 48)) >> 24);
    return top >= (1ll << 23) || top < -(1ll << 23);
}

// A block's digits dig[0 .. 6], read and cleared by the control warp.
struct Digits
{
    int4 d;
    int top; // d4, or the mark of a chunk out of range
    int mag; // the chunks' magnitudes (225: below 2^26, in a cluster 60: below 2^24)
};
__device__ __forceinline__ Digits take(int *dig)
{
    Digits r;
    int bad;
    [[maybe_unused]] int pad;
    const unsigned at = smem_u32(dig);
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.d.x), "=r"(r.d.y), "=r"(r.d.z), "=r"(r.d.w)
                 : "r"(at)
                 : "memory");
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.top), "=r"(bad), "=r"(r.mag), "=r"(pad)
                 : "r"(at + 16u)
                 : "memory");
    if (bad)
        r.top = kTopBad;
    __syncwarp();
    if ((threadIdx.x & 31) < 7)
        dig[threadIdx.x & 31] = 0;
    return r;
}
__device__ __forceinline__ bool decode(const Digits &v, int s, Raw &r)
{
    return combine(v.d.x, v.d.y, v.d.z, v.d.w + (long long)v.top * (1ll << 24), s, r);
}

// The same digits as a record, carried so that a cluster's 16 add up in 32 bits: what
// is above d3's 24 bits (a block's 60 chunks: below 2^20, or kTopBad) is in the
// upper bytes of the first three, bit 31 of the first saying that it is not zero.
__device__ __forceinline__ int4 carried(const Digits &v)
{
    const int up = v.top + (v.d.w >> 24);
    const unsigned f = (unsigned(up) & 0x7fffffu) | (up != 0 ? 0x800000u : 0u);
    int4 c = v.d;
    c.y += c.x >> 24;
    c.z += c.y >> 24;
    c.w = (c.w & 0xffffff) + (c.z >> 24);
    c.x = int(unsigned(c.x & 0xffffff) | (f & 0xff0000u) << 8);
    c.y = int(unsigned(c.y & 0xffffff) | (f & 0xff00u) << 16);
    c.z = int(unsigned(c.z & 0xffffff) | f << 24);
    return c;
}
// The same of r.r, in which nothing cancels: a block's sum past d3's 24 bits makes the
// total out of range by itself, so the upper bytes are free for r.z's magnitudes.
__device__ __forceinline__ int4 carried_with(const Digits &v, int mag)
{
    int4 c = v.d;
    c.y += c.x >> 24;
    c.z += c.y >> 24;
    c.w += c.z >> 24;
    if ((v.top | (v.d.w >> 24)) != 0)
        c.w = 1 << 26;
    c.x = (c.x & 0xffffff) | mag << 24;
    c.y = (c.y & 0xffffff) | (mag >> 8) << 24;
    c.z = (c.z & 0xffffff) | (mag >> 16) << 24;
    return c;
}
__device__ __forceinline__ bool decode_with(const int4 *rec, int nblk, int s, Raw &r,
                                            unsigned long long &mag)
{
    int4 c = make_int4(0, 0, 0, 0);
    if ((threadIdx.x & 31) < nblk)
        c = rec[threadIdx.x & 31];
    mag = __reduce_add_sync(kFull, __byte_perm(__byte_perm(c.x, c.y, 0x73), c.z, 0x3710) & 0xffffffu);
    const int d0 = __reduce_add_sync(kFull, c.x & 0xffffff),
              d1 = __reduce_add_sync(kFull, c.y & 0xffffff),
              d2 = __reduce_add_sync(kFull, c.z & 0xffffff), d3 = __reduce_add_sync(kFull, c.w);
    return combine(d0, d1, d2, d3, s, r);
}
// Total of a cluster's nblk records.
__device__ __forceinline__ bool decode(const int4 *rec, int nblk, int s, Raw &r)
{
    int4 c = make_int4(0, 0, 0, 0);
    if ((threadIdx.x & 31) < nblk)
        c = rec[threadIdx.x & 31];
    int up = 0;
    if (__any_sync(kFull, c.x < 0))
    {
        const unsigned f = (unsigned(c.x) >> 8 & 0x7f0000u) | (unsigned(c.y) >> 16 & 0xff00u) |
                           unsigned(c.z) >> 24;
        up = __reduce_add_sync(kFull, int(f << 9) >> 9);
        c.x &= 0xffffff;
        c.y &= 0xffffff;
        c.z &= 0xffffff;
    }
    const int d0 = __reduce_add_sync(kFull, c.x), d1 = __reduce_add_sync(kFull, c.y),
              d2 = __reduce_add_sync(kFull, c.z), d3 = __reduce_add_sync(kFull, c.w);
    return combine(d0, d1, d2, d3 + (long long)up * (1ll << 24), s, r);
}

// Word k of a block's sum: added to the team's by lane k.
__device__ __forceinline__ void word_add(unsigned long long *words, const Digits &v, int k)
{
    const int d = k == 0 ? v.d.x : k == 1 ? v.d.y : k == 2 ? v.d.z : v.d.w;
    const unsigned long long w =
        kOne + kBias +
        (unsigned long long)(d + (long long)(k == 3 ? v.top : 0) * (1ll << 24));
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(words + k), "l"(w)
                 : "memory");
}
// The magnitudes: a word each.
__device__ __forceinline__ void mag_add(unsigned long long *word, int mag)
{
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(word),
                 "l"(kOne + (unsigned long long)mag)
                 : "memory");
}
__device__ __forceinline__ bool mags_in(const unsigned long long *p, unsigned long long target,
                                        unsigned long long (&m)[2])
{
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                 : "=l"(m[0]), "=l"(m[1])
                 : "l"(p)
                 : "memory");
    return min(m[0] >> kCountShift, m[1] >> kCountShift) >= target;
}
// A team's sum words, the same in every lane (one 32-byte request a poll: the
// team's polls and reductions queue at one L2 slice).
struct Words
{
    unsigned long long w[4];
    __device__ __forceinline__ void load(const unsigned long long *p)
    {
        asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                     : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                     : "l"(p)
                     : "memory");
    }
    // every block's contribution is in
    __device__ __forceinline__ bool all_in(unsigned long long target) const
    {
        return min(min(w[0] >> kCountShift, w[1] >> kCountShift),
                   min(w[2] >> kCountShift, w[3] >> kCountShift)) >= target;
    }
    __device__ __forceinline__ bool decode(int nblk, int s, Raw &r) const
    {
        const unsigned long long b = (unsigned long long)nblk * kBias;
        return combine((long long)((w[0] & kSumMask) - b), (long long)((w[1] & kSumMask) - b),
                       (long long)((w[2] & kSumMask) - b), (long long)((w[3] & kSumMask) - b), s,
                       r);
    }
};

__device__ __forceinline__ bool is_noise(const Raw &v, unsigned long long mag)
{
    static_assert(kCancelUnit >= 48, "the upper part holds it");
    return fx_cancels(v.hi >> (kCancelUnit - 48), mag);
}

// ---- scalars without the FP64 pipe.  |value| = (hi + lo 2^-24) 2^e with hi
// in [2^23, 2^24): its top 48 bits, the rest dropped (relative error 2^-47).
struct Top48
{
    unsigned hi, lo;
    int e;
    bool neg;
};
__device__ __forceinline__ Top48 top48(const Raw &v)
{
    Top48 r;
    unsigned long long hi = (unsigned long long)v.hi, lo = v.lo;
    // the usual range (a sum's last value has 2^70 units): 32-bit shifts
    if (unsigned(hi >> 32) == 0u && unsigned(hi) != 0u)
    {
        const unsigned h = unsigned(hi), m = unsigned(lo >> 16), l = unsigned(lo) << 16;
        const int c = __clz(int(h));
        const unsigned w0 = __funnelshift_l(m, h, c), w1 = __funnelshift_l(l, m, c);
        r.neg = false;
        r.hi = w0 >> 8;
        r.lo = (w0 & 0xffu) << 16 | w1 >> 16;
        r.e = 48 + 32 - c - 24 - v.s;
        return r;
    }
    r.neg = v.hi < 0;
    if (r.neg)
    {
        lo = (0ull - lo) & 0xffffffffffffull;
        hi = 0ull - hi - (lo != 0ull ? 1ull : 0ull);
    }
    int base = 48;
    if (hi == 0ull)
    {
        hi = lo;
        lo = 0ull;
        base = 0;
    }
    const int nb = 64 - __clzll((long long)hi); // bits of hi
    const unsigned long long t = nb <= 48 ? hi << (48 - nb) | lo >> nb : hi >> (nb - 48);
    r.hi = unsigned(t >> 24);
    r.lo = unsigned(t) & 0xffffffu;
    r.e = base + nb - 24 - v.s;
    return r;
}
// An order of the magnitudes that a relative difference above 2^-22 decides.
__device__ __forceinline__ long long key(const Top48 &t)
{
    return ((long long)t.e << 24) + (long long)(t.hi - 0x800000u);
}
// fx_scale of the FP64 value: from its exponent, unless the rounding to FP64
// could have carried into it (or the sum left the range where it rounds once).
__device__ __forceinline__ int scale_of(const Raw &v, const Top48 &t)
{
    if (t.hi == 0u || (t.hi == 0xffffffu && t.lo == 0xffffffu) || v.hi >= (1ll << 37) ||
        v.hi <= -(1ll << 37))
        return fx_scale(value(v));
    return max(-900, min(900, kFxTop - (t.e + 23)));
}

// float(a / b), the quotient of the FP64 values rounded to FP64 and then to
// FP32, as the drivers that divide in FP64 form it.  The quotient is formed
// as q1 + q2 (FP32 quotient, then its remainder over b): within 2^-43 of the
// exact one.  Where that leaves the rounding to FP32 open (the sum lies
// within 2^-38 of a midpoint: one time in ~10,000), or the result is not in
// the normal range, *ok = false and the caller divides in FP64.  rb: about
// 1 / b.hi.
// (hi as a float by its bits; lo to 23 of them)
__device__ __forceinline__ float hi_f(const Top48 &t)
{
    return __uint_as_float(0x4b000000u | (t.hi & 0x7fffffu));
}
__device__ __forceinline__ float lo_f(const Top48 &t)
{
    return (__uint_as_float(0x4b000000u | t.lo >> 1) - 0x1p23f) * 0x1p-23f;
}
__device__ __forceinline__ float recip(const Top48 &b) { return __fdividef(1.f, hi_f(b)); }
__device__ __forceinline__ float ratio(const Top48 &a, const Top48 &b, float rb, bool *ok)
{
    const float ah = hi_f(a), al = lo_f(a), bh = hi_f(b), bl = lo_f(b);
    const float q1 = ah * rb;
    const float rem = fmaf(-q1, bl, fmaf(-q1, bh, ah) + al);
    const float q2 = rem * rb;
    const float f = q1 + q2;
    const float e = q2 - (f - q1); // what the rounding of f left off, exactly
    const unsigned fb = __float_as_uint(f);
    const float half_ulp = f >= 1.f ? 0x1p-24f : 0x1p-25f;
    const int ex = int(fb >> 23) + (a.e - b.e);
    *ok = a.hi != 0u && b.hi != 0u && (fb & 0x7fffffu) != 0u &&
          half_ulp - fabsf(e) > 0x1p-38f && ex > 1 && ex < 254;
    const unsigned r = (fb & 0x7fffffu) | unsigned(ex) << 23 |
                       (a.neg != b.neg ? 0x80000000u : 0u);
    return __uint_as_float(r);
}

// What the warps of a block share; in a cluster also the blocks' sum records
// (p.q; r.z; r.r; p.q's magnitudes), the barriers they and the z rows are counted on,
// and where a row of z goes: the blocks whose columns touch rows of this one.
template <bool CLUSTER> struct Shared
{
    alignas(16) int4 rec[4][CLUSTER ? kClusterMax : 1];
    alignas(8) unsigned long long bar[3];
    TeamPeer peer[CLUSTER ? kClusterMax : 1];
    int npeer;
    float af, bf;
    int stop, err, go;
};

// Block start: the descriptor and the shared state; false (after the cluster
// has met twice) when there is nothing to solve.
template <bool CLUSTER>
__device__ __forceinline__ bool team_begin(InstDesc *const *descs, const TeamBlock &w, InstDesc &d,
                                           Shared<CLUSTER> &sh)
{
    if (threadIdx.x == 0)
    {
        sh.stop = 0;
        sh.err = 0;
        sh.go = 0;
        if (!CLUSTER || w.inst >= 0)
        {
            d = *descs[w.inst];
            sh.go = __ldcg(&d.st->active);
        }
        if (CLUSTER)
        {
            for (int i = 0; i < 3; i++)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(sh.bar + i))
                             : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();
    if (CLUSTER)
        cluster_sync();
    if (!sh.go && CLUSTER)
        cluster_sync();
    return sh.go != 0;
}

// One thread of a cluster's block: the blocks that need rows of this one, and
// the first count of its own halo rows.  z_at: the z buffer of a block whose
// halo has that many rows, as an offset in its shared memory.
template <class F>
__device__ __forceinline__ void find_peers(const TeamBlock *work, const TeamBlock &w,
                                           Shared<true> &sh, F z_at)
{
    const unsigned bar = smem_u32(sh.bar + 2);
    int n = 0;
    for (int j = 0; j < w.nblk; j++)
    {
        const TeamBlock o = work[blockIdx.x - w.rank + j];
        if (j == w.rank || o.halo0 >= w.row1 || o.halo1 <= w.row0)
            continue;
        // row i of this block is entry i - halo0 of block j's range, and
        // that less its own rows in front of it in its z buffer
        const int own = o.row0 < w.row0 ? o.row1 - o.row0 : 0;
        sh.peer[n++] = TeamPeer{max(o.halo0, w.row0), min(o.halo1, w.row1),
                                peer_addr(z_at(o.halo1 - o.halo0), j) -
                                    16u * unsigned(o.halo0 + own),
                                peer_addr(bar, j)};
    }
    sh.npeer = n;
    const int nhalo = (w.halo1 - w.halo0) - (w.row1 - w.row0);
    if (nhalo > 0)
        mbar_expect(bar, 16u * unsigned(nhalo));
}
// A row of z to the blocks that need it.
__device__ __forceinline__ void push_row(const Shared<true> &sh, int row, float3 z)
{
    for (int j = 0; j < sh.npeer; j++)
    {
        const TeamPeer o = sh.peer[j];
        if (row >= o.row0 && row < o.row1)
            peer_store(o.z + 16u * unsigned(row), o.bar, __float_as_int(z.x),
                       __float_as_int(z.y), __float_as_int(z.z), 0);
    }
}

// The control warp of a block: takes the digits the workers have added,
// exchanges them with the team, forms alpha, beta and the end of the solve, and
// posts them.
template <bool CLUSTER>
__device__ __forceinline__ void control_warp(const InstDesc &d, const TeamBlock &w, TeamSync *sync,
                                             const SpinCfg &sc, int it0, bool multi,
                                             Shared<CLUSTER> &sh, int (*dig)[8], int *scale)
{
    InstState *st = d.st;
    const int lane = threadIdx.x & 31;
    constexpr int kAll = kTeamThreads;
    unsigned long long(*words)[16] = CLUSTER ? nullptr : sync[blockIdx.x - w.rank].words;
    const unsigned bar_p = smem_u32(sh.bar), bar_z = smem_u32(sh.bar + 1);
    // this lane's peer: block lane % 16, sum lane / 16 (p.q and its magnitudes; r.z and r.r)
    const int pr_ = lane & (kClusterMax - 1), pq_ = lane / kClusterMax;
    unsigned to_p = 0, to_z = 0, at_p = 0, at_z = 0;
    if (CLUSTER && pr_ < w.nblk)
    {
        to_p = peer_addr(bar_p, pr_);
        to_z = peer_addr(bar_z, pr_);
        at_p = peer_addr(smem_u32(&sh.rec[3 * pq_][w.rank]), pr_);
        at_z = peer_addr(smem_u32(&sh.rec[1 + pq_][w.rank]), pr_);
    }
    unsigned phase = 0;
    // the scalars as exact sums: what alpha and beta were formed from too
    Raw pq = raw(__ldcg(&st->pq)), rho = raw(__ldcg(&st->rho)), rr = raw(__ldcg(&st->rr));
    Raw rho_b = rho, rho_a = rho, pq_a = pq;
    const double alpha0 = __ldcg(&st->alpha), beta0 = __ldcg(&st->beta);
    bool have_a = false, have_b = false;
    // the convergence threshold on ||r||^2
    const double bb = __ldcg(&st->bb);
    double thr = 0.0;
    if (d.rel_tol2 > 0.0)
        thr = d.rel_tol2 * bb;
    if (d.abs_tol2 > 0.0)
        thr = fmax(thr, d.abs_tol2);
    const bool tests = d.rel_tol2 > 0.0 || d.abs_tol2 > 0.0;
    const Top48 thr48 = top48(raw(thr));
    const long long thr_key = key(thr48) + 2;
    const int check_every = d.check_every, max_iters = d.max_iters;
    int to_check = check_every - 1 - (it0 + check_every - 1) % check_every;
    Top48 rho48 = top48(rho);
    float rb_rho = recip(rho48);
    bool rr_was_zero = rr.hi == 0 && rr.lo == 0ull;
    int s_pq = fx_scale(__ldcg(&st->pq)), s_rho = fx_scale(__ldcg(&st->rho)),
        s_rr = fx_scale(__ldcg(&st->rr));
    const unsigned long long target = (unsigned long long)w.nblk + sc.extra;
    int it = it0, stop = 0;
    if (lane < 3)
        scale[lane] = lane == 0 ? s_pq : lane == 1 ? s_rho : s_rr;
    if (lane < 24)
        dig[lane >> 3][lane & 7] = 0;
    // the end of the solve is told at the next alpha (the workers' step
    // towards it changes nothing that is kept)
    bar_sync(6, kAll); // the workers have filled shared memory
    for (;;)
    {
        unsigned long long *wd = CLUSTER ? nullptr : words[it & 3];
        // ---- p.q and alpha
        bar_sync(2, kAll);
        if (*(volatile int *)&sh.err)
            stop = 9;
        float af = 0.f;
        Top48 pq48 = rho48;
        unsigned long long mag[2] = {0ull, 0ull};
        if (!stop)
        {
            const Digits v = take(dig[0]);
            mag[0] = (unsigned long long)v.mag;
            bool bad = false;
            if (!multi)
                bad = decode(v, s_pq, pq);
            else if (CLUSTER)
            {
                const int4 c = carried(v);
                if (lane == 0)
                    mbar_expect(bar_p, 32u * (unsigned(w.nblk) + sc.extra));
                __syncwarp();
                if (pr_ < w.nblk)
                    peer_store(at_p, to_p, pq_ ? v.mag : c.x, c.y, c.z, c.w);
                if (mbar_wait(bar_p, phase, sc.limit))
                    bad = decode(sh.rec[0], w.nblk, s_pq, pq);
                else
                    stop = 9;
                __syncwarp();
            }
            else
            {
                if (lane < 4)
                    word_add(wd, v, lane);
                Words x;
                unsigned n = 0;
                for (;;)
                {
                    x.load(wd);
                    if (x.all_in(target))
                    {
                        bad = x.decode(w.nblk, s_pq, pq);
                        break;
                    }
                    if (++n > sc.limit)
                    {
                        stop = 9;
                        break;
                    }
                    if (n > 256)
                        __nanosleep(32);
                }
            }
            if (!stop)
            {
                pq48 = top48(pq);
                bool ok;
                af = ratio(rho48, pq48, recip(pq48), &ok);
                if (bad)
                    stop = 6;
                else if (pq48.hi == 0u)
                    stop = 7;
                else if (!ok)
                    af = float(value(rho) / value(pq));
            }
        }
        if (lane == 0)
        {
            sh.af = af;
            sh.stop = stop;
        }
        __syncwarp();
        bar_arrive(3, kAll);
        if (stop)
            break;
        rho_a = rho;
        pq_a = pq;
        have_a = true;
        s_pq = scale_of(pq, pq48);
        if (lane == 0)
            scale[0] = s_pq;
        bool noise = false;
        if (CLUSTER) // (while the workers form z)
        {
            if (multi)
                mag[0] = __reduce_add_sync(kFull,
                                           lane < w.nblk ? unsigned(sh.rec[3][lane].x) : 0u);
            noise = is_noise(pq, mag[0]);
        }
        // ---- r.z, r.r and beta
        bar_sync(4, kAll);
        if (*(volatile int *)&sh.err)
            stop = 9;
        float bf = 0.f;
        Raw rz = rho;
        Top48 new48 = rho48;
        Digits v2;
        Words x, y;
        bool bad = false;
        unsigned n = 0;
        if (!stop)
        {
            const Digits v1 = take(dig[1]);
            v2 = take(dig[2]);
            mag[1] = (unsigned long long)v1.mag;
            if (!multi)
                bad = decode(v1, s_rho, rz);
            else if (CLUSTER)
            {
                const int4 c1 = carried(v1), c2 = carried_with(v2, v1.mag);
                const int4 c = pq_ ? c2 : c1;
                if (lane == 0)
                    mbar_expect(bar_z, 32u * (unsigned(w.nblk) + sc.extra));
                __syncwarp();
                if (pr_ < w.nblk)
                    peer_store(at_z, to_z, c.x, c.y, c.z, c.w);
                if (mbar_wait(bar_z, phase, sc.limit))
                    bad = decode(sh.rec[1], w.nblk, s_rho, rz);
                else
                    stop = 9;
                __syncwarp();
            }
            else
            {
                if (lane < 8)
                    word_add(wd + 4 + (lane & 4), lane < 4 ? v1 : v2, lane & 3);
                else if (lane < 10)
                    mag_add(wd + 4 + lane, lane == 8 ? int(mag[0]) : v1.mag);
                for (;;)
                {
                    x.load(wd + 4);
                    if (x.all_in(target))
                    {
                        bad = x.decode(w.nblk, s_rho, rz);
                        break;
                    }
                    if (++n > sc.limit)
                    {
                        stop = 9;
                        break;
                    }
                    if (n > 256)
                        __nanosleep(32);
                }
            }
            if (!stop)
            {
                new48 = top48(rz);
                bool ok;
                bf = ratio(new48, rho48, rb_rho, &ok);
                if (!ok)
                    bf = rho48.hi == 0u ? 0.f : float(value(rz) / value(rho));
            }
        }
        if (lane == 0)
            sh.bf = bf;
        __syncwarp();
        bar_arrive(5, kAll);
        // ---- r.r, the convergence test and the next scales, while the
        // workers form p and A p
        phase ^= 1u;
        if (!stop && multi && !CLUSTER)
            for (;;)
            {
                y.load(wd + 8);
                if (mags_in(wd + 12, target, mag) && y.all_in(target))
                    break;
                if (++n > sc.limit)
                {
                    stop = 9;
                    break;
                }
            }
        if (stop)
            continue; // a wait gave up: told at the next alpha
        bad |= !multi    ? decode(v2, s_rr, rr)
               : CLUSTER ? decode_with(sh.rec[2], w.nblk, s_rr, rr, mag[1])
                         : y.decode(w.nblk, s_rr, rr);
        if (!CLUSTER)
            noise = is_noise(pq, mag[0] & kSumMask);
        // (no branches: these are between two exchanges)
        bad = (int(bad) | int(noise) | int(is_noise(rz, mag[1] & kSumMask)) |
               int(rho48.hi == 0u && new48.hi != 0u) |
               int(rr_was_zero && (rr.hi | (long long)rr.lo) != 0)) != 0;
        it++;
        rho_b = rho;
        have_b = true;
        rho = rz;
        rho48 = new48;
        rb_rho = recip(rho48);
        const Top48 r48 = top48(rr);
        rr_was_zero = r48.hi == 0u;
        s_rho = scale_of(rho, rho48);
        s_rr = scale_of(rr, r48);
        if (lane == 0)
        {
            scale[1] = s_rho;
            scale[2] = s_rr;
        }
        const bool check = to_check == 0 || it >= max_iters;
        to_check = to_check == 0 ? check_every - 1 : to_check - 1;
        if (bad)
            stop = 6;
        else
        {
            if (check && tests &&
                (r48.hi == 0u || thr48.hi == 0u || key(r48) <= thr_key))
            {
                const double v = value(rr);
                if ((d.rel_tol2 > 0.0 && v <= d.rel_tol2 * bb) ||
                    (d.abs_tol2 > 0.0 && v <= d.abs_tol2))
                    stop = 1;
            }
            if (!stop && it >= max_iters)
                stop = 8;
            if (!stop && sc.iters != 0u && unsigned(it - it0) >= sc.iters)
                stop = kLeave;
        }
    }
    if (lane == 0)
    {
        if (stop == 9)
            atomicExch(&st->bar_err, 1);
        if (w.rank == 0)
        {
            const double rho_d = value(rho), b_d = value(rho_b);
            st->iter = it;
            st->status = stop == 1 || stop == kLeave ? 0 : stop;
            st->rho = rho_d;
            st->rr = value(rr);
            st->pq = value(pq);
            st->alpha = have_a ? value(rho_a) / value(pq_a) : alpha0;
            st->beta = have_b ? (b_d == 0.0 ? 0.0 : rho_d / b_d) : beta0;
            if (stop == kLeave)
                st->beta = 0.0; // z holds the next p
            else
                st->active = 0;
        }
    }
    if (CLUSTER)
    {
        // (a block that gave up leaves its shared memory to the peers' stores that
        // are still on their way)
        if (stop == 9)
            for (int i = 0; i < 32; i++)
                __nanosleep(1000);
        cluster_sync();
        // a wait of another block alone gave up, after the first one's last sum: the
        // solve is not to go on from that block's rows
        if (lane == 0 && w.rank == 0 && stop != 9 && atomicAdd(&st->bar_err, 0) != 0)
        {
            st->status = 9;
            st->active = 0;
        }
    }
}

__device__ __forceinline__ float3 pick(bool on, float3 a, float3 b)
{
    return make_float3(on ? a.x : b.x, on ? a.y : b.y, on ? a.z : b.z);
}

} // namespace

// K: chunks of 32 rows per warp (a block owns at most K * kTeamWorkers rows).
// SKEW: the launch set holds a dihedral-bending instance; skew block parts
// are kept and applied where an instance has them.
// The first RW blocks of a row are in registers (where a thread has one row),
// the others in shared memory: its bandwidth (11 wavefronts per slot and warp,
// 5 of them for p and the column) bounds the SpMV of a full block.
// CLUSTER: every team is one thread-block cluster (the launch's cluster size,
// idle blocks included) and exchanges sums and z rows through its blocks'
// shared memory: ~400 cycles a sum instead of ~1,500.  Teams are independent,
// so a launch may have more of them than fit on the GPU at once.
template <int K, int RW, bool SKEW, bool CLUSTER>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_pcg_team(InstDesc *const *descs, const TeamBlock *work, TeamSync *sync, SpinCfg sc)
{
    constexpr int kAll = kTeamThreads;
    constexpr int RC = RW > 0 ? 5 : 0; // slots past the RW whose offsets of p are in registers
    extern __shared__ float4 sm_dyn[];
    __shared__ InstDesc d;
    alignas(16) __shared__ int s_dig[3][8]; // digits of the block's sums: p.q, r.z, r.r
    __shared__ int s_scale[3];   // and their scales
    __shared__ Shared<CLUSTER> sh;
    const TeamBlock w = work[blockIdx.x];
    if (!team_begin(descs, w, d, sh))
        return;
    InstState *st = d.st;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrow = w.row1 - w.row0, nch = (nrow + 31) >> 5;
    const int nh = w.halo1 - w.halo0, W = max(d.width - RW, 0); // slots in shared memory
    const bool skew = SKEW && d.Aw;
    // the test hook's extra arrivals make a team of one wait too
    const bool multi = w.nblk > 1 || sc.extra != 0u;
    const int it0 = __ldcg(&st->iter);
    // shared memory: p over the halo (z of its rows that other blocks own),
    // then the rows' blocks by slot
    const int nhalo = nh - nrow;
    float4 *sp = sm_dyn;
    float4 *sz = sp + nh;
    // chunk by chunk and slot by slot a record of 32 rows: blocks (16 and 8
    // bytes), byte offsets of p (and skew parts), so that a walk over the slots
    // has constant strides
    constexpr int kRec = team_slot_bytes(false);
    const int rec = team_slot_bytes(skew);
    float4 *sM0 = CLUSTER ? sz + nhalo : sz; // inverse diagonal blocks
    float2 *sM1 = reinterpret_cast<float2 *>(sM0 + nrow);
    char *sA = reinterpret_cast<char *>(sM1 + ((nrow + 1) & ~1));

    if (warp == kWarps)
    {
        control_warp<CLUSTER>(d, w, sync, sc, it0, multi, sh, s_dig, s_scale);
        return;
    }

    // ---------------------------------------------------- workers
    const int own0 = w.row0 - w.halo0;
    const unsigned bar_h = smem_u32(sh.bar + 2);
    if constexpr (CLUSTER)
        if (tid == 0)
            find_peers(work, w, sh, [](int halo) { return smem_u32(sm_dyn) + 16u * unsigned(halo); });
    unsigned hphase = 0;
    float3 x[K], r[K], z[K], p[K];
    int len[K];
    float bf = float(__ldcg(&st->beta));
    {
        const float4 *pold = (it0 & 1) ? d.p1 : d.p0;
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = (warp + k * kWarps) * 32 + lane, row = w.row0 + li;
            len[k] = 0;
            x[k] = r[k] = z[k] = p[k] = make_float3(0.f, 0.f, 0.f);
            if (li < nrow)
            {
                len[k] = d.rowinfo[row] & 255;
                x[k] = xyz(d.dx[row]);
                r[k] = xyz(d.r[row]);
                z[k] = xyz(d.z[row]);
                sM0[li] = d.M0[row];
                sM1[li] = d.M1[row];
                if (it0 > 0)
                    p[k] = xyz(__ldcg(pold + row));
            }
        }
        // a solve handed over in its middle: p_old over the halo
        if (it0 > 0)
            for (int i = tid; i < nhalo; i += kWorkers)
            {
                const int j = i < own0 ? i : i + nrow;
                sp[j] = __ldcg(pold + w.halo0 + j);
            }
    }
    // the rows' blocks: lower slots from their transposed position
    const int wl = d.width_lo, wu = d.width_up;
    auto block_of = [&](int s, int row, int info, uint32_t &oa) -> int {
        if (s < ((info >> 8) & 255))
        {
            const uint32_t ref = d.lref[lo_idx(s, row, wl)];
            oa = lref_block(ref, wu);
            return lref_col(ref) - w.halo0;
        }
        oa = up_idx(s - ((info >> 8) & 255), row, wu);
        return d.colu[oa] - w.halo0;
    };
    float rA[RW + 1][6], rw[RW + 1][3];
    unsigned rc[RW + RC + 1];
    if (RW > 0)
    {
        const int li = warp * 32 + lane, row = w.row0 + li;
        const int info = li < nrow ? d.rowinfo[row] : 0;
#pragma unroll
        for (int s = 0; s < RW; s++)
        {
            rc[s] = li < nrow ? unsigned(own0 + li) * 16u : 0u;
#pragma unroll
            for (int i = 0; i < 6; i++)
                rA[s][i] = 0.f;
            rw[s][0] = rw[s][1] = rw[s][2] = 0.f;
            if (s < (info & 255))
            {
                uint32_t oa;
                rc[s] = unsigned(block_of(s, row, info, oa)) * 16u;
                load_sym(d.A0, d.A1, oa, rA[s]);
                if (SKEW && skew)
                {
                    const float4 aw = d.Aw[oa];
                    rw[s][0] = aw.x;
                    rw[s][1] = aw.y;
                    rw[s][2] = aw.z;
                }
            }
        }
#pragma unroll
        for (int s = RW; s < RW + RC; s++)
        {
            uint32_t oa;
            rc[s] = li < nrow ? unsigned(own0 + li) * 16u : 0u;
            if (s < (info & 255))
                rc[s] = unsigned(block_of(s, row, info, oa)) * 16u;
        }
    }
    const int ds0 = RW > 0 && warp * 32 + lane < nrow
                        ? (d.rowinfo[w.row0 + warp * 32 + lane] >> 8) & 255
                        : 0;
    {
#pragma unroll 2
        for (int u = warp; u < W * nch; u += kWarps)
        {
            const int c = u / W, s = u - c * W, li = c * 32 + lane, row = w.row0 + li;
            const int info = li < nrow ? d.rowinfo[row] : 0, slot = s + RW;
            char *at = sA + size_t(u) * rec;
            float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), aw = a0;
            float2 a1 = make_float2(0.f, 0.f);
            // past a row's last slot: a zero block at the row's own column
            int col = li < nrow ? own0 + li : 0;
            if (slot < (info & 255))
            {
                uint32_t oa;
                col = block_of(slot, row, info, oa);
                a0 = d.A0[oa];
                a1 = d.A1[oa];
                if (SKEW && skew)
                {
                    aw = d.Aw[oa];
                    // the transposed block's skew part changes sign
                    aw.w = slot < ((info >> 8) & 255) ? -1.f : 1.f;
                }
            }
            reinterpret_cast<float4 *>(at)[lane] = a0;
            reinterpret_cast<float2 *>(at + 512)[lane] = a1;
            reinterpret_cast<unsigned *>(at + 768)[lane] = unsigned(col) * 16u;
            if (SKEW && skew)
                reinterpret_cast<float4 *>(at + kRec)[lane] = aw;
        }
    }
    // halo rows of z of the first iteration (written before this launch)
    float3 hz[kHaloAhead];
    if (CLUSTER)
        for (int i = tid; i < nhalo; i += kWorkers)
            sz[i] = __ldcg(d.z + w.halo0 + (i < own0 ? i : i + nrow));
    else
#pragma unroll
    for (int u = 0; u < kHaloAhead; u++)
    {
        const int i = tid + u * kWorkers;
        hz[u] = make_float3(0.f, 0.f, 0.f);
        if (i < nhalo)
            hz[u] = xyz(__ldcg(d.z + w.halo0 + (i < own0 ? i : i + nrow)));
    }
    bar_sync(6, kAll);
    for (unsigned tag = unsigned(it0);; tag++)
    {
        // ---- p = z + beta p_old over the halo and the own rows
        const bool first = bf == 0.f;
        for (int i = tid, u = 0; i < nhalo; i += kWorkers, u++)
        {
            const int j = i < own0 ? i : i + nrow;
            float3 zz;
            if (CLUSTER)
                zz = xyz(sz[i]);
            else if (u < kHaloAhead)
                zz = u == 0 ? hz[0] : u == 1 ? hz[1] : hz[2];
            else if (tag == unsigned(it0))
                zz = xyz(__ldcg(d.z + w.halo0 + j));
            else
                zz = poll_row(d.z + w.halo0 + j, tag, sc.limit, &sh.err);
            sp[j] = f4(first ? zz : pform(zz, bf, xyz(sp[j])));
        }
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = (warp + k * kWarps) * 32 + lane;
            if (li < nrow)
            {
                p[k] = first ? z[k] : pform(z[k], bf, p[k]);
                sp[own0 + li] = f4(p[k]);
            }
        }
        bar_sync(1, kWorkers);
        // ---- q = A p; p.q per 32-row chunk
        float3 q[K];
        float part[K];
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int ch = warp + k * kWarps, li = ch * 32 + lane;
            q[k] = make_float3(0.f, 0.f, 0.f);
            part[k] = 0.f;
            if (ch < nch)
            {
                // kAhead slots at a time, loads first; past a row's last slot
                // the blocks are zero (a branch per slot made the walk three
                // times as long)
                constexpr int kAhead = K > 1 || SKEW ? 4 : 8;
                auto p_at = [&](unsigned off) {
                    return *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(sp) +
                                                             off);
                };
#pragma unroll
                for (int s0 = 0; s0 < RW; s0 += kAhead)
                {
                    float4 pc[kAhead];
#pragma unroll
                    for (int i = 0; i < kAhead; i++)
                        if (s0 + i < RW)
                            pc[i] = p_at(rc[s0 + i]);
#pragma unroll
                    for (int i = 0; i < kAhead; i++)
                    {
                        const int s = s0 + i;
                        if (s >= RW)
                            continue;
                        q[k] = q[k] + symv(rA[s], xyz(pc[i]));
                        if (SKEW && skew)
                        {
                            const float3 cw = skewv(
                                make_float4(rw[s][0], rw[s][1], rw[s][2], 0.f), xyz(pc[i]));
                            q[k] = s < ds0 ? q[k] - cw : q[k] + cw;
                        }
                    }
                }
                // N slots of this lane's row from at on; their offsets of p in
                // registers where the first of them is rc's
                auto walk = [&](const char *at, auto count, auto known) {
                    constexpr int N = decltype(count)::value, C = decltype(known)::value;
                    float4 u[N], pc[N];
                    float2 v[N];
#pragma unroll
                    for (int i = 0; i < N; i++)
                    {
                        const char *a = at + i * (SKEW ? rec : kRec);
                        pc[i] = p_at(C >= 0 ? rc[C >= 0 ? C + i : 0]
                                            : reinterpret_cast<const unsigned *>(a + 768)[lane]);
                        u[i] = reinterpret_cast<const float4 *>(a)[lane];
                        v[i] = reinterpret_cast<const float2 *>(a + 512)[lane];
                    }
#pragma unroll
                    for (int i = 0; i < N; i++)
                    {
                        const float A[6] = {u[i].x, u[i].y, u[i].z, u[i].w, v[i].x, v[i].y};
                        q[k] = q[k] + symv(A, xyz(pc[i]));
                        if (SKEW && skew)
                        {
                            const float4 aw =
                                reinterpret_cast<const float4 *>(at + i * rec + kRec)[lane];
                            const float3 cw = skewv(aw, xyz(pc[i]));
                            q[k] = aw.w < 0.f ? q[k] - cw : q[k] + cw;
                        }
                    }
                };
                const int top = __reduce_max_sync(kFull, len[k] - RW);
                const char *at = sA + ch * W * rec;
                using std::integral_constant;
                int s0 = 0;
                if (RC > 0 && top >= RC)
                {
                    walk(at, integral_constant<int, RC ? RC : 1>(), integral_constant<int, RW>());
                    s0 = RC;
                    at += RC * rec;
                }
                for (; s0 + kAhead <= top; s0 += kAhead, at += kAhead * rec)
                    walk(at, integral_constant<int, kAhead>(), integral_constant<int, -1>());
                for (; s0 < top; s0++, at += rec)
                    walk(at, integral_constant<int, 1>(), integral_constant<int, -1>());
                part[k] = warp_sum(li < nrow ? fdot(p[k], q[k]) : 0.f);
            }
        }
        chunks_add<K>(s_dig, s_scale, part);
        bar_arrive(2, kAll);
        // the sum words of iteration it + 2 were last polled in iteration
        // it - 2, which every block of the team has left (its r.z words of
        // it - 1 are in): cleared here, and ordered before this block's next
        // arrivals, by a warp that is waiting anyway
        if (!CLUSTER && multi && w.rank == 0 && warp == kWarps - 1)
        {
            if (lane < 16)
                sync[blockIdx.x].words[(tag + 2u) & 3u][lane] = 0ull;
            __threadfence();
        }
        float4 m0[K]; // (in flight while alpha is awaited)
        float2 m1[K];
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = min((warp + k * kWarps) * 32 + lane, nrow - 1);
            m0[k] = sM0[li];
            m1[k] = sM1[li];
        }
        bar_sync(3, kAll);
        if (*(volatile int *)&sh.stop)
            break;
        const float af = *(volatile float *)&sh.af;
        // ---- r -= alpha q, z = M^-1 r; r.z and r.r per chunk (dx += alpha p
        // once they are on their way)
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int ch = warp + k * kWarps, li = ch * 32 + lane;
            part[k] = 0.f;
            if (ch < nch)
            {
                float pr = 0.f, prr = 0.f;
                if (li < nrow)
                {
                    r[k] = make_float3(fmaf(-af, q[k].x, r[k].x), fmaf(-af, q[k].y, r[k].y),
                                       fmaf(-af, q[k].z, r[k].z));
                    const float M[6] = {m0[k].x, m0[k].y, m0[k].z, m0[k].w, m1[k].x, m1[k].y};
                    z[k] = symv(M, r[k]);
                    if (!CLUSTER && multi)
                        st_row(d.z + w.row0 + li, z[k], tag + 1u);
                    if constexpr (CLUSTER)
                        push_row(sh, w.row0 + li, z[k]);
                    pr = fdot(r[k], z[k]);
                    prr = fdot(r[k], r[k]);
                }
                part[k] = warp_sum2(pr, prr);
            }
        }
        chunks_add2<K>(s_dig, s_scale, part);
        bar_arrive(4, kAll);
#pragma unroll
        for (int k = 0; k < K; k++)
            x[k] = make_float3(fmaf(af, p[k].x, x[k].x), fmaf(af, p[k].y, x[k].y),
                               fmaf(af, p[k].z, x[k].z));
        // the halo rows of the new z, while the sums are under way
#pragma unroll
        for (int u = 0; u < (CLUSTER ? 0 : kHaloAhead); u++)
        {
            const int i = tid + u * kWorkers;
            if (i < nhalo)
                hz[u] = poll_row(d.z + w.halo0 + (i < own0 ? i : i + nrow), tag + 1u, sc.limit,
                                 &sh.err);
        }
        if (CLUSTER && nhalo > 0)
        {
            if (!mbar_wait(bar_h, hphase, sc.limit))
                sh.err = 1;
            hphase ^= 1u;
        }
        bar_sync(5, kAll);
        // (every worker has seen the phase: the next one may be counted)
        if (CLUSTER && nhalo > 0 && tid == 0)
            mbar_expect(bar_h, 16u * unsigned(nhalo));
        bf = *(volatile float *)&sh.bf;
    }
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int li = (warp + k * kWarps) * 32 + lane, row = w.row0 + li;
        if (li < nrow)
        {
            d.dx[row] = f4(x[k]);
            d.r[row] = f4(r[k]);
            // a solve that goes on later starts from its next p, formed above
            if (*(volatile int *)&sh.stop == kLeave)
                d.z[row] = f4(p[k]);
        }
    }
    if (CLUSTER)
        cluster_sync(); // peers may still be storing here
}

// The same solve for blocks with more rows than fit with their whole matrix:
// only the diagonal and upper blocks are kept, each read by its own row and by
// the rows whose lower block is its transpose.  Where not even those fit, the
// planes [u0, u1) of them are on chip (the first upper ones, which serve lower
// slots too; the work list says which) and the others come from L2, as do the
// lower blocks whose transposed row another block owns, but for the last rows
// in front of this block's that fit as well.  A column and the transposed
// block's plane share one 16-bit word.  K: rows per thread.
template <int K, bool SKEW, bool CLUSTER>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_pcg_half(InstDesc *const *descs, const TeamBlock *work, TeamSync *sync, SpinCfg sc)
{
    constexpr int kAll = kTeamThreads;
    extern __shared__ float4 sm_dyn[];
    __shared__ InstDesc d;
    alignas(16) __shared__ int s_dig[3][8];
    __shared__ int s_scale[3];
    __shared__ Shared<CLUSTER> sh;
    const TeamBlock w = work[blockIdx.x];
    if (!team_begin(descs, w, d, sh))
        return;
    InstState *st = d.st;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrow = w.row1 - w.row0, nch = (nrow + 31) >> 5, rp = nch << 5;
    const int nh = w.halo1 - w.halo0, nhalo = nh - nrow;
    const bool skew = SKEW && d.Aw;
    const bool multi = w.nblk > 1 || sc.extra != 0u;
    const int it0 = __ldcg(&st->iter);
    // on chip: planes [u0, u1), of this block's rows and of the last `ext` rows
    // in front of them (other blocks' rows that lower slots refer to)
    const int u0 = w.p_global & 15, u1 = w.p_global >> 4 & 15, ext = w.p_global >> 8;
    const int re = rp + ext; // rows of a plane
    const int wl = d.width_lo, wu = d.width_up;
    // p over the halo in 12 bytes an entry (x and y, then z)
    float2 *spx = reinterpret_cast<float2 *>(sm_dyn);
    float *spz = reinterpret_cast<float *>(spx + nh);
    auto p_get = [&](int j) {
        const float2 v = spx[j];
        return make_float3(v.x, v.y, spz[j]);
    };
    auto p_set = [&](int j, float3 v) {
        spx[j] = make_float2(v.x, v.y);
        spz[j] = v.z;
    };
    float4 *sz = sm_dyn + half_p_quads(nh);
    // plane by plane the rows' stored blocks (24 bytes; with skew parts 40):
    // read 8 bytes at a time, conflict-free at any row
    const int kb = SKEW && skew ? 40 : 24;
    char *sU = reinterpret_cast<char *>(CLUSTER ? sz + nhalo : sz);
    // chunk by chunk and slot by slot 32 words: the lower slots' (column | plane
    // << 12), then the upper planes' columns
    unsigned short *scol =
        reinterpret_cast<unsigned short *>(sU + size_t(u1 - u0) * re * kb);
    if (warp == kWarps)
    {
        control_warp<CLUSTER>(d, w, sync, sc, it0, multi, sh, s_dig, s_scale);
        return;
    }
    const int own0 = w.row0 - w.halo0;
    // A warp's k-th chunk: the first kWarps chunks in turn, then from the last warp
    // on (the first chunks have the lower slots that other blocks own)
    auto chunk = [&](int k) { return k * kWarps + (k == 0 ? warp : kWarps - 1 - warp); };
    const unsigned bar_h = smem_u32(sh.bar + 2);
    if constexpr (CLUSTER)
        if (tid == 0)
            find_peers(work, w, sh, [](int halo) { return smem_u32(sm_dyn) + 16u * unsigned(half_p_quads(halo)); });
    unsigned hphase = 0;
    float3 x[K], r[K], z[K];
    int info[K];
    const float4 *pold = (it0 & 1) ? d.p1 : d.p0;
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int li = chunk(k) * 32 + lane, row = w.row0 + li;
        info[k] = 0;
        x[k] = r[k] = z[k] = make_float3(0.f, 0.f, 0.f);
        if (li < nrow)
        {
            info[k] = d.rowinfo[row];
            x[k] = xyz(d.dx[row]);
            r[k] = xyz(d.r[row]);
            z[k] = xyz(d.z[row]);
        }
    }
    if (it0 > 0) // a solve handed over in its middle
        for (int i = tid; i < nh; i += kWorkers)
            p_set(i, xyz(__ldcg(pold + w.halo0 + i)));
    unsigned far = 0u; // chunks of this warp with a lower slot whose block is not on chip
#pragma unroll 2
    for (int u = warp; u < (wl + wu) * nch; u += kWarps)
    {
        const int c = u / (wl + wu), s = u - c * (wl + wu), li = c * 32 + lane,
                  row = w.row0 + li;
        const int inf = li < nrow ? d.rowinfo[row] : 0, ds = (inf >> 8) & 255;
        const int uu = s - wl; // upper plane
        // past a row's last slot: its own column and a block on chip (not used),
        // or a zero block
        unsigned word = unsigned(own0 + min(li, nrow - 1)) | (s < wl ? unsigned(u0) << 12 : 0u);
        if (s < wl)
        {
            if (s < ds)
            {
                const uint32_t ref = d.lref[lo_idx(s, row, wl)];
                word = unsigned(lref_col(ref) - w.halo0) | (ref >> 24) << 12;
            }
        }
        else
        {
            float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), aw = a0;
            float2 a1 = make_float2(0.f, 0.f);
            const bool here = uu >= u0 && uu < u1;
            if (uu < (inf & 255) - ds)
            {
                const uint32_t oa = up_idx(uu, row, wu);
                word = unsigned(d.colu[oa] - w.halo0);
                if (here)
                {
                    a0 = d.A0[oa];
                    a1 = d.A1[oa];
                    if (SKEW && skew)
                        aw = d.Aw[oa];
                }
            }
            if (here)
            {
                float2 *o = reinterpret_cast<float2 *>(sU + (size_t(uu - u0) * re + ext + li) * kb);
                o[0] = make_float2(a0.x, a0.y);
                o[1] = make_float2(a0.z, a0.w);
                o[2] = a1;
                if (SKEW && skew)
                {
                    o[3] = make_float2(aw.x, aw.y);
                    o[4] = make_float2(aw.z, 0.f);
                }
            }
        }
        scol[size_t(u) * 32 + lane] = (unsigned short)word;
    }
    for (int i = tid; i < ext; i += kWorkers)
    {
        const int row = w.row0 - ext + i, inf = d.rowinfo[row],
                  ne = (inf & 255) - ((inf >> 8) & 255);
        for (int uu = u0; uu < min(u1, ne); uu++)
        {
            const uint32_t oa = up_idx(uu, row, wu);
            const float4 a0 = d.A0[oa];
            float2 *o = reinterpret_cast<float2 *>(sU + (size_t(uu - u0) * re + i) * kb);
            o[0] = make_float2(a0.x, a0.y);
            o[1] = make_float2(a0.z, a0.w);
            o[2] = d.A1[oa];
            if (SKEW && skew)
            {
                const float4 aw = d.Aw[oa];
                o[3] = make_float2(aw.x, aw.y);
                o[4] = make_float2(aw.z, 0.f);
            }
        }
    }
    bar_sync(1, kWorkers);
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int ch = chunk(k);
        bool any = false;
        if (ch < nch)
            for (int s = 0; s < ((info[k] >> 8) & 255); s++)
            {
                const unsigned wd = scol[(size_t(ch) * (wl + wu) + s) * 32 + lane];
                any |= int(wd & 4095u) < own0 - ext ||
                       (wd >> 12) - unsigned(u0) >= unsigned(u1 - u0);
            }
        far |= __any_sync(kFull, any) ? 1u << k : 0u;
    }
    // halo rows of z of the first iteration (written before this launch)
    float3 hz[kHaloAhead];
    if (CLUSTER)
        for (int i = tid; i < nhalo; i += kWorkers)
            sz[i] = __ldcg(d.z + w.halo0 + (i < own0 ? i : i + nrow));
    else
#pragma unroll
        for (int u = 0; u < kHaloAhead; u++)
        {
            const int i = tid + u * kWorkers;
            hz[u] = make_float3(0.f, 0.f, 0.f);
            if (i < nhalo)
                hz[u] = xyz(__ldcg(d.z + w.halo0 + (i < own0 ? i : i + nrow)));
        }
    float bf = float(__ldcg(&st->beta));
    bar_sync(6, kAll);
    for (unsigned tag = unsigned(it0);; tag++)
    {
        // ---- p = z + beta p_old over the halo and the own rows
        const bool first = bf == 0.f;
        for (int i = tid, u = 0; i < nhalo; i += kWorkers, u++)
        {
            const int j = i < own0 ? i : i + nrow;
            float3 zz;
            if (CLUSTER)
                zz = xyz(sz[i]);
            else if (u < kHaloAhead)
                zz = u == 0 ? hz[0] : u == 1 ? hz[1] : hz[2];
            else if (tag == unsigned(it0))
                zz = xyz(__ldcg(d.z + w.halo0 + j));
            else
                zz = poll_row(d.z + w.halo0 + j, tag, sc.limit, &sh.err);
            p_set(j, first ? zz : pform(zz, bf, p_get(j)));
        }
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = chunk(k) * 32 + lane;
            if (li < nrow)
                p_set(own0 + li, first ? z[k] : pform(z[k], bf, p_get(own0 + li)));
        }
        bar_sync(1, kWorkers);
        // ---- q = A p; p.q per 32-row chunk
        float3 q[K];
        float part[K];
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int ch = chunk(k), li = ch * 32 + lane, row = w.row0 + li;
            q[k] = make_float3(0.f, 0.f, 0.f);
            part[k] = 0.f;
            if (ch >= nch)
                continue;
            const int ds = (info[k] >> 8) & 255, ne = (info[k] & 255) - ds;
            const int top_l = __reduce_max_sync(kFull, ds), top_u = __reduce_max_sync(kFull, ne);
            struct Block
            {
                float A[6];
                float4 w;
            };
            auto add = [&](const Block &b, float3 pc, bool lower, bool on) {
                float3 t = q[k] + symv(b.A, pc);
                if (SKEW && skew)
                {
                    const float3 cw = skewv(b.w, pc);
                    t = lower ? t - cw : t + cw;
                }
                q[k] = pick(on, t, q[k]);
            };
            auto on_chip = [&](const char *at) {
                const float2 *o = reinterpret_cast<const float2 *>(at);
                const float2 e0 = o[0], e1 = o[1], e2 = o[2];
                Block b{{e0.x, e0.y, e1.x, e1.y, e2.x, e2.y}, {0.f, 0.f, 0.f, 0.f}};
                if (SKEW && skew)
                {
                    const float2 e3 = o[3], e4 = o[4];
                    b.w = make_float4(e3.x, e3.y, e4.x, 0.f);
                }
                return b;
            };
            auto from_l2 = [&](bool on, int u, int r) {
                Block b{{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                if (on)
                {
                    const uint32_t oa = up_idx(u, r, wu);
                    const float4 a0 = __ldg(d.A0 + oa);
                    const float2 a1 = __ldg(d.A1 + oa);
                    b.A[0] = a0.x;
                    b.A[1] = a0.y;
                    b.A[2] = a0.z;
                    b.A[3] = a0.w;
                    b.A[4] = a1.x;
                    b.A[5] = a1.y;
                    if (SKEW && skew)
                        b.w = __ldg(d.Aw + oa);
                }
                return b;
            };
            // upper planes that are not on chip: the first kPre in flight from here
            constexpr int kPre = 2;
            Block f[kPre];
#pragma unroll
            for (int i = 0; i < kPre; i++)
            {
                const int u = i == 0 ? 0 : u1 + i - 1;
                f[i] = from_l2((i > 0 || u0 > 0) && u < ne, u, row);
            }
            // lower slots, kLow at a time, loads first
            const unsigned short *cc = scol + size_t(ch) * (wl + wu) * 32 + lane;
            constexpr int kLow = 3;
            const char *sUl = sU - (own0 - ext + u0 * re) * kb; // entry c, plane u at (u re + c) kb
            if (!(far >> k & 1u))
                for (int s0 = 0; s0 < top_l; s0 += kLow)
                {
                    Block b[kLow];
                    float3 pc[kLow];
#pragma unroll
                    for (int i = 0; i < kLow; i++)
                    {
                        const unsigned wd = cc[min(s0 + i, top_l - 1) * 32];
                        pc[i] = p_get(wd & 4095u);
                        b[i] = on_chip(sUl + int((wd >> 12) * unsigned(re) + (wd & 4095u)) * kb);
                    }
#pragma unroll
                    for (int i = 0; i < kLow; i++)
                        add(b[i], pc[i], true, s0 + i < ds);
                }
            else
                for (int s0 = 0; s0 < top_l; s0 += kLow)
                {
                    Block b[kLow];
                    float3 pc[kLow];
#pragma unroll
                    for (int i = 0; i < kLow; i++)
                    {
                        const unsigned wd = cc[min(s0 + i, top_l - 1) * 32];
                        const int c = int(wd & 4095u), u = int(wd >> 12);
                        pc[i] = p_get(c);
                        if (c >= own0 - ext && unsigned(u - u0) < unsigned(u1 - u0))
                            b[i] = on_chip(sUl + (u * re + c) * kb);
                        else
                            b[i] = from_l2(s0 + i < ds, u, c + w.halo0);
                    }
#pragma unroll
                    for (int i = 0; i < kLow; i++)
                        add(b[i], pc[i], true, s0 + i < ds);
                }
            // upper slots in order (past a row's last one the blocks are zero)
            const unsigned short *cu = cc + wl * 32;
            if (u0 > 0)
                add(f[0], p_get(cu[0]), false, true);
            const int top_r = min(top_u, u1);
            const char *at = sU + (ext + li) * kb;
            const unsigned short *cr = cu + u0 * 32;
            auto walk = [&](auto count) {
                constexpr int N = decltype(count)::value;
                Block b[N];
                float3 pc[N];
#pragma unroll
                for (int i = 0; i < N; i++)
                {
                    pc[i] = p_get(cr[i * 32]);
                    b[i] = on_chip(at + i * re * kb);
                }
#pragma unroll
                for (int i = 0; i < N; i++)
                    add(b[i], pc[i], false, true);
                at += N * re * kb;
                cr += N * 32;
            };
            int u = u0;
            for (; u + 3 <= top_r; u += 3)
                walk(std::integral_constant<int, 3>());
            for (; u < top_r; u++)
                walk(std::integral_constant<int, 1>());
#pragma unroll
            for (int i = 1; i < kPre; i++)
                if (u1 + i - 1 < top_u)
                    add(f[i], p_get(cu[(u1 + i - 1) * 32]), false, true);
            for (u = u1 + kPre - 1; u < top_u; u++)
                add(from_l2(u < ne, u, row), p_get(cu[u * 32]), false, true);
            const float3 pv = p_get(own0 + min(li, nrow - 1));
            part[k] = warp_sum(li < nrow ? fdot(pv, q[k]) : 0.f);
        }
        chunks_add<K>(s_dig, s_scale, part);
        bar_arrive(2, kAll);
        if (!CLUSTER && multi && w.rank == 0 && warp == kWarps - 1)
        {
            // the sum words of iteration it + 2 (see k_pcg_team)
            if (lane < 16)
                sync[blockIdx.x].words[(tag + 2u) & 3u][lane] = 0ull;
            __threadfence();
        }
        // the inverse diagonal blocks, in flight while alpha is awaited
        float4 m0[K];
        float2 m1[K];
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = chunk(k) * 32 + lane;
            m0[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            m1[k] = make_float2(0.f, 0.f);
            if (li < nrow)
            {
                m0[k] = __ldg(d.M0 + w.row0 + li);
                m1[k] = __ldg(d.M1 + w.row0 + li);
            }
        }
        bar_sync(3, kAll);
        if (*(volatile int *)&sh.stop)
            break;
        const float af = *(volatile float *)&sh.af;
        // ---- r -= alpha q, z = M^-1 r; r.z and r.r per chunk (dx += alpha p
        // once they are on their way)
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int ch = chunk(k), li = ch * 32 + lane;
            part[k] = 0.f;
            if (ch < nch)
            {
                float pr = 0.f, prr = 0.f;
                if (li < nrow)
                {
                    r[k] = make_float3(fmaf(-af, q[k].x, r[k].x), fmaf(-af, q[k].y, r[k].y),
                                       fmaf(-af, q[k].z, r[k].z));
                    const float M[6] = {m0[k].x, m0[k].y, m0[k].z, m0[k].w, m1[k].x, m1[k].y};
                    z[k] = symv(M, r[k]);
                    if constexpr (CLUSTER)
                        push_row(sh, w.row0 + li, z[k]);
                    else if (multi)
                        st_row(d.z + w.row0 + li, z[k], tag + 1u);
                    pr = fdot(r[k], z[k]);
                    prr = fdot(r[k], r[k]);
                }
                part[k] = warp_sum2(pr, prr);
            }
        }
        chunks_add2<K>(s_dig, s_scale, part);
        bar_arrive(4, kAll);
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = chunk(k) * 32 + lane;
            if (li < nrow)
            {
                const float3 p = p_get(own0 + li);
                x[k] = make_float3(fmaf(af, p.x, x[k].x), fmaf(af, p.y, x[k].y),
                                   fmaf(af, p.z, x[k].z));
            }
        }
        // the halo rows of the new z, while the sums are under way
        if (CLUSTER)
        {
            if (nhalo > 0 && !mbar_wait(bar_h, hphase, sc.limit))
                sh.err = 1;
            hphase ^= 1u;
        }
        else
#pragma unroll
            for (int u = 0; u < kHaloAhead; u++)
            {
                const int i = tid + u * kWorkers;
                if (i < nhalo)
                    hz[u] = poll_row(d.z + w.halo0 + (i < own0 ? i : i + nrow), tag + 1u,
                                     sc.limit, &sh.err);
            }
        bar_sync(5, kAll);
        if (CLUSTER && nhalo > 0 && tid == 0)
            mbar_expect(bar_h, 16u * unsigned(nhalo));
        bf = *(volatile float *)&sh.bf;
    }
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int li = chunk(k) * 32 + lane, row = w.row0 + li;
        if (li < nrow)
        {
            d.dx[row] = f4(x[k]);
            d.r[row] = f4(r[k]);
            if (*(volatile int *)&sh.stop == kLeave)
                d.z[row] = f4(p_get(own0 + li));
        }
    }
    if (CLUSTER)
        cluster_sync();
}

// The same solve for blocks with more rows than k_pcg_half takes, the matrix read
// from memory (sets without skew parts).  On chip are p over the halo and q, then z,
// in one place of shared memory, and up to kWideRows rows a thread r and dx in
// registers and the inverse diagonal blocks in shared memory as well.  z goes to
// memory only for rows that another block's columns touch.  K: most rows per thread.
//
// What bounds it: reading the stored blocks and the columns (220 bytes a row of a
// grid) and the transposed rows' blocks again, from L2 and past ~650^2 from HBM, by as
// many loads as the registers hold.  So a warp has a group's loads in flight
// together: the upper planes' addresses need no column, and a chunk's lower references
// are fetched one chunk ahead.  Groups of 3 next to r and dx in registers (groups of 4
// spill: 640^2 28.0 us per iteration, 26.6 with 3); where the matrix does not stay in
// L2 r and dx are better read as well and the registers hold groups of 6: 1024^2 92.0
// us (4: 98.7, 5: 95.1; 3 with r in registers 99.7), 760^2 42.3 (48.3).
// us per iteration, before (k_pcg_persistent_gm): 545^2 27.5 -> 18.9, 640^2 44.4 ->
// 26.6, 680^2 47.9 -> 35.4, 760^2 59.7 -> 42.3, 800^2 69.3 -> 46.9, 1024^2 100.3 -> 92.0.
template <int K>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_pcg_wide(InstDesc *const *descs, const TeamBlock *work, TeamSync *sync, SpinCfg sc)
{
    constexpr int kAll = kTeamThreads;
    constexpr bool kHold = wide_hold(K); // r, dx and the inverse diagonal blocks on chip
    extern __shared__ float4 sm_dyn[];
    __shared__ InstDesc d;
    alignas(16) __shared__ int s_dig[3][8];
    __shared__ int s_scale[3];
    __shared__ Shared<false> sh;
    const TeamBlock w = work[blockIdx.x];
    if (!team_begin(descs, w, d, sh))
        return;
    InstState *st = d.st;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = lane >> 3;
    const int nrow = w.row1 - w.row0, nch = (nrow + 31) >> 5, rp = nch << 5;
    const int nh = w.halo1 - w.halo0, nhalo = nh - nrow;
    const bool multi = w.nblk > 1 || sc.extra != 0u;
    const int it0 = __ldcg(&st->iter);
    const int wl = d.width_lo, wu = d.width_up;
    float2 *spx = reinterpret_cast<float2 *>(sm_dyn);
    float *spz = reinterpret_cast<float *>(spx + nh);
    auto p_get = [&](int j) {
        const float2 v = spx[j];
        return make_float3(v.x, v.y, spz[j]);
    };
    auto p_set = [&](int j, float3 v) {
        spx[j] = make_float2(v.x, v.y);
        spz[j] = v.z;
    };
    float2 *sqx = reinterpret_cast<float2 *>(sm_dyn + half_p_quads(nh));
    float *sqz = reinterpret_cast<float *>(sqx + rp);
    auto q_get = [&](int j) {
        const float2 v = sqx[j];
        return make_float3(v.x, v.y, sqz[j]);
    };
    auto q_set = [&](int j, float3 v) {
        sqx[j] = make_float2(v.x, v.y);
        sqz[j] = v.z;
    };
    float2 *sM = reinterpret_cast<float2 *>(sqz + rp); // three of rp
    if (warp == kWarps)
    {
        control_warp<false>(d, w, sync, sc, it0, multi, sh, s_dig, s_scale);
        return;
    }
    const int own0 = w.row0 - w.halo0;
    // rows below need0 or from need1 on have readers in other blocks
    int need0 = w.row0, need1 = w.row1;
    for (int j = lane; j < w.nblk; j += 32)
    {
        const TeamBlock &o = work[int(blockIdx.x) - w.rank + j];
        if (o.row1 <= w.row0)
            need0 = max(need0, o.halo1);
        else if (o.row0 >= w.row1)
            need1 = min(need1, o.halo0);
    }
    need0 = __reduce_max_sync(kFull, need0);
    need1 = __reduce_min_sync(kFull, need1);
    float3 x[kHold ? K : 1], r[kHold ? K : 1];
    const float4 *pold = (it0 & 1) ? d.p1 : d.p0;
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int li = (k * kWarps + warp) * 32 + lane, row = w.row0 + li;
        if constexpr (kHold)
            x[k] = r[k] = make_float3(0.f, 0.f, 0.f);
        if (li < nrow)
        {
            q_set(li, xyz(d.z[row]));
            if constexpr (kHold)
            {
                r[k] = xyz(d.r[row]);
                x[k] = xyz(d.dx[row]);
                const float4 m0 = d.M0[row];
                sM[li] = make_float2(m0.x, m0.y);
                sM[rp + li] = make_float2(m0.z, m0.w);
                sM[2 * rp + li] = d.M1[row];
            }
        }
    }
    if (it0 > 0) // a solve handed over in its middle
        for (int i = tid; i < nh; i += kWorkers)
            p_set(i, xyz(__ldcg(pold + w.halo0 + i)));
    bar_sync(1, kWorkers);
    // halo rows of z of the first iteration (written before this launch)
    float3 hz[kHaloAhead];
#pragma unroll
    for (int u = 0; u < kHaloAhead; u++)
    {
        const int i = tid + u * kWorkers;
        hz[u] = make_float3(0.f, 0.f, 0.f);
        if (i < nhalo)
            hz[u] = xyz(__ldcg(d.z + w.halo0 + (i < own0 ? i : i + nrow)));
    }
    float bf = float(__ldcg(&st->beta));
    bar_sync(6, kAll);
    for (unsigned tag = unsigned(it0);; tag++)
    {
        // ---- p = z + beta p_old over the halo and the own rows
        const bool first = bf == 0.f;
        for (int i = tid, u = 0; i < nhalo; i += kWorkers, u++)
        {
            const int j = i < own0 ? i : i + nrow;
            float3 zz;
            if (u < kHaloAhead)
                zz = u == 0 ? hz[0] : u == 1 ? hz[1] : hz[2];
            else if (tag == unsigned(it0))
                zz = xyz(__ldcg(d.z + w.halo0 + j));
            else
                zz = poll_row(d.z + w.halo0 + j, tag, sc.limit, &sh.err);
            p_set(j, first ? zz : pform(zz, bf, p_get(j)));
        }
        // (a thread's first row, formed anew: else the addresses and bounds of all its
        // rows are kept in registers from one iteration to the next)
        int li0 = warp * 32 + lane;
        asm volatile("" : "+r"(li0));
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = k * kWorkers + li0;
            if (li < nrow)
            {
                const float3 z = q_get(li);
                p_set(own0 + li, first ? z : pform(z, bf, p_get(own0 + li)));
            }
        }
        // (the first chunk's references, in flight over the barrier)
        constexpr int G = kHold ? 3 : 6, kRef = kHold ? 2 * G : G;
        uint32_t next_ref[kRef];
        int next_info = 0;
        auto fetch = [&](int ch) {
            const int row = min(w.row0 + ch * 32 + lane, w.row1 - 1);
            next_info = __ldg(d.rowinfo + row);
#pragma unroll
            for (int i = 0; i < kRef; i++)
                next_ref[i] = i < wl ? __ldg(d.lref + lo_idx(i, row, wl)) : 0u;
        };
        fetch(min(warp, nch - 1));
        bar_sync(1, kWorkers);
        // ---- q = A p; p.q per 32-row chunk
        int dig = 0;
        float v4 = 0.f; // four chunks' sums, one per group of 8 lanes
#pragma unroll 1
        for (int k = 0; k < K; k++)
        {
            const int ch = k * kWarps + warp, li = ch * 32 + lane, row = w.row0 + li;
            if (ch >= nch)
                break;
            const int inf = li < nrow ? next_info : 0;
            const int ds = (inf >> 8) & 255, ne = (inf & 255) - ds;
            struct Block
            {
                float4 a0;
                float2 a1;
            };
            float3 q = make_float3(0.f, 0.f, 0.f);
            auto load = [&](Block &b, bool on, uint32_t oa) {
                b.a0 = make_float4(0.f, 0.f, 0.f, 0.f);
                b.a1 = make_float2(0.f, 0.f);
                if (on)
                {
                    b.a0 = __ldg(d.A0 + oa);
                    b.a1 = __ldg(d.A1 + oa);
                }
            };
            auto add = [&](const Block &b, float3 pc, bool on) {
                const float A[6] = {b.a0.x, b.a0.y, b.a0.z, b.a0.w, b.a1.x, b.a1.y};
                q = pick(on, q + symv(A, pc), q);
            };
            // the upper planes' first group and the lower ones' first two groups
            // know their addresses
            Block up[G], lo[G];
            int cu[G], cl[G];
            auto lower = [&](int i, bool on, uint32_t ref) {
                load(lo[i], on, lref_block(ref, wu));
                cl[i] = on ? lref_col(ref) - w.halo0 : own0;
            };
            auto upper = [&](int i, int u) {
                const uint32_t oa = up_idx(u, row, wu);
                load(up[i], u < ne, oa);
                cu[i] = u < ne ? __ldg(d.colu + oa) - w.halo0 : own0;
            };
            uint32_t ref[kRef];
#pragma unroll
            for (int i = 0; i < kRef; i++)
                ref[i] = next_ref[i];
#pragma unroll
            for (int i = 0; i < G; i++)
                lower(i, i < ds, ref[i]);
#pragma unroll
            for (int i = 0; i < G; i++)
                upper(i, i);
            fetch(min(ch + kWarps, nch - 1));
#pragma unroll
            for (int i = 0; i < G; i++)
                add(lo[i], p_get(cl[i]), i < ds);
            if constexpr (kRef > G)
                if (wl > G)
                {
#pragma unroll
                    for (int i = 0; i < G; i++)
                        lower(i, G + i < ds, ref[G + i]);
#pragma unroll
                    for (int i = 0; i < G; i++)
                        add(lo[i], p_get(cl[i]), G + i < ds);
                }
            for (int s = kRef; s < wl; s++)
            {
                lower(0, s < ds, s < ds ? __ldg(d.lref + lo_idx(s, row, wl)) : 0u);
                add(lo[0], p_get(cl[0]), s < ds);
            }
            for (int u = 0;;)
            {
#pragma unroll
                for (int i = 0; i < G; i++)
                    add(up[i], p_get(cu[i]), u + i < ne);
                u += G;
                if (u >= wu)
                    break;
#pragma unroll
                for (int i = 0; i < G; i++)
                    if (u + i < wu)
                        upper(i, u + i);
            }
            q_set(li, q);
            const float3 pv = p_get(own0 + min(li, nrow - 1));
            const float part = warp_sum(li < nrow ? fdot(pv, q) : 0.f);
            v4 = grp == (k & 3) ? part : v4;
            if ((k & 3) == 3 || k == K - 1 || ch + kWarps >= nch)
            {
                int t;
                if (chunk_digit(v4, s_scale[0], t) && grp <= (k & 3))
                    dig += t;
            }
        }
        dig += __shfl_xor_sync(kFull, dig, 8);
        dig += __shfl_xor_sync(kFull, dig, 16);
        digits_add(s_dig[0], dig, grp == 0);
        bar_arrive(2, kAll);
        if (multi && w.rank == 0 && warp == kWarps - 1)
        {
            // the sum words of iteration it + 2 (see k_pcg_team)
            if (lane < 16)
                sync[blockIdx.x].words[(tag + 2u) & 3u][lane] = 0ull;
            __threadfence();
        }
        // (not on chip: kAhead rows' inverse diagonal blocks and r in flight)
        constexpr int kAhead = 6;
        float4 m0[kAhead];
        float2 m1[kAhead];
        float4 rr[kAhead];
        auto fetch_m = [&](int k) {
            const int row = w.row0 + min((k * kWarps + warp) * 32 + lane, nrow - 1);
            m0[k % kAhead] = __ldg(d.M0 + row);
            m1[k % kAhead] = __ldg(d.M1 + row);
            rr[k % kAhead] = d.r[row];
        };
        if constexpr (!kHold)
#pragma unroll
            for (int k = 0; k < kAhead; k++)
                fetch_m(k);
        bar_sync(3, kAll);
        if (*(volatile int *)&sh.stop)
            break;
        const float af = *(volatile float *)&sh.af;
        // ---- r -= alpha q, z = M^-1 r; r.z and r.r per chunk (dx += alpha p
        // once they are on their way)
        dig = 0;
        const int s2 = s_scale[1 + (grp >> 1)];
        float last = 0.f;
        int own = nrow - li0;
        asm volatile("" : "+r"(li0), "+r"(own));
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int li = k * kWorkers + li0, row = w.row0 + li;
            float part = 0.f;
            if (k * kWorkers - lane < own) // the warp's chunk has rows
            {
                float pr = 0.f, prr = 0.f;
                if (k * kWorkers < own)
                {
                    const float3 q = q_get(li);
                    float3 &rv = r[kHold ? k : 0];
                    if constexpr (!kHold)
                        rv = xyz(rr[k % kAhead]);
                    rv = make_float3(fmaf(-af, q.x, rv.x), fmaf(-af, q.y, rv.y),
                                     fmaf(-af, q.z, rv.z));
                    if constexpr (!kHold)
                        d.r[row] = f4(rv);
                    float M[6];
                    if constexpr (kHold)
                    {
                        const float2 m0 = sM[li], m1 = sM[rp + li], m2 = sM[2 * rp + li];
                        M[0] = m0.x;
                        M[1] = m0.y;
                        M[2] = m1.x;
                        M[3] = m1.y;
                        M[4] = m2.x;
                        M[5] = m2.y;
                    }
                    else
                    {
                        M[0] = m0[k % kAhead].x;
                        M[1] = m0[k % kAhead].y;
                        M[2] = m0[k % kAhead].z;
                        M[3] = m0[k % kAhead].w;
                        M[4] = m1[k % kAhead].x;
                        M[5] = m1[k % kAhead].y;
                    }
                    const float3 z = symv(M, rv);
                    q_set(li, z);
                    if (row < need0 || row >= need1)
                        st_row(d.z + row, z, tag + 1u);
                    pr = fdot(rv, z);
                    prr = fdot(rv, rv);
                }
                part = warp_sum2(pr, prr);
            }
            if constexpr (!kHold)
                if (k + kAhead < K)
                    fetch_m(k + kAhead);
            if (k & 1 || k == K - 1)
            {
                int t;
                if (chunk_digit(k & 1 ? (grp & 1 ? part : last) : part, s2, t) &&
                    (k & 1 || !(grp & 1)))
                    dig += t;
            }
            last = part;
        }
        dig += __shfl_xor_sync(kFull, dig, 8);
        digits_add(s_dig[1 + (grp >> 1)], dig, !(grp & 1));
        bar_arrive(4, kAll);
        if constexpr (kHold)
        {
#pragma unroll
            for (int k = 0; k < K; k++)
            {
                const int li = (k * kWarps + warp) * 32 + lane;
                if (li < nrow)
                {
                    const float3 p = p_get(own0 + li);
                    x[k] = make_float3(fmaf(af, p.x, x[k].x), fmaf(af, p.y, x[k].y),
                                       fmaf(af, p.z, x[k].z));
                }
            }
        }
        else
        {
            constexpr int kX = 4;
#pragma unroll 1
            for (int k0 = 0; k0 * kWarps + warp < nch; k0 += kX)
            {
                float4 v[kX];
#pragma unroll
                for (int k = 0; k < kX; k++)
                    v[k] = d.dx[w.row0 + min(((k0 + k) * kWarps + warp) * 32 + lane, nrow - 1)];
#pragma unroll
                for (int k = 0; k < kX; k++)
                {
                    const int li = ((k0 + k) * kWarps + warp) * 32 + lane;
                    if (li < nrow)
                    {
                        const float3 p = p_get(own0 + li);
                        d.dx[w.row0 + li] = make_float4(fmaf(af, p.x, v[k].x), fmaf(af, p.y, v[k].y),
                                                        fmaf(af, p.z, v[k].z), 0.f);
                    }
                }
            }
        }
        // the halo rows of the new z, while the sums are under way
#pragma unroll
        for (int u = 0; u < kHaloAhead; u++)
        {
            const int i = tid + u * kWorkers;
            if (i < nhalo)
                hz[u] = poll_row(d.z + w.halo0 + (i < own0 ? i : i + nrow), tag + 1u, sc.limit,
                                 &sh.err);
        }
        bar_sync(5, kAll);
        bf = *(volatile float *)&sh.bf;
    }
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int li = (k * kWarps + warp) * 32 + lane, row = w.row0 + li;
        if (li < nrow)
        {
            if constexpr (kHold)
            {
                d.dx[row] = f4(x[k]);
                d.r[row] = f4(r[k]);
            }
            if (*(volatile int *)&sh.stop == kLeave)
                d.z[row] = f4(p_get(own0 + li));
        }
    }
}

template <int K> const void *half_kernel(bool skew, bool cluster)
{
    return cluster ? (skew ? (const void *)k_pcg_half<K, true, true>
                           : (const void *)k_pcg_half<K, false, true>)
                   : (skew ? (const void *)k_pcg_half<K, true, false>
                           : (const void *)k_pcg_half<K, false, false>);
}

template <int K> const void *row_kernel(bool skew, bool cluster)
{
    constexpr int T = K < 1 ? 1 : K;
    return cluster ? (skew ? (const void *)k_pcg_team<T, team_reg_slots(K, true), true, true>
                           : (const void *)k_pcg_team<T, team_reg_slots(K, false), false, true>)
                   : (skew ? (const void *)k_pcg_team<T, team_reg_slots(K, true), true, false>
                           : (const void *)k_pcg_team<T, team_reg_slots(K, false), false, false>);
}

const void *team_kernel(int k, bool half, bool skew, bool cluster)
{
    if (half && k > 4)
        return k == kWideRows ? (const void *)k_pcg_wide<kWideRows>
                              : (const void *)k_pcg_wide<kWidestRows>;
    if (half)
        return k <= 2   ? half_kernel<2>(skew, cluster)
               : k == 3 ? half_kernel<3>(skew, cluster)
                        : half_kernel<4>(skew, cluster);
    return k == 0   ? row_kernel<0>(skew, cluster)
           : k == 1 ? row_kernel<1>(skew, cluster)
                    : row_kernel<2>(skew, cluster);
}

} // namespace cloth
