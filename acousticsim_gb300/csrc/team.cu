// Persistent block-Jacobi PCG with the matrix on chip (k_pcg_team).
//
// One cooperative launch runs every PCG iteration of every instance of a
// launch set.  A block owns a contiguous row range of one instance and keeps
// everything it iterates on next to its SM: the rows' 3x3 blocks and local
// column indices and p over the block's column range (halo) in shared memory,
// dx, r, z, p and the inverse diagonal block of its rows in registers.  Per
// iteration only boundary rows of z and two team sums cross the L2.
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
//     this GPU's narrow FP64 pipe); the FP64 scalars that the next fixed-point
//     scales and the result need are formed while the other warps compute.
// The arithmetic is that of the other PCG drivers, bit for bit.
//
// Measured (one GB300, us per PCG iteration over a whole step, before: the
// kernel that reads the matrix from L2 and forms the scalars in FP64): 20x20
// 11.8 -> 4.6, 97x61 11.8 -> 4.5, 193x255 12.4 -> 4.9, 128x128 with dihedral
// bending 14.1 -> 5.1.
#include "internal.h"
#include "pcg_math.cuh"

namespace cloth {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWorkers = kTeamWorkers;
constexpr int kWarps = kWorkers / 32;
constexpr int kHaloAhead = 2; // halo rows per thread polled before beta is known

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

// ---- team sums.  A sum is the exact total of fixed-point chunk sums, 96 bits
// and a sign, in units of 2^-s (fx_split).  Three words carry it: bits 0-31,
// 32-63 and the rest (biased), each with the number of blocks that added to
// it in its top byte, and the number of blocks that saw a chunk out of range
// (or Inf / NaN) in bits 40-55 of the second.
typedef __int128 i128;
constexpr int kCountShift = 56;
constexpr unsigned long long kOne = 1ull << kCountShift;
constexpr unsigned long long kBias = 1ull << 44;
constexpr unsigned long long kBad = 1ull << 40;

__device__ __forceinline__ i128 shl(long long v, int n)
{
    return i128((unsigned __int128)(i128(v)) << n);
}

struct Total
{
    long long H;          // bits 32.. (wraps where the sum is out of range)
    unsigned long long L; // bits 0-31
    int s;
    bool bad;
};

__device__ __forceinline__ double total_value(const Total &t) { return fx_value(t.H, t.L, t.s); }

// The block's chunk sums c[0 .. n) at scale s: 24-bit digits per lane, added
// over the warp by the integer reduce instructions.
__device__ __forceinline__ i128 fold(const float *c, int n, int s, bool &bad)
{
    unsigned d0 = 0, d1 = 0, d2 = 0, b = 0;
    int d3 = 0;
    for (int ch = threadIdx.x & 31; ch < n; ch += 32)
    {
        const float v = c[ch];
        long long h;
        unsigned long long l;
        fx_split(v, s, h, l);
        const int e = int((__float_as_uint(v) >> 23) & 0xffu);
        if (e == 255 || e - 127 + s >= 95)
            b = 1u;
        d0 += unsigned(l) & 0xffffffu;
        d1 += (unsigned(l) >> 24) | (unsigned(h) & 0xffffu) << 8;
        d2 += unsigned(h >> 16) & 0xffffffu;
        d3 += int(h >> 40);
    }
    d0 = __reduce_add_sync(kFull, d0);
    d1 = __reduce_add_sync(kFull, d1);
    d2 = __reduce_add_sync(kFull, d2);
    d3 = __reduce_add_sync(kFull, d3);
    bad = __any_sync(kFull, b) != 0;
    return i128(d0) + (i128(d1) << 24) + (i128(d2) << 48) + shl(d3, 72);
}

__device__ __forceinline__ Total make_total(i128 v, int s, bool bad)
{
    Total t;
    t.H = (long long)(v >> 32);
    t.L = (unsigned long long)v & 0xffffffffull;
    t.s = s;
    t.bad = bad || (v >> 95) != ((v >> 95) ? i128(-1) : i128(0));
    return t;
}

// Word k (0-2) of a block's contribution.
__device__ __forceinline__ unsigned long long sum_word(i128 v, bool bad, int k)
{
    if (k == 0)
        return kOne + ((unsigned long long)v & 0xffffffffull);
    if (k == 1)
        return kOne + ((unsigned long long)(v >> 32) & 0xffffffffull) + (bad ? kBad : 0ull);
    return kOne + kBias + (unsigned long long)(long long)(v >> 64);
}

// Team total of NQ quantities: lanes 0 .. 3 NQ - 1 add one word each and poll
// it until every block's arrival is in.  Returns false when the wait gave up.
template <int NQ>
__device__ __forceinline__ bool team_total(unsigned long long *words, const i128 (&v)[NQ],
                                           const bool (&bad)[NQ], const int (&s)[NQ], int nblk,
                                           const SpinCfg &sc, Total (&out)[NQ])
{
    const int lane = threadIdx.x & 31;
    unsigned long long w = 0ull;
    if (lane < 3 * NQ)
    {
        const int q = NQ == 1 ? 0 : lane / 3, k = lane - 3 * q;
        i128 vq = v[0];
        bool bq = bad[0];
        if (NQ > 1 && q)
        {
            vq = v[NQ - 1];
            bq = bad[NQ - 1];
        }
        w = sum_word(vq, bq, k);
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(words + lane), "l"(w)
                     : "memory");
    }
    const unsigned long long target = (unsigned long long)nblk + sc.extra;
    unsigned n = 0;
    for (;;)
    {
        bool here = true;
        if (lane < 3 * NQ)
        {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
                         : "=l"(w)
                         : "l"(words + lane)
                         : "memory");
            here = (w >> kCountShift) >= target;
        }
        if (__all_sync(kFull, here))
            break;
        if (++n > sc.limit)
            return false;
        if (n > 256)
            __nanosleep(32);
    }
    w &= kOne - 1;
#pragma unroll
    for (int q = 0; q < NQ; q++)
    {
        const unsigned long long w0 = __shfl_sync(kFull, w, 3 * q),
                                 w1 = __shfl_sync(kFull, w, 3 * q + 1),
                                 w2 = __shfl_sync(kFull, w, 3 * q + 2);
        const long long hi = (long long)(w2 - (unsigned long long)nblk * kBias);
        const i128 t = i128(w0) + (i128(w1 & (kBad - 1)) << 32) + shl(hi, 64);
        out[q] = make_total(t, s[q], (w1 >> 40) != 0);
    }
    return true;
}

// ---- scalars without the FP64 pipe.  |value| = (hi + lo 2^-24) 2^e with hi
// in [2^23, 2^24): its top 48 bits, the rest dropped (relative error 2^-47).
struct Top48
{
    unsigned hi, lo;
    int e;
    bool neg;
};
__device__ __forceinline__ Top48 top48(const Total &t)
{
    Top48 r;
    i128 v = shl(t.H, 32) + i128(t.L);
    r.neg = v < 0;
    if (r.neg)
        v = -v;
    const unsigned long long vh = (unsigned long long)(v >> 64), vl = (unsigned long long)v;
    const int nb = vh ? 128 - __clzll((long long)vh) : 64 - __clzll((long long)vl);
    const int sh = nb - 48;
    const unsigned long long m =
        sh > 0 ? (unsigned long long)((unsigned __int128)v >> sh) : vl << -sh;
    r.hi = unsigned(m >> 24);
    r.lo = unsigned(m) & 0xffffffu;
    r.e = nb - 24 - t.s;
    return r;
}
__device__ __forceinline__ Top48 top48(double d)
{
    Top48 r;
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const unsigned long long m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) >> 5;
    const int e = int((b >> 52) & 0x7ff);
    r.neg = (b >> 63) != 0;
    r.hi = e ? unsigned(m >> 24) : 0u;
    r.lo = unsigned(m) & 0xffffffu;
    r.e = e - 1023 - 23;
    return r;
}
// An order of the magnitudes that a relative difference above 2^-22 decides.
__device__ __forceinline__ long long key(const Top48 &t)
{
    return ((long long)t.e << 24) + (long long)(t.hi - 0x800000u);
}

// float(a / b), the quotient of the FP64 values rounded to FP64 and then to
// FP32, as the drivers that divide in FP64 form it.  The quotient is formed
// as q1 + q2 (FP32 quotient, then its remainder over b): within 2^-43 of the
// exact one.  Where that leaves the rounding to FP32 open (the sum lies
// within 2^-38 of a midpoint: one time in ~10,000), or the result is not in
// the normal range, *ok = false and the caller divides in FP64.
__device__ __forceinline__ float ratio(const Top48 &a, const Top48 &b, bool *ok)
{
    const float ah = float(a.hi), al = float(a.lo) * 0x1p-24f;
    const float bh = float(b.hi), bl = float(b.lo) * 0x1p-24f;
    const float rb = __fdividef(1.f, bh);
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

} // namespace

// K: chunks of 32 rows per warp (a block owns at most K * kTeamWorkers rows).
// SKEW: the launch set holds a dihedral-bending instance; skew block parts
// are kept and applied where an instance has them.
template <int K, bool SKEW>
__global__ void __launch_bounds__(kTeamThreads, 1)
    k_pcg_team(InstDesc *const *descs, const TeamBlock *work, TeamSync *sync, SpinCfg sc)
{
    constexpr int kAll = kTeamThreads;
    extern __shared__ float4 sm_dyn[];
    __shared__ InstDesc d;
    __shared__ float cpart[3][K * kWarps]; // FP32 sums of the 32-row chunks: p.q, r.z, r.r
    __shared__ float s_af, s_bf;
    __shared__ int s_stop, s_err, s_go;
    const TeamBlock w = work[blockIdx.x];
    if (threadIdx.x == 0)
    {
        d = *descs[w.inst];
        s_stop = 0;
        s_err = 0;
        s_go = __ldcg(&d.st->active);
    }
    __syncthreads();
    InstState *st = d.st;
    if (!s_go)
        return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrow = w.row1 - w.row0, nch = (nrow + 31) >> 5, rp = nch << 5;
    const int nh = w.halo1 - w.halo0, W = d.width;
    const bool skew = SKEW && d.Aw;
    // the test hook's extra arrivals make a team of one wait too
    const bool multi = w.nblk > 1 || sc.extra != 0u;
    const int it0 = __ldcg(&st->iter);
    // shared memory: p over the halo, then the rows' blocks by slot
    float4 *sp = sm_dyn;
    float4 *sA0 = sp + nh;
    float4 *sAw = sA0 + size_t(W) * rp;
    float2 *sA1 = reinterpret_cast<float2 *>(skew ? sAw + size_t(W) * rp : sAw);
    unsigned short *scol = reinterpret_cast<unsigned short *>(sA1 + size_t(W) * rp);

    if (warp == kWarps)
    {
        // ------------------------------------------------ control warp
        unsigned long long(*words)[16] = sync[blockIdx.x - w.rank].words;
        double rho = __ldcg(&st->rho), rr = __ldcg(&st->rr), pq = __ldcg(&st->pq);
        const double alpha0 = __ldcg(&st->alpha), beta0 = __ldcg(&st->beta);
        double rho_prev = 0.0, rho_alpha = 0.0, pq_alpha = 0.0; // what beta and alpha came from
        bool have_a = false, have_b = false;
        // the convergence threshold on ||r||^2
        const double bb = __ldcg(&st->bb);
        double thr = 0.0;
        if (d.rel_tol2 > 0.0)
            thr = d.rel_tol2 * bb;
        if (d.abs_tol2 > 0.0)
            thr = fmax(thr, d.abs_tol2);
        const bool tests = d.rel_tol2 > 0.0 || d.abs_tol2 > 0.0;
        const Top48 thr48 = top48(thr);
        const long long thr_key = key(thr48) + 2;
        Top48 rho48 = top48(rho);
        int s_pq = fx_scale(pq), s_rho = fx_scale(rho), s_rr = fx_scale(rr);
        int it = it0, status = 0;
        bar_sync(6, kAll); // the workers have filled shared memory
        for (;;)
        {
            unsigned long long *wd = words[it & 3];
            // ---- p.q and alpha
            bar_sync(2, kAll);
            int stop = *(volatile int *)&s_err ? 9 : 0;
            Total tq[1];
            if (!stop)
            {
                bool bad[1];
                i128 v[1];
                v[0] = fold(cpart[0], nch, s_pq, bad[0]);
                const int s[1] = {s_pq};
                if (!multi)
                    tq[0] = make_total(v[0], s_pq, bad[0]);
                else if (!team_total<1>(wd, v, bad, s, w.nblk, sc, tq))
                    stop = 9;
            }
            float af = 0.f;
            if (!stop)
            {
                if (tq[0].bad)
                    stop = 6;
                else if (tq[0].H == 0 && tq[0].L == 0ull)
                    stop = 7;
                else
                {
                    bool ok;
                    af = ratio(rho48, top48(tq[0]), &ok);
                    if (!ok)
                        af = float(rho / total_value(tq[0]));
                }
            }
            if (lane == 0)
            {
                s_af = af;
                s_stop = stop;
            }
            __syncwarp();
            bar_arrive(3, kAll);
            if (stop != 9)
                pq = total_value(tq[0]);
            if (stop)
            {
                status = stop;
                break;
            }
            rho_alpha = rho;
            pq_alpha = pq;
            have_a = true;
            const int s_pq_next = fx_scale(pq);
            // the buffer of iteration it + 2 was last polled in iteration
            // it - 2, which every block of the team has left: cleared here,
            // ordered before this block's next arrivals by the fence below
            if (w.rank == 0 && lane < 16)
                words[(it + 2) & 3][lane] = 0ull;
            const bool check = (it % d.check_every) == 0 || it + 1 >= d.max_iters;
            // ---- r.z, r.r and beta
            bar_sync(4, kAll);
            stop = *(volatile int *)&s_err ? 9 : 0;
            Total tz[2];
            if (!stop)
            {
                bool bad[2];
                i128 v[2];
                v[0] = fold(cpart[1], nch, s_rho, bad[0]);
                v[1] = fold(cpart[2], nch, s_rr, bad[1]);
                const int s[2] = {s_rho, s_rr};
                if (!multi)
                {
                    tz[0] = make_total(v[0], s_rho, bad[0]);
                    tz[1] = make_total(v[1], s_rr, bad[1]);
                }
                else if (!team_total<2>(wd + 4, v, bad, s, w.nblk, sc, tz))
                    stop = 9;
            }
            float bf = 0.f;
            Top48 new48 = rho48;
            bool tested = false;
            if (!stop)
            {
                new48 = top48(tz[0]);
                bool ok;
                bf = ratio(new48, rho48, &ok);
                if (!ok)
                    bf = rho == 0.0 ? 0.f : float(total_value(tz[0]) / rho);
                if (tz[0].bad || tz[1].bad)
                    stop = 6;
                else
                {
                    if (check && tests)
                    {
                        const bool zero = tz[1].H == 0 && tz[1].L == 0ull;
                        if (zero || thr48.hi == 0u || key(top48(tz[1])) <= thr_key)
                            tested = true;
                    }
                    if (tested)
                    {
                        const double v = total_value(tz[1]);
                        if ((d.rel_tol2 > 0.0 && v <= d.rel_tol2 * bb) ||
                            (d.abs_tol2 > 0.0 && v <= d.abs_tol2))
                            stop = 1;
                    }
                    if (!stop && it + 1 >= d.max_iters)
                        stop = 8;
                }
            }
            if (lane == 0)
            {
                s_bf = bf;
                s_stop = stop;
            }
            __syncwarp();
            bar_arrive(5, kAll);
            if (stop == 9)
            {
                status = 9;
                break;
            }
            it++;
            // FP64 scalars: the next scales, and the state that is reported
            rho_prev = rho;
            have_b = true;
            rho = total_value(tz[0]);
            rr = total_value(tz[1]);
            rho48 = new48;
            s_pq = s_pq_next;
            s_rho = fx_scale(rho);
            s_rr = fx_scale(rr);
            if (stop)
            {
                status = stop == 1 ? 0 : stop;
                break;
            }
            if (multi && w.rank == 0)
                __threadfence();
        }
        if (lane == 0)
        {
            if (status == 9)
                atomicExch(&st->bar_err, 1);
            if (w.rank == 0)
            {
                st->iter = it;
                st->status = status;
                st->rho = rho;
                st->rr = rr;
                st->pq = pq;
                st->alpha = have_a ? rho_alpha / pq_alpha : alpha0;
                st->beta = have_b ? (rho_prev == 0.0 ? 0.0 : rho / rho_prev) : beta0;
                st->active = 0;
            }
        }
        return;
    }

    // ---------------------------------------------------- workers
    const int own0 = w.row0 - w.halo0, nhalo = nh - nrow;
    float3 x[K], r[K], z[K], p[K];
    float M[K][6];
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
                load_sym(d.M0, d.M1, row, M[k]);
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
        // the rows' blocks: lower slots from their transposed position
        const int wl = d.width_lo, wu = d.width_up;
#pragma unroll 2
        for (int u = warp; u < W * nch; u += kWarps)
        {
            const int s = u / nch, li = (u - s * nch) * 32 + lane, row = w.row0 + li;
            if (li >= nrow)
                continue;
            const int info = d.rowinfo[row], ds = (info >> 8) & 255;
            if (s >= (info & 255))
                continue;
            uint32_t oa;
            int c;
            if (s < ds)
            {
                const uint32_t ref = d.lref[lo_idx(s, row, wl)];
                oa = lref_block(ref, wu);
                c = lref_col(ref);
            }
            else
            {
                oa = up_idx(s - ds, row, wu);
                c = d.colu[oa];
            }
            const size_t o = size_t(s) * rp + li;
            sA0[o] = d.A0[oa];
            sA1[o] = d.A1[oa];
            if (SKEW && skew)
            {
                float4 aw = d.Aw[oa];
                aw.w = s < ds ? -1.f : 1.f; // the transposed block's skew part changes sign
                sAw[o] = aw;
            }
            scol[o] = (unsigned short)(c - w.halo0);
        }
    }
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
                zz = u == 0 ? hz[0] : hz[1];
            else if (tag == unsigned(it0))
                zz = xyz(__ldcg(d.z + w.halo0 + j));
            else
                zz = poll_row(d.z + w.halo0 + j, tag, sc.limit, &s_err);
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
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int ch = warp + k * kWarps, li = ch * 32 + lane;
            q[k] = make_float3(0.f, 0.f, 0.f);
            if (ch < nch)
            {
                const float4 *a0 = sA0 + li;
                const float2 *a1 = sA1 + li;
                const unsigned short *cc = scol + li;
                // the next slots' blocks and columns are in flight while the
                // products of these form
#pragma unroll 4
                for (int s = 0; s < len[k]; s++)
                {
                    const size_t o = size_t(s) * rp;
                    const float4 u = a0[o];
                    const float2 v = a1[o];
                    const float3 pc = xyz(sp[cc[o]]);
                    const float A[6] = {u.x, u.y, u.z, u.w, v.x, v.y};
                    q[k] = q[k] + symv(A, pc);
                    if (SKEW && skew)
                    {
                        const float4 aw = sAw[o + li];
                        const float3 cw = skewv(aw, pc);
                        q[k] = aw.w < 0.f ? q[k] - cw : q[k] + cw;
                    }
                }
                const float part = warp_sum(li < nrow ? fdot(p[k], q[k]) : 0.f);
                if (lane == 0)
                    cpart[0][ch] = part;
            }
        }
        bar_arrive(2, kAll);
        bar_sync(3, kAll);
        if (*(volatile int *)&s_stop)
            break;
        const float af = *(volatile float *)&s_af;
        // ---- dx += alpha p, r -= alpha q, z = M^-1 r; r.z and r.r per chunk
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            const int ch = warp + k * kWarps, li = ch * 32 + lane;
            if (ch < nch)
            {
                float pr = 0.f, prr = 0.f;
                if (li < nrow)
                {
                    x[k] = make_float3(fmaf(af, p[k].x, x[k].x), fmaf(af, p[k].y, x[k].y),
                                       fmaf(af, p[k].z, x[k].z));
                    r[k] = make_float3(fmaf(-af, q[k].x, r[k].x), fmaf(-af, q[k].y, r[k].y),
                                       fmaf(-af, q[k].z, r[k].z));
                    z[k] = symv(M[k], r[k]);
                    if (multi)
                        st_row(d.z + w.row0 + li, z[k], tag + 1u);
                    pr = fdot(r[k], z[k]);
                    prr = fdot(r[k], r[k]);
                }
                pr = warp_sum(pr);
                prr = warp_sum(prr);
                if (lane == 0)
                {
                    cpart[1][ch] = pr;
                    cpart[2][ch] = prr;
                }
            }
        }
        bar_arrive(4, kAll);
        // the halo rows of the new z, while the sums are under way
#pragma unroll
        for (int u = 0; u < kHaloAhead; u++)
        {
            const int i = tid + u * kWorkers;
            if (i < nhalo)
                hz[u] = poll_row(d.z + w.halo0 + (i < own0 ? i : i + nrow), tag + 1u, sc.limit,
                                 &s_err);
        }
        bar_sync(5, kAll);
        if (*(volatile int *)&s_stop)
            break;
        bf = *(volatile float *)&s_bf;
    }
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int li = (warp + k * kWarps) * 32 + lane, row = w.row0 + li;
        if (li < nrow)
        {
            d.dx[row] = f4(x[k]);
            d.r[row] = f4(r[k]);
        }
    }
}

const void *team_kernel(int chunks_per_warp, bool skew)
{
    if (chunks_per_warp <= 1)
        return skew ? (const void *)k_pcg_team<1, true> : (const void *)k_pcg_team<1, false>;
    return skew ? (const void *)k_pcg_team<2, true> : (const void *)k_pcg_team<2, false>;
}

} // namespace cloth
