/*
 * txg_boxcar.cu -- boxcar matched filter over dedispersed series, the Boxcar::match /
 * Boxcar::run step (src/singlepulse/boxcar.cpp:158-296), fused with the S/N threshold and
 * candidate compaction that feed Cluster::run (cluster.cpp:89-112).
 *
 * One CTA per DM row.  The row is staged in shared memory, its mean/variance reduced
 * (FP32 runs combined in FP64), then the running sum of (x - mean) is formed in place by a
 * block scan (per-thread FP32 chunks, FP64 chunk offsets added as a float pair) and every
 * sample i keeps the
 * largest S = (c[i+wh] - c[i-wl]) * sqrt(1/(wn*var)) over the width ladder, later widths
 * winning ties (S >= best, best starting at 0) as in boxcar.cpp:253-262.  Rows with
 * var <= 0 yield zeros (boxcar.cpp:242).  The IQR statistics (boxcar.cpp:215-227) come from
 * an exact radix selection of the three order statistics.  Points with S > thre are appended
 * to the candidate list with a warp-aggregated atomic; dense mxS/mxwn are optional.  Where only
 * the points are wanted, upper bounds over blocks of samples decide which widths are scored.
 */
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdlib>

#include "txg_device.cuh"
#include "txg_internal.h"

namespace txg {

namespace {

constexpr int BX_THREADS = 512;
constexpr int BX_U = 4;  /* samples per thread per pass, tracked search: width parameters
                          * loaded once for all */
constexpr int BX_UF = 8; /* the same for the maximum-only search */
constexpr unsigned FULL = 0xffffffffu;
constexpr size_t BX_SMEM_MAX = 200 * 1024; /* longest row kept whole */
constexpr size_t BX_SMEM_TOP = 216 * 1024; /* with its bounds; + ~10 KB static stays under 227 KB */
constexpr int BX_RUN = 32; /* row statistics: FP32 runs per thread before each FP64 addition */

/* Block sums of a and b in every thread: an xor butterfly in each warp, then over the warps.  The
 * lower half of a warp reduces a and the upper half b, so each level is one addition for both
 * (the first exchanges the halves); the sums are those of two butterflies. */
__device__ __forceinline__ void block_sum2_d(double &a, double &b, double *red)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int NW = BX_THREADS / 32;
    double v = __dadd_rn(lane < 16 ? a : b, __shfl_xor_sync(FULL, lane < 16 ? b : a, 16));
#pragma unroll
    for (int off = 8; off >= 1; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(FULL, v, off));
    if ((lane & 15) == 0) red[(lane >> 4) * NW + w] = v;
    __syncthreads();
    if (threadIdx.x < 32) { /* lanes 0..15 the warps' a, 16..31 their b */
        static_assert(NW == 16, "a half warp holds one sum of every warp");
        v = red[lane];
#pragma unroll
        for (int off = 8; off >= 1; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(FULL, v, off));
        if ((lane & 15) == 0) red[lane] = v;
    }
    __syncthreads();
    a = red[0];
    b = red[16];
}

/* Statistics of row[0..n) in the fixed pattern: thread t takes samples t, t + BX_THREADS, ...
 * in FP32 runs of BX_RUN, each added to its FP64 sums, then the block sums.  The samples are
 * stored in c on the way when it is given (eight loads in flight). */
__device__ __forceinline__ void row_stats(const float *__restrict__ row, long n, float *c, double *red,
                                          float2 *mv, float &mean, float &var)
{
    double s1 = 0., s2 = 0.;
    long i = threadIdx.x;
    while (i < n) {
        float r1 = 0.f, r2 = 0.f;
        for (int h = 0; h < BX_RUN / 8 && i < n; h++) {
            if (i + 7 * BX_THREADS < n) {
                float v[8];
#pragma unroll
                for (int r = 0; r < 8; r++) v[r] = row[i + r * BX_THREADS];
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    if (c) c[i + r * BX_THREADS] = v[r];
                    r1 = __fadd_rn(r1, v[r]);
                    r2 = __fadd_rn(r2, __fmul_rn(v[r], v[r]));
                }
                i += 8 * BX_THREADS;
            } else {
                for (int r = 0; r < 8 && i < n; r++, i += BX_THREADS) {
                    const float v = row[i];
                    if (c) c[i] = v;
                    r1 = __fadd_rn(r1, v);
                    r2 = __fadd_rn(r2, __fmul_rn(v, v));
                }
            }
        }
        s1 = i < (long)(BX_RUN + 1) * BX_THREADS ? f2d(r1) : __dadd_rn(s1, f2d(r1)); /* first run: 0 + r */
        s2 = i < (long)(BX_RUN + 1) * BX_THREADS ? f2d(r2) : __dadd_rn(s2, f2d(r2));
    }
    block_sum2_d(s1, s2, red);
    if (threadIdx.x < 32) { /* two lanes: an FP64 division by the whole CTA costs microseconds */
        const double q = __ddiv_rn(threadIdx.x & 1 ? s2 : s1, (double)n);
        const double m = __shfl_sync(FULL, q, 0);
        if (threadIdx.x == 1) *mv = make_float2(__double2float_rn(m), __double2float_rn(__dsub_rn(q, __dmul_rn(m, m))));
    }
    __syncthreads();
    mean = mv->x;
    var = mv->y;
}

/* f(c[i]) for i = a .. b-1 in order, a the start of the thread's chunk of L shared-memory words:
 * lanes whose chunks start in the same bank (L and 32 have the factor g in common) run g steps
 * or fewer apart, so that a step's accesses hit different banks (16-sample chunks: 31 steps of
 * one wavefront instead of 16 of sixteen). */
template <typename F> __device__ __forceinline__ void chunk_walk(float *c, int a, int b, int L, F f)
{
    const int g = L & 31 ? L & -L : 32, skew = (threadIdx.x & 31) * g >> 5;
    const unsigned len = b - a;
    float *p = c + a - skew;
#pragma unroll 4
    for (int k = 0; k < L + g - 1; k++)
        if ((unsigned)(k - skew) < len) f(p[k]);
}

/* Exclusive FP64 scan of the BX_THREADS chunk totals by one warp. */
__device__ __forceinline__ void chunk_scan(double *chunk_off)
{
    const int tid = threadIdx.x;
    const int per = BX_THREADS / 32;
    double run = 0.;
    for (int q = 0; q < per; q++) run = __dadd_rn(run, chunk_off[tid * per + q]);
    double incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(FULL, incl, off);
        if (tid >= off) incl = __dadd_rn(incl, y);
    }
    /* exclusive prefix = the left neighbour's inclusive sum */
    const double left = __shfl_up_sync(FULL, incl, 1);
    double ex = tid == 0 ? 0. : left;
    for (int q = 0; q < per; q++) {
        const double v = chunk_off[tid * per + q];
        chunk_off[tid * per + q] = ex;
        ex = __dadd_rn(ex, v);
    }
}

/* Width w's parameters: wl, wh, end of the visited range, wn; and sqrt(1/(wn*var)). */
__device__ __forceinline__ void width_params(int wn, long n, float var, bool avx2_tail, int4 &p, float &tw)
{
    const int wl = wn / 2 + 1, wh = (wn - 1) / 2;
    tw = __double2float_rn(__dsqrt_rn(__ddiv_rn(1., (double)__fmul_rn((float)wn, var))));
    long hi = n - wh;
    if (avx2_tail) {
        const long len = n - wh - wl;
        const long nv = len >= 0 ? len / 8 : 0; /* C division truncates toward zero */
        hi = nv > 0 ? wl + 8 * nv : wl;
    }
    p = make_int4(wl, wh, (int)hi, wn);
}

/* float -> unsigned key with the same ordering */
__device__ __forceinline__ unsigned fkey(float f)
{
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(unsigned k)
{
    unsigned u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

/* The three order statistics of the IQR (ranks n/4, n/2, n-1-n/4, 0-based) of row[0..n), exactly,
 * by 4 rounds of 8-bit radix selection on the ordered keys.  The three share every round's pass
 * over the row (the first round's counts are the same for all), and a warp each finds its
 * digit, eight counts per lane and a scan: one thread walking the 256 counts of one statistic
 * at a time took most of the kernel (701 rows of 4995 samples: 119 us, so 38). */
struct Select3 {
    unsigned hist[3][256];
    unsigned pref[3], rank[3];
};
static_assert(sizeof(Select3) <= BX_THREADS * sizeof(double), "it lies where the chunk offsets go later");

__device__ __forceinline__ void select3(const float *row, long n, Select3 &s, float (&q)[3])
{
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < 3) {
        s.pref[tid] = 0;
        s.rank[tid] = (unsigned)(tid == 0 ? n / 4 : tid == 1 ? n / 2 : n - 1 - n / 4);
    }
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int b = tid; b < 3 * 256; b += BX_THREADS) (&s.hist[0][0])[b] = 0;
        __syncthreads();
        if (shift == 24) {
            for (long i = tid; i < n; i += BX_THREADS) atomicAdd(&s.hist[0][fkey(row[i]) >> 24], 1u);
        } else {
            const unsigned p0 = s.pref[0] >> (shift + 8), p1 = s.pref[1] >> (shift + 8), p2 = s.pref[2] >> (shift + 8);
            for (long i = tid; i < n; i += BX_THREADS) {
                const unsigned key = fkey(row[i]), m = key >> (shift + 8), d = (key >> shift) & 255u;
                if (m == p0) atomicAdd(&s.hist[0][d], 1u);
                if (m == p1) atomicAdd(&s.hist[1][d], 1u);
                if (m == p2) atomicAdd(&s.hist[2][d], 1u);
            }
        }
        __syncthreads();
        if (tid < 3 * 32) {
            const int t = tid >> 5;
            const unsigned *h = s.hist[shift == 24 ? 0 : t];
            unsigned cnt[8], tot = 0;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                cnt[u] = h[8 * lane + u];
                tot += cnt[u];
            }
            unsigned incl = tot;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned y = __shfl_up_sync(FULL, incl, off);
                if (lane >= off) incl += y;
            }
            const unsigned rk = s.rank[t];
            unsigned acc = incl - tot;
            __syncwarp();
            if (rk >= acc && rk < incl) {
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    if (rk >= acc && rk < acc + cnt[u]) {
                        s.pref[t] |= (unsigned)(8 * lane + u) << shift;
                        s.rank[t] = rk - acc;
                    }
                    acc += cnt[u];
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < 3; t++) q[t] = fkey_inv(s.pref[t]);
}

/* Median and IQR variance of row[0..n) (boxcar.cpp:215-227) by exact selection. */
__device__ __forceinline__ void row_stats_iqr(const float *row, long n, Select3 &sel, float2 *mv, float &mean, float &var)
{
    float q[3];
    select3(row, n, sel, q);
    mean = q[1];
    if (threadIdx.x == 0) {
        const double d = __ddiv_rn((double)__fsub_rn(q[2], q[0]), 1.349);
        mv->y = __double2float_rn(__dmul_rn(d, d));
    }
    __syncthreads();
    var = mv->y;
}

/* Best S over the width ladder for U samples i = i0 + u*BX_THREADS, with its width (later
 * widths win ties).  CHECK selects the per-width range test (needed near the row ends); AVX2
 * reproduces the unordered-compare blend of the -mavx2 build. */
template <bool CHECK, bool AVX2, int U>
__device__ __forceinline__ void widths_pass(const float *__restrict__ c, int coff, int i0, int iend,
                                            int nw, const int4 *__restrict__ wpar,
                                            const float *__restrict__ temp_w, float *best, int *bw)
{
    /* c[j - coff] holds the running sum at sample j; samples at or past iend are skipped */
    for (int w = 0; w < nw; w++) {
        const int4 p = wpar[w];
        const float tw = temp_w[w];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * BX_THREADS;
            if (!CHECK || (i >= p.x && i < p.z && i < iend)) {
                const float S = __fmul_rn(__fsub_rn(c[i - coff + p.y], c[i - coff - p.x]), tw);
                if (S >= best[u]) {
                    best[u] = S;
                    bw[u] = p.w;
                } else if (AVX2 && !(S < best[u])) {
                    best[u] = 0.f;
                    bw[u] = 0;
                }
            }
        }
    }
}

/* The same search keeping only the best S (S is never NaN: var > 0 and the sums are finite,
 * so the maximum is that of the tracked search). */
template <bool CHECK, int U>
__device__ __forceinline__ void widths_max(const float *__restrict__ c, int coff, int i0, int iend,
                                           int nw, const int4 *__restrict__ wpar,
                                           const float *__restrict__ temp_w, float *best)
{
    for (int w = 0; w < nw; w++) {
        const int4 p = wpar[w];
        const float tw = temp_w[w];
        const int hz = min(p.z, iend);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + u * BX_THREADS;
            if (!CHECK || (i >= p.x && i < hz)) {
                const float S = __fmul_rn(__fsub_rn(c[i - coff + p.y], c[i - coff - p.x]), tw);
                best[u] = fmaxf(best[u], S);
            }
        }
    }
}

/* The width of a point above the threshold, for the searches that keep only its best S: the
 * tracked search keeps the last width whose S reaches the final best (>= with best starting at
 * 0), the largest w with S_w == best, or width 0 when none equals it (best stayed 0).  The warp
 * finds it for each hit in turn, one width per lane, with the same arithmetic as the search. */
__device__ __forceinline__ int hit_width(const float *__restrict__ c, int coff, int i, int iend, bool hit, float best,
                                         int nw, const int4 *__restrict__ wpar, const float *__restrict__ temp_w)
{
    const int lane = threadIdx.x & 31;
    int bw = 0;
    unsigned hm = __ballot_sync(FULL, hit);
    while (hm) {
        const int src = __ffs(hm) - 1;
        hm &= hm - 1;
        const int is = __shfl_sync(FULL, i, src);
        const float bs = __shfl_sync(FULL, best, src);
        int wf = -1;
        for (int w0 = 0; w0 < nw; w0 += 32) {
            const int w = w0 + lane;
            bool eq = false;
            if (w < nw) {
                const int4 p = wpar[w];
                if (is >= p.x && is < min(p.z, iend))
                    eq = __fmul_rn(__fsub_rn(c[is - coff + p.y], c[is - coff - p.x]), temp_w[w]) == bs;
            }
            const unsigned e = __ballot_sync(FULL, eq);
            if (e) wf = w0 + 31 - __clz(e);
        }
        if (lane == src) bw = wf >= 0 ? wpar[wf].w : 0;
    }
    return bw;
}

/* Appends the warp's hits to the candidate list, one atomic per warp. */
__device__ __forceinline__ void append_hits(bool hit, long k, int i, int bw, float best, txg_cand *__restrict__ cand,
                                            int *__restrict__ ncand, long cap)
{
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(FULL, hit);
    if (!m) return;
    int basei = 0;
    if (lane == __ffs(m) - 1) basei = atomicAdd(ncand, __popc(m));
    basei = __shfl_sync(FULL, basei, __ffs(m) - 1);
    if (hit) {
        const long slot = basei + __popc(m & ((1u << lane) - 1u));
        if (slot < cap) cand[slot] = txg_cand{(int32_t)k, (int32_t)i, bw, best};
    }
}

/* Width search over samples [s_lo, iend) of row k, the running sum at c[j - coff]; every
 * width is in range for samples in [lo_all, hi_all).  Points with S > thre are appended to
 * the candidate list (warp-aggregated atomic), dense mxS/mxwn written when given.  TRACK keeps
 * the best width at every step (the dense output and the AVX2 blend need it); otherwise the
 * pass keeps only the maximum S and the width of each point above the threshold is found
 * afterwards with the same arithmetic. */
template <bool AVX2, bool TRACK>
__device__ __forceinline__ void search_row(const float *__restrict__ c, int coff, int s_lo, int iend,
                                           int lo_all, int hi_all, int nw, const int4 *__restrict__ wpar,
                                           const float *__restrict__ temp_w, bool active, float thre,
                                           long k, long n, txg_cand *__restrict__ cand,
                                           int *__restrict__ ncand, long cap, float *__restrict__ mxS,
                                           int32_t *__restrict__ mxwn)
{
    constexpr int U = TRACK ? BX_U : BX_UF;
    const int tid = threadIdx.x;
    for (int base = s_lo; base < iend; base += BX_THREADS * U) {
        float best[U];
        int bw[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            best[u] = 0.f;
            bw[u] = 0;
        }
        if (active) {
            const int i0 = base + tid;
            const bool inner = base >= lo_all && base + BX_THREADS * U <= hi_all && base + BX_THREADS * U <= iend;
            if (TRACK) {
                if (inner)
                    widths_pass<false, AVX2, U>(c, coff, i0, iend, nw, wpar, temp_w, best, bw);
                else
                    widths_pass<true, AVX2, U>(c, coff, i0, iend, nw, wpar, temp_w, best, bw);
            } else {
                if (inner)
                    widths_max<false, U>(c, coff, i0, iend, nw, wpar, temp_w, best);
                else
                    widths_max<true, U>(c, coff, i0, iend, nw, wpar, temp_w, best);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = base + tid + u * BX_THREADS;
            if (TRACK && i < iend && mxS) {
                mxS[k * n + i] = best[u];
                mxwn[k * n + i] = bw[u];
            }
            const bool hit = i < iend && best[u] > thre;
            if (!TRACK) bw[u] = hit_width(c, coff, i, iend, hit, best[u], nw, wpar, temp_w);
            append_hits(hit, k, i, bw[u], best[u], cand, ncand, cap);
        }
    }
}

/* ---- search that skips widths by upper bounds ---------------------------------------------- */
/* Only points with S > thre are wanted, and in noise almost no (sample, width) pair comes near
 * it, so scoring all of them (two shared-memory loads and three operations a pair) is mostly
 * wasted: 2000 noise rows of 13156 samples and 30 widths at threshold 7 took 322 us that way and
 * take 96 so, of 3289 samples and 23 widths 115 and 62, 600 of 62496 and 25 358 and 133.  For a block of BB
 * samples and a width two upper bounds on S are cheap:
 *   - the largest running sum where the samples' upper ends lie minus the smallest where their
 *     lower ends lie, times the width's factor (subtraction and product are monotone, so the
 *     bound holds for the rounded S), good for wide boxes;
 *   - for boxes of BB samples or fewer, n16 * m16 + n4 * m4 + n1 * m1, m_k being the largest
 *     k-sample difference of the running sum in the block and its neighbours and
 *     n16, n4, n1 the box's length in sixteens, fours and ones; BX_SLACK covers the roundings.
 * In noise 0.15 of a block's 30 widths pass both; with BB 64 it is 0.02, but a row has twice the
 * blocks (143 us).  The search then takes less than the row's statistics and running sum, which
 * the FP64 unit bounds (a warp instruction holds a scheduler's for about 60 cycles).
 * A width is scored, with the plain search's arithmetic, only where neither bound rules it out;
 * a point above the threshold keeps its maximum and width, since every skipped S is <= thre. */
constexpr int BB = 128;
constexpr float BX_SLACK = 1.000002f; /* > (1 + 2^-24)^8: S, the m_k and the bound's own sums */

__host__ __device__ constexpr int bound_blocks(long nc) { return (int)((nc + BB - 1) / BB); }
constexpr int BX_BOUND_FLOATS = 6; /* per block: hi, lo and a float4 of the neighbourhood's m_k */

__device__ __forceinline__ int okey(float f)
{
    const int u = __float_as_int(f);
    return u ^ ((u >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float okey_inv(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
__device__ __forceinline__ float max_nan(float a, float b) /* a NaN if either is */
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

/* hi[], lo[] (as ordered keys, so that a NaN counts as the largest and is never ruled out) and
 * nbh[] = (m1, m4, m16 over the block and its neighbours, not below 0) of all blocks of
 * c[0..nc); ends with a barrier.  Out-of-range partners are clamped into the row: a shorter
 * difference there only loosens the bound. */
__device__ __forceinline__ void block_bounds(const float *__restrict__ c, int nc, int *__restrict__ hi,
                                             int *__restrict__ lo, float4 *__restrict__ nbh)
{
    const int lane = threadIdx.x & 31, nb = bound_blocks(nc);
    for (int b = threadIdx.x >> 5; b < nb; b += BX_THREADS / 32) {
        float h = -INFINITY, l = INFINITY;
        int k1 = 0, k4 = 0, k16 = 0;
        /* positive floats order as their bits; a negative one is below 0 as an integer too */
        auto take = [&](float v, float v1, float v4, float v16) {
            h = max_nan(h, v);
            l = fminf(l, v);
            k1 = max(k1, __float_as_int(__fsub_rn(v, v1)));
            k4 = max(k4, __float_as_int(__fsub_rn(v, v4)));
            k16 = max(k16, __float_as_int(__fsub_rn(v, v16)));
        };
        if (b > 0 && (b + 1) * BB <= nc) {
            const float *p = c + b * BB + lane;
#pragma unroll
            for (int q = 0; q < BB / 32; q++) take(p[q * 32], p[q * 32 - 1], p[q * 32 - 4], p[q * 32 - 16]);
        } else {
            for (int q = 0; q < BB / 32; q++) {
                const int i = min(b * BB + q * 32 + lane, nc - 1);
                take(c[i], c[max(i - 1, 0)], c[max(i - 4, 0)], c[max(i - 16, 0)]);
            }
        }
        const int kh = __reduce_max_sync(FULL, okey(h)), kl = __reduce_min_sync(FULL, okey(l));
        k1 = __reduce_max_sync(FULL, k1);
        k4 = __reduce_max_sync(FULL, k4);
        k16 = __reduce_max_sync(FULL, k16);
        if (lane == 0) {
            hi[b] = kh;
            lo[b] = kl;
            nbh[b] = make_float4(__int_as_float(k1), __int_as_float(k4), __int_as_float(k16), 0.f);
        }
    }
    __syncthreads();
    /* the neighbourhood's maxima, in place: every thread reads before any writes */
    for (int b0 = 0; b0 < nb; b0 += BX_THREADS) {
        const int b = b0 + threadIdx.x;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (b < nb) {
            const float4 l = nbh[max(b - 1, 0)], m = nbh[b], r = nbh[min(b + 1, nb - 1)];
            /* as integers, so that a NaN (above infinity) stays the largest; the left
             * neighbour of a pass's first block may hold its own neighbourhood's already */
            auto mx = [](float x, float y, float z) {
                return __int_as_float(max(max(__float_as_int(x), __float_as_int(y)), __float_as_int(z)));
            };
            v = make_float4(mx(l.x, m.x, r.x), mx(l.y, m.y, r.y), mx(l.z, m.z, r.z), 0.f);
        }
        __syncthreads();
        if (b < nb) nbh[b] = v;
        __syncthreads();
    }
}

/* The maximum-only search of search_row over the samples [s_lo, iend) of row k, c[j - coff] the
 * running sum at sample j for j - coff in [0, nc), by one warp per block of BB samples. */
__device__ __forceinline__ void search_bounded(const float *__restrict__ c, int coff, int nc, int s_lo, int iend,
                                               int nw, const int4 *__restrict__ wpar,
                                               const float *__restrict__ temp_w, const int *__restrict__ hi,
                                               const int *__restrict__ lo, const float4 *__restrict__ nbh,
                                               float thre, long k, txg_cand *__restrict__ cand,
                                               int *__restrict__ ncand, long cap)
{
    constexpr int Q = BB / 32;
    const int lane = threadIdx.x & 31, nb = bound_blocks(nc);
    const int b1 = (iend - 1 - coff) / BB;
    int4 p = make_int4(0, 0, 0, 0); /* the lane's width; up to 32 of them stay in registers */
    float tw = 0.f;
    if (lane < nw) {
        p = wpar[lane];
        tw = temp_w[lane];
    }
    for (int b = (s_lo - coff) / BB + (threadIdx.x >> 5); b <= b1; b += BX_THREADS / 32) {
        const int base = b * BB; /* local index of the block's first sample */
        const float4 m = nbh[b];
        float best[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) best[q] = 0.f;
        for (int w0 = 0; w0 < nw; w0 += 32) {
            bool score = false;
            if (w0 + lane < nw) { /* a width per lane */
                if (w0 > 0 || nw > 32) {
                    p = wpar[w0 + lane];
                    tw = temp_w[w0 + lane];
                }
                const int u0 = (base + p.y) / BB, u1 = min((base + BB - 1 + p.y) / BB, nb - 1);
                const int v0 = max(base - p.x, 0) / BB, v1 = base + BB - 1 - p.x;
                if (p.w < 1) {
                    score = true; /* no box: nothing is known about it */
                } else if (u0 < nb && v1 >= 0) {
                    const float S = __fmul_rn(
                        __fsub_rn(okey_inv(max(hi[u0], hi[u1])), okey_inv(min(lo[v0], lo[v1 / BB]))), tw);
                    const float B = (float)(p.w >> 4) * m.z + (float)((p.w >> 2) & 3) * m.y + (float)(p.w & 3) * m.x;
                    score = !(S <= thre) && !(p.w <= BB && B * tw * BX_SLACK <= thre);
                }
            }
            unsigned todo = __ballot_sync(FULL, score);
            while (todo) {
                const int w = w0 + __ffs(todo) - 1;
                todo &= todo - 1;
                const int4 pw = wpar[w];
                const float tww = temp_w[w];
                const int hz = min(pw.z, iend);
#pragma unroll
                for (int q = 0; q < Q; q++) {
                    const int i = coff + base + q * 32 + lane;
                    if (i >= pw.x && i >= s_lo && i < hz)
                        best[q] = fmaxf(best[q], __fmul_rn(__fsub_rn(c[i - coff + pw.y], c[i - coff - pw.x]), tww));
                }
            }
        }
        float top = best[0];
#pragma unroll
        for (int q = 1; q < Q; q++) top = fmaxf(top, best[q]);
        if (!__any_sync(FULL, top > thre)) continue;
#pragma unroll 1
        for (int q = 0; q < Q; q++) {
            const int i = coff + base + q * 32 + lane;
            const bool hit = best[q] > thre;
            const int bw = hit_width(c, coff, i, iend, hit, best[q], nw, wpar, temp_w);
            append_hits(hit, k, i, bw, best[q], cand, ncand, cap);
        }
    }
}

/* Below this threshold noise defeats the bounds and the plain search is as fast (2000 noise rows
 * of 13156 samples and 30 widths, bounded / plain: 211 / 321 us at 4, 328 / 415 at 3; of 3289 and
 * 23: 82 / 100 at 4, 103 / 102 at 3.5, 124 / 112 at 3). */
constexpr float BX_BOUND_THRE = 4.f;

/* Samples where every width is in range: [lo, hi). */
__device__ __forceinline__ void common_range(int nw, const int4 *wpar, int n, int &lo, int &hi)
{
    lo = 0;
    hi = n;
    for (int w = 0; w < nw; w++) {
        lo = max(lo, wpar[w].x);
        hi = min(hi, wpar[w].z);
    }
}

template <bool AVX2, bool TRACK, bool BOUND>
__global__ void __launch_bounds__(BX_THREADS, BOUND ? 3 : 4)
k_boxcar(const float *__restrict__ tim, long ldt, long n, const int32_t *__restrict__ vwn,
         int nw, int iqr, float thre, txg_cand *__restrict__ cand,
         int *__restrict__ ncand, long cap, float *__restrict__ mxS, int32_t *__restrict__ mxwn)
{
    chain_wait();
    extern __shared__ __align__(16) float c[];
    __shared__ double red[2 * BX_THREADS / 32];
    __shared__ float2 mv;
    __shared__ double chunk_off[BX_THREADS];
    __shared__ float temp_w[256];
    __shared__ int4 wpar[256]; /* wl, wh, end of the visited range, wn */
    __shared__ int lo_all, hi_all; /* samples where every width is in range */
    const long k = blockIdx.x;
    const int tid = threadIdx.x;
    const float *row = tim + k * ldt;

    float mean, var;
    if (!iqr) {
        row_stats(row, n, c, red, &mv, mean, var);
    } else {
        for (long i = tid; i < n; i += BX_THREADS) c[i] = row[i];
        __syncthreads();
        row_stats_iqr(c, n, *reinterpret_cast<Select3 *>(chunk_off), &mv, mean, var);
    }

    /* running sum of (x - mean): thread t owns the contiguous chunk [t*L, (t+1)*L) */
    const int L = (int)((n + BX_THREADS - 1) / BX_THREADS);
    const int a = min((long)tid * L, n), b = min((long)a + L, n);
    float loc = 0.f;
    chunk_walk(c, a, b, L, [&](float &v) { loc = __fadd_rn(loc, __fsub_rn(v, mean)); });
    chunk_off[tid] = f2d(loc);
    __syncthreads();
    if (tid < 32) { /* the scan, and beside it the widths' parameters */
        chunk_scan(chunk_off);
    } else {
        for (int w = tid - 32; w < nw; w += BX_THREADS - 32) width_params(vwn[w], n, var, AVX2, wpar[w], temp_w[w]);
    }
    __syncthreads();
    {
        /* the chunk's FP64 offset as a float pair: c[i] = (hi + run) + lo, two FP32 adds per
         * sample (the FP64 pipe is a small fraction of the FP32 one on this part) */
        const double off = chunk_off[tid];
        const float oh = __double2float_rn(off), ol = __double2float_rn(__dsub_rn(off, f2d(oh)));
        float run = 0.f;
        chunk_walk(c, a, b, L, [&](float &v) {
            run = __fadd_rn(run, __fsub_rn(v, mean));
            v = __fadd_rn(__fadd_rn(oh, run), ol);
        });
    }
    if (!BOUND && tid == 0) common_range(nw, wpar, (int)n, lo_all, hi_all);
    __syncthreads();
    if (BOUND) {
        if (!(var > 0.f)) return; /* no S: thre >= 0 */
        const int nb = bound_blocks(n);
        float4 *nbh = reinterpret_cast<float4 *>(c + (n + 3) / 4 * 4);
        int *hi = reinterpret_cast<int *>(nbh + nb), *lo = hi + nb;
        block_bounds(c, (int)n, hi, lo, nbh);
        search_bounded(c, 0, (int)n, 0, (int)n, nw, wpar, temp_w, hi, lo, nbh, thre, k, cand, ncand, cap);
    } else {
        search_row<AVX2, TRACK>(c, 0, 0, (int)n, lo_all, hi_all, nw, wpar, temp_w, var > 0.f, thre, k, n, cand,
                                ncand, cap, mxS, mxwn);
    }
}

/* ---- rows longer than one CTA's shared memory ------------------------------------------ */
/* The single-CTA kernel's arithmetic depends only on n: statistics by the fixed run pattern,
 * and the running sum over BX_THREADS chunks of L = ceil(n/BX_THREADS) samples (FP32 inside a
 * chunk, FP64 chunk offsets added as a float pair).  k_boxcar_prep computes, per row, the same
 * statistics and chunk offsets from global memory; k_boxcar_seg rebuilds the running sum of a
 * segment of chunks plus a halo of the widest boxcar and runs the same width passes: results
 * are identical to k_boxcar's.  scratch row k: [0, BX_THREADS) chunk offsets, [BX_THREADS] mean and var. */
constexpr int SEG_CHUNKS = 32; /* chunks per segment CTA */

/* Shared memory: per warp `pc` chunks of the row (a warp's chunks are consecutive, so a pass's
 * load is one contiguous, coalesced piece; reading a chunk per thread straight from memory
 * touched 32 lines per load).  pc divides 32: 8, or fewer where 16 warps' pieces would not fit. */
static int prep_chunks(long L)
{
    int pc = 8;
    while (pc > 1 && (size_t)(BX_THREADS / 32) * pc * L * sizeof(float) > BX_SMEM_TOP) pc /= 2;
    return pc;
}

__global__ void __launch_bounds__(BX_THREADS)
k_boxcar_prep(const float *__restrict__ tim, long ldt, long n, int iqr, int pc, double *__restrict__ scratch)
{
    chain_wait();
    extern __shared__ __align__(16) float c[];
    __shared__ double red[2 * BX_THREADS / 32];
    __shared__ float2 mv;
    __shared__ double chunk_off[BX_THREADS];
    const long k = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const float *row = tim + k * ldt;
    float mean, var;
    if (!iqr) {
        row_stats(row, n, nullptr, red, &mv, mean, var);
    } else {
        row_stats_iqr(row, n, *reinterpret_cast<Select3 *>(chunk_off), &mv, mean, var);
    }
    const long L = (n + BX_THREADS - 1) / BX_THREADS;
    float *piece = c + (size_t)wp * pc * L;
    for (int q0 = 0; q0 < 32; q0 += pc) { /* the warp's 32 chunks */
        const long p0 = min((wp * 32L + q0) * L, n), p1 = min(p0 + pc * L, n);
        __syncwarp();
#pragma unroll 8
        for (long i = p0 + lane; i < p1; i += 32) piece[i - p0] = row[i];
        __syncwarp();
        if (lane < pc) {
            const long a = min(p0 + lane * L, p1), b = min(a + L, p1);
            float loc = 0.f;
#pragma unroll 4
            for (long i = a; i < b; i++) loc = __fadd_rn(loc, __fsub_rn(piece[i - p0], mean));
            chunk_off[wp * 32 + q0 + lane] = f2d(loc);
        }
    }
    __syncthreads();
    if (tid < 32) chunk_scan(chunk_off);
    __syncthreads();
    double *out = scratch + k * (BX_THREADS + 1);
    out[tid] = chunk_off[tid];
    if (tid == 0) {
        float *o = reinterpret_cast<float *>(out + BX_THREADS);
        o[0] = mean;
        o[1] = var;
    }
}

template <bool AVX2, bool TRACK, bool BOUND>
__global__ void __launch_bounds__(BX_THREADS)
k_boxcar_seg(const float *__restrict__ tim, long ldt, long n, const int32_t *__restrict__ vwn,
             int nw, float thre, const double *__restrict__ scratch, txg_cand *__restrict__ cand,
             int *__restrict__ ncand, long cap, float *__restrict__ mxS, int32_t *__restrict__ mxwn)
{
    chain_wait();
    extern __shared__ __align__(16) float c[];
    __shared__ float temp_w[256];
    __shared__ int4 wpar[256];
    __shared__ int lo_all, hi_all, wlmax_sh, whmax_sh;
    const long k = blockIdx.x;
    const int tid = threadIdx.x;
    const float *row = tim + k * ldt;
    const double *sc = scratch + k * (BX_THREADS + 1);
    const float mean = reinterpret_cast<const float *>(sc + BX_THREADS)[0];
    const float var = reinterpret_cast<const float *>(sc + BX_THREADS)[1];
    const long L = (n + BX_THREADS - 1) / BX_THREADS;
    const long s_lo = (long)blockIdx.y * SEG_CHUNKS * L;
    if (s_lo >= n) return;
    if (BOUND && !(var > 0.f)) return; /* no S: thre >= 0 */
    const long s_hi = min(n, s_lo + (long)SEG_CHUNKS * L);

    if (tid == 0) wlmax_sh = whmax_sh = 0;
    __syncthreads();
    for (int w = tid; w < nw; w += BX_THREADS) {
        width_params(vwn[w], n, var, AVX2, wpar[w], temp_w[w]);
        atomicMax(&wlmax_sh, wpar[w].x);
        atomicMax(&whmax_sh, wpar[w].y);
    }
    __syncthreads();
    if (!BOUND && tid == 0) common_range(nw, wpar, (int)n, lo_all, hi_all);
    /* running sum over the segment and its halo, rebuilt chunk by chunk from the offsets: the
     * samples of the chunks are brought in first, coalesced (f_lo: first sample of the first
     * chunk), then summed in place */
    const long h_lo = max(0L, s_lo - wlmax_sh), h_hi = min(n, s_hi + whmax_sh);
    const long ch0 = h_lo / L, f_lo = ch0 * L;
#pragma unroll 4
    for (long i = f_lo + tid; i < h_hi; i += BX_THREADS) c[i - f_lo] = row[i];
    __syncthreads();
    for (long ch = ch0 + tid; ch * L < h_hi; ch += BX_THREADS) {
        const long a = ch * L, b = min(a + L, h_hi);
        const double off = sc[ch];
        const float oh = __double2float_rn(off), ol = __double2float_rn(__dsub_rn(off, (double)oh));
        float run = 0.f;
#pragma unroll 4
        for (long i = a; i < b; i++) {
            run = __fadd_rn(run, __fsub_rn(c[i - f_lo], mean));
            c[i - f_lo] = __fadd_rn(__fadd_rn(oh, run), ol);
        }
    }
    __syncthreads();
    if (BOUND) {
        const int nc = (int)(h_hi - f_lo), nb = bound_blocks(nc);
        float4 *nbh = reinterpret_cast<float4 *>(c + (nc + 3) / 4 * 4);
        int *hi = reinterpret_cast<int *>(nbh + nb), *lo = hi + nb;
        block_bounds(c, nc, hi, lo, nbh);
        search_bounded(c, (int)f_lo, nc, (int)s_lo, (int)s_hi, nw, wpar, temp_w, hi, lo, nbh, thre, k, cand, ncand, cap);
    } else {
        search_row<AVX2, TRACK>(c, (int)f_lo, (int)s_lo, (int)s_hi, lo_all, hi_all, nw, wpar, temp_w, var > 0.f,
                                thre, k, n, cand, ncand, cap, mxS, mxwn);
    }
}

} // namespace

size_t boxcar_max_samples() { return (BX_SMEM_MAX) / sizeof(float); }

size_t boxcar_scratch_doubles(long ndm) { return (size_t)ndm * (BX_THREADS + 1); }

/* Shared memory for nc samples: the running sum and, for the bounded search, its blocks' bounds. */
static size_t boxcar_smem(long nc, bool bound)
{
    return ((size_t)(nc + 3) / 4 * 4 + (bound ? (size_t)BX_BOUND_FLOATS * bound_blocks(nc) : 0)) * sizeof(float);
}

/* A segment's samples: its chunks, the halo of the widest boxcar and the rest of the chunk that
 * the halo starts in. */
static long seg_samples(long n, int maxwn)
{
    const long L = (n + BX_THREADS - 1) / BX_THREADS;
    return (SEG_CHUNKS + 1) * L + maxwn + 2;
}

bool boxcar_supported(long n, int maxwn, int nw)
{
    if (n <= 0 || n >= (1L << 31) || nw > 256) return false;
    if ((size_t)n <= boxcar_max_samples()) return true;
    const long L = (n + BX_THREADS - 1) / BX_THREADS;
    const long seg = (long)SEG_CHUNKS * L;
    return (size_t)(seg + maxwn + 2) * sizeof(float) <= BX_SMEM_MAX && (n + seg - 1) / seg <= 65535;
}

static bool force_segmented()
{
    const char *e = getenv("TXG_BOXCAR_SEGMENTED");
    return e && e[0] == '1';
}

int launch_boxcar(const float *tim, long ldt, long ndm, long n, const int32_t *vwn, int nw,
                  int maxwn, int iqr, int avx2_tail, float thre, txg_cand *cand, int *ncand,
                  long cap, float *mxS, int32_t *mxwn, double *scratch, int *err, cudaStream_t st)
{
    (void)err;
    if (n <= 0 || ndm <= 0) return TXG_OK;
    if (nw > 256 || n >= (1L << 31)) return TXG_ERR_UNSUPPORTED;
    /* rows so long that the bounds do not fit beside them search plainly */
    const bool want = !avx2_tail && !mxS && thre >= BX_BOUND_THRE;
    if ((size_t)n <= boxcar_max_samples() && !(force_segmented() && scratch)) {
        const bool bound = want && boxcar_smem(n, true) <= BX_SMEM_TOP;
        const size_t smem = boxcar_smem(n, bound);
#define TXG_BX(A, T, B)                                                                               \
    do {                                                                                              \
        cudaFuncSetAttribute(k_boxcar<A, T, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BX_SMEM_TOP); \
        launch_chained(k_boxcar<A, T, B>, (unsigned)ndm, BX_THREADS, smem, st, tim, ldt, n, vwn, nw, iqr, thre, \
                       cand, ncand, cap, mxS, mxwn);                                                  \
    } while (0)
        if (avx2_tail)
            TXG_BX(true, true, false);
        else if (mxS)
            TXG_BX(false, true, false);
        else if (bound)
            TXG_BX(false, false, true);
        else
            TXG_BX(false, false, false);
#undef TXG_BX
        return TXG_OK;
    }
    /* long rows: statistics and chunk offsets per row, then segments of SEG_CHUNKS chunks */
    if (!scratch) return TXG_ERR_UNSUPPORTED;
    const long L = (n + BX_THREADS - 1) / BX_THREADS;
    const long seg = (long)SEG_CHUNKS * L;
    const long nseg = (n + seg - 1) / seg;
    if (!boxcar_supported(n, maxwn, nw)) return TXG_ERR_UNSUPPORTED;
    const long nc = seg_samples(n, maxwn);
    const bool bound = want && boxcar_smem(nc, true) <= BX_SMEM_TOP;
    const size_t smem = boxcar_smem(nc, bound), psmem = (size_t)(BX_THREADS / 32) * prep_chunks(L) * L * sizeof(float);
    if (smem > BX_SMEM_TOP || psmem > BX_SMEM_TOP) return TXG_ERR_UNSUPPORTED;
    cudaFuncSetAttribute(k_boxcar_prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psmem);
    launch_chained(k_boxcar_prep, (unsigned)ndm, BX_THREADS, psmem, st, tim, ldt, n, iqr, prep_chunks(L), scratch);
    dim3 grid((unsigned)ndm, (unsigned)nseg);
#define TXG_BXS(A, T, B)                                                                              \
    do {                                                                                              \
        cudaFuncSetAttribute(k_boxcar_seg<A, T, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        launch_chained(k_boxcar_seg<A, T, B>, grid, BX_THREADS, smem, st, tim, ldt, n, vwn, nw, thre, scratch, \
                       cand, ncand, cap, mxS, mxwn);                                                  \
    } while (0)
    if (avx2_tail)
        TXG_BXS(true, true, false);
    else if (mxS)
        TXG_BXS(false, true, false);
    else if (bound)
        TXG_BXS(false, false, true);
    else
        TXG_BXS(false, false, false);
#undef TXG_BXS
    return TXG_OK;
}

} // namespace txg
