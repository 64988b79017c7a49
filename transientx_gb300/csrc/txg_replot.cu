/*
 * txg_replot.cu -- the per-candidate chain of replot_fil (src/singlepulse/replot_fil.cpp:409-457)
 * on the GPU, batched over candidates: Candidate::zdot, get_stats, dedisperse (incoherent),
 * shrink_to_fit, azap, zap, normalize, clip, kadaneF, downsample, optimize (the DM-time Hough
 * transform of include/hough_transform.h), matched_filter and peak_search
 * (src/singlepulse/candidate.cpp:56-1200).
 *
 * Every kernel restates one Candidate method for one polarisation with the reference's own
 * mixture of float and double arithmetic (each expression rounded as the C++ evaluates it;
 * this file is compiled without multiply-add contraction), so results equal the reference's.
 * Candidates of a batch share the launches: blockIdx.y is the candidate, and each candidate's
 * rows keep their original pitch while its nbin and nchan shrink.  The small per-candidate
 * decisions the reference makes on the host (delays, the chop length, the azap quantiles, the
 * Hough shift plan) are made on the host here too.
 */
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <vector>

#include "txg_device.cuh"
#include "txg_internal.h"

namespace txg {

namespace {

/* device view of one candidate */
struct RpMeta {
    long off;   /* first float of its rows in the data buffers */
    long pitch; /* row pitch (its original nbin) */
    long nbin;  /* current samples */
    int nchan;  /* current channels */
    int pad;
    long coff;  /* first entry of its per-channel arrays (original nchan of them) */
    long hoff;  /* first float of its DM-time rows (nchans x nbin) */
    int nchans; /* rows of the Hough transform: nchan rounded up to a power of two */
    int levels; /* log2(nchans) */
    long soff;  /* first entry of its shift plan (levels x nchans) */
    long roff;  /* first entry of its row order hrange (nchans) */
    long rowoff; /* first of its S/N-map rows among the batch's */
};

inline unsigned nblk(long n, int b) { return (unsigned)((n + b - 1) / b); }

/* ---- sequential per-row chains ----------------------------------------------------------- */
/* The reference's statistics, running sums and kadane scans are chains: each sample's float or
 * double operation needs the previous one's result, so a row is one lane's work.  What need
 * not be serial is everything beside the chain.  A CTA of four warps takes 32 rows: warps 2 and 3
 * copy RT-sample tiles of them into shared memory by cp.async, one coalesced 128-byte row piece
 * per instruction, RNB - 1 tiles ahead, and prepare what the chains can be given ready (products,
 * differences); warps 0 and 1 each run a chain, every lane along its own row of the tile
 * (33-word pitch: no bank conflicts).  A chain then runs at its arithmetic's latency, about 5
 * cycles a float and 60 a double operation (conversions included, hence f2d).  One thread per
 * row straight from memory waited for an uncoalesced load at every sample; one warp per 32 rows
 * doing all of it spent most of its issue slots on the staging.  Candidate of 256 channels x
 * 2187 samples, us: zdot sums 1520 / 352 / 169, fit 1121 / 376 / 179, statistics (both) 1472 /
 * 354 / 118, boxcar chains of 256 x 625 samples 3112 (with the search) / 364 / 221. */
constexpr int RT = 32;
constexpr int RNB = 4;
constexpr int RP_THREADS = 128;
typedef float RpTile[RT][RT + 1];
typedef double RpTileD[RT][RT + 1];

__device__ __forceinline__ void rp_cp4(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void rp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void rp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(RNB - 2) : "memory"); }

struct RpNone {
    __device__ void operator()(int, int, int, float) const {}
};
struct RpNoTile {
    __device__ void operator()(long, int) const {}
};

/* Walks samples t = 0 .. cnt-1 of 32 rows (nrow of them exist; the others' values are undefined):
 * stream k's sample is (start + off[k] + t) mod n of the row, start = first[row] (shared memory,
 * or 0 without), start + off[k] + cnt <= 3n.  prep(b, row, q, v) runs once for every sample of
 * stream 0 on warps 2 and 3, before the chains come to it (b: tile parity, q: place in the
 * tile); step(t, q, b, v) on both chain warps; after(tl, b) on warp 1 when warp 0 has finished
 * tile tl.  tile: K * RNB tiles.  Starts and ends with a barrier. */
template <int K, typename Prep, typename Step, typename After>
__device__ __forceinline__ void rp_scan(RpTile *tile, const float *rows, long pitch, int nrow, long n, const int *first,
                                        const long (&off)[K], long cnt, Prep prep, Step step, After after)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long ntl = (cnt + RT - 1) / RT;
    auto stage = [&](long tl) {
        if (tl < ntl) {
            const long t = tl * RT + lane;
            const int b = (int)(tl % RNB);
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (first) {
#pragma unroll 4
                    for (int r = (w - 2) * 16; r < min(nrow, (w - 1) * 16); r++) {
                        long i = first[r] + off[k] + t;
                        i = i >= n ? i - n : i;
                        i = i >= n ? i - n : i;
                        if (t < cnt) rp_cp4(&tile[k * RNB + b][r][lane], rows + r * pitch + i);
                    }
                } else {
                    long i = off[k] + t;
                    i = i >= n ? i - n : i;
                    i = i >= n ? i - n : i;
                    const float *src = rows + (w - 2) * 16 * pitch + i;
                    float *dst = &tile[k * RNB + b][(w - 2) * 16][lane];
                    const int nr = min(nrow - (w - 2) * 16, 16);
                    if (t < cnt)
#pragma unroll 4
                        for (int r = 0; r < nr; r++, src += pitch, dst += RT + 1) rp_cp4(dst, src);
                }
            }
        }
        rp_commit(); /* one group per tile, empty past the end */
    };
    __syncthreads(); /* the previous scan's tiles are read no more */
    if (w >= 2)
        for (int b = 0; b < RNB - 1; b++) stage(b);
    for (long tl = 0; tl < ntl; tl++) {
        const int b = (int)(tl % RNB), par = (int)(tl & 1);
        if (w >= 2) {
            rp_wait();
            __syncwarp(); /* the warp's rows of tile tl are there */
            for (int r = (w - 2) * 16; r < min(nrow, (w - 1) * 16); r++) prep(par, r, lane, tile[b][r][lane]);
        }
        __syncthreads(); /* tile tl is there for all; tile tl-1 is read no more */
        if (w >= 2) {
            stage(tl + RNB - 1);
        } else {
            if (w == 1 && tl > 0) after(tl - 1, par ^ 1);
            const long t0 = tl * RT;
            const int nq = (int)min((long)RT, cnt - t0);
            float v[K];
            if (nq == RT) {
#pragma unroll 8
                for (int q = 0; q < RT; q++) {
#pragma unroll
                    for (int k = 0; k < K; k++) v[k] = tile[k * RNB + b][lane][q];
                    step(t0 + q, q, par, v);
                }
            } else {
                for (int q = 0; q < nq; q++) {
#pragma unroll
                    for (int k = 0; k < K; k++) v[k] = tile[k * RNB + b][lane][q];
                    step(t0 + q, q, par, v);
                }
            }
        }
    }
    __syncthreads();
    if (w == 1 && ntl > 0) after(ntl - 1, (int)((ntl - 1) & 1));
}

/* Candidate::zdot, first loop (candidate.cpp:837-859): per channel, double mean (warp 0) and
 * (float square) power (warp 1); std 1 where it is 0. */
__global__ void __launch_bounds__(RP_THREADS) k_rp_zdot_sums(const float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                             double *__restrict__ mean, double *__restrict__ std)
{
    chain_wait();
    __shared__ RpTile tile[RNB];
    __shared__ double mean_sh[32];
    const RpMeta c = m[blockIdx.y];
    const int j0 = blockIdx.x * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5, j = j0 + lane;
    if (j0 >= c.nchan) return;
    double acc = 0.;
    rp_scan<1>(tile, buf + c.off + (long)j0 * c.pitch, c.pitch, min(32, c.nchan - j0), c.nbin, nullptr, {0}, c.nbin,
               RpNone(), [&](long, int, int, const float(&v)[1]) { acc += f2d(w ? v[0] * v[0] : v[0]); }, RpNoTile());
    acc /= c.nbin;
    if (w == 0) mean_sh[lane] = acc;
    __syncthreads();
    if (j >= c.nchan || w > 1) return;
    if (w == 0) {
        mean[c.coff + j] = acc;
    } else {
        acc -= mean_sh[lane] * mean_sh[lane];
        acc = sqrt(acc);
        if (acc == 0.) acc = 1.;
        std[c.coff + j] = acc;
    }
}

/* its second half, one CTA per channel: x = (x - mean) / std in double, stored as float after
 * each step */
__global__ void __launch_bounds__(256) k_rp_zdot_norm(float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                      const double *__restrict__ mean, const double *__restrict__ std)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= c.nchan) return;
    float *r = buf + c.off + (long)j * c.pitch;
    const double mu = mean[c.coff + j], sd = std[c.coff + j];
    for (long i = threadIdx.x; i < c.nbin; i += blockDim.x) r[i] = (float)((float)(r[i] - mu) / sd);
}

/* zdot's zero-DM series: s[i] = sum over channels in order (double), / nchan (:857-864) */
__global__ void k_rp_zdot_s(const float *__restrict__ buf, const RpMeta *__restrict__ m,
                            double *__restrict__ s, long soff_stride)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nbin) return;
    const float *p = buf + c.off + i;
    double acc = 0.;
    int j = 0;
    for (; j + 16 <= c.nchan; j += 16) { /* sixteen loads in flight, added in channel order */
        float v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = p[(long)(j + r) * c.pitch];
#pragma unroll
        for (int r = 0; r < 16; r++) acc += v[r];
    }
    for (; j < c.nchan; j++) acc += p[(long)j * c.pitch];
    acc /= c.nchan;
    s[blockIdx.y * soff_stride + i] = acc;
}

/* zdot's least-squares fit (:866-885): the sums over each channel, xe by warp 0 and xs by warp 1 from
 * the products of warps 2 and 3; and by the last CTA of a candidate those of s, se and ss, which
 * are the same for every channel (32 samples and squares read and formed at a time). */
__global__ void __launch_bounds__(RP_THREADS) k_rp_zdot_fit(const float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                            const double *__restrict__ s_all, long soff_stride,
                                                            double *__restrict__ xe_all, double *__restrict__ xs_all,
                                                            double2 *__restrict__ ses)
{
    chain_wait();
    __shared__ RpTile tile[RNB];
    __shared__ RpTileD prod[2];
    const RpMeta c = m[blockIdx.y];
    const double *s = s_all + blockIdx.y * soff_stride;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (blockIdx.x == gridDim.x - 1) {
        if (w > 1) return;
        double acc = 0., v = lane < c.nbin ? s[lane] : 0.;
        for (long i = 0; i < c.nbin; i += 32) {
            const double p = w ? v * v : v;
            v = i + 32 + lane < c.nbin ? s[i + 32 + lane] : 0.;
            const int nq = (int)min(32L, c.nbin - i);
            for (int q = 0; q < nq; q++) acc += __shfl_sync(0xffffffffu, p, q);
        }
        if (lane == 0) (w ? ses[blockIdx.y].y : ses[blockIdx.y].x) = acc;
        return;
    }
    const int j0 = blockIdx.x * 32, j = j0 + lane;
    if (j0 >= c.nchan) return;
    double acc = 0., sv = 0.;
    long tp = -1; /* the tile whose s the lane holds */
    rp_scan<1>(tile, buf + c.off + (long)j0 * c.pitch, c.pitch, min(32, c.nchan - j0), c.nbin, nullptr, {0}, c.nbin,
               [&](int par, int r, int q, float v) {
                   if (r == (w - 2) * 16) { /* the warp's first row: the next tile */
                       tp++;
                       sv = tp * RT + q < c.nbin ? s[tp * RT + q] : 0.;
                   }
                   prod[par][r][q] = f2d(v) * sv;
               },
               [&](long, int q, int par, const float(&v)[1]) { acc += w ? prod[par][lane][q] : f2d(v[0]); }, RpNoTile());
    if (j >= c.nchan) return;
    if (w == 0) xe_all[c.coff + j] = acc;
    if (w == 1) xs_all[c.coff + j] = acc;
}

/* the fit's coefficients and its subtraction (:880-895), one CTA per channel */
__global__ void __launch_bounds__(256) k_rp_zdot_sub(float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                     const double *__restrict__ s_all, long soff_stride,
                                                     const double *__restrict__ xe_all,
                                                     const double *__restrict__ xs_all,
                                                     const double2 *__restrict__ ses)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= c.nchan) return;
    float *r = buf + c.off + (long)j * c.pitch;
    const double *s = s_all + blockIdx.y * soff_stride;
    const double xe = xe_all[c.coff + j], xs = xs_all[c.coff + j], se = ses[blockIdx.y].x, ss = ses[blockIdx.y].y;
    double alpha = 0., beta = 0.;
    const double tmp = se * se - ss * c.nbin;
    if (tmp != 0) {
        alpha = (xe * se - xs * c.nbin) / tmp;
        beta = (xs * se - xe * ss) / tmp;
    }
    for (long i = threadIdx.x; i < c.nbin; i += blockDim.x) r[i] = (float)(r[i] - (alpha * s[i] + beta));
}

/* Candidate::get_stats (:429-534) for one polarisation: the half-length window of least sum
 * (circular), then over that window either skewness, kurtosis and lag-1 autocorrelation in
 * float (SHAPE, what azap reads) or mean and variance in double (what normalize reads). */
template <bool SHAPE>
__global__ void __launch_bounds__(RP_THREADS) k_rp_stats(const float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                         double *__restrict__ mean, double *__restrict__ var,
                                                         float *__restrict__ skew, float *__restrict__ kurt,
                                                         float *__restrict__ ac)
{
    chain_wait();
    __shared__ RpTile tile[2 * RNB];
    __shared__ int first[32];
    __shared__ float shape[32];
    __shared__ double mu_sh[32];
    const RpMeta c = m[blockIdx.y];
    const int j0 = blockIdx.x * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5, j = j0 + lane;
    if (j0 >= c.nchan) return;
    const float *rows = buf + c.off + (long)j0 * c.pitch;
    const int nrow = min(32, c.nchan - j0);
    const long nbin = c.nbin, h = nbin / 2;
    /* data_sumif starts at 0 and adds the data: 0.f + x.  Both chain warps find the window. */
    float boxsum = 0.;
    rp_scan<1>(tile, rows, c.pitch, nrow, nbin, nullptr, {0}, h, RpNone(),
               [&](long, int, int, const float(&v)[1]) { boxsum += 0.f + v[0]; }, RpNoTile());
    float mn = boxsum;
    int istart = 0;
    rp_scan<2>(tile, rows, c.pitch, nrow, nbin, nullptr, {0, h}, nbin, RpNone(),
               [&](long i, int, int, const float(&v)[2]) {
                   boxsum -= 0.f + v[0];
                   boxsum += 0.f + v[1];
                   if (boxsum < mn) {
                       mn = boxsum;
                       istart = (int)i + 1;
                   }
               },
               RpNoTile());
    if (w == 0) first[lane] = istart;
    const long q = c.coff + j;
    if (SHAPE) { /* warp 0: variance and skewness, warp 1: kurtosis and autocorrelation */
        const float tmp_mean = mn / h;
        float a = 0., b = 0., last = 0;
        rp_scan<1>(tile, rows, c.pitch, nrow, nbin, first, {0}, h, RpNone(),
                   [&](long, int, int, const float(&v)[1]) {
                       const float t = (0.f + v[0]) - tmp_mean;
                       const float t2 = t * t, t3 = t2 * t, t4 = t3 * t;
                       a += w ? t4 : t2;
                       b += w ? t * last : t3;
                       last = t;
                   },
                   RpNoTile());
        if (w == 0) shape[lane] = a / h; /* the variance */
        __syncthreads();
        if (w > 1 || j >= c.nchan) return;
        const float tmp_var = shape[lane];
        if (tmp_var <= 0) {
            if (w) a = 0.;
            b = 0.;
        }
        if (w == 0) {
            float sk = b;
            sk /= h;
            sk /= tmp_var * sqrtf(tmp_var);
            skew[q] = sk;
        } else {
            float ku = a, a1 = b;
            ku /= h;
            ku /= tmp_var * tmp_var;
            ku -= 3.;
            a1 /= h - 1;
            a1 /= tmp_var;
            kurt[q] = ku;
            ac[q] = a1;
        }
    } else { /* warp 0: mean, warp 1: mean square */
        double acc = 0.;
        rp_scan<1>(tile, rows, c.pitch, nrow, nbin, first, {0}, h, RpNone(),
                   [&](long, int, int, const float(&v)[1]) { acc += f2d(w ? v[0] * v[0] : v[0]); }, RpNoTile());
        acc /= h;
        if (w == 0) mu_sh[lane] = acc;
        __syncthreads();
        if (w > 1 || j >= c.nchan) return;
        if (w == 0) mean[q] = acc;
        else var[q] = acc - mu_sh[lane] * mu_sh[lane];
    }
}

/* Candidate::dedisperse, incoherent branch (:106-140): row j rotated left by its delay; the
 * first keep[candidate] samples, all that the chop which follows leaves.  One CTA per channel. */
__global__ void __launch_bounds__(256) k_rp_dedisp(const float *__restrict__ src, float *__restrict__ dst,
                                                   const RpMeta *__restrict__ m, const int *__restrict__ delay,
                                                   const long *__restrict__ keep)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= c.nchan) return;
    const long o = c.off + (long)j * c.pitch, d = delay[c.coff + j], n = keep[blockIdx.y];
    for (long i = threadIdx.x; i < n; i += blockDim.x) dst[o + i] = src[o + (i + d < c.nbin ? i + d : i + d - c.nbin)];
}

/* data *= weights[j] (azap :610-621, zap :641-653), one CTA per channel */
__global__ void __launch_bounds__(256) k_rp_scale(float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                  const float *__restrict__ w)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= c.nchan) return;
    float *r = buf + c.off + (long)j * c.pitch;
    const float f = w[c.coff + j];
    for (long i = threadIdx.x; i < c.nbin; i += blockDim.x) r[i] *= f;
}

/* Candidate::normalize (:536-567), one CTA per channel */
__global__ void __launch_bounds__(256) k_rp_normalize(float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                      const double *__restrict__ mean,
                                                      const double *__restrict__ var)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= c.nchan) return;
    float *r = buf + c.off + (long)j * c.pitch;
    const double mu = mean[c.coff + j], v = var[c.coff + j];
    const float sd = v <= 0. ? 1.f : (float)sqrt(v); /* x / 1 is x */
    for (long i = threadIdx.x; i < c.nbin; i += blockDim.x) r[i] = (float)(r[i] - mu) / sd;
}

/* Candidate::clip (:656-708): td x fd sums (fd outer, td inner) above thre zero their cells */
__global__ void k_rp_clip(float *__restrict__ buf, const RpMeta *__restrict__ m, int td, int fd,
                          float thre)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const long nsds = c.nbin / td, ncds = c.nchan / fd;
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ncds * nsds) return;
    const long j = e / nsds, i = e - j * nsds;
    float acc = 0.;
    for (int k = 0; k < fd; k++)
        for (int n = 0; n < td; n++) acc += buf[c.off + (j * fd + k) * c.pitch + i * td + n];
    if (acc > thre)
        for (int k = 0; k < fd; k++)
            for (int n = 0; n < td; n++) buf[c.off + (j * fd + k) * c.pitch + i * td + n] = 0.;
}

/* Candidate::kadaneF (:710-829): the td x fd sums (fd outer, td inner), one CTA per downsampled
 * channel; ds: scratch rows of stride `dstride` per channel */
__global__ void __launch_bounds__(128) k_rp_kadane_ds(const float *__restrict__ buf, const RpMeta *__restrict__ m,
                                                      int td, int fd, float *__restrict__ ds, long dstride)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const long nsds = c.nbin / td, ncds = c.nchan / fd;
    const long j = blockIdx.x;
    if (j >= ncds) return;
    for (long i = threadIdx.x; i < nsds; i += blockDim.x) {
        float acc = 0.;
        for (int k = 0; k < fd; k++)
            for (int n = 0; n < td; n++) acc += buf[c.off + (j * fd + k) * c.pitch + i * td + n];
        ds[(c.coff + j) * dstride + i] = acc;
    }
}

/* kadane<float> of the XLibs helpers as the reference tree's callers use it (a new maximum
 * needs a strictly larger sum, the running sum restarts after it drops below zero), on the
 * positive sums by warp 0 and the negated ones by warp 1, then the S/N test with no minimum
 * window (replot_fil passes nwidth 0): ranges[4*channel + 2*sign] = first and last-plus-one
 * sample, -1 where nothing is zapped */
__global__ void __launch_bounds__(RP_THREADS) k_rp_kadane_scan(const float *__restrict__ ds,
                                                               const RpMeta *__restrict__ m, int td, int fd,
                                                               float threshold, long dstride, long *__restrict__ ranges)
{
    chain_wait();
    __shared__ RpTile tile[RNB];
    const RpMeta c = m[blockIdx.y];
    const long nsds = c.nbin / td, ncds = c.nchan / fd;
    const int w = threadIdx.x >> 5;
    const long j0 = (long)blockIdx.x * 32, j = j0 + (threadIdx.x & 31);
    if (j0 >= ncds) return;
    float best = -INFINITY, cur = 0;
    int cs = 0, start = 0, end = -1;
    rp_scan<1>(tile, ds + (c.coff + j0) * dstride, dstride, (int)min(32L, ncds - j0), max(nsds, 1L), nullptr, {0}, nsds,
               RpNone(),
               [&](long i, int, int, const float(&v)[1]) {
                   cur = cur + (w ? -v[0] : v[0]);
                   if (cur > best) {
                       best = cur;
                       start = cs;
                       end = (int)i;
                   }
                   if (cur < 0) {
                       cur = 0;
                       cs = (int)i + 1;
                   }
               },
               RpNoTile());
    if (j >= ncds || w > 1) return;
    const float var = (float)(td * fd);
    const long wn = (long)end - start + 1;
    float snr2 = 0.;
    if (wn > 0) snr2 = best * best / (wn * var);
    const bool zap = snr2 > threshold * threshold;
    long *o = ranges + 4 * (c.coff + j) + 2 * w;
    o[0] = zap ? (long)start * td : -1;
    o[1] = zap ? (long)(end + 1) * td : -1;
}

/* its zapping, one CTA per channel */
__global__ void __launch_bounds__(128) k_rp_kadane_apply(float *__restrict__ buf, const RpMeta *__restrict__ m, int fd,
                                                         const long *__restrict__ ranges)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const int j = blockIdx.x;
    if (j >= c.nchan / fd * fd) return;
    const long *o = ranges + 4 * (c.coff + j / fd);
    float *r = buf + c.off + (long)j * c.pitch;
    for (int p = 0; p < 2; p++)
        if (o[2 * p] >= 0)
            for (long i = o[2 * p] + threadIdx.x; i < o[2 * p + 1]; i += blockDim.x) r[i] = 0.;
}

/* Candidate::downsample(1, fd) (:381-427): channel sums in order, out of place */
__global__ void k_rp_fsum(const float *__restrict__ src, float *__restrict__ dst,
                          const RpMeta *__restrict__ m, int fd)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y]; /* geometry before the downsample */
    const long nc = c.nchan / fd;
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nc * c.nbin) return;
    const long j = e / c.nbin, i = e - j * c.nbin;
    float acc = 0.;
    for (int jj = 0; jj < fd; jj++) acc += src[c.off + (j * fd + jj) * c.pitch + i];
    dst[c.off + j * c.pitch + i] = acc;
}

/* One level of the transform of hough_transform.h:29-55 (depth = levels-1-t), one CTA per output
 * row: for block irow of 2*nrowsub rows, row k of the first half becomes x0 + rot(y, d0) and row
 * k of the second half x0 + rot(y, d1), y being the old second-half row and
 * rot(y, d)[i] = y[(i+d) mod ncol].  The first level reads Candidate::optimize's input
 * (:899-966): the channels, frequency-descending, rows past them zero.  A candidate's last
 * level writes the transform's output order, row hrange[r]; later levels of a batch whose
 * other candidates have more rows copy it. */
__global__ void __launch_bounds__(256) k_rp_hough_level(const float *__restrict__ buf, const float *__restrict__ hin,
                                                        float *__restrict__ hout, const RpMeta *__restrict__ m,
                                                        const int *__restrict__ shift,
                                                        const int *__restrict__ hrange,
                                                        const int *__restrict__ flip, int t)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const long ncol = c.nbin, r = blockIdx.x;
    if (r >= c.nchans) return;
    if (t >= c.levels) {
        for (long i = threadIdx.x; i < ncol; i += blockDim.x)
            hout[c.hoff + r * ncol + i] = hin[c.hoff + r * ncol + i];
        return;
    }
    const long nrowsub = 1L << t;
    const long blk = r / (2 * nrowsub), k = r - blk * 2 * nrowsub;
    const long d = shift[c.soff + (long)t * c.nchans + blk * 2 * nrowsub + k];
    const long x0 = k < nrowsub ? r : r - nrowsub, y = x0 + nrowsub;
    const bool fl = flip[blockIdx.y];
    auto row = [&](long j) -> const float * {
        if (t > 0) return hin + c.hoff + j * ncol;
        return j < c.nchan ? buf + c.off + (fl ? c.nchan - 1 - j : j) * c.pitch : nullptr;
    };
    const float *xr = row(x0), *yr = row(y);
    float *o = hout + c.hoff + (t == c.levels - 1 ? (long)hrange[c.roff + r] : r) * ncol;
    for (long i = threadIdx.x; i < ncol; i += blockDim.x) {
        const long iy = i + d < ncol ? i + d : i + d - ncol;
        const float a = xr ? xr[i] : 0.f, b = yr ? yr[iy] : 0.f;
        /* the input rows are 0 + data */
        o[i] = t > 0 ? a + b : (0.f + a) + (0.f + b);
    }
}

/* peak_search's profile (:1115-1129): sum of the channels in order, from 0 */
__global__ void k_rp_profile(const float *__restrict__ buf, float *__restrict__ h,
                             const RpMeta *__restrict__ m)
{
    chain_wait();
    const RpMeta c = m[blockIdx.y];
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.nbin) return;
    const float *p = buf + c.off + i;
    float acc = 0.;
    int j = 0;
    for (; j + 16 <= c.nchan; j += 16) { /* sixteen loads in flight, added in channel order */
        float v[16];
#pragma unroll
        for (int r = 0; r < 16; r++) v[r] = p[(long)(j + r) * c.pitch];
#pragma unroll
        for (int r = 0; r < 16; r++) acc += v[r];
    }
    for (; j < c.nchan; j++) acc += p[(long)j * c.pitch];
    h[c.hoff + i] = acc;
}

/* The chains of matched_filter / peak_search (:1000-1030, :1131-1150): per row the double mean
 * (warp 0) and mean square (warp 1; a float's square is exact in a double, so the fused multiply-add
 * rounds like the separate ones), then twice round the row the float running sum of (x - mean),
 * each addition in double: warps 2 and 3 form the differences, warp 0 adds, warp 1 writes the
 * finished tile.  csum: 2*nbin floats per row. */
__global__ void __launch_bounds__(RP_THREADS) k_rp_csum(const float *__restrict__ h, const RpMeta *__restrict__ m,
                                                        const int *__restrict__ rows, double *__restrict__ var_all,
                                                        float *__restrict__ csump)
{
    chain_wait();
    __shared__ RpTile tile[RNB];
    __shared__ RpTileD diff[2];
    __shared__ RpTile outt[2];
    __shared__ double mean_sh[32];
    const RpMeta c = m[blockIdx.y];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long j0 = (long)blockIdx.x * 32, j = j0 + lane;
    if (j0 >= rows[blockIdx.y]) return;
    const long nbin = c.nbin;
    const int nrow = (int)min(32L, rows[blockIdx.y] - j0);
    const float *tim = h + c.hoff + j0 * nbin;
    float *cs = csump + (c.hoff + j0 * nbin) * 2;
    double acc = 0.;
    rp_scan<1>(tile, tim, nbin, nrow, nbin, nullptr, {0}, nbin, RpNone(),
               [&](long, int, int, const float(&x)[1]) {
                   const double v = f2d(x[0]);
                   acc = w ? __fma_rn(v, v, acc) : acc + v;
               },
               RpNoTile());
    acc /= nbin;
    if (w == 0) mean_sh[lane] = acc;
    __syncthreads();
    if (w == 1 && lane < nrow) var_all[c.rowoff + j] = acc - mean_sh[lane] * mean_sh[lane];
    float csum = 0.;
    rp_scan<1>(tile, tim, nbin, nrow, nbin, nullptr, {0}, 2 * nbin,
               [&](int par, int r, int q, float v) { diff[par][r][q] = f2d(v) - mean_sh[r]; },
               [&](long, int q, int par, const float(&)[1]) {
                   if (w) return;
                   csum = (float)(f2d(csum) + diff[par][lane][q]);
                   outt[par][lane][q] = csum;
               },
               [&](long tl, int par) {
                   const long t = tl * RT + lane;
                   if (t < 2 * nbin)
#pragma unroll 4
                       for (int r = 0; r < nrow; r++) cs[r * 2 * nbin + t] = outt[par][r][lane];
               });
}

/* best of a row or candidate: the first largest S in row-major order (the scan of :1065-1078) */
struct RpBest {
    long idx;
    float S;
    int wn;
};
__device__ __forceinline__ bool rp_before(float S, long i, float T, long k) { return S > T || (S == T && i < k); }

/* The boxcar search of one row (:1031-1063, :1151-1180), one CTA per row: S over the float
 * ladder from the circular running sum, S >= best keeps the later width.  Widths in chunks of
 * RP_W, their factors computed once per CTA; a sample's best lives in the map between chunks. */
constexpr int RP_W = 128;

__global__ void __launch_bounds__(256) k_rp_match(const RpMeta *__restrict__ m, const int *__restrict__ rows,
                                                  const float *__restrict__ vwn, const int *__restrict__ nbox,
                                                  long wstride, const double *__restrict__ var_all,
                                                  const float *__restrict__ csump, float *__restrict__ snr,
                                                  int *__restrict__ wid, RpBest *__restrict__ rbest)
{
    chain_wait();
    __shared__ float temp[RP_W];
    __shared__ int wns[RP_W];
    __shared__ RpBest red[8];
    const RpMeta c = m[blockIdx.y];
    const long j = blockIdx.x;
    if (j >= rows[blockIdx.y]) return;
    const long nbin = c.nbin;
    const float *cs = csump + (c.hoff + j * nbin) * 2;
    float *vS = snr + c.hoff + j * nbin;
    int *vw = wid + c.hoff + j * nbin;
    const double var = var_all[c.rowoff + j];
    const int nw = var > 0 ? nbox[blockIdx.y] : 0;
    const float *lad = vwn + blockIdx.y * wstride;
    RpBest mine{0x7fffffffffffffffL, -1.f, 0};
    for (int w0 = 0; w0 == 0 || w0 < nw; w0 += RP_W) {
        const int nc = min(RP_W, nw - w0);
        __syncthreads();
        for (int w = threadIdx.x; w < nc; w += blockDim.x) {
            const int wn = (int)lad[w0 + w];
            wns[w] = wn;
            temp[w] = (float)sqrt(1. / (wn * var));
        }
        __syncthreads();
        for (long i = threadIdx.x; i < nbin; i += blockDim.x) {
            float b = w0 ? vS[i] : 0.f;
            int bw = w0 ? vw[i] : 0;
#pragma unroll 4
            for (int w = 0; w < nc; w++) {
                const int wn = wns[w], wl = wn / 2 + 1, wh = (wn - 1) / 2;
                const long k = i >= wl ? i : i + nbin;
                const float S = (cs[k + wh] - cs[k - wl]) * temp[w];
                if (S >= b) {
                    b = S;
                    bw = wn;
                }
            }
            vS[i] = b;
            vw[i] = bw;
            if (w0 + RP_W >= nw && rp_before(b, i, mine.S, mine.idx)) mine = RpBest{i, b, bw};
        }
    }
    /* the row's first largest S (never a NaN: a NaN score fails S >= best) */
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    for (int off = 16; off >= 1; off >>= 1) {
        const RpBest o{__shfl_xor_sync(0xffffffffu, mine.idx, off), __shfl_xor_sync(0xffffffffu, mine.S, off),
                       __shfl_xor_sync(0xffffffffu, mine.wn, off)};
        if (rp_before(o.S, o.idx, mine.S, mine.idx)) mine = o;
    }
    if (lane == 0) red[wp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 8; q++)
            if (rp_before(red[q].S, red[q].idx, mine.S, mine.idx)) mine = red[q];
        mine.idx += j * nbin;
        rbest[c.rowoff + j] = mine;
    }
}

/* the candidate's best from its rows' */
__global__ void __launch_bounds__(256) k_rp_best(const RpMeta *__restrict__ m, const int *__restrict__ rows,
                                                 const RpBest *__restrict__ rbest, RpBest *__restrict__ best)
{
    chain_wait();
    __shared__ RpBest red[256];
    const RpMeta c = m[blockIdx.x];
    RpBest mine{0x7fffffffffffffffL, -1.f, 0};
    for (long j = threadIdx.x; j < rows[blockIdx.x]; j += blockDim.x) {
        const RpBest o = rbest[c.rowoff + j];
        if (rp_before(o.S, o.idx, mine.S, mine.idx)) mine = o;
    }
    red[threadIdx.x] = mine;
    __syncthreads();
    for (int h = 128; h >= 1; h >>= 1) {
        if (threadIdx.x < h) {
            const RpBest o = red[threadIdx.x + h];
            if (rp_before(o.S, o.idx, mine.S, mine.idx)) red[threadIdx.x] = mine = o;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) best[blockIdx.x] = mine;
}

} // namespace

} // namespace txg

using namespace txg;

namespace {

/* host mirror of one candidate through the chain */
struct RpHost {
    long off, pitch, nbin, coff;
    int nchan;
    double tbin, dm;
    float width;
    std::vector<double> f;
    /* Hough geometry (step 12) */
    int nchans = 1, levels = 0;
    long hoff = 0, soff = 0, roff = 0, rowoff = 0, rows = 1;
    double dms = 0., ddm = 0.;
};

double rp_dmdelay(double dm, double fh, double fl) { return 4.148741601e3 * dm * (1. / (fl * fl) - 1. / (fh * fh)); }

/* get_shiftplan of hough_transform.h:57-101, as written */
void rp_shiftplan(std::vector<std::vector<int>> &shiftplan, std::vector<int> &hrange, int nrow, int ncol,
                  const std::function<int(int, int, int)> &get_shift)
{
    int nrow_tmp = nrow;
    int nrowsub_tmp = nrow / nrow_tmp;
    hrange.assign(nrow, 0);
    for (long k = 0; k < nrowsub_tmp; k++) hrange[k] = k * nrow_tmp;
    std::vector<int> xrange_tmp(nrow, 0);
    for (long j = 0; j < nrow; j++) xrange_tmp[j] = j;
    int n = (int)std::log2(nrow);
    for (long l = 0; l < n; l++) {
        std::vector<int> shift_tmp(nrow_tmp * nrowsub_tmp);
        for (long j = 0; j < nrow_tmp / 2; j++) {
            for (long k = 0; k < nrowsub_tmp; k++) {
                hrange[k] = hrange[k];
                hrange[k + nrowsub_tmp] = hrange[k] + nrow_tmp / 2;
            }
            for (long k = 0; k < nrowsub_tmp * 2; k++) {
                int s = get_shift(xrange_tmp[j * 2], xrange_tmp[j * 2 + 1], hrange[k]) % ncol;
                if (s < 0) s += ncol;
                shift_tmp[j * (nrowsub_tmp * 2) + k] = s;
            }
            xrange_tmp[j] = xrange_tmp[j * 2];
        }
        shiftplan.push_back(shift_tmp);
        nrowsub_tmp <<= 1;
        nrow_tmp >>= 1;
    }
}

/* azap's IQR cut of one statistic (candidate.cpp:573-597): q1 the n/4-th smallest, q3 the
 * n/4-th largest, by nth_element as the reference takes them */
void rp_quartiles(const float *v, int n, float &q1, float &q3)
{
    std::vector<float> s(v, v + n);
    std::nth_element(s.begin(), s.begin() + s.size() / 4, s.end(), std::less<float>());
    q1 = s[s.size() / 4];
    std::nth_element(s.begin(), s.begin() + s.size() / 4, s.end(), std::greater<float>());
    q3 = s[s.size() / 4];
}

} // namespace

extern "C" int txg_replot(const txg_replot_opts *o, const txg_replot_cand *cands, int64_t n,
                          txg_replot_result *out, float *snrmap, int64_t snrmap_cap, float *data_out,
                          int64_t data_cap)
{
    if (!o || !cands || !out || n <= 0) return set_arg_error("null options, candidates or results");
    const bool kad = o->kadane[0] > 0, clp = o->clip[0] > 0;
    if ((kad && (o->kadane[1] < 1)) || (clp && (o->clip[1] < 1)) || o->fd < 1 || o->nwidth < 1 ||
        o->nzap < 0 || o->nzap > 16)
        return set_arg_error("kadane/clip td and fd, fd and nw must be positive; at most 16 zap ranges");
    const int upto = o->upto > 0 ? o->upto : 12;
    std::vector<RpHost> H(n);
    long total = 0, tchan = 0, maxnbin = 0;
    for (long b = 0; b < n; b++) {
        const txg_replot_cand &c = cands[b];
        if (!c.data || !c.frequencies || c.nchan < 2 || c.nbin < 4 || !(c.tbin > 0.) || !(c.width > 0.f))
            return set_arg_error("candidate " + std::to_string(b) + ": need data, frequencies, nchan >= 2, nbin >= 4, tbin > 0, width > 0");
        if (c.nchan / o->fd < 2) return set_arg_error("fd leaves fewer than 2 channels");
        RpHost &h = H[b];
        h.off = total;
        h.pitch = h.nbin = c.nbin;
        h.nchan = c.nchan;
        h.coff = tchan;
        h.tbin = c.tbin;
        h.dm = c.dm;
        h.width = c.width;
        h.f.assign(c.frequencies, c.frequencies + c.nchan);
        total += (long)c.nchan * c.nbin;
        tchan += c.nchan;
        maxnbin = std::max(maxnbin, (long)c.nbin);
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return set_cuda_error(cudaErrorNoDevice, "txg_replot", __FILE__, __LINE__);

    Scratch mem;
    float *buf[2] = {nullptr, nullptr}, *skew, *kurt, *ac, *w;
    double *mean, *var;
    int *delay;
    RpMeta *dmeta;
    cudaError_t e = cudaSuccess;
#define RP_TRY(x)                                                                  \
    do {                                                                           \
        e = (x);                                                                   \
        if (e != cudaSuccess) return set_cuda_error(e, #x, __FILE__, __LINE__);    \
    } while (0)
    RP_TRY(mem.open());
    const cudaStream_t st = mem.st;
    RP_TRY(mem.alloc(&buf[0], total));
    RP_TRY(mem.alloc(&buf[1], total));
    RP_TRY(mem.alloc(&mean, tchan));
    RP_TRY(mem.alloc(&var, tchan));
    RP_TRY(mem.alloc(&skew, tchan));
    RP_TRY(mem.alloc(&kurt, tchan));
    RP_TRY(mem.alloc(&ac, tchan));
    RP_TRY(mem.alloc(&w, tchan));
    RP_TRY(mem.alloc(&delay, tchan));
    RP_TRY(mem.alloc(&dmeta, n));
    for (long b = 0; b < n; b++)
        RP_TRY(cudaMemcpyAsync(buf[0] + H[b].off, cands[b].data, sizeof(float) * H[b].nchan * H[b].nbin,
                               cudaMemcpyHostToDevice, st));
    int cur = 0;
    std::vector<RpMeta> meta(n);
    auto push_meta = [&]() -> cudaError_t {
        for (long b = 0; b < n; b++) {
            const RpHost &h = H[b];
            RpMeta &m = meta[b];
            m.off = h.off;
            m.pitch = h.pitch;
            m.nbin = h.nbin;
            m.nchan = h.nchan;
            m.pad = 0;
            m.coff = h.coff;
            m.hoff = h.hoff;
            m.nchans = h.nchans;
            m.levels = h.levels;
            m.soff = h.soff;
            m.roff = h.roff;
            m.rowoff = h.rowoff;
        }
        return cudaMemcpyAsync(dmeta, meta.data(), sizeof(RpMeta) * n, cudaMemcpyHostToDevice, st);
    };
    auto maxchan = [&]() {
        int mc = 0;
        for (auto &h : H) mc = std::max(mc, h.nchan);
        return mc;
    };
    auto per32 = [&](int rows) { return nblk(rows, 32); }; /* CTAs of the row scans */
    auto maxelem = [&]() {
        long me = 0;
        for (auto &h : H) me = std::max(me, (long)h.nchan * h.nbin);
        return me;
    };
    const unsigned NB = (unsigned)n;
    RP_TRY(push_meta());
    std::vector<float> w_h(tchan, 1.f);

    /* 1: zdot */
    if (o->zdot) {
        double *zs, *xe, *xs;
        double2 *ses;
        RP_TRY(mem.alloc(&zs, (size_t)n * maxnbin));
        RP_TRY(mem.alloc(&xe, tchan));
        RP_TRY(mem.alloc(&xs, tchan));
        RP_TRY(mem.alloc(&ses, n));
        launch_chained(k_rp_zdot_sums, dim3(per32(maxchan()), NB), RP_THREADS, 0, st, buf[cur], dmeta, mean, var);
        launch_chained(k_rp_zdot_norm, dim3(maxchan(), NB), 256, 0, st, buf[cur], dmeta, mean, var);
        launch_chained(k_rp_zdot_s, dim3(nblk(maxnbin, 64), NB), 64, 0, st, buf[cur], dmeta, zs, maxnbin);
        launch_chained(k_rp_zdot_fit, dim3(per32(maxchan()) + 1, NB), RP_THREADS, 0, st, buf[cur], dmeta, zs, maxnbin,
                       xe, xs, ses);
        launch_chained(k_rp_zdot_sub, dim3(maxchan(), NB), 256, 0, st, buf[cur], dmeta, zs, maxnbin,
                       xe, xs, ses);
        RP_TRY(cudaGetLastError());
    }
    /* 2: get_stats (their skewness, kurtosis, autocorrelation drive azap) */
    std::vector<float> sk_h(tchan), ku_h(tchan), ac_h(tchan);
    if (upto >= 2) {
        launch_chained(k_rp_stats<true>, dim3(per32(maxchan()), NB), RP_THREADS, 0, st, buf[cur], dmeta,
                       mean, var, skew, kurt, ac);
        RP_TRY(cudaGetLastError());
        RP_TRY(cudaMemcpyAsync(sk_h.data(), skew, sizeof(float) * tchan, cudaMemcpyDeviceToHost, st));
        RP_TRY(cudaMemcpyAsync(ku_h.data(), kurt, sizeof(float) * tchan, cudaMemcpyDeviceToHost, st));
        RP_TRY(cudaMemcpyAsync(ac_h.data(), ac, sizeof(float) * tchan, cudaMemcpyDeviceToHost, st));
    }
    /* 4 (decided first, the rotation below then writes no more than it leaves):
     * shrink_to_fit(2*nw, pow2bin, kadane td) (:234-264) */
    std::vector<long> cut(n);
    for (long b = 0; b < n; b++) {
        const RpHost &h = H[b];
        cut[b] = h.nbin;
        if (upto < 4) continue;
        const int nw2 = 2 * o->nwidth, factor = kad ? o->kadane[0] : 1;
        long nbin_new = (long)(nw2 * h.width / h.tbin);
        if (o->pow2bin) nbin_new = (long)std::pow(2, std::ceil(std::log2(nbin_new)));
        nbin_new = (long)(std::ceil(nbin_new / factor) * factor);
        if (nbin_new < h.nbin) cut[b] = nbin_new;
        if (cut[b] < 4) {
            return set_arg_error("the chop to 2*nw*width leaves fewer than 4 samples");
        }
    }
    /* 3: dedisperse at the candidate DM (incoherent) */
    if (upto >= 3) {
        std::vector<int> dl(tchan);
        for (long b = 0; b < n; b++) {
            const RpHost &h = H[b];
            const double fmax = *std::max_element(h.f.begin(), h.f.end());
            for (int j = 0; j < h.nchan; j++) {
                int d = (int)std::round(rp_dmdelay(h.dm, fmax, h.f[j]) / h.tbin);
                d %= h.nbin;
                if (d < 0) d += h.nbin;
                dl[h.coff + j] = d;
            }
        }
        RP_TRY(cudaMemcpyAsync(delay, dl.data(), sizeof(int) * tchan, cudaMemcpyHostToDevice, st));
        long *dcut;
        RP_TRY(mem.alloc(&dcut, n));
        RP_TRY(cudaMemcpyAsync(dcut, cut.data(), sizeof(long) * n, cudaMemcpyHostToDevice, st));
        launch_chained(k_rp_dedisp, dim3(maxchan(), NB), 256, 0, st, buf[cur], buf[cur ^ 1], dmeta, delay, dcut);
        RP_TRY(cudaGetLastError());
        RP_TRY(cudaStreamSynchronize(st)); /* dl goes out of scope */
        cur ^= 1;
    }
    if (upto >= 4) {
        for (long b = 0; b < n; b++) H[b].nbin = cut[b];
        RP_TRY(push_meta());
    }
    /* 5: azap(zapthre) with the statistics of step 2 */
    if (upto >= 5) {
        RP_TRY(cudaStreamSynchronize(st));
        const float t = o->zapthre;
        for (auto &h : H) {
            float k1, k3, s1, s3, a1, a3;
            rp_quartiles(ku_h.data() + h.coff, h.nchan, k1, k3);
            rp_quartiles(sk_h.data() + h.coff, h.nchan, s1, s3);
            rp_quartiles(ac_h.data() + h.coff, h.nchan, a1, a3);
            const float kR = k3 - k1, sR = s3 - s1, aR = a3 - a1;
            for (int j = 0; j < h.nchan; j++) {
                const float ku = ku_h[h.coff + j], sk = sk_h[h.coff + j], a = ac_h[h.coff + j];
                if ((ku < k1 - t * kR) || (ku > k3 + t * kR) || (sk < s1 - t * sR) || (sk > s3 + t * sR) ||
                    (a < a1 - t * aR) || (a > a3 + t * aR))
                    w_h[h.coff + j] = 0.;
            }
        }
        RP_TRY(cudaMemcpyAsync(w, w_h.data(), sizeof(float) * tchan, cudaMemcpyHostToDevice, st));
        launch_chained(k_rp_scale, dim3(maxchan(), NB), 256, 0, st, buf[cur], dmeta, w);
        RP_TRY(cudaGetLastError());
    }
    /* 6: zap(zaplist): weights keep azap's zeros */
    if (upto >= 6 && o->nzap > 0) {
        RP_TRY(cudaStreamSynchronize(st));
        for (auto &h : H)
            for (int j = 0; j < h.nchan; j++)
                for (int z = 0; z < o->nzap; z++)
                    if (h.f[j] >= o->zap[z][0] && h.f[j] <= o->zap[z][1]) w_h[h.coff + j] = 0;
        RP_TRY(cudaMemcpyAsync(w, w_h.data(), sizeof(float) * tchan, cudaMemcpyHostToDevice, st));
        launch_chained(k_rp_scale, dim3(maxchan(), NB), 256, 0, st, buf[cur], dmeta, w);
        RP_TRY(cudaGetLastError());
    }
    /* 7, 8: get_stats, normalize */
    if (upto >= 7)
        launch_chained(k_rp_stats<false>, dim3(per32(maxchan()), NB), RP_THREADS, 0, st, buf[cur], dmeta,
                       mean, var, skew, kurt, ac);
    if (upto >= 8)
        launch_chained(k_rp_normalize, dim3(maxchan(), NB), 256, 0, st, buf[cur], dmeta, mean, var);
    RP_TRY(cudaGetLastError());
    /* 9: clip */
    if (upto >= 9 && clp) {
        const int td = o->clip[0], fd = o->clip[1];
        const float thre = (float)((float)o->clip[2] * std::sqrt(td * fd));
        launch_chained(k_rp_clip, dim3(nblk(maxelem(), 256), NB), 256, 0, st, buf[cur], dmeta, td, fd, thre);
        RP_TRY(cudaGetLastError());
    }
    /* 10: kadaneF (nwidth 0, as replot_fil calls it) */
    if (upto >= 10 && kad) {
        const int td = o->kadane[0], fd = o->kadane[1];
        long dstride = 1, ncmax = 0;
        for (auto &h : H) {
            dstride = std::max(dstride, h.nbin / td);
            ncmax = std::max(ncmax, (long)h.nchan / fd);
        }
        if (ncmax > 0) {
            float *ds;
            long *rng;
            RP_TRY(mem.alloc(&ds, (size_t)tchan * dstride));
            RP_TRY(mem.alloc(&rng, (size_t)tchan * 4));
            launch_chained(k_rp_kadane_ds, dim3(ncmax, NB), 128, 0, st, buf[cur], dmeta, td, fd, ds, dstride);
            launch_chained(k_rp_kadane_scan, dim3(per32((int)ncmax), NB), RP_THREADS, 0, st, ds, dmeta, td, fd,
                                                                                 (float)o->kadane[2], dstride, rng);
            launch_chained(k_rp_kadane_apply, dim3(maxchan(), NB), 128, 0, st, buf[cur], dmeta, fd, rng);
            RP_TRY(cudaGetLastError());
        }
    }
    /* 11: downsample(1, fd) */
    if (upto >= 11 && o->fd > 1) {
        launch_chained(k_rp_fsum, dim3(nblk(maxelem(), 256), NB), 256, 0, st, buf[cur], buf[cur ^ 1], dmeta, o->fd);
        RP_TRY(cudaGetLastError());
        cur ^= 1;
        for (auto &h : H) {
            const int nc = h.nchan / o->fd;
            std::vector<double> fn(nc, 0.);
            for (int j = 0; j < nc; j++) {
                for (int jj = 0; jj < o->fd; jj++) fn[j] += h.f[j * o->fd + jj];
                fn[j] /= o->fd;
            }
            h.f.swap(fn);
            h.nchan = nc;
        }
        RP_TRY(push_meta());
    }
    /* 12: optimize + matched_filter, or peak_search */
    std::vector<RpBest> best(n);
    long hsize = 0, nrows = 0;
    std::vector<int> rows_h(n, 1);
    float *hb[2] = {nullptr, nullptr}, *dsnr = nullptr, *csump = nullptr, *dvwn = nullptr;
    int *dwidm = nullptr, *drows = nullptr, *dnbox = nullptr;
    if (upto >= 12) {
        std::vector<int> shifts, hranges, flip(n, 0);
        for (long b = 0; b < n; b++) {
            RpHost &h = H[b];
            h.hoff = hsize;
            if (!o->nopt) {
                const double fmx = *std::max_element(h.f.begin(), h.f.end());
                const double fmn = *std::min_element(h.f.begin(), h.f.end());
                const double tmp = rp_dmdelay(1., fmx, fmn);
                const double dmrange = (h.nbin * h.tbin) / tmp;
                h.dms = std::max(0., h.dm - dmrange / 2.);
                const double dme = h.dm + dmrange / 2.;
                h.nchans = (int)std::pow(2, std::ceil(std::log2(h.nchan)));
                h.levels = (int)std::log2(h.nchans);
                h.ddm = (dme - h.dms) / h.nchans;
                std::vector<double> fP(h.nchans, 0.);
                const double foff = h.f[1] - h.f[0];
                if (foff < 0.) {
                    for (int j = 0; j < h.nchan; j++) fP[j] = h.f[j];
                    for (int j = h.nchan; j < h.nchans; j++) fP[j] = h.f[0] + j * foff;
                } else {
                    flip[b] = 1;
                    for (int j = 0; j < h.nchan; j++) fP[j] = h.f[h.nchan - 1 - j];
                    for (int j = h.nchan; j < h.nchans; j++) fP[j] = h.f[0] + (h.nchan - 1 - j) * foff;
                }
                const double dms = h.dms, ddm = h.ddm, dm = h.dm, tbin = h.tbin;
                std::function<int(int, int, int)> gs = [&](int x0, int x1, int p) {
                    return (int)std::round(rp_dmdelay(dms + p * ddm - dm, fP[x0], fP[x1]) / tbin);
                };
                std::vector<std::vector<int>> plan;
                std::vector<int> hr;
                rp_shiftplan(plan, hr, h.nchans, (int)h.nbin, gs);
                h.soff = (long)shifts.size();
                for (auto &lv : plan) shifts.insert(shifts.end(), lv.begin(), lv.end());
                h.roff = (long)hranges.size();
                hranges.insert(hranges.end(), hr.begin(), hr.end());
                h.rows = h.nchans;
            } else {
                h.nchans = 1;
                h.levels = 0;
                h.rows = 1;
                h.dms = h.dm;
                h.ddm = 0.;
            }
            rows_h[b] = (int)h.rows;
            h.rowoff = nrows;
            nrows += h.rows;
            hsize += h.rows * h.nbin;
        }
        int *dshift, *dhr, *dflip;
        RP_TRY(mem.alloc(&hb[0], hsize));
        RP_TRY(mem.alloc(&hb[1], hsize));
        RP_TRY(mem.alloc(&dsnr, hsize));
        RP_TRY(mem.alloc(&dwidm, hsize));
        RP_TRY(mem.alloc(&csump, 2 * hsize));
        RP_TRY(mem.alloc(&dshift, shifts.size()));
        RP_TRY(mem.alloc(&dhr, hranges.size()));
        RP_TRY(mem.alloc(&dflip, n));
        RP_TRY(mem.alloc(&drows, n));
        RP_TRY(push_meta());
        if (!shifts.empty())
            RP_TRY(cudaMemcpyAsync(dshift, shifts.data(), sizeof(int) * shifts.size(), cudaMemcpyHostToDevice, st));
        if (!hranges.empty())
            RP_TRY(cudaMemcpyAsync(dhr, hranges.data(), sizeof(int) * hranges.size(), cudaMemcpyHostToDevice, st));
        RP_TRY(cudaMemcpyAsync(dflip, flip.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
        RP_TRY(cudaMemcpyAsync(drows, rows_h.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
        int hc = 0; /* which of hb holds the rows the boxcar reads */
        int maxlevels = 0;
        for (auto &h : H) maxlevels = std::max(maxlevels, h.levels);
        const int maxrows = *std::max_element(rows_h.begin(), rows_h.end());
        if (!o->nopt) {
            for (int t = 0; t < maxlevels; t++) {
                launch_chained(k_rp_hough_level, dim3(maxrows, NB), 256, 0, st, buf[cur], hb[hc], hb[hc ^ 1], dmeta, dshift, dhr,
                                                                   dflip, t);
                hc ^= 1;
            }
        } else {
            launch_chained(k_rp_profile, dim3(nblk(maxnbin, 128), NB), 128, 0, st, buf[cur], hb[0], dmeta);
        }
        RP_TRY(cudaGetLastError());
        /* boxcar width ladder of matched_filter / peak_search (:979-993), a float vector */
        const float wfactor = (float)(1. / ((1. - o->snrloss) * (1. - o->snrloss)));
        long wstride = 1;
        std::vector<std::vector<float>> lads(n);
        for (long b = 0; b < n; b++) {
            std::vector<float> &v = lads[b];
            v.push_back(1);
            while (true) {
                int w1 = (int)v.back();
                int w2 = (int)(w1 * wfactor);
                w2 = w2 < w1 + 1 ? w1 + 1 : w2;
                if (w2 > H[b].nbin / 2) break;
                v.push_back((float)w2);
            }
            wstride = std::max(wstride, (long)v.size());
        }
        std::vector<float> lad_h((size_t)n * wstride, 0.f);
        std::vector<int> nbox_h(n);
        for (long b = 0; b < n; b++) {
            std::copy(lads[b].begin(), lads[b].end(), lad_h.begin() + b * wstride);
            nbox_h[b] = (int)lads[b].size();
        }
        RP_TRY(mem.alloc(&dvwn, lad_h.size()));
        RP_TRY(mem.alloc(&dnbox, n));
        RP_TRY(cudaMemcpyAsync(dvwn, lad_h.data(), sizeof(float) * lad_h.size(), cudaMemcpyHostToDevice, st));
        RP_TRY(cudaMemcpyAsync(dnbox, nbox_h.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
        double *dvar;
        RpBest *drbest, *dbest;
        RP_TRY(mem.alloc(&dvar, nrows));
        RP_TRY(mem.alloc(&drbest, nrows));
        RP_TRY(mem.alloc(&dbest, n));
        launch_chained(k_rp_csum, dim3(per32(maxrows), NB), RP_THREADS, 0, st, hb[hc], dmeta, drows, dvar, csump);
        launch_chained(k_rp_match, dim3(maxrows, NB), 256, 0, st, dmeta, drows, dvwn, dnbox, wstride, dvar, csump, dsnr, dwidm,
                                                     drbest);
        launch_chained(k_rp_best, NB, 256, 0, st, dmeta, drows, drbest, dbest);
        RP_TRY(cudaGetLastError());
        RP_TRY(cudaMemcpyAsync(best.data(), dbest, sizeof(RpBest) * n, cudaMemcpyDeviceToHost, st));
        RP_TRY(cudaStreamSynchronize(st));
        for (long b = 0; b < n; b++) {
            const RpHost &h = H[b];
            const long maxdmid = best[b].idx / h.nbin, maxtid = best[b].idx % h.nbin;
            out[b].snr = best[b].S;
            out[b].width = (float)(best[b].wn * h.tbin);
            out[b].dm_maxsnr = o->nopt ? h.dm : h.dms + maxdmid * h.ddm;
            out[b].maxtid = maxtid;
            out[b].ndm = (int)h.rows;
            out[b].dms = h.dms;
            out[b].ddm = h.ddm;
        }
        if (snrmap) {
            long pos = 0;
            for (long b = 0; b < n && pos < snrmap_cap; b++) {
                const long cnt = std::min(H[b].rows * H[b].nbin, (long)snrmap_cap - pos);
                RP_TRY(copy_out(snrmap + pos, dsnr + H[b].hoff, sizeof(float) * cnt));
                pos += cnt;
            }
        }
    }
    for (long b = 0; b < n; b++) {
        out[b].nbin = H[b].nbin;
        out[b].nchan = H[b].nchan;
        if (upto < 12) {
            out[b].snr = 0.f;
            out[b].width = 0.f;
            out[b].dm_maxsnr = 0.;
            out[b].maxtid = 0;
            out[b].ndm = 0;
            out[b].dms = out[b].ddm = 0.;
        }
    }
    if (data_out) {
        RP_TRY(cudaStreamSynchronize(st));
        long pos = 0;
        for (long b = 0; b < n && pos < data_cap; b++) {
            const RpHost &h = H[b];
            const long cnt = std::min((long)h.nchan * h.nbin, (long)data_cap - pos);
            RP_TRY(cudaMemcpy2D(data_out + pos, sizeof(float) * h.nbin, buf[cur] + h.off, sizeof(float) * h.pitch,
                                sizeof(float) * h.nbin, (size_t)(cnt / h.nbin), cudaMemcpyDeviceToHost));
            pos += cnt;
        }
    }
    RP_TRY(cudaStreamSynchronize(st));
#undef RP_TRY
    return TXG_OK;
}
