/*
 * txg_dedisp.cu -- two-stage subband dedispersion (the RealTime::SubbandDedispersion role,
 * call sites singlepulse.cpp:230-238,328,338 and boxcar.cpp:183).
 *
 * Stage 1: for subband s, coarse-DM group g and new output time t
 *     sub[g][s][t] = sum_{j in s, ascending} x_j[t + d1[g][j]]
 * written into a per-(g,s) ring of modulus R (time index t mod R), stored as T
 * (float, bf16 or half; accumulation is always FP32).
 * Stage 2: for fine DM k of group g and output sample i of the gated block
 *     tim[k][i] = sum_{s ascending} sub[g][s][t0 + i + d2[k][s]].
 *
 * By default stage 1 copies a subband's channel windows to shared memory with cp.async and from
 * there, as lanes of sixteen samples, to tensor memory, from which the sums are read at any column
 * (k_stage1t).  Its other shapes and stage 2 stage their input windows in shared memory with the
 * bulk-copy engine (cp.async.bulk global->shared, completion tracked by an mbarrier with a bounded
 * wait): one window per channel row (stage 1) or per subband ring segment (stage 2), so each
 * input element crosses HBM/L2 once per CTA tile.  A wait that runs out sets *err and the
 * CTA returns without touching its outputs.
 */
#include <algorithm>
#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "txg_device.cuh"
#include "txg_internal.h"

namespace txg {

namespace {

/* ---- storage conversions -------------------------------------------------------------- */
template <typename T> __device__ __forceinline__ T to_store(float v);
template <> __device__ __forceinline__ float to_store<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 to_store<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half to_store<__half>(float v) { return __float2half_rn(v); }
__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }

/* ---- bulk copy + mbarrier helpers (PTX) ------------------------------------------------ */
__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

/* Orders earlier generic-proxy accesses of shared memory before later bulk copies into it. */
__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

/* 4-byte asynchronous global->shared copies (completion per thread by group). */
__device__ __forceinline__ void cp_async4(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
/* the same, 16 bytes (both addresses 16-byte aligned) */
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

/* Nanosecond clock of the GPU. */
__device__ __forceinline__ uint64_t gtimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

/* A window copy lands in microseconds; a wait that has not seen its phase complete after this
 * long gives up (the kernel then reports an error instead of hanging). */
constexpr uint64_t MBAR_LIMIT_NS = 2000000000ull;

/* Bounded wait on phase `parity`: gives up (returns false) after limit_ns of the GPU clock,
 * or after 2^30 polls should that clock not advance. */
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint64_t limit_ns = MBAR_LIMIT_NS)
{
    const uint64_t t0 = gtimer();
    uint32_t done = 0;
    for (long it = 0; it < (1L << 30); it++) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if (gtimer() - t0 > limit_ns) return false;
    }
    return false;
}

/* ---- stage 1 ---------------------------------------------------------------------------- */
constexpr int S1_THREADS = 128;
constexpr int S1_U = 2;                       /* samples per thread */
constexpr int S1_TT = S1_THREADS * S1_U;      /* samples per CTA */
constexpr int S1_GPC = 16;                    /* coarse-DM groups per CTA */

/* grid: x = time tiles, y = subband, z = group chunks.  xh points at buffer column 0; output
 * sample u of channel j reads column u + col0 + d1[g][j].  Shared memory: channel windows
 * [cj][wmax] floats followed by the chunk's d1 [cj][S1_GPC]. */
template <typename T>
__global__ void __launch_bounds__(S1_THREADS)
k_stage1(const float *__restrict__ xh, long ldh, long col0, int C, long N, int nsub, int ng,
         const int32_t *__restrict__ sub_start, const int32_t *__restrict__ d1, int cj,
         long wmax, T *__restrict__ ring, long R, long tbase_mod, int *err)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int span_sh;
    float *win = reinterpret_cast<float *>(smraw);
    const int s = blockIdx.y;
    const long u0 = (long)blockIdx.x * S1_TT;
    const int g0 = blockIdx.z * S1_GPC;
    const int gn = min(S1_GPC, ng - g0);
    const int j0 = sub_start[s], j1 = sub_start[s + 1];
    int32_t *dsm = reinterpret_cast<int32_t *>(win + (size_t)cj * wmax);
    const int tid = threadIdx.x;
    /* copies start on a 16-byte boundary; al = elements skipped in front */
    const long cstart = (u0 + col0) & ~3L;
    const int al = (int)(u0 + col0 - cstart);

    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();

    float acc[S1_GPC][S1_U];
#pragma unroll
    for (int g = 0; g < S1_GPC; g++)
#pragma unroll
        for (int q = 0; q < S1_U; q++) acc[g][q] = 0.f;

    uint32_t phase = 0;
    for (int jc = j0; jc < j1; jc += cj) {
        const int jn = min(cj, j1 - jc);
        /* window span: the largest delay of the chunk's channels in the last group */
        if (tid == 0) span_sh = 0;
        __syncthreads();
        for (int jj = tid; jj < jn; jj += S1_THREADS)
            atomicMax(&span_sh, d1[(size_t)(g0 + gn - 1) * C + jc + jj]);
        for (int e = tid; e < jn * S1_GPC; e += S1_THREADS) {
            int jj = e / S1_GPC, g = e % S1_GPC;
            dsm[e] = g < gn ? d1[(size_t)(g0 + g) * C + jc + jj] : 0;
        }
        __syncthreads();
        const long W = ((long)S1_TT + span_sh + al + 3) / 4 * 4; /* <= wmax */
        if (tid == 0) {
            const uint32_t bytes = (uint32_t)(W * sizeof(float));
            fence_proxy_async();
            mbar_expect_tx(&bar, bytes * (uint32_t)jn);
            for (int jj = 0; jj < jn; jj++)
                bulk_g2s(win + (size_t)jj * W, xh + (long)(jc + jj) * ldh + cstart, bytes, &bar);
        }
        bool ok = mbar_wait(&bar, phase);
        phase ^= 1;
        if (!__syncthreads_and(ok)) {
            if (tid == 0) atomicExch(err, 1);
            mbar_wait(&bar, phase ^ 1); /* let copies still in flight land (bounded) */
            return;
        }
        for (int jj = 0; jj < jn; jj++) {
            const float *wr = win + (size_t)jj * W + al + tid;
            const int4 *dv = reinterpret_cast<const int4 *>(dsm + jj * S1_GPC);
#pragma unroll
            for (int gq = 0; gq < S1_GPC / 4; gq++) {
                const int4 d = dv[gq];
                const int dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (int r = 0; r < 4; r++)
#pragma unroll
                    for (int q = 0; q < S1_U; q++)
                        acc[gq * 4 + r][q] =
                            __fadd_rn(acc[gq * 4 + r][q], wr[dd[r] + q * S1_THREADS]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int g = 0; g < S1_GPC; g++) {
        if (g < gn) {
            T *out = ring + ((size_t)(g0 + g) * nsub + s) * R;
#pragma unroll
            for (int q = 0; q < S1_U; q++) {
                long u = u0 + tid + q * S1_THREADS;
                if (u < N) {
                    long t = tbase_mod + u;
                    t = t >= R ? t - R : t;
                    out[t] = to_store<T>(acc[g][q]);
                }
            }
        }
    }
}

/* Stage 1 with the subband's whole channel window resident in shared memory: one CTA per
 * (TH*U-sample tile, subband) loads every channel row of the subband once (so each input
 * element crosses HBM once per tile) and then walks all coarse-DM groups, GS*GPT at a time:
 * the CTA's GS thread sets share the window and take GPT groups each.  Each output adds its
 * channels in ascending order from 0.0f. */
template <typename T, int TH, int U, int GS, int GPT>
__global__ void __launch_bounds__(TH * GS)
k_stage1r(const float *__restrict__ xh, long ldh, long col0, int C, long N, int nsub, int ng,
          const int32_t *__restrict__ sub_start, const int32_t *__restrict__ d1, long wmax,
          int maxch, T *__restrict__ ring, long R, long tbase_mod, int *err)
{
    constexpr int NT = TH * GS, TT = TH * U, GPC = GS * GPT;
    static_assert(GPT % 4 == 0, "delays are read four at a time");
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int span_sh;
    float *win = reinterpret_cast<float *>(smraw);
    int32_t *dsm = reinterpret_cast<int32_t *>(win + (size_t)maxch * wmax); /* 2 x [maxch][GPC] */
    const int s = blockIdx.y;
    const long u0 = (long)blockIdx.x * TT;
    const int j0 = sub_start[s], j1 = sub_start[s + 1], jn = j1 - j0;
    const int tid = threadIdx.x, lt = tid % TH, gs = tid / TH;
    const long cstart = (u0 + col0) & ~3L;
    const int al = (int)(u0 + col0 - cstart);
    const int nch = (ng + GPC - 1) / GPC;
    /* delays of chunk c (groups past the end repeat the last one) into table buffer c & 1 */
    auto fetch = [&](int c) {
        if (c < nch) {
            const int g0 = c * GPC, gn = min(GPC, ng - g0);
            int32_t *dt = dsm + (size_t)(c & 1) * maxch * GPC;
#pragma unroll 1
            for (int e = tid; e < jn * GPC; e += NT) {
                const int jj = e / GPC, g = e % GPC;
                cp_async4(&dt[e], &d1[(size_t)(g0 + (g < gn ? g : gn - 1)) * C + j0 + jj]);
            }
        }
        cp_async_commit();
    };

    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        span_sh = 0;
    }
    fetch(0);
    __syncthreads();
    for (int jj = tid; jj < jn; jj += NT) atomicMax(&span_sh, d1[(size_t)(ng - 1) * C + j0 + jj]);
    __syncthreads();
    const long W = ((long)TT + span_sh + al + 3) / 4 * 4; /* <= wmax */
    if (tid == 0) {
        const uint32_t bytes = (uint32_t)(W * sizeof(float));
        mbar_expect_tx(&bar, bytes * (uint32_t)jn);
        for (int jj = 0; jj < jn; jj++)
            bulk_g2s(win + (size_t)jj * W, xh + (long)(j0 + jj) * ldh + cstart, bytes, &bar);
    }
    const bool ok = mbar_wait(&bar, 0);
    if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicExch(err, 1);
        mbar_wait(&bar, 0);
        cp_async_wait_all();
        return;
    }
    for (int c = 0; c < nch; c++) {
        const int g0 = c * GPC, gn = min(GPC, ng - g0);
        cp_async_wait_all(); /* this thread's copies of chunk c */
        __syncthreads();     /* everyone's; and buffer (c+1)&1 is no longer read */
        fetch(c + 1);        /* overlaps this chunk's sums */
        const int32_t *dtab = dsm + (size_t)(c & 1) * maxch * GPC;
        /* the thread's samples in pairs (q, q + 1): one packed FP32 add (add.rn.f32x2, each
         * half rounded as __fadd_rn) serves two samples of a group */
        constexpr int UH = (U + 1) / 2;
        float2 acc[GPT][UH];
#pragma unroll
        for (int g = 0; g < GPT; g++)
#pragma unroll
            for (int q = 0; q < UH; q++) acc[g][q] = make_float2(0.f, 0.f);
        for (int jj = 0; jj < jn; jj++) {
            const float *wr = win + (size_t)jj * W + al + lt;
            const int4 *dv = reinterpret_cast<const int4 *>(dtab + jj * GPC + gs * GPT);
            int dd[GPT];
#pragma unroll
            for (int gq = 0; gq < GPT / 4; gq++) {
                const int4 d = dv[gq];
                dd[4 * gq] = d.x;
                dd[4 * gq + 1] = d.y;
                dd[4 * gq + 2] = d.z;
                dd[4 * gq + 3] = d.w;
            }
            /* neighbouring coarse-DM groups often share a channel's delay (it moves by a
             * third of a sample per group on average): the window values are loaded again only
             * where the delay changes (a branch uniform over the thread set) */
            float2 v[UH];
#pragma unroll
            for (int g = 0; g < GPT; g++) {
                if (g == 0 || dd[g] != dd[g - 1]) {
#pragma unroll
                    for (int q = 0; q < UH; q++) {
                        v[q].x = wr[dd[g] + 2 * q * TH];
                        v[q].y = 2 * q + 1 < U ? wr[dd[g] + (2 * q + 1) * TH] : 0.f;
                    }
                }
#pragma unroll
                for (int q = 0; q < UH; q++) {
                    if (2 * q + 1 < U)
                        acc[g][q] = __fadd2_rn(acc[g][q], v[q]);
                    else
                        acc[g][q].x = __fadd_rn(acc[g][q].x, v[q].x);
                }
            }
        }
#pragma unroll
        for (int g = 0; g < GPT; g++) {
            const int gc = gs * GPT + g;
            if (gc < gn) {
                T *out = ring + ((size_t)(g0 + gc) * nsub + s) * R;
#pragma unroll
                for (int q = 0; q < U; q++) {
                    const long u = u0 + lt + q * TH;
                    if (u < N) {
                        long t = tbase_mod + u;
                        t = t >= R ? t - R : t;
                        out[t] = to_store<T>((q & 1) ? acc[g][q / 2].y : acc[g][q / 2].x);
                    }
                }
            }
        }
    }
}

/* ---- tensor memory as a file of shiftable windows ------------------------------------------ */
/* A dedispersion sum reads one window at many offsets: each (channel, delay) pair adds the same
 * samples, shifted.  Read from shared memory that is one 4-byte word per addition, or per
 * distinct delay, and the 128 bytes a clock of that pipe bound the kernel at a quarter of the
 * FP32 add rate.  Tensor memory gives each of an SM's four schedulers 128 bytes a clock of its
 * own, and one tcgen05.ld.32x32b.x16 reads 16 consecutive columns from any start column into
 * every lane's registers: with consecutive samples of a lane in consecutive columns, a shift
 * by d samples is a start column d further on, costs one instruction for 512 samples and
 * leaves them aligned for the packed add.  Measured on the GB300 with 16 warps per SM: 12.4
 * clocks per x16 load and scheduler, load and eight packed adds together at 0.76 of the add
 * rate (0.58 with the windows' filling beside them). */
__device__ __forceinline__ void tm_alloc(uint32_t *slot, int cols) /* one warp */
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tm_free(uint32_t t, int cols) /* the same warp */
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t), "r"(cols));
}
__device__ __forceinline__ void tm_ld16(uint32_t (&r)[16], uint32_t t)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                 "%13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15])
                 : "r"(t)
                 : "memory");
}
__device__ __forceinline__ void tm_st8(uint32_t t, const float (&v)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t),
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tm_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
/* The 160 threads whose warps share a scheduler (and with it 32 lanes of tensor memory) meet:
 * what any of them stored is there for the others' loads, and their loads are done. */
__device__ __forceinline__ void tm_team_sync(int team)
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync %0, 160;" ::"r"(team + 1) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
/* acc[q] += the pair of samples (2q, 2q + 1) of a loaded window */
__device__ __forceinline__ void tm_acc(float2 (&acc)[8], const uint32_t (&r)[16])
{
#pragma unroll
    for (int q = 0; q < 8; q++)
        acc[q] = __fadd2_rn(acc[q], make_float2(__uint_as_float(r[2 * q]), __uint_as_float(r[2 * q + 1])));
}
/* Sixteen consecutive samples to 64-byte (float) or 32-byte (16-bit) aligned memory. */
__device__ __forceinline__ void store16(float *o, const float2 (&a)[8])
{
#pragma unroll
    for (int q = 0; q < 4; q++)
        reinterpret_cast<float4 *>(o)[q] = make_float4(a[2 * q].x, a[2 * q].y, a[2 * q + 1].x, a[2 * q + 1].y);
}
__device__ __forceinline__ uint32_t pack2(float2 v, __half *)
{
    const __half2 h = __floats2half2_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack2(float2 v, __nv_bfloat16 *)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t *>(&h);
}
template <typename T> __device__ __forceinline__ void store16(T *o, const float2 (&a)[8])
{
#pragma unroll
    for (int q = 0; q < 2; q++)
        reinterpret_cast<uint4 *>(o)[q] = make_uint4(pack2(a[4 * q], o), pack2(a[4 * q + 1], o),
                                                     pack2(a[4 * q + 2], o), pack2(a[4 * q + 3], o));
}

/* ---- stage 1 from tensor memory ----------------------------------------------------------- */
/* CTA = (512-sample tile, subband).  Lane l of every warp owns samples 16l .. 16l+15 of the tile; a
 * warp that adds has four consecutive coarse-DM groups (a quad), and the four such warps of a
 * scheduler (a team) take consecutive quads.  The subband's channel windows are copied into
 * shared memory once (one word of padding per 16, so that the lanes' starts fall in different
 * banks) and stay while the teams walk all passes of up to 64 groups, each at its own pace.
 * Per pass and block of `nb` channels the team's fifth warp, one block ahead, copies the piece
 * of each channel that the team's quads need (16 samples and the spread of their delays) into
 * the team's columns; the others add it at their groups' offsets.  A group with its
 * neighbour's delay adds the values that are still in registers (two thirds of the steps
 * between groups are 0 in the searches' plans).
 *
 * 1024 channels, 256 groups, 13156 samples, 16-bit subbands: 433 us with the best shared-memory
 * shape below, 286 us so; 4096 channels and the searches' three rows, per row: 917 us and 785.
 * Issue and latency bound it (2.1 of 4 instructions a clock, FP32 adds a third of them; 86
 * registers leave five warps a scheduler).  Measured and not kept: the quads' common prefixes of
 * equal delays summed once (a quarter fewer additions, but more branches and register moves:
 * 346 us), one load per group without the branches (294 us), two loads in flight (293 us), loads
 * one ahead (298 us), two groups a warp at eight warps a scheduler (342 us), the adding warps
 * also filling (297 us). */
constexpr int S1T_TT = 512;    /* samples per CTA */
constexpr int S1T_THREADS = 640; /* 16 warps that add and 4 that fill */
constexpr int S1T_COLS = 256;  /* columns of one of the two window buffers */
constexpr int S1T_PASS = 64;   /* table entries (groups) per pass */
/* words of a channel window beside its subband's largest delay: the tile and the rest of the
 * last eight columns that a fill writes */
constexpr int S1T_HALO = S1T_TT + 8;
static_assert(S1T_TT == 32 * 16, "a lane holds 16 samples");

/* rel: [channel][pass][64] column offsets from the set's window start; first: [channel][pass][4]
 * that start, the delay of the set's first group rounded down to 8 (so that eight columns never
 * straddle a padding word).  qpt: quads per team.  span: the largest delay of each subband. */
template <typename T>
__global__ void __launch_bounds__(S1T_THREADS, 1)
k_stage1t(const float *__restrict__ xh, long ldh, long col0, int C, long N, int nsub, int ng,
          const int32_t *__restrict__ sub_start, const uint16_t *__restrict__ rel,
          const int32_t *__restrict__ first, int npass, int qpt, int cw, int nb,
          const int32_t *__restrict__ span, int maxch, T *__restrict__ ring, long R, long tbase_mod)
{
    chain_wait();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ uint32_t tm_slot;
    /* the shuffle tells the compiler that all of a warp has the same wp */
    const int tid = threadIdx.x, lane = tid & 31, wp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int team = wp & 3, m = wp >> 2;
    /* tables [channel][pass] x (64 offsets, 4 window starts), then the channel windows */
    uint2 *rel_sm = reinterpret_cast<uint2 *>(smraw);
    int32_t *first_sm = reinterpret_cast<int32_t *>(rel_sm + (size_t)maxch * npass * 16);
    float *win = reinterpret_cast<float *>(first_sm + (size_t)maxch * npass * 4);
    const int words = S1T_HALO + span[blockIdx.y], pitch = words + (words >> 4) + 1;
    const int s = blockIdx.y, j0 = sub_start[s], jn = sub_start[s + 1] - j0;
    /* tiles start where the ring index is a multiple of 16, so that a lane's samples are one
     * aligned piece of the ring; samples before 0 are not stored */
    const long u0 = (long)blockIdx.x * S1T_TT - (tbase_mod & 15);

    if (wp == 0) tm_alloc(&tm_slot, 2 * S1T_COLS);
    for (int e = tid; e < jn * npass * 8; e += S1T_THREADS) /* 16 bytes each */
        cp_async16(rel_sm + 2 * e, rel + (size_t)j0 * npass * S1T_PASS + 8 * e);
    for (int e = tid; e < jn * npass; e += S1T_THREADS)
        cp_async16(first_sm + 4 * e, first + (size_t)j0 * npass * 4 + 4 * e);
    for (int jj = wp; jj < jn; jj += S1T_THREADS / 32) {
        float *d = win + (size_t)jj * pitch;
        const float *x = xh + (long)(j0 + jj) * ldh;
        const long c0 = u0 + col0; /* columns before the buffer hold no stored sample */
        int n = lane;
        for (; n < words && c0 + n < 0; n += 32) d[n + (n >> 4)] = 0.f;
        x += c0;
#pragma unroll 4
        for (; n < words; n += 32) cp_async4(d + n + (n >> 4), x + n);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm = tm_slot + ((uint32_t)(32 * team) << 16);
    const int nblk = (jn + nb - 1) / nb;
    /* passes in which the team has groups; its steps are (pass, block of channels) */
    int mypass = 0;
    while (mypass < npass && (mypass * 4 + team) * qpt * 4 < ng) mypass++;
    const int nstep = mypass * nblk;

    if (m == 4) { /* the team's filling warp: the windows of a step's channels */
        const float *lane_win = win + 17 * lane;
        const int32_t *fp = first_sm + team;
        /* the set's last group, the furthest, in the upper half */
        const uint32_t *lp = reinterpret_cast<const uint32_t *>(rel_sm) + team * 8 + 2 * qpt - 1;
        int n0 = *fp;
        uint32_t last = *lp;
        for (int i = 0, ps = 0, b = 0; i < nstep; i++) {
            const int j1 = b * nb, je = min(jn, j1 + nb);
            uint32_t t = tm + (i & 1) * S1T_COLS;
            const float *row = lane_win + j1 * pitch;
            b = b + 1 < nblk ? b + 1 : 0;
            const int pn = b ? ps : ps + 1;
            for (int jj = j1; jj < je; jj++, t += cw, row += pitch) {
                /* 16 samples and the spread of the set's delays; n0 is a multiple of 8: a padding
                 * word before every other eight */
                const int wcols = 16 + (int)(last >> 16);
                const float *x = row + n0 + (n0 >> 4), *y = x + (n0 >> 3 & 1), *z = x + 17;
                float v[24];
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = x[q];
#pragma unroll
                for (int q = 0; q < 8; q++) v[8 + q] = y[8 + q];
#pragma unroll
                for (int q = 0; q < 8; q++) v[16 + q] = z[q];
                const int odd = n0 & 8;
                { /* the next channel's table entries */
                    const int jx = jj + 1 < je ? jj + 1 : b * nb, px = jj + 1 < je ? ps : min(pn, npass - 1);
                    n0 = fp[(jx * npass + px) * 4];
                    last = lp[(jx * npass + px) * 32];
                }
                tm_st8(t, *reinterpret_cast<float(*)[8]>(v));
                tm_st8(t + 8, *reinterpret_cast<float(*)[8]>(v + 8));
                tm_st8(t + 16, *reinterpret_cast<float(*)[8]>(v + 16));
                for (int c = 24; c < wcols; c += 8) {
                    const float *w = x + c + ((odd + c) >> 4);
                    float u[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) u[q] = w[q];
                    tm_st8(t + c, u);
                }
            }
            ps = pn;
            tm_wait_st();
            tm_team_sync(team);
        }
    } else {
        int i = 0;
        for (int ps = 0; ps < mypass; ps++) {
            const int quad = (ps * 4 + team) * qpt + m;
            const bool mine = m < qpt && 4 * quad < ng;
            float2 acc[4][8];
#pragma unroll
            for (int g = 0; g < 4; g++)
#pragma unroll
                for (int q = 0; q < 8; q++) acc[g][q] = make_float2(0.f, 0.f);
            const uint2 *r = rel_sm + ps * 16 + team * 4 + m;
            for (int j0b = 0; j0b < jn; j0b += nb) {
                tm_team_sync(team); /* the block's windows are there, the other buffer is read no more */
                uint32_t t = tm + (i++ & 1) * S1T_COLS;
                const int n = min(nb, jn - j0b);
                if (mine) {
                    uint2 w = *r;
                    w.x = __shfl_sync(0xffffffffu, w.x, 0);
                    w.y = __shfl_sync(0xffffffffu, w.y, 0);
#pragma unroll 1
                    for (int k = 0; k < n; k++, t += cw) {
                        const uint32_t c0 = w.x & 0xffffu, c1 = w.x >> 16, c2 = w.y & 0xffffu, c3 = w.y >> 16;
                        r += npass * 16;
                        if (k + 1 < n) w = *r;
                        uint32_t v[16];
                        tm_ld16(v, t + c0);
                        w.x = __shfl_sync(0xffffffffu, w.x, 0);
                        w.y = __shfl_sync(0xffffffffu, w.y, 0);
                        tm_wait_ld();
                        tm_acc(acc[0], v);
                        if (c1 != c0) {
                            tm_ld16(v, t + c1);
                            tm_wait_ld();
                        }
                        tm_acc(acc[1], v);
                        if (c2 != c1) {
                            tm_ld16(v, t + c2);
                            tm_wait_ld();
                        }
                        tm_acc(acc[2], v);
                        if (c3 != c2) {
                            tm_ld16(v, t + c3);
                            tm_wait_ld();
                        }
                        tm_acc(acc[3], v);
                    }
                }
            }
            if (mine) {
                const long u = u0 + 16 * lane;
                long tr = tbase_mod + u;
                tr = tr >= R ? tr - R : tr;
                T *o = ring + ((size_t)(4 * quad) * nsub + s) * R + tr;
                /* samples [lo, hi) of the sixteen are the block's */
                const int lo = u < 0 ? (int)-u : 0, hi = u + 16 <= N ? 16 : (int)max(N - u, 0L);
                const bool whole = lo == 0 && hi == 16;
#pragma unroll
                for (int g = 0; g < 4; g++, o += (size_t)nsub * R) {
                    if (4 * quad + g >= ng) break;
                    if (whole) {
                        store16(o, acc[g]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            if (q >= lo && q < hi) o[q] = to_store<T>((q & 1) ? acc[g][q / 2].y : acc[g][q / 2].x);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wp == 0) tm_free(tm_slot, 2 * S1T_COLS);
}

/* ---- 16-bit pairs ---------------------------------------------------------------------- */
/* FP32 += one 16-bit value (exact conversion, one rounding), PTX mixed-precision add. */
__device__ __forceinline__ void addp(float &lo_acc, float &hi_acc, uint32_t v, __half)
{
    asm("{ .reg .b16 l, h; mov.b32 {l, h}, %2; add.rn.f32.f16 %0, l, %0; add.rn.f32.f16 %1, h, %1; }"
        : "+f"(lo_acc), "+f"(hi_acc)
        : "r"(v));
}
__device__ __forceinline__ void addp(float &lo_acc, float &hi_acc, uint32_t v, __nv_bfloat16)
{
    asm("{ .reg .b16 l, h; mov.b32 {l, h}, %2; add.rn.f32.bf16 %0, l, %0; add.rn.f32.bf16 %1, h, %1; }"
        : "+f"(lo_acc), "+f"(hi_acc)
        : "r"(v));
}

/* Odd-aligned pair copy of a 16-bit window: o[k] = (e[2k+1], e[2k+2]) as one word. */
__device__ __forceinline__ void build_odd(const uint32_t *e, uint32_t *o, long nwords, int tid, int nth)
{
    for (int k = tid; k < nwords / 4; k += nth) {
        const uint4 v = reinterpret_cast<const uint4 *>(e)[k];
        const uint32_t n = e[4 * k + 4];
        reinterpret_cast<uint4 *>(o)[k] = make_uint4(__byte_perm(v.x, v.y, 0x5432), __byte_perm(v.y, v.z, 0x5432),
                                                     __byte_perm(v.z, v.w, 0x5432), __byte_perm(v.w, n, 0x5432));
    }
}

/* ---- stage 2 ---------------------------------------------------------------------------- */
constexpr int S2_THREADS = 128;
constexpr int S2_U = 2;                  /* samples per thread */
constexpr int S2_TT = S2_THREADS * S2_U;

/* grid: x = time tiles, y = (group, DM chunk of KPC); TH threads take U samples each of the
 * S2_TT-sample tile.  Shared memory: for a chunk of `sc`
 * subbands their ring windows (each S2_TT + d2[klast][s] - d2[kfirst][s] plus alignment),
 * then the d2 offsets [sc][KPC] and the window bookkeeping.  Each output adds its subbands
 * in ascending order from 0.0f. */
template <typename T, int KPC, int TH, int U>
__global__ void __launch_bounds__(TH)
k_stage2(const T *__restrict__ ring, long R, int nsub, int G, long ndm, long nout,
         const int32_t *__restrict__ d2, long t0_mod, int sc, long wtot_max,
         float *__restrict__ tim, long ldt, int *err)
{
    chain_wait();
    static_assert(TH * U == S2_TT && TH >= 32, "the tile is S2_TT samples");
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    T *win = reinterpret_cast<T *>(smraw);
    int32_t *doff = reinterpret_cast<int32_t *>(smraw + ((wtot_max * sizeof(T) + 15) / 16) * 16);
    int32_t *wbeg = doff + sc * KPC;
    int32_t *wts = wbeg + sc, *wal = wts + sc, *wlen = wal + sc, *wpos = wlen + sc;
    const int tid = threadIdx.x;
    const int nkc = (G + KPC - 1) / KPC;
    const int g = blockIdx.y / nkc, kc = blockIdx.y % nkc;
    const long k0 = (long)g * G + (long)kc * KPC;
    const long kend = min((long)(g + 1) * G, ndm);
    const int kn = (int)min((long)KPC, kend - k0);
    if (kn <= 0) return;
    const long u0 = (long)blockIdx.x * S2_TT;

    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();

    float acc[KPC][U];
#pragma unroll
    for (int k = 0; k < KPC; k++)
#pragma unroll
        for (int q = 0; q < U; q++) acc[k][q] = 0.f;

    uint32_t phase = 0;
    constexpr int EPC = 16 / (int)sizeof(T); /* elements per 16 bytes */
    for (int s0 = 0; s0 < nsub; s0 += sc) {
        const int sn = min(sc, nsub - s0);
        for (int e = tid; e < sn * KPC; e += TH) {
            const int ss = e / KPC, k = e % KPC;
            const int lo = d2[(size_t)k0 * nsub + s0 + ss];
            doff[e] = d2[(size_t)(k0 + (k < kn ? k : kn - 1)) * nsub + s0 + ss] - lo;
        }
        /* window of each subband: ring start rounded down to 16 bytes, length, offset */
        for (int ss = tid; ss < sn; ss += TH) {
            const int s = s0 + ss;
            const long lo = d2[(size_t)k0 * nsub + s];
            const long hi = d2[(size_t)(k0 + kn - 1) * nsub + s];
            long tstart = (t0_mod + u0 + lo) % R;
            const long al = tstart % EPC;
            tstart -= al;
            wts[ss] = (int32_t)tstart;
            wal[ss] = (int32_t)al;
            wlen[ss] = (int32_t)(((long)S2_TT + (hi - lo) + al + EPC - 1) / EPC * EPC);
        }
        __syncthreads();
        if (tid < 32) { /* exclusive prefix of the lengths (one warp) */
            int carry = 0;
            for (int base = 0; base < sn; base += 32) {
                const int ss = base + tid;
                const int v = ss < sn ? wlen[ss] : 0;
                int incl = v;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, incl, off);
                    if (tid >= off) incl += y;
                }
                if (ss < sn) wpos[ss] = carry + incl - v;
                carry += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (tid == 0) {
                fence_proxy_async();
                mbar_expect_tx(&bar, (uint32_t)(carry * (int)sizeof(T)));
            }
        }
        __syncthreads();
        for (int ss = tid; ss < sn; ss += TH) {
            const T *row = ring + ((size_t)g * nsub + s0 + ss) * R;
            const long pos = wpos[ss], len = wlen[ss], tstart = wts[ss];
            wbeg[ss] = (int32_t)(pos + wal[ss]);
            /* split at the ring end; R is a multiple of 32 elements and exceeds len, so both
             * parts are whole 16-byte units inside the row */
            const long first = min(len, R - tstart);
            fence_proxy_async();
            bulk_g2s(win + pos, row + tstart, (uint32_t)(first * sizeof(T)), &bar);
            if (first < len)
                bulk_g2s(win + pos + first, row, (uint32_t)((len - first) * sizeof(T)), &bar);
        }
        __syncthreads();
        bool ok = mbar_wait(&bar, phase);
        phase ^= 1;
        if (!__syncthreads_and(ok)) {
            if (tid == 0) atomicExch(err, 2);
            mbar_wait(&bar, phase ^ 1);
            return;
        }
        for (int ss = 0; ss < sn; ss++) {
            const T *wr = win + wbeg[ss] + tid;
            const int4 *dv = reinterpret_cast<const int4 *>(doff + ss * KPC);
            int dd[KPC];
#pragma unroll
            for (int kq = 0; kq < KPC / 4; kq++) {
                const int4 d = dv[kq];
                dd[4 * kq] = d.x;
                dd[4 * kq + 1] = d.y;
                dd[4 * kq + 2] = d.z;
                dd[4 * kq + 3] = d.w;
            }
            /* DMs past the end of a partial group repeat the last offset; their sums are
             * discarded, and no per-DM branch keeps all loads free to issue together */
#pragma unroll
            for (int k = 0; k < KPC; k++)
#pragma unroll
                for (int q = 0; q < U; q++)
                    acc[k][q] = __fadd_rn(acc[k][q], to_f(wr[dd[k] + q * TH]));
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < KPC; k++) {
        if (k < kn) {
#pragma unroll
            for (int q = 0; q < U; q++) {
                const long u = u0 + tid + q * TH;
                if (u < nout) tim[(k0 + k) * ldt + u] = acc[k][q];
            }
        }
    }
}

/* Stage 2 on a 16-bit ring, two consecutive samples per 32-bit shared-memory load: the
 * subband windows are held as even-aligned pairs (bulk copies) and odd-aligned pairs (built
 * in shared memory).  Same order of additions as k_stage2.  An addition takes a 16-bit operand
 * as it is; the instructions beside it bound the kernel (2.6 an addition, with 3 warps a scheduler),
 * so a DM's offset is one of bytes, that one addition brings to the loads' common base, and the odd
 * copies are made from 16-byte words: 823 -> 788 us for 5000 DMs of 128 subbands x 13156
 * samples (bfloat16, 4096 channels), 598 -> 515 for 64 subbands of 1024 channels (float16). */
template <typename T, int KPC, int TH, int UP>
__global__ void __launch_bounds__(TH)
k_stage2p(const T *__restrict__ ring, long R, int nsub, int G, long ndm, long nout,
          const int32_t *__restrict__ d2, long t0_mod, int sc, long wtot_max,
          float *__restrict__ tim, long ldt, int *err)
{
    chain_wait();
    constexpr int TT = 2 * TH * UP;
    static_assert(TT == S2_TT && TH >= 32, "the tile is S2_TT samples");
    constexpr int EPC = 8; /* 16-bit elements per 16 bytes */
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    uint32_t *words = reinterpret_cast<uint32_t *>(smraw);
    T *win = reinterpret_cast<T *>(smraw);
    /* even pairs: wtot_max halves + one pad word; odd pairs: wtot_max/2 words */
    const long ewords = wtot_max / 2 + 4;
    uint32_t *ow = words + ewords;
    int32_t *doff = reinterpret_cast<int32_t *>(ow + wtot_max / 2);
    int32_t *wts = doff + sc * KPC, *wal = wts + sc, *wlen = wal + sc, *wpos = wlen + sc;
    const int tid = threadIdx.x;
    const int nkc = (G + KPC - 1) / KPC;
    const int g = blockIdx.y / nkc, kc = blockIdx.y % nkc;
    const long k0 = (long)g * G + (long)kc * KPC;
    const long kend = min((long)(g + 1) * G, ndm);
    const int kn = (int)min((long)KPC, kend - k0);
    if (kn <= 0) return;
    const long u0 = (long)blockIdx.x * TT;

    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();

    float acc[KPC][2 * UP];
#pragma unroll
    for (int k = 0; k < KPC; k++)
#pragma unroll
        for (int q = 0; q < 2 * UP; q++) acc[k][q] = 0.f;

    uint32_t phase = 0;
    for (int s0 = 0; s0 < nsub; s0 += sc) {
        const int sn = min(sc, nsub - s0);
        /* windows: ring start rounded down to 16 bytes, length covering the last pair */
        for (int ss = tid; ss < sn; ss += TH) {
            const int s = s0 + ss;
            const long lo = d2[(size_t)k0 * nsub + s];
            const long hi = d2[(size_t)(k0 + kn - 1) * nsub + s];
            long tstart = (t0_mod + u0 + lo) % R;
            const long al = tstart % EPC;
            tstart -= al;
            wts[ss] = (int32_t)tstart;
            wal[ss] = (int32_t)al;
            wlen[ss] = (int32_t)(((long)TT + (hi - lo) + al + 2 + EPC - 1) / EPC * EPC);
        }
        __syncthreads();
        if (tid < 32) { /* exclusive prefix of the lengths (one warp) */
            int carry = 0;
            for (int base = 0; base < sn; base += 32) {
                const int ss = base + tid;
                const int v = ss < sn ? wlen[ss] : 0;
                int incl = v;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, incl, off);
                    if (tid >= off) incl += y;
                }
                if (ss < sn) wpos[ss] = carry + incl - v;
                carry += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (tid == 0) {
                fence_proxy_async();
                mbar_expect_tx(&bar, (uint32_t)(carry * (int)sizeof(T)));
            }
        }
        __syncthreads();
        /* byte offsets of each (subband, DM): even or odd copy by the parity */
        for (int e = tid; e < sn * KPC; e += TH) {
            const int ss = e / KPC, k = e % KPC;
            const int lo = d2[(size_t)k0 * nsub + s0 + ss];
            const int h = wpos[ss] + wal[ss] + d2[(size_t)(k0 + (k < kn ? k : kn - 1)) * nsub + s0 + ss] - lo;
            doff[e] = 4 * ((h & 1) ? (int)ewords + h / 2 : h / 2);
        }
        for (int ss = tid; ss < sn; ss += TH) {
            const T *row = ring + ((size_t)g * nsub + s0 + ss) * R;
            const long pos = wpos[ss], len = wlen[ss], tstart = wts[ss];
            const long first = min(len, R - tstart);
            fence_proxy_async();
            bulk_g2s(win + pos, row + tstart, (uint32_t)(first * sizeof(T)), &bar);
            if (first < len)
                bulk_g2s(win + pos + first, row, (uint32_t)((len - first) * sizeof(T)), &bar);
        }
        __syncthreads();
        bool ok = mbar_wait(&bar, phase);
        phase ^= 1;
        if (!__syncthreads_and(ok)) {
            if (tid == 0) atomicExch(err, 2);
            mbar_wait(&bar, phase ^ 1);
            return;
        }
        {
            const long nw = (wpos[sn - 1] + wlen[sn - 1]) / 2;
            build_odd(words, ow, nw, tid, TH);
        }
        __syncthreads();
        const unsigned char *wr = smraw + 4 * tid;
        for (int ss = 0; ss < sn; ss++) {
            const int4 *dv = reinterpret_cast<const int4 *>(doff + ss * KPC);
            int dd[KPC];
#pragma unroll
            for (int kq = 0; kq < KPC / 4; kq++) {
                const int4 d = dv[kq];
                dd[4 * kq] = d.x;
                dd[4 * kq + 1] = d.y;
                dd[4 * kq + 2] = d.z;
                dd[4 * kq + 3] = d.w;
            }
#pragma unroll
            for (int k = 0; k < KPC; k++)
#pragma unroll
                for (int q = 0; q < UP; q++) 
                    addp(acc[k][2 * q], acc[k][2 * q + 1],
                         *reinterpret_cast<const uint32_t *>(wr + dd[k] + 4 * q * TH), T());
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < KPC; k++) {
        if (k < kn) {
#pragma unroll
            for (int q = 0; q < 2 * UP; q++) {
                const long u = u0 + 2 * (tid + (q >> 1) * TH) + (q & 1);
                if (u < nout) tim[(k0 + k) * ldt + u] = acc[k][q];
            }
        }
    }
}

inline unsigned nblk(long n, int b) { return (unsigned)((n + b - 1) / b); }

constexpr size_t SMEM_BUDGET = 100 * 1024;     /* chunked stage 1: two CTAs per SM */
constexpr size_t RESIDENT_BUDGET = 200 * 1024; /* whole-subband stage-1 windows */
constexpr size_t S1T_SMEM = 224 * 1024;        /* k_stage1t: tables and windows */

} // namespace

/* Largest window any stage-1 CTA needs: tile + maxd1 + alignment (delays grow with the
 * group index).  xh points at column 0 of the channel buffer; col0 = H - maxd1.  When the
 * widest subband's full window fits in shared memory the resident kernel reads every channel
 * row once; otherwise the chunked kernel (channel chunks, 16 groups per CTA) is used.  Every
 * precision sums the FP32 block; only the ring's element type differs. */
template <typename T, int TH, int U, int GS, int GPT>
static bool stage1r_try(const float *xh, long ldh, long col0, int C, long N, int nsub, int ng,
                        const int32_t *sub_start, const int32_t *d1, long maxd1, int maxch, T *ring,
                        long R, long tbase_mod, int *err, cudaStream_t st)
{
    const long tt = (long)TH * U;
    const long wr = (tt + maxd1 + 3 + 3) / 4 * 4;
    const size_t smem = (size_t)maxch * wr * sizeof(float) + 2 * (size_t)maxch * GS * GPT * sizeof(int32_t);
    if (smem > RESIDENT_BUDGET) return false;
    auto kern = k_stage1r<T, TH, U, GS, GPT>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<dim3(nblk(N, (int)tt), nsub), TH * GS, smem, st>>>(xh, ldh, col0, C, N, nsub, ng, sub_start,
                                                              d1, wr, maxch, ring, R, tbase_mod, err);
    return true;
}

template <typename T>
static void stage1_chunked(const float *xh, long ldh, long col0, int C, long N, int nsub, int ng,
                           const int32_t *sub_start, const int32_t *d1, long maxd1, int maxch,
                           T *ring, long R, long tbase_mod, int *err, cudaStream_t st)
{
    long wmax = ((long)S1_TT + maxd1 + 3 + 3) / 4 * 4;
    size_t per = wmax * sizeof(float) + S1_GPC * sizeof(int32_t);
    int cj = (int)((SMEM_BUDGET - 64) / per);
    if (cj > maxch) cj = maxch;
    if (cj < 1) cj = 1;
    size_t smem = (size_t)cj * wmax * sizeof(float) + (size_t)cj * S1_GPC * sizeof(int32_t);
    dim3 grid(nblk(N, S1_TT), nsub, nblk(ng, S1_GPC));
    cudaFuncSetAttribute(k_stage1<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_stage1<T><<<grid, S1_THREADS, smem, st>>>(xh, ldh, col0, C, N, nsub, ng, sub_start, d1, cj,
                                                wmax, ring, R, tbase_mod, err);
}

static size_t stage1t_smem(int maxch, int npass, int span)
{
    const long words = S1T_HALO + span, pitch = words + words / 16 + 1;
    return (size_t)maxch * (npass * (S1T_PASS * sizeof(uint16_t) + 4 * sizeof(int32_t)) + pitch * sizeof(float));
}

/* The tables of k_stage1t for a row, or none (false) where it does not apply: tables and windows
 * do not fit in shared memory, a team's groups spread over more than 112 samples in a channel, or
 * delays do not grow with the group. */
bool stage1t_tables(const int32_t *d1, int C, int nsub, int ng, const int32_t *sub_start, int maxch, Stage1T &t)
{
    t = Stage1T();
    const int quads = (ng + 3) / 4, npass = (quads + 15) / 16, qpt = (quads + 4 * npass - 1) / (4 * npass);
    t.span.assign(nsub, 0);
    int widest = 0;
    for (int s = 0; s < nsub; s++) {
        for (int j = sub_start[s]; j < sub_start[s + 1]; j++)
            t.span[s] = std::max(t.span[s], d1[(size_t)(ng - 1) * C + j]);
        widest = std::max(widest, t.span[s]);
    }
    if (stage1t_smem(maxch, npass, widest) > S1T_SMEM) return false;
    t.rel.assign((size_t)C * npass * S1T_PASS, 0);
    t.first.assign((size_t)C * npass * 4, 0);
    auto delay = [&](int g, int j) { return d1[(size_t)std::min(g, ng - 1) * C + j]; };
    int spread = 0;
    for (int j = 0; j < C; j++)
        for (int set = 0; set < 4 * npass; set++) {
            const int g0 = set * qpt * 4, d0 = delay(g0, j) & ~7;
            t.first[(size_t)j * npass * 4 + set] = d0;
            for (int k = 0, prev = d0; k < 4 * qpt; k++) {
                const int d = delay(g0 + k, j);
                if (d < prev) return false;
                prev = d;
                spread = std::max(spread, d - d0);
                if (spread > 112) return false;
                t.rel[((size_t)j * npass + set / 4) * S1T_PASS + (set % 4) * 16 + k] = (uint16_t)(d - d0);
            }
        }
    t.npass = npass;
    t.qpt = qpt;
    t.cw = std::max((16 + spread + 7) / 8 * 8, 24); /* a fill writes 24 columns or more */
    t.nb = S1T_COLS / t.cw;
    t.widest = widest;
    return true;
}

template <typename T>
static void stage1t(const Stage1TDev &t, const float *xh, long ldh, long col0, int C, long N, int nsub, int ng,
                    const int32_t *sub_start, int maxch, T *ring, long R, long tbase_mod, cudaStream_t st)
{
    const size_t smem = stage1t_smem(maxch, t.npass, t.widest);
    auto kern = k_stage1t<T>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(kern, dim3(nblk(N + (tbase_mod & 15), S1T_TT), nsub), S1T_THREADS, smem, st, xh, ldh, col0, C, N,
                   nsub, ng, sub_start, t.rel, t.first, t.npass, t.qpt, t.cw, t.nb, t.span, maxch, ring, R, tbase_mod);
}

/* Resident launch shapes (threads per set x samples per thread, thread sets x groups each),
 * the same for every ring precision:
 *   0 = from tensor memory (k_stage1t), where it does not apply 32x16 16x4 (18), 1 = 256x2 1x16, 2 = 512x1 1x16, 3 = 256x2 2x8, 4 = 256x2 2x16,
 *   5 = 256x1 2x8, 6 = 256x2 4x4, 7 = 128x4 4x8, 8 = 256x4 2x8, 9 = 128x4 2x8, 10 = 128x4 8x4,
 *   11 = 64x8 8x4, 12 = 64x8 4x4, 13 = 64x8 16x4, 14 = 64x8 8x8, 15 = 64x16 8x4,
 *   16 = 256x2 4x8, 17 = 32x8 16x8
 * Every channel step loads the thread's delays (broadcast 16-byte loads, two shared-memory
 * wavefronts each) and then one window element per sample for each distinct delay among its
 * groups: many samples per thread and one warp per set keep the delay loads a small share of
 * the shared-memory traffic (measured on the 4096-channel workload: 32x16 16x4 took stage 1
 * from 185 to 159 ms per 20 blocks against 256x2 4x8; loading only where the delay changes,
 * 159 to 114 ms; a sweep of all shapes on the GB300 kept 32x16 16x4, the 1024-thread 64x8
 * 16x4 at 60 registers being 3 % slower).  A shape whose windows do not fit falls back to
 * 256x2 1x16, then to the chunked kernel (any negative variant selects the chunked kernel
 * directly). */
template <typename T>
static void stage1_dispatch(const float *xh, long ldh, long col0, int C, long N,
                            int nsub, int ng, const int32_t *sub_start, const int32_t *d1, long maxd1,
                            int maxch, T *ring, long R, long tbase_mod, int var, const Stage1TDev &t, int *err,
                            cudaStream_t st)
{
    if (var == 0 && t.npass > 0) {
        stage1t<T>(t, xh, ldh, col0, C, N, nsub, ng, sub_start, maxch, ring, R, tbase_mod, st);
        return;
    }
    if (var < 0) { /* the chunked kernel, whatever fits */
        stage1_chunked<T>(xh, ldh, col0, C, N, nsub, ng, sub_start, d1, maxd1, maxch, ring, R, tbase_mod, err, st);
        return;
    }
    bool done = false;
#define TXG_ARGS xh, ldh, col0, C, N, nsub, ng, sub_start, d1, maxd1, maxch, ring, R, tbase_mod, err, st
    switch (var) {
    case 1: break;
    case 2: done = stage1r_try<T, 512, 1, 1, 16>(TXG_ARGS); break;
    case 3: done = stage1r_try<T, 256, 2, 2, 8>(TXG_ARGS); break;
    case 4: done = stage1r_try<T, 256, 2, 2, 16>(TXG_ARGS); break;
    case 5: done = stage1r_try<T, 256, 1, 2, 8>(TXG_ARGS); break;
    case 6: done = stage1r_try<T, 256, 2, 4, 4>(TXG_ARGS); break;
    case 7: done = stage1r_try<T, 128, 4, 4, 8>(TXG_ARGS); break;
    case 8: done = stage1r_try<T, 256, 4, 2, 8>(TXG_ARGS); break;
    case 9: done = stage1r_try<T, 128, 4, 2, 8>(TXG_ARGS); break;
    case 10: done = stage1r_try<T, 128, 4, 8, 4>(TXG_ARGS); break;
    case 11: done = stage1r_try<T, 64, 8, 8, 4>(TXG_ARGS); break;
    case 12: done = stage1r_try<T, 64, 8, 4, 4>(TXG_ARGS); break;
    case 13: done = stage1r_try<T, 64, 8, 16, 4>(TXG_ARGS); break;
    case 14: done = stage1r_try<T, 64, 8, 8, 8>(TXG_ARGS); break;
    case 15: done = stage1r_try<T, 64, 16, 8, 4>(TXG_ARGS); break;
    case 16: done = stage1r_try<T, 256, 2, 4, 8>(TXG_ARGS); break;
    case 17: done = stage1r_try<T, 32, 8, 16, 8>(TXG_ARGS); break;
    default: done = stage1r_try<T, 32, 16, 16, 4>(TXG_ARGS); break;
    }
    if (!done) done = stage1r_try<T, 256, 2, 1, 16>(TXG_ARGS);
#undef TXG_ARGS
    if (!done) stage1_chunked<T>(xh, ldh, col0, C, N, nsub, ng, sub_start, d1, maxd1, maxch, ring, R, tbase_mod, err, st);
}

void launch_stage1(const float *xh, long ldh, long col0, int C, long N, int nsub,
                   int ng, const int32_t *sub_start, const int32_t *d1, long maxd1, int maxch, void *ring,
                   long R, long tbase_mod, int prec, int var, const Stage1TDev &t, int *err, cudaStream_t st)
{
    if (prec == TXG_PREC_BF16)
        stage1_dispatch<__nv_bfloat16>(xh, ldh, col0, C, N, nsub, ng, sub_start, d1, maxd1, maxch,
                                       (__nv_bfloat16 *)ring, R, tbase_mod, var, t, err, st);
    else if (prec == TXG_PREC_FP16)
        stage1_dispatch<__half>(xh, ldh, col0, C, N, nsub, ng, sub_start, d1, maxd1, maxch,
                                (__half *)ring, R, tbase_mod, var, t, err, st);
    else
        stage1_dispatch<float>(xh, ldh, col0, C, N, nsub, ng, sub_start, d1, maxd1, maxch,
                               (float *)ring, R, tbase_mod, var, t, err, st);
}


/* DMs per stage-2 CTA for a group of G fine DMs (one chunk per group when G <= 32). */
constexpr int S2_MAXK = 32; /* most DMs a stage-2 CTA sums */

/* DMs a stage-2 CTA sums: a whole group of up to 16, else the part of a group that leaves the
 * fewest sums over (they are computed and dropped); of equal ones the smallest for FP32, whose time
 * is the shared-memory reads', and the largest for 16-bit pairs, whose windows are copied twice.
 * us, this choice (with stage2_kb's windows) against 8, 16, 24 or 32 DMs: 16-bit groups of 40 of
 * 8192 channels 427 / 726, of 56 1501 / 1885, of 24 of 4096 channels 287 / 348; FP32 groups of
 * 4 of 256 channels 109 / 168, of 24 of 4096 channels 366 / 406. */
static int stage2_kpc(int G, bool pairs)
{
    if (G <= 16) return (G + 3) / 4 * 4;
    int best = 0, left = 0;
    for (int i = 0; i < 6; i++) {
        const int k = pairs ? 28 - 4 * i : 8 + 4 * i, pad = (G + k - 1) / k * k - G;
        if (!best || pad < left) best = k, left = pad;
    }
    return best;
}

/* Window budget of a stage-2 CTA in KB: small where few accumulators let many CTAs run on an SM
 * (one-warp CTAs of 8 DMs, 1024 channels in FP16: 481 us with 12 KB, 516 with 18), large where wide
 * CTAs share long windows (28 DMs of 8192 channels: 1501 us with 36 KB, 1627 with 18). */
static int stage2_kb(int k, int G, bool pairs)
{
    if (k > 16) return pairs && k == 20 ? 24 : 36;
    if (pairs) return k <= 12 ? 12 : 18;
    return k <= 8 && G <= 8 ? 12 : 18;
}

/* Largest d2 spread inside any S2_MAXK DMs of a group, over all groups and subbands. */
long stage2_span(const int32_t *d2h, int nsub, int G, long ndm)
{
    long span = 0;
    for (long g0 = 0; g0 < ndm; g0 += G)
        for (long k0 = g0; k0 < min(g0 + (long)G, ndm); k0++) {
            long k1 = min(min(k0 + S2_MAXK, g0 + (long)G), ndm) - 1;
            for (int s = 0; s < nsub; s++) {
                long d = (long)d2h[k1 * nsub + s] - d2h[k0 * nsub + s];
                span = d > span ? d : span;
            }
        }
    return span;
}

/* ---- subband series of one DM (get_subdata) and candidate bands ------------------------ */
template <typename T>
__global__ void k_subdata(const T *__restrict__ ring, long R, int nsub, int G, const int32_t *__restrict__ d2,
                          long k, long t0_mod, long nout, float *__restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    if (i >= nout) return;
    const long g = k / G;
    const long t = (t0_mod + i + d2[(size_t)k * nsub + s]) % R;
    out[(size_t)s * nout + i] = to_f(ring[((size_t)g * nsub + s) * R + t]);
}

/* One CTA per candidate: per subband, the sum over samples (isamp-wn, isamp+wn) of the
 * subband sample divided by its channel count, ascending from 0.0f. */
template <typename T>
__global__ void k_cand_vpf(const T *__restrict__ ring, long R, int nsub, int G,
                           const int32_t *__restrict__ d2, const int32_t *__restrict__ sub_start,
                           long t0_mod, long nout, const txg_cand *__restrict__ c,
                           float *__restrict__ vpf)
{
    const txg_cand cd = c[blockIdx.x];
    const long k = cd.idm, g = k / G;
    const long lo = max(0L, (long)cd.isamp - cd.wn + 1), hi = min(nout, (long)cd.isamp + cd.wn);
    for (int s = threadIdx.x; s < nsub; s += blockDim.x) {
        const float cnt = (float)(sub_start[s + 1] - sub_start[s]);
        const T *row = ring + ((size_t)g * nsub + s) * R;
        const long d = d2[(size_t)k * nsub + s];
        float acc = 0.f;
        for (long i = lo; i < hi; i++) acc = __fadd_rn(acc, __fdiv_rn(to_f(row[(t0_mod + i + d) % R]), cnt));
        vpf[(size_t)blockIdx.x * nsub + s] = acc;
    }
}

template <typename T>
static void subdata_impl(const void *ring, long R, int nsub, int G, const int32_t *d2, long k,
                         long t0_mod, long nout, float *out, cudaStream_t st)
{
    dim3 grid(nblk(nout, 256), nsub);
    k_subdata<T><<<grid, 256, 0, st>>>((const T *)ring, R, nsub, G, d2, k, t0_mod, nout, out);
}

void launch_subdata(const void *ring, long R, int nsub, int G, const int32_t *d2, long k,
                    long t0_mod, long nout, int prec, float *out, cudaStream_t st)
{
    if (prec == TXG_PREC_BF16)
        subdata_impl<__nv_bfloat16>(ring, R, nsub, G, d2, k, t0_mod, nout, out, st);
    else if (prec == TXG_PREC_FP16)
        subdata_impl<__half>(ring, R, nsub, G, d2, k, t0_mod, nout, out, st);
    else
        subdata_impl<float>(ring, R, nsub, G, d2, k, t0_mod, nout, out, st);
}

void launch_cand_vpf(const void *ring, long R, int nsub, int G, const int32_t *d2,
                     const int32_t *sub_start, long t0_mod, long nout, const txg_cand *c, long n,
                     int prec, float *vpf, cudaStream_t st)
{
    if (n <= 0) return;
    if (prec == TXG_PREC_BF16)
        k_cand_vpf<__nv_bfloat16><<<(unsigned)n, 128, 0, st>>>((const __nv_bfloat16 *)ring, R, nsub, G, d2,
                                                               sub_start, t0_mod, nout, c, vpf);
    else if (prec == TXG_PREC_FP16)
        k_cand_vpf<__half><<<(unsigned)n, 128, 0, st>>>((const __half *)ring, R, nsub, G, d2, sub_start,
                                                        t0_mod, nout, c, vpf);
    else
        k_cand_vpf<float><<<(unsigned)n, 128, 0, st>>>((const float *)ring, R, nsub, G, d2, sub_start,
                                                       t0_mod, nout, c, vpf);
}

/* Ring length a stage-2 window may need (the ring must be longer, so a window wraps once). */
long stage2_window(long span) { return (long)S2_TT + span + 16; }

template <typename T, int KPC, int TH>
static void stage2_impl(const void *ring, long R, int nsub, int G, long ndm, long nout,
                        const int32_t *d2, long span, long t0_mod, float *tim, long ldt, size_t budget,
                        int *err, cudaStream_t st)
{
    const long epc = 16 / (long)sizeof(T);
    const long wlen = ((long)S2_TT + span + 2 * epc) / epc * epc;
    const size_t per = wlen * sizeof(T) + KPC * sizeof(int32_t) + 5 * sizeof(int32_t);
    int sc = (int)((budget - 64) / per);
    if (sc > nsub) sc = nsub;
    if (sc < 1) sc = 1;
    const long wtot = (long)sc * wlen;
    const size_t smem = ((wtot * sizeof(T) + 15) / 16) * 16 + (size_t)sc * KPC * 4 + (size_t)sc * 5 * 4;
    const int nkc = (G + KPC - 1) / KPC;
    const long ng = (ndm + G - 1) / G;
    dim3 grid(nblk(nout, S2_TT), (unsigned)(ng * nkc));
    auto kern = k_stage2<T, KPC, TH, S2_TT / TH>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(kern, grid, TH, smem, st, (const T *)ring, R, nsub, G, ndm, nout, d2, t0_mod, sc, wtot, tim, ldt,
                   err);
}

/* 16-bit ring: pair kernel, TH threads of UP pairs over the S2_TT-sample tile, windows doubled
 * by the odd copy. */
template <typename T, int KPC, int TH>
static void stage2p_impl(const void *ring, long R, int nsub, int G, long ndm, long nout,
                         const int32_t *d2, long span, long t0_mod, float *tim, long ldt, size_t budget,
                         int *err, cudaStream_t st)
{
    constexpr int UP = S2_TT / 2 / TH;
    const long wlen = ((long)S2_TT + span + 2 + 7 + 7) / 8 * 8; /* halves */
    const size_t per = wlen * 4 + KPC * sizeof(int32_t) + 4 * sizeof(int32_t);
    int sc = (int)((budget - 80) / per);
    if (sc > nsub) sc = nsub;
    if (sc < 1) sc = 1;
    const long wtot = (long)sc * wlen;
    const size_t smem = (size_t)(wtot / 2 + 4) * 4 + (size_t)(wtot / 2) * 4 + (size_t)sc * KPC * 4 +
                        (size_t)sc * 4 * 4;
    const int nkc = (G + KPC - 1) / KPC;
    const long ng = (ndm + G - 1) / G;
    dim3 grid(nblk(nout, S2_TT), (unsigned)(ng * nkc));
    auto kern = k_stage2p<T, KPC, TH, UP>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_chained(kern, grid, TH, smem, st, (const T *)ring, R, nsub, G, ndm, nout, d2, t0_mod, sc, wtot, tim, ldt,
                   err);
}

/* FP32 threads per CTA by variant: 0 = 32 (8 samples each; DM chunks wider than 16 take 64),
 * 1 = 64 (4), 2 = 128 (2; 64 for wider chunks).  Fewer threads with more samples each load the
 * per-subband delays (broadcast 16-byte loads) for more additions: on the 4096-channel workload
 * variant 0 with 18 KB per CTA took stage 2 from 91 to 81 ms per 20 blocks against 128 threads
 * with 36 KB. */
template <typename T, int K>
static void stage2_var(int var, const void *ring, long R, int nsub, int G, long ndm, long nout,
                       const int32_t *d2, long span, long t0_mod, float *tim, long ldt, size_t budget,
                       int *err, cudaStream_t st)
{
    if constexpr (K <= 16) {
        if (var == 0) {
            stage2_impl<T, K, 32>(ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st);
            return;
        }
    }
    if constexpr (K <= 16) {
        if (var == 2) {
            stage2_impl<T, K, 128>(ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st);
            return;
        }
    }
    stage2_impl<T, K, 64>(ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st);
}

/* 16-bit pair kernel by variant: 0 = 32 threads of 4 pairs (DM chunks wider than 16: 64 of
 * 2), 1 = 64 of 2, 2 = 128 of 1 (64 of 2 for wider chunks).  Variant 0 with 18 KB per CTA:
 * 71 -> 65 ms per 20 blocks of the 4096-channel workload against variant 2 with 36 KB. */
template <typename T, int K>
static void stage2p_var(int var, const void *ring, long R, int nsub, int G, long ndm, long nout,
                        const int32_t *d2, long span, long t0_mod, float *tim, long ldt, size_t budget,
                        int *err, cudaStream_t st)
{
    if constexpr (K <= 16) {
        if (var == 0) {
            stage2p_impl<T, K, 32>(ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st);
            return;
        }
    }
    if constexpr (K <= 16) {
        if (var == 2) {
            stage2p_impl<T, K, 128>(ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st);
            return;
        }
    }
    stage2p_impl<T, K, 64>(ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st);
}

template <typename T, bool PAIRS>
static void stage2_dispatch(int var, const void *ring, long R, int nsub, int G, long ndm, long nout,
                            const int32_t *d2, long span, long t0_mod, float *tim, long ldt,
                            int kb, int *err, cudaStream_t st)
{
    /* variants 3-5: the thread shapes of 0-2 with at most 8 DMs per CTA: fewer accumulators, so
     * more CTAs per SM, each subband window loaded by more CTAs; every DM's sum is the same */
    const int kfull = stage2_kpc(G, PAIRS);
    int kuse = var >= 3 ? std::min(kfull, 8) : kfull;
    if ((ndm + G - 1) / G * ((G + kuse - 1) / kuse) > 65535 && G > 16) kuse = S2_MAXK; /* the grid's y */
    const int v = var >= 3 ? var - 3 : var;
    const size_t budget = (size_t)(kb >= 8 ? kb : stage2_kb(kuse, G, PAIRS)) * 1024;
#define TXG_S2(K)                                                                                   \
    if constexpr (PAIRS)                                                                            \
        stage2p_var<T, K>(v, ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st); \
    else                                                                                            \
        stage2_var<T, K>(v, ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, budget, err, st)
    switch (kuse) {
    case 4: TXG_S2(4); break;
    case 8: TXG_S2(8); break;
    case 12: TXG_S2(12); break;
    case 16: TXG_S2(16); break;
    case 20: TXG_S2(20); break;
    case 24: TXG_S2(24); break;
    case 28: TXG_S2(28); break;
    default: TXG_S2(32); break;
    }
#undef TXG_S2
}

/* One CTA waits, with the bounded wait of the window copies, for a 256-byte bulk copy whose
 * barrier expects 256 + extra bytes: with extra > 0 the phase never completes (the copy lands,
 * nothing else comes), the wait runs out after limit_ns and the CTA reports it in status[0]. */
__global__ void k_wait_selftest(const uint8_t *__restrict__ src, int extra, uint64_t limit_ns,
                                int *__restrict__ status)
{
    __shared__ __align__(16) unsigned char buf[256];
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, 256u + (uint32_t)extra);
        bulk_g2s(buf, src, 256u, &bar);
    }
    const bool ok = mbar_wait(&bar, 0, limit_ns);
    if (!__syncthreads_and(ok)) {
        if (threadIdx.x == 0) status[0] = 1;
        return;
    }
    if (threadIdx.x == 0) status[0] = buf[0] == src[0] && buf[255] == src[255] ? 0 : 2;
}

void launch_wait_selftest(const uint8_t *src, int extra, long limit_ms, int *status, cudaStream_t st)
{
    k_wait_selftest<<<1, 32, 0, st>>>(src, extra, (uint64_t)limit_ms * 1000000ull, status);
}

void launch_stage2(const void *ring, long R, int nsub, int G, long ndm, long nout,
                   const int32_t *d2, long span, long t0_mod, int prec, int s2_var, int s2_kb,
                   float *tim, long ldt, int *err, cudaStream_t st)
{
    if (prec == TXG_PREC_BF16)
        stage2_dispatch<__nv_bfloat16, true>(s2_var, ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt,
                                             s2_kb, err, st);
    else if (prec == TXG_PREC_FP16)
        stage2_dispatch<__half, true>(s2_var, ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, s2_kb,
                                      err, st);
    else
        stage2_dispatch<float, false>(s2_var, ring, R, nsub, G, ndm, nout, d2, span, t0_mod, tim, ldt, s2_kb,
                                      err, st);
}

} // namespace txg
