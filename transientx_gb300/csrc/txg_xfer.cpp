/*
 * txg_xfer.cpp -- host side of copies and short-lived device memory: large copies between host
 * buffers by several threads, first touch of large pageable outputs by several threads, and a
 * stream with scratch memory from a bounded per-device pool for the calls that own no handle.
 */
#include <cuda.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

#include "txg_internal.h"

namespace txg {

namespace {

constexpr size_t PART = 1 << 20; /* bytes worth a thread */
constexpr unsigned MAX_THREADS = 4;

/* f(begin, end) over [0, n) in parts of whole pages, by the caller and up to three more threads. */
template <typename F> void in_parts(size_t n, F f)
{
    size_t k = std::min<size_t>(MAX_THREADS, n / PART);
    if (k > 1) k = std::min<size_t>(k, std::thread::hardware_concurrency() / 2);
    if (k < 2) {
        f((size_t)0, n);
        return;
    }
    const size_t part = (n / k + 65535) / 65536 * 65536;
    std::thread th[MAX_THREADS];
    size_t from = 0;
    unsigned started = 0;
    try {
        for (; started + 1 < k && from + part < n; started++, from += part) th[started] = std::thread(f, from, from + part);
    } catch (...) { /* fewer threads: the caller does the rest */
    }
    f(from, n);
    for (unsigned t = 0; t < started; t++) th[t].join();
}

} // namespace

/* A pageable block goes to pinned staging by several threads once each has 1 MB to copy: pushes of
 * 512 channels x 7812 float samples (16 MB) with dense results read back took 2.4 to 3.3 ms by one
 * thread and 1.8 with four here and in copy_out. */
void host_copy(void *dst, const void *src, size_t n)
{
    in_parts(n, [=](size_t a, size_t b) { memcpy((char *)dst + a, (const char *)src + a, b - a); });
}

/* The pages of a pageable buffer that is about to be written are populated first by several
 * threads: a copy from the device into fresh memory otherwise takes their faults one by one
 * (26 MB of S/N maps: a call of 13.4 ms took 4.9 with this and the scratch pool).  What the buffer holds stays until the copy.  Pinned,
 * managed and device memory are left to the copy itself, and so is what the kernel cannot populate. */
static void populate(void *dst, size_t n)
{
#ifdef MADV_POPULATE_WRITE
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type != cudaMemoryTypeUnregistered) {
        cudaGetLastError();
        return;
    }
    const uintptr_t page = (uintptr_t)std::max(4096L, sysconf(_SC_PAGESIZE));
    const uintptr_t first = (uintptr_t)dst / page * page, end = ((uintptr_t)dst + n + page - 1) / page * page;
    in_parts(end - first, [=](size_t a, size_t b) { (void)madvise((void *)(first + a), b - a, MADV_POPULATE_WRITE); });
#else
    (void)dst, (void)n;
#endif
}

cudaError_t copy_out(void *dst, const void *dev, size_t n)
{
    if (n >= 2 * PART) populate(dst, n);
    return cudaMemcpy(dst, dev, n, cudaMemcpyDeviceToHost);
}

/* ---- scratch ---------------------------------------------------------------------------- */
namespace {

constexpr int MAX_DEV = 64;
constexpr unsigned long long POOL_KEEP = 256ull << 20; /* bytes a device's pool keeps between calls */

/* An id of the current context that no later one has; 0 if it cannot be had. */
unsigned long long context_id()
{
    using Fn = CUresult (*)(CUcontext, unsigned long long *);
    static const Fn fn = [] {
        void *q = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &q, 12000, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess)
            q = nullptr;
        return (Fn)q;
    }();
    unsigned long long id = 0;
    return fn && fn(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

/* The current device's scratch pool, made at the first use; null where there is none, and in a
 * context other than the first use's (the pool does not outlive cudaDeviceReset): scratch then
 * comes from cudaMalloc.  One pool serves all threads: memory goes from one stream to another only
 * after the first has ended with it.  A txg_boxcar call of 1000 x 8193 samples took 1.19 ms with
 * cudaMalloc and cudaFree and takes 0.81 with the pool. */
cudaMemPool_t current_pool()
{
    static std::mutex m;
    static struct {
        bool tried;
        unsigned long long ctx;
        cudaMemPool_t pool;
    } tab[MAX_DEV];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) return nullptr;
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lk(m);
    auto &t = tab[dev];
    if (!t.tried) {
        t.tried = true;
        t.ctx = ctx;
        int ok = 0;
        cudaMemPoolProps pr{};
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = dev;
        unsigned long long keep = POOL_KEEP;
        if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess || !ok ||
            cudaMemPoolCreate(&t.pool, &pr) != cudaSuccess)
            t.pool = nullptr;
        else
            cudaMemPoolSetAttribute(t.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        cudaGetLastError(); /* a missing pool is no error of the call */
    }
    return ctx && ctx == t.ctx ? t.pool : nullptr;
}

} // namespace

void scratch_trim()
{
    if (cudaMemPool_t p = current_pool()) cudaMemPoolTrimTo(p, 0);
}

cudaError_t Scratch::open()
{
    const cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) pool_ = current_pool();
    return e;
}

cudaError_t Scratch::get(void **p, size_t bytes)
{
    bytes = std::max<size_t>(bytes, 16);
    cudaError_t e = pool_ ? cudaMallocFromPoolAsync(p, bytes, pool_, st) : cudaMalloc(p, bytes);
    if (pool_ && e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaMemPoolTrimTo(pool_, 0);
        e = cudaMallocFromPoolAsync(p, bytes, pool_, st);
    }
    if (e == cudaSuccess) ptr_.push_back(*p);
    return e;
}

Scratch::~Scratch()
{
    if (!st) return;
    cudaStreamSynchronize(st);
    for (void *p : ptr_) {
        if (pool_) cudaFreeAsync(p, st);
        else cudaFree(p);
    }
    if (pool_) cudaStreamSynchronize(st); /* what is above the kept size goes back here */
    cudaStreamDestroy(st);
}

} // namespace txg
