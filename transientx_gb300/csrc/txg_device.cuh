/*
 * txg_device.cuh -- device helpers shared by the kernel files.
 */
#ifndef TXG_DEVICE_CUH
#define TXG_DEVICE_CUH

namespace txg {

/* The exact double of a float by integer operations: a conversion, like every FP64 instruction,
 * holds a scheduler's FP64 unit for about 60 cycles on this part. */
__device__ __forceinline__ double f2d(float f)
{
    const unsigned u = __float_as_uint(f), mag = u & 0x7fffffffu;
    if (mag - 0x00800000u >= 0x7f000000u && mag) return (double)f; /* subnormal, infinite, NaN */
    return __hiloint2double((int)((u & 0x80000000u) | (mag ? (mag >> 3) + 0x38000000u : 0u)), (int)(u << 29));
}

/* A block is a chain of twenty and more short kernels, and on the smallest formats most of its time
 * is the gaps between them.  So a kernel of the chain may be launched while the one before it still
 * runs, and starts with this wait for that one to have ended (and its writes to be seen); since
 * every one starts so, all earlier ones have ended too.  us a call: 64 channels 205 -> 176, 1000
 * channels with filters 373 -> 336, a file of 256 channels 2604 -> 2446.  (Letting the next kernel
 * come as soon as all blocks of one have started is no gain: 178, 353, 2606; its waiting blocks take
 * the room of other rows'.) */
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline void launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kern, static_cast<P>(args)...);
}

} // namespace txg

#endif
