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

} // namespace txg

#endif
