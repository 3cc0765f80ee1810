// store16.cuh — 16-bit wavefield storage as the z-marching kernels see it
// (kernels_ztwin16.cu, kernels_zpair.cu): value h of field g reads back as
// float(h) * 2^e_g, and v is stored as RN16(v * 2^-e_g), binary16 saturating
// at +-65504 — the roundings of kernels_half.cu and of the oracle.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "../../include/sgfd.h"
#include "sgfd_internal.h"

namespace sgfd {

template <int ST>
struct H16 {
    __device__ __forceinline__ static float h2f(uint32_t h) {
        if (ST == SGFD_STORE_BF16) return __uint_as_float(h << 16);
        return __half2float(__ushort_as_half((unsigned short)h));
    }
    __device__ __forceinline__ static uint32_t f2h(float w) {
        if (ST == SGFD_STORE_BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(w));
        return __half_as_ushort(__float2half_rn(fminf(fmaxf(w, -65504.0f), 65504.0f)));
    }
};

// Largest |v| (as unsigned float bits) of the warp's active lanes into field
// g's running maximum of the CTA, in shared memory (the rescale steps of 16-bit
// storage, as kernels_half.cu notes them); the CTA adds its maxima to the
// global ones once (flush_max16).
__device__ __forceinline__ void note_bits16s(unsigned *smax, int g, unsigned v) {
    const unsigned mask = __activemask();
    const unsigned bits = __reduce_max_sync(mask, v);
    if ((threadIdx.x & 31) == __ffs(mask) - 1) atomicMax(smax + g, bits);
}
__device__ __forceinline__ void note_max16s(unsigned *smax, int g, float v) {
    note_bits16s(smax, g, __float_as_uint(fabsf(v)));
}
// Two values at once (the second only if `second`), compared as bits: fmaxf
// would drop a NaN, whose bits are the largest and keep the field's exponent.
// (Masks, not fabsf: the 64 x 8 stress update spills 92 bytes with it, 80 so.)
__device__ __forceinline__ void note_max16s(unsigned *smax, int g, float2 v, bool second) {
    const unsigned a = __float_as_uint(v.x) & 0x7fffffffu, b = __float_as_uint(v.y) & (second ? 0x7fffffffu : 0u);
    note_bits16s(smax, g, a > b ? a : b);
}
// After a barrier: threads 0..8 add the CTA's maxima to the global ones.
__device__ __forceinline__ void flush_max16(const HalfState &hs, const unsigned *smax) {
    if (threadIdx.x < 9 && smax[threadIdx.x] != 0u) atomicMax(hs.amax + threadIdx.x, smax[threadIdx.x]);
}

}  // namespace sgfd
