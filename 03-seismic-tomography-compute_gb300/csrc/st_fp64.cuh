// FP64 helpers for kernels bound by the FP64 pipe, which takes a warp's operation
// in 16 cycles on this GPU.
#pragma once

#include <cuda_runtime.h>

namespace stg {

// Whether |x| lies in 2^-300 .. 2^300.
__device__ __forceinline__ bool moderate(double x) {
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return h - (723u << 20) < (600u << 20);
}

// x / d, correctly rounded, from y = 1 / d correctly rounded: two steps of
// Markstein's correction ("Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): the first leaves the quotient within one unit in
// the last place, so the second's remainder is exact and its rounding correct.
// Five operations where a division takes about ten; for moderate d, and |x| zero
// or from 2^-400 to 2^400.
__device__ __forceinline__ double quotient_of(double x, double d, double y) {
    double q = __dmul_rn(x, y);
    q = __fma_rn(__fma_rn(-q, d, x), y, q);
    return __fma_rn(__fma_rn(-q, d, x), y, q);
}

// Finite, tested on the bits.
__device__ __forceinline__ bool finite_bits(double x) {
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}

}  // namespace stg
