// Packed pairs of floats (sm_100's f32x2 instructions) for kernels whose products and sums must
// round one by one. Each half rounds exactly as the scalar operation does, and a pair takes one
// issue slot; the lane rate is the scalar one (220-240 lane operations per ns and SM measured
// either way), so they pay where instruction issue bounds a kernel.
#pragma once

#include <cuda_runtime.h>

namespace nrb {

// The assembler contracts mul.rn.f32x2 followed by add.rn.f32x2 into one fused operation, rounding
// modifiers or not (measured: 59% of the sums of three products differ from the scalar ones), and
// sees through a literal -0. A product is therefore a fused multiply-add of -0 read from constant
// memory: a * b + (-0) rounds to a * b for every a and b, the sign of a zero product included, and
// leaves nothing to contract (measured: no sum differs).
static __constant__ unsigned long long kNegZeroPair = 0x8000000080000000ull;

struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2(float both) { return f2(both, both); }
__device__ __forceinline__ void split(F2 a, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(kNegZeroPair));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

}  // namespace nrb
