// Smoothing constants of a period, as the crate forms them in f64 and rounds to
// f32, without f64 arithmetic on the device.  Every thread of a recurrence
// kernel needs them, and on GB300 an f64 divide is some 20 instructions of a pipe
// with two lanes per SM.  For p below 2^24 the f32 quotient of the (exact)
// integers is the same number: such a quotient lies at least 2^-50 from any f32
// rounding boundary, farther than the f64 forms' own errors.
#pragma once

namespace vta {
namespace coef {

constexpr int kExact = 1 << 24;

__device__ __forceinline__ float wilder(int p) {  // 1 / p
    return p < kExact ? __fdiv_rn(1.f, (float)p) : (float)(1.0 / (double)p);
}
__device__ __forceinline__ float wilder_keep(int p) {  // 1 - 1 / p
    return p < kExact ? __fdiv_rn((float)(p - 1), (float)p) : (float)(1.0 - 1.0 / (double)p);
}
__device__ __forceinline__ float ema(int p) {  // 2 / (p + 1)
    return p < kExact - 1 ? __fdiv_rn(2.f, (float)(p + 1)) : (float)(2.0 / ((double)p + 1.0));
}
__device__ __forceinline__ float ema_keep(int p) {  // 1 - 2 / (p + 1)
    return p < kExact - 1 ? __fdiv_rn((float)(p - 1), (float)(p + 1)) : (float)(1.0 - 2.0 / ((double)p + 1.0));
}

}  // namespace coef
}  // namespace vta
