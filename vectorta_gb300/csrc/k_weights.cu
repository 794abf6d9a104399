// Per-combo weight rows of the weighted-window moving averages, generated on
// the device and right-aligned into a [n_combos][kmax] f32 matrix
// (zero-padded on the left), normalised so each row sums to one.
//
// Weight definitions follow the crate:
//   ALMA   w_i = exp(-(i - m)^2 / (2 s^2)), m = offset (p-1), s = p / sigma
//          (alma.rs:1426-1437)
//   WMA    w_i = (i + 1) / (p (p + 1) / 2)                       (wma.rs:295-336)
//   SWMA   symmetric triangle = box(a) * box(b)        (swma.rs:320-400, 406-482)
//   PWMA   binomial row C(p-1, r) / sum                  (pwma.rs:1367-1408)
//   SINWMA w_k = sin((k+1) pi / (p+1)) / sum             (sinwma.rs:271-289)
//   TRIMA  box(m1) * box(m2), m1 = (p+1)/2, m2 = p - m1 + 1 (trima.rs:277-364)
//
// Arithmetic: GB300's FP64 rate is a small fraction of its FP32 rate, so the
// per-combo constants (ALMA's centre m and 1/(2 s^2)) come in f64 from the
// host and the rest is FP32.  Each weight is evaluated in
// double-single FP32 (error-free products through FMA): the ALMA exponent
// e = (i - m)^2 / (2 s^2) is carried as e_hi + e_lo and exponentiated as
// expf(-e_hi) * (1 - e_lo), and the row sum is accumulated as a double-single
// value, so the stored f32 weights stay within ~2 ulp of the f64 ones.
#include "wwma_weights.cuh"

namespace vta {

namespace {

constexpr int kWThreads = 256;

using namespace wts;

// One warp per combo (kWThreads / 32 combos per block): raw weights summed in
// double-single across the lanes, then a second pass writes raw * (1 / sum).
// The per-combo f64 constants and the reciprocal are formed by lane 0 only.
__global__ void __launch_bounds__(kWThreads) k_weights(int kind, const int* periods, const double* pa,
                                                       const double* pb, int n_combos, int kmax, float* w) {
    const int lane = threadIdx.x & 31;
    const int c = blockIdx.x * (kWThreads / 32) + (threadIdx.x >> 5);
    if (c >= n_combos) return;  // whole warp (no block-wide barrier below)
    const int p = periods[c];
    const RowConst rc = row_const(kind, pa, pb, c);
    DS s{0.f, 0.f};
    for (int i = lane; i < p; i += 32) s = ds_add(s, raw_weight(kind, i, p, rc));
    const DS inv = row_inv(s);
    float* row = w + (size_t)c * kmax;
    const int lead = kmax - p;
    for (int k = lane; k < kmax; k += 32) {
        const int i = k - lead;
        float v = 0.f;
        if (i >= 0) {
            const DS r = ds_mul(raw_weight(kind, i, p, rc), inv);
            v = r.hi + r.lo;
        }
        row[k] = v;
    }
}

}  // namespace

vta_status launch_weights(int kind, const int* periods, const double* pa, const double* pb, int n_combos,
                          int kmax, float* w, cudaStream_t st) {
    k_weights<<<ceil_div(n_combos, kWThreads / 32), kWThreads, 0, st>>>(kind, periods, pa, pb, n_combos, kmax, w);
    return check_launch("k_weights");
}

}  // namespace vta
