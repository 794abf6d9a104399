// Series preparation kernels: per-series first-valid scan for time-major
// inputs and the blocked FP64 prefix scan behind the SMA/variance windows.
//
// The prefix is the only FP64 bulk arithmetic of the library (GB300's FP64
// rate is a small fraction of FP32): one f64 add per element in a 3-phase
// scan (block reduce -> scan of block sums -> block scan + offset), then the
// result is packed as double-single float2 (hi = f32(P), lo = f32(P - hi)) so
// the per-output window kernels work in FP32 only.
#include <algorithm>

#include "vta_internal.h"

namespace vta {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanBlock = kScanThreads * kScanItems;  // elements per block

// First valid row per series: a block owns 32 series (a warp's lanes, so each
// row is one 128-byte load) and its warps examine 8 rows each, up to 256 rows a
// round, until every series of the block is found.  Bound by memory latency: a
// NaN lead of up to 256 rows costs one round trip (one thread per series, 16
// rows a trip, took 22 us for 3,000 series with leads up to 250, 50 us over
// high / low / close; now 3.6 and 5.7).  Where the series alone fill the GPU, past
// two blocks of 32 warps per SM, 4 warps: the rows behind short leads are read
// for nothing (50,000 series x 250 rows, 32 warps / 4: ALMA(14) 73 / 62 us,
// Donchian(14) 78 / 56).
constexpr int kFvWarps = 32, kFvWideWarps = 4, kFvRows = 8;

int first_valid_threads(int cols) { return 32 * (ceil_div(cols, 32) > 2u * kNumSMs ? kFvWideWarps : kFvWarps); }

// ALL: c together with h and l (first), beside c alone (first_c, may be null).
template <bool ALL>
__global__ void __launch_bounds__(32 * kFvWarps)
k_first_valid_tm(const float* __restrict__ h, const float* __restrict__ l, const float* __restrict__ c, int cols,
                 int rows, const int* len, int* first, int* first_c, int* first_nan, int* first_big) {
    __shared__ int fa[32], fc[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, round = (blockDim.x >> 5) * kFvRows;
    const int s = blockIdx.x * 32 + lane;
    const int L = s < cols ? (len ? len[s] : rows) : 0;
    if (warp == 0) fa[lane] = fc[lane] = L;
    __syncthreads();
    for (int t0 = 0;; t0 += round) {
        if (L - t0 > warp * kFvRows) {
            const int tb = t0 + warp * kFvRows, m = L - tb;  // m rows left
            float hv[kFvRows], lv[kFvRows], cv[kFvRows];
#pragma unroll
            for (int j = 0; j < kFvRows; ++j) {  // all the loads before any test (rows clamped into the series)
                const size_t i = (size_t)(tb + min(j, m - 1)) * cols + s;
                cv[j] = __ldg(c + i);
                hv[j] = ALL ? __ldg(h + i) : 0.f;
                lv[j] = ALL ? __ldg(l + i) : 0.f;
            }
            int ba = L, bc = L;
#pragma unroll
            for (int j = kFvRows - 1; j >= 0; --j) {
                const bool ok = (j < m) & !isnan(cv[j]);
                if (ok) bc = tb + j;
                if (ok & !isnan(hv[j]) & !isnan(lv[j])) ba = tb + j;
            }
            if (ba < L) atomicMin(&fa[lane], ba);
            if (ALL && bc < L) atomicMin(&fc[lane], bc);
        }
        __syncthreads();
        // done once found or past the end (a round's finds are below the next one's)
        const bool more = fa[lane] == L && L - t0 > round;
        if (!__syncthreads_or(more)) break;
    }
    if (warp == 0 && s < cols) {
        first[s] = fa[lane];
        if (first_c) first_c[s] = fc[lane];
        if (first_nan) first_nan[s] = rows;
        if (first_big) first_big[s] = rows;
    }
}

// First NaN after each series' first valid row, and first value of magnitude
// above `limit` (infinite ones too): first_nan[s] and first_big[s] (may be null)
// hold `rows` (set by k_first_valid_tm) and are lowered to the row.  Blocks of
// 128 series x 64 rows read the whole matrix once (one thread per series
// walking its rows took 1,073 us for 3,000 x 2,520; now 11).
constexpr int kFnRows = 64, kFnBatch = 16;

__global__ void __launch_bounds__(128)
k_first_nan_tm(const float* __restrict__ x, int cols, int rows, const int* __restrict__ first, int* first_nan,
               int* first_big, float limit) {
    const int s = blockIdx.x * 128 + threadIdx.x;
    if (s >= cols) return;
    const int f = first[s];
    int found = rows, big = rows;
    for (long long t0 = (long long)blockIdx.y * kFnRows; t0 < rows; t0 += (long long)gridDim.y * kFnRows) {
        const int t1 = (int)min(t0 + kFnRows, (long long)rows);
        if (t1 - 1 < f) continue;
        for (int tb = (int)t0; tb < t1; tb += kFnBatch) {
            const int m = t1 - tb;
            float v[kFnBatch];
#pragma unroll
            for (int j = 0; j < kFnBatch; ++j) v[j] = __ldg(x + (size_t)(tb + min(j, m - 1)) * cols + s);
#pragma unroll
            for (int j = 0; j < kFnBatch; ++j) {
                if (j < m && tb + j > f && isnan(v[j])) found = min(found, tb + j);
                if (j < m && fabsf(v[j]) > limit) big = min(big, tb + j);
            }
        }
    }
    if (found < rows) atomicMin(first_nan + s, found);
    if (first_big && big < rows) atomicMin(first_big + s, big);
}

__device__ __forceinline__ double prefix_value(const float* x, int i, int first, int kind) {
    if (i < first) return 0.0;
    const double v = (double)x[i];
    switch (kind) {
        case PK_X: return v;
        case PK_X2: return v * v;
        case PK_NAN: return isnan(x[i]) ? 1.0 : 0.0;
        case PK_GAIN:
        case PK_LOSS: {
            if (i == first) return 0.0;
            const double d = v - (double)x[i - 1];
            if (!isfinite(d)) return __longlong_as_double(0x7ff8000000000000ll);
            if (kind == PK_GAIN) return d > 0.0 ? d : 0.0;
            return d < 0.0 ? -d : 0.0;
        }
    }
    return 0.0;
}

__device__ __forceinline__ double warp_incl_scan(double v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Block-wide exclusive scan of one double per thread (true exclusive: a NaN
// in thread i reaches threads > i only); leaves the block total in *total.
__device__ double block_excl_scan(double v, double* total) {
    constexpr int kW = kScanThreads / 32;
    __shared__ double wsum[kW];
    __shared__ double wtot;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double inc = warp_incl_scan(v);
    double exc = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) exc = 0.0;
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const double w = lane < kW ? wsum[lane] : 0.0;
        const double wi = warp_incl_scan(w);
        double we = __shfl_up_sync(0xffffffffu, wi, 1);
        if (lane == 0) we = 0.0;
        if (lane < kW) wsum[lane] = we;  // exclusive warp offsets
        if (lane == kW - 1) wtot = wi;
    }
    __syncthreads();
    const double res = wsum[warp] + exc;
    *total = wtot;
    __syncthreads();
    return res;
}

__global__ void k_prefix_reduce(const float* __restrict__ x, int n, int first, int kind,
                                double* block_sums) {
    const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + k;
        if (i < n) s += prefix_value(x, i, first, kind);
    }
    double total;
    block_excl_scan(s, &total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// Exclusive scan of the block sums in place (single block, any count).
__global__ void k_prefix_scan_blocks(double* block_sums, int nb) {
    double carry = 0.0;
    for (int base = 0; base < nb; base += kScanThreads) {
        const int i = base + threadIdx.x;
        const double v = i < nb ? block_sums[i] : 0.0;
        double total;
        const double exc = block_excl_scan(v, &total);
        if (i < nb) block_sums[i] = carry + exc;
        carry += total;
    }
}

__global__ void k_prefix_apply(const float* __restrict__ x, int n, int first, int kind,
                               const double* __restrict__ block_offsets, double* out_f64,
                               float2* out_ds) {
    const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
    double v[kScanItems];
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + k;
        v[k] = i < n ? prefix_value(x, i, first, kind) : 0.0;
        s += v[k];
    }
    double total;
    double run = block_offsets[blockIdx.x] + block_excl_scan(s, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int i = base + k;
        run += v[k];
        if (i < n) {
            if (out_f64) out_f64[i] = run;
            if (out_ds) {
                const float hi = (float)run;
                const float lo = (float)(run - (double)hi);
                out_ds[i] = make_float2(hi, lo);
            }
        }
    }
}

}  // namespace

vta_status launch_first_valid_tm(const float* x_tm, int cols, int rows, int* first, cudaStream_t st,
                                 int* first_nan, int* first_big, float limit) {
    k_first_valid_tm<false><<<ceil_div(cols, 32), first_valid_threads(cols), 0, st>>>(nullptr, nullptr, x_tm, cols, rows, nullptr,
                                                                         first, nullptr, first_nan, first_big);
    VTA_TRY(check_launch("k_first_valid_tm"));
    if (!first_nan) return VTA_OK;
    const unsigned ny = std::min(ceil_div(rows, kFnRows), 65535u);
    k_first_nan_tm<<<dim3(ceil_div(cols, 128), ny), 128, 0, st>>>(x_tm, cols, rows, first, first_nan, first_big,
                                                                  limit);
    return check_launch("k_first_nan_tm");
}

vta_status launch_first_valid_tm_hlc(const float* h, const float* l, const float* c, int cols,
                                     int rows, int* first, cudaStream_t st, const int* len, int* first_c) {
    k_first_valid_tm<true><<<ceil_div(cols, 32), first_valid_threads(cols), 0, st>>>(h, l, c, cols, rows, len, first, first_c,
                                                                        nullptr, nullptr);
    return check_launch("k_first_valid_tm_hlc");
}

size_t prefix_tmp_doubles(int n) { return ceil_div(n, kScanBlock) + 1; }

vta_status launch_prefix_f64(const float* x, int n, int first, int kind, double* out_f64,
                             float2* out_ds, double* block_tmp, cudaStream_t st) {
    const int nb = (int)ceil_div(n, kScanBlock);
    k_prefix_reduce<<<nb, kScanThreads, 0, st>>>(x, n, first, kind, block_tmp);
    VTA_TRY(check_launch("k_prefix_reduce"));
    k_prefix_scan_blocks<<<1, kScanThreads, 0, st>>>(block_tmp, nb);
    VTA_TRY(check_launch("k_prefix_scan_blocks"));
    k_prefix_apply<<<nb, kScanThreads, 0, st>>>(x, n, first, kind, block_tmp, out_f64, out_ds);
    return check_launch("k_prefix_apply");
}

// Row-major [rows][cols] -> [cols][rows] through 32 x 33 shared tiles (one
// coalesced read and one coalesced write per element).
namespace {
__global__ void k_transpose(const float* __restrict__ in, int rows, int cols, float* __restrict__ out) {
    __shared__ float tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = r0 + j, c = c0 + threadIdx.x;
        if (r < rows && c < cols) tile[j][threadIdx.x] = in[(size_t)r * cols + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = c0 + j, r = r0 + threadIdx.x;
        if (r < rows && c < cols) out[(size_t)c * rows + r] = tile[threadIdx.x][j];
    }
}
}  // namespace

vta_status launch_transpose(const float* in, int rows, int cols, float* out, cudaStream_t st) {
    if (rows <= 0 || cols <= 0) return VTA_OK;
    const dim3 grid(ceil_div(cols, 32), ceil_div(rows, 32));
    if (grid.y > 65535) return fail(VTA_ERR_LAUNCH_CONFIG_TOO_LARGE, "transpose: too many rows");
    k_transpose<<<grid, dim3(32, 8), 0, st>>>(in, rows, cols, out);
    return check_launch("k_transpose");
}

}  // namespace vta
