// Nearest-rank percentile sweeps of one series: every (length, percentage)
// combo of a batch call over the same x.
//
//   out[c][t] = sorted(window)[k], window = the non-NaN values of
//   x[t - len + 1 .. t], k = round(p * count) - 1 clamped to [0, count - 1]
//   (percentile_nearest_rank.rs:190-266).  Selection only, so the outputs are
//   inputs bit for bit.
//
// Per slab of time tiles:
//   k_pnr_ranks  ranks the values of each tile's input span [t0 - lmax + 1,
//                t0 + T) among themselves once for all combos (ties by
//                position, so ranks are distinct);
//   k_pnr_grow   dense length axes: a thread owns one time and walks the
//                combos of one percentage by length, entering the values by
//                which each window is longer than the one before.  Nothing
//                ever leaves a window and the lanes write consecutive times;
//   k_pnr_slide  sparse axes: a thread owns one combo over a run of times; a
//                step drops the leaving value and enters the next one.
// Both hold a window as a bitmap over the span's ranks with a cursor on its
// k-th set bit, which a new value moves by one set bit or not at all.  A
// summary word marks the nonempty bitmap words, so the next / previous set
// bit is at most two words away however sparse the window is.
//
// Why ranks: a step costs a few dozen instructions whatever the window
// length, where keeping the window's values sorted costs O(len) a step.
// Bound by instruction issue.  Lengths 15..264 (250 combos) on 100k bars:
// 36.4 ms with one sorted array per thread in global memory -> 0.148 ms
// (ranks 0.021).  The 28 lengths 10..64 step 2 on 200k bars: 0.051 ms.
#include <algorithm>
#include <cmath>
#include <numeric>

#include "pnr_ops.cuh"
#include "vta_internal.h"

namespace vta {
namespace {

constexpr int kSwThreads = 128;
constexpr int kSwStage = 16;  // times staged per thread between row writes
constexpr int kGrowTile = 256;  // times (threads) per block of the growing walk
constexpr uint16_t kNoRank = 0xffff;

__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

struct PnrTiles {
    const float* x;
    int n, lmax;
    int tile0;       // first tile of this slab
    int T, S, spad;  // times per tile, span T + lmax - 1, and its row pitch
    uint16_t* rank;  // [slab tiles][spad]
    float* val;      // [slab tiles][spad]: the span's values in rank order
};

// Rank of each span value by counting the smaller ones (and the equal ones
// before it): S compares per value, two instructions each, against shared
// memory broadcasts.  For spans of a few hundred values that is less work
// than a block-wide sort and has no dependent passes.
__global__ void __launch_bounds__(512) k_pnr_ranks(PnrTiles a) {
    extern __shared__ __align__(16) float xs[];  // [spad]
    const int tile = blockIdx.x;
    const int base = (a.tile0 + tile) * a.T - (a.lmax - 1);
    for (int i = threadIdx.x; i < a.spad; i += blockDim.x) {
        const int g = base + i;
        xs[i] = (i < a.S && g >= 0 && g < a.n) ? __ldg(a.x + g) : qnan();
    }
    __syncthreads();
    uint16_t* rk = a.rank + (size_t)tile * a.spad;
    float* sv = a.val + (size_t)tile * a.spad;
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < a.spad; i += blockDim.x) {
        const float v = xs[i];  // (NaN compares false: it is counted by nobody)
        int cnt = 0;
        const int w0 = i - lane;  // the warp's 32 values: [w0, w0 + 32)
        for (int j = 0; j < w0; j += 4) {
            const float4 u = *reinterpret_cast<const float4*>(xs + j);
            cnt += (u.x <= v) + (u.y <= v) + (u.z <= v) + (u.w <= v);
        }
        for (int j = w0; j < w0 + 32; ++j) {
            const float u = xs[j];
            cnt += (u < v) || (u == v && j < i);
        }
        for (int j = w0 + 32; j < a.spad; j += 4) {
            const float4 u = *reinterpret_cast<const float4*>(xs + j);
            cnt += (u.x < v) + (u.y < v) + (u.z < v) + (u.w < v);
        }
        if (isnan(v)) {
            rk[i] = kNoRank;
        } else {
            rk[i] = (uint16_t)cnt;
            sv[cnt] = v;
        }
    }
}

struct PnrSlide {
    PnrTiles t;
    int first, n_combos;
    const int* lengths;
    const float* pfrac;
    int nsub, Q;    // a tile's T times in nsub runs of Q
    int groups;     // blocks per tile: ceil(n_combos * nsub / kSwThreads)
    int nwords;     // bitmap words per thread
    float* out;
};

// Bit operations of the two bitmap forms: 32-bit words with a 32-bit summary
// (spans up to 1,024 ranks) and 64-bit ones (up to 4,096).
__device__ __forceinline__ int low_bit(uint32_t w) { return __ffs((int)w) - 1; }
__device__ __forceinline__ int low_bit(uint64_t w) { return __ffsll((long long)w) - 1; }
__device__ __forceinline__ int high_bit(uint32_t w) { return 31 - __clz((int)w); }
__device__ __forceinline__ int high_bit(uint64_t w) { return 63 - __clzll((long long)w); }
__device__ __forceinline__ int pop(uint32_t w) { return __popc(w); }
__device__ __forceinline__ int pop(uint64_t w) { return __popcll(w); }

template <class W, int kStride>
struct RankSet {
    static constexpr int kLog = sizeof(W) == 4 ? 5 : 6;
    static constexpr int kMask = (1 << kLog) - 1;
    W* bits;  // this thread's column: word w at bits[w * kStride]
    W sum;    // bit w: word w is not zero
    __device__ __forceinline__ W& word(int w) const { return bits[w * kStride]; }
    __device__ __forceinline__ void set(int r) {
        const int w = r >> kLog;
        word(w) |= (W)1 << (r & kMask);
        sum |= (W)1 << w;
    }
    __device__ __forceinline__ void clear(int r) {
        const int w = r >> kLog;
        const W v = word(w) & ~((W)1 << (r & kMask));
        word(w) = v;
        if (v == 0) sum &= ~((W)1 << w);
    }
    __device__ __forceinline__ bool has(int r) const { return (word(r >> kLog) >> (r & kMask)) & 1; }
    // smallest member > r; r itself when there is none
    __device__ __forceinline__ int next(int r) const {
        int w = r >> kLog;
        W v = word(w) & (~(W)1 << (r & kMask));
        if (v == 0) {
            const W s = sum & (~(W)1 << w);
            if (s == 0) return r;
            w = low_bit(s);
            v = word(w);
        }
        return (w << kLog) + low_bit(v);
    }
    // largest member < r; r itself when there is none
    __device__ __forceinline__ int prev(int r) const {
        int w = r >> kLog;
        W v = word(w) & (((W)1 << (r & kMask)) - 1);
        if (v == 0) {
            const W s = sum & (((W)1 << w) - 1);
            if (s == 0) return r;
            w = high_bit(s);
            v = word(w);
        }
        return (w << kLog) + high_bit(v);
    }
    // The cursor's step in a full window: the smallest member > r (up) or the
    // largest < r, one code path for both so that the lanes do not diverge.
    // (The member exists: the caller moves toward a value it has just counted.)
    __device__ __forceinline__ int step(int r, bool up) const {
        int w = r >> kLog;
        const int b = r & kMask;
        W v = word(w) & (up ? (~(W)1 << b) : (((W)1 << b) - 1));
        if (v == 0) {
            const W s = sum & (up ? (~(W)1 << w) : (((W)1 << w) - 1));
            if (s == 0) return r;
            w = high_bit(up ? s & (~s + 1) : s);
            v = word(w);
        }
        return (w << kLog) + high_bit(up ? v & (~v + 1) : v);
    }
    // the k-th member (from 0; k < size)
    __device__ int select(int k, int nwords) const {
        for (int w = 0; w < nwords; ++w) {
            W v = word(w);
            const int c = pop(v);
            if (k < c) {
                for (; k > 0; --k) v &= v - 1;
                return (w << kLog) + low_bit(v);
            }
            k -= c;
        }
        return 0;
    }
};

// Threads take (combo, run) items, combos fastest, so a warp's lanes share
// the run's times (the entering rank is one broadcast load).  Outputs are
// staged 16 times per lane and written as 64-byte row segments.
template <class W>
__global__ void __launch_bounds__(kSwThreads) k_pnr_slide(PnrSlide a) {
    extern __shared__ __align__(16) unsigned char sw_smem[];
    const int spad = a.t.spad;
    float* sv = reinterpret_cast<float*>(sw_smem);                    // [spad]
    uint16_t* rk = reinterpret_cast<uint16_t*>(sv + spad);            // [spad] (spad is a multiple of 32)
    W* bits = reinterpret_cast<W*>(rk + spad);                        // [nwords][kSwThreads]
    float* stage = reinterpret_cast<float*>(bits + (size_t)a.nwords * kSwThreads);
    const int tid = threadIdx.x, lane = tid & 31;
    float* row = stage + tid * (kSwStage + 1);
    const float* wrow = stage + (tid - lane) * (kSwStage + 1);
    const int tile = blockIdx.x / a.groups, group = blockIdx.x - tile * a.groups;
    const int t0 = (a.t.tile0 + tile) * a.t.T;
    const int base = t0 - (a.t.lmax - 1);
    {
        const uint4* gr = reinterpret_cast<const uint4*>(a.t.rank + (size_t)tile * spad);
        const uint4* gv = reinterpret_cast<const uint4*>(a.t.val + (size_t)tile * spad);
        for (int i = tid; i < spad / 8; i += kSwThreads) reinterpret_cast<uint4*>(rk)[i] = gr[i];
        for (int i = tid; i < spad / 4; i += kSwThreads) reinterpret_cast<uint4*>(sv)[i] = gv[i];
    }
    RankSet<W, kSwThreads> set{bits + tid, 0};
    for (int w = 0; w < a.nwords; ++w) set.word(w) = 0;
    __syncthreads();
    int gap = 0;  // the span holds a NaN (or runs past an end of the series)
    for (int i = tid; i < a.t.S; i += kSwThreads) gap |= rk[i] == kNoRank;
    gap = __syncthreads_or(gap);

    const int item = group * kSwThreads + tid;
    const int j = item / a.n_combos, c = item - j * a.n_combos;
    const bool live = j < a.nsub && t0 + j * a.Q < a.t.n;
    const int q0 = live ? t0 + j * a.Q : t0;
    const int q1 = live ? q0 + min(a.Q, a.t.n - q0) : q0;
    const int len = live ? a.lengths[c] : 1;
    const double pf = live ? (double)a.pfrac[c] : 0.5;
    const int kfull = pnr::rank(pf, len);
    const int ti = max(q0, a.first + len - 1);  // this run's first output that is not warm-up
    int wl = 0, r = 0, below = 0;               // window size; the cursor and the members under it
    if (ti < q1) {
        for (int i = ti - len + 1 - base; i <= ti - base; ++i) {
            const int e = rk[i];
            if (e != kNoRank) {
                set.set(e);
                ++wl;
            }
        }
        if (wl > 0) {
            below = wl == len ? kfull : pnr::rank(pf, wl);
            r = set.select(below, a.nwords);
        }
    }
    float* orow = a.out + (size_t)c * a.t.n + q0;
    const uint16_t* in = rk + (q0 - base);
    // no gap and every lane past its warm-up: all the warp's windows are full,
    // and the cursor moves only when the two ranks lie on its two sides
    // (a lane without an item follows along on an empty set)
    const bool full = !gap && __all_sync(0xffffffffu, !live || ti == q0);
    for (int s0 = 0; s0 < a.Q; s0 += kSwStage) {
        if (full) {
            if (s0 == 0) row[0] = sv[r];
            const uint16_t* ip = in + s0;
#pragma unroll 4
            for (int s = s0 == 0 ? 1 : 0; s < kSwStage; ++s) {
                const int ro = ip[s - len], ri = ip[s];
                set.clear(ro);
                set.set(ri);
                const bool up = ro <= r && ri > r;
                if (up || (ro >= r && ri < r)) r = set.step(r, up);
                row[s] = sv[r];
            }
        }
        for (int s = 0; s < (full ? 0 : kSwStage); ++s) {
            const int t = q0 + s0 + s;
            float v = qnan();
            if (t >= ti && t < q1) {
                if (t > ti) {
                    const int ro = in[s0 + s - len], ri = in[s0 + s];
                    if (ro != kNoRank) {
                        set.clear(ro);
                        below -= ro < r;
                        --wl;
                    }
                    if (ri != kNoRank) {
                        set.set(ri);
                        below += ri < r;
                        ++wl;
                    }
                    if (wl > 0) {
                        const int k = wl == len ? kfull : pnr::rank(pf, wl);
                        if (below > k) {
                            do {
                                r = set.prev(r);
                                --below;
                            } while (below > k);
                        } else {
                            bool member = set.has(r);
                            while (!member || below < k) {
                                below += member;
                                r = set.next(r);
                                member = true;
                            }
                        }
                    }
                }
                if (wl > 0) v = sv[r];
            }
            row[s] = v;
        }
        __syncwarp();
        const int m = min(kSwStage, q1 - (q0 + s0));  // this lane's values to write
#pragma unroll 4
        for (int l = 0; l < 32; l += 2) {  // two rows a store: 16 lanes each
            const int src = l + (lane >> 4), h = lane & 15;
            const int ml = __shfl_sync(0xffffffffu, m, src);
            float* o = reinterpret_cast<float*>(
                __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(orow), src));
            if (h < ml) o[s0 + h] = wrow[src * (kSwStage + 1) + h];
        }
        __syncwarp();
    }
}

// One combo of the growing walk: its length, output row and full-window rank.
// The walk visits a percentage's combos by ascending length.
struct GrowItem {
    int len, row, kfull;
    float pf;
};
struct PnrGrow {
    PnrTiles t;
    int first;
    const int4* items;  // GrowItem
    const int2* runs;  // [gridDim.y] item ranges, each within one percentage
    int nwords;
    float* out;
};

template <class W>
__global__ void __launch_bounds__(kGrowTile) k_pnr_grow(PnrGrow a) {
    extern __shared__ __align__(16) unsigned char sw_smem[];
    const int spad = a.t.spad;
    float* sv = reinterpret_cast<float*>(sw_smem);          // [spad]
    uint16_t* rk = reinterpret_cast<uint16_t*>(sv + spad);  // [spad]
    W* bits = reinterpret_cast<W*>(rk + spad);              // [nwords][kGrowTile]
    const int tid = threadIdx.x, tile = blockIdx.x;
    {
        const uint4* gr = reinterpret_cast<const uint4*>(a.t.rank + (size_t)tile * spad);
        const uint4* gv = reinterpret_cast<const uint4*>(a.t.val + (size_t)tile * spad);
        for (int i = tid; i < spad / 8; i += kGrowTile) reinterpret_cast<uint4*>(rk)[i] = gr[i];
        for (int i = tid; i < spad / 4; i += kGrowTile) reinterpret_cast<uint4*>(sv)[i] = gv[i];
    }
    RankSet<W, kGrowTile> set{bits + tid, 0};
    for (int w = 0; w < a.nwords; ++w) set.word(w) = 0;
    const int t = (a.t.tile0 + tile) * kGrowTile + tid;
    __syncthreads();
    if (t >= a.t.n) return;
    const int2 run = a.runs[blockIdx.y];
    float* out = a.out + t;
    int cur = 0, wl = 0, r = -1, below = 0;  // values entered; window size; cursor (-1: none yet) and members under it
    const uint16_t* at = rk + tid + a.t.lmax - 1;  // x[t - cur]
    for (int e = run.x; e < run.y; ++e) {
        const int4 raw = __ldg(a.items + e);
        const GrowItem it{raw.x, raw.y, raw.z, __int_as_float(raw.w)};
        for (; cur < it.len; ++cur, --at) {
            const int ri = *at;
            if (ri != kNoRank) {
                set.set(ri);
                below += ri < r;
                ++wl;
            }
        }
        float v = qnan();
        if (wl > 0) {
            const int k = wl == it.len ? it.kfull : pnr::rank((double)it.pf, wl);
            if (r < 0) {
                r = set.select(k, a.nwords);
                below = k;
            }
            while (below != k) {
                const bool up = below < k;
                r = set.step(r, up);
                below += up ? 1 : -1;
            }
            if (t >= a.first + it.len - 1) v = sv[r];
        }
        out[(size_t)it.row * a.t.n] = v;
    }
}

constexpr int kMaxSpan = 4096;              // ranks of the 64-bit bitmap form
constexpr int kMinTile = 256, kMaxTile = 1024;
constexpr size_t kMaxGridY = 65535;         // runs of a launch of the growing walk
constexpr size_t kSlabBytes = size_t(128) << 20;  // ranks and values of one slab of tiles

// Times per tile: the largest of 256, 512, 1024 that is at most the longest
// window (a run starts by entering its window's len members, so tiles not
// shorter than the window keep that below one step in two) and keeps the
// span within the bitmap.
int tile_times(int lmax) {
    int T = kMaxTile;
    while (T > kMinTile && (T > lmax || T + lmax - 1 > kMaxSpan)) T >>= 1;
    return T;
}

// The tiles of a sweep of series length n and longest window lmax, T times
// each, with the slab that kSlabBytes hold.
struct Geo {
    int T, S, spad;
    long long tiles, slab;
    size_t bytes;  // ranks and values of a slab
};
Geo geo(int n, int lmax, int T) {
    Geo g{};
    g.T = T;
    g.S = T + lmax - 1;
    g.spad = (g.S + 31) & ~31;
    g.tiles = ceil_div(n, T);
    const size_t per = (size_t)g.spad * (sizeof(float) + sizeof(uint16_t));
    g.slab = std::min<long long>(g.tiles, (long long)std::max<size_t>(1, kSlabBytes / per));
    g.bytes = (size_t)g.slab * per;
    return g;
}

// Which walk: the growing one enters the longest window's values per time and
// percentage whatever the number of combos, the sliding one pays two bitmap
// updates and the row staging per output and its own window's entry per run.
// Growing / sliding at 100k bars, 264 the longest length: 250 lengths 147 / 161
// us, 165 lengths 111 / 123, 85 lengths 96 / 92, 43 lengths 80 / 76, one length
// 37 / 47; 50k bars, 101 lengths 1000..2000: 542 / 369.  So growing up to 2.5
// values entered per combo; and for up to 12 combos, whose sliding runs are
// short (11 lengths 600..700 on 50k bars: 92 / 99).
bool grow_better(long long entered, int n_combos) { return 2 * entered <= 5LL * n_combos || n_combos <= 12; }

}  // namespace

// Longest window the rank sweep takes: its span has to fit the bitmap.
// (Times are int: the last tile may run kMaxTile past n.)
bool pnr_sweep_ok(int n, int lmax) { return kMinTile + lmax - 1 <= kMaxSpan && n <= INT32_MAX - kMaxTile; }

PnrPlan pnr_plan(int n, const std::vector<int>& lengths, const std::vector<float>& pfrac, int num_sms) {
    PnrPlan p;
    const int nc = (int)lengths.size();
    p.lmax = *std::max_element(lengths.begin(), lengths.end());
    std::vector<int> order(nc);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return pfrac[x] != pfrac[y] ? pfrac[x] < pfrac[y] : lengths[x] < lengths[y];
    });
    long long entered = 0;  // values a growing walk enters per time
    int npf = 0;
    for (int i = 0; i < nc; ++i)
        if (i + 1 == nc || pfrac[order[i + 1]] != pfrac[order[i]]) {
            entered += lengths[order[i]];
            ++npf;
        }
    p.grow = grow_better(entered, nc);
    const Geo g = geo(n, p.lmax, p.grow ? kGrowTile : tile_times(p.lmax));
    p.work_bytes = g.bytes + 256;
    if (!p.grow) return p;
    // runs: one per percentage, cut further until the blocks make about four
    // per SM; a cut run enters its first window anew (eight: 3 to 10% slower)
    const long long want = std::max(1LL, (4LL * num_sms) / std::max(1LL, g.tiles * npf));
    for (int i0 = 0; i0 < nc;) {
        int i1 = i0;
        while (i1 < nc && pfrac[order[i1]] == pfrac[order[i0]]) ++i1;
        const int parts = (int)std::max(1LL, std::min<long long>(want, (i1 - i0) / 8));
        for (int q = 0; q < parts; ++q)
            p.runs.push_back({i0 + (int)((long long)(i1 - i0) * q / parts),
                              i0 + (int)((long long)(i1 - i0) * (q + 1) / parts)});
        i0 = i1;
    }
    for (int c : order) {
        const long long raw = (long long)std::round(std::fma((double)pfrac[c], (double)lengths[c], 0.0)) - 1;
        const int k = raw <= 0 ? 0 : (int)std::min<long long>(raw, lengths[c] - 1);
        p.items.push_back({lengths[c], c, k, 0});
        std::memcpy(&p.items.back().w, &pfrac[c], sizeof(float));
    }
    return p;
}

vta_status launch_pnr_sweep(const PnrArgs& p, const PnrPlan& plan, const int4* items, const int2* runs, int num_sms,
                            cudaStream_t st) {
    const Geo g = geo(p.n, plan.lmax, plan.grow ? kGrowTile : tile_times(plan.lmax));
    PnrTiles t{};
    t.x = p.x;
    t.n = p.n;
    t.lmax = plan.lmax;
    t.T = g.T;
    t.S = g.S;
    t.spad = g.spad;
    t.val = p.scratch;
    t.rank = reinterpret_cast<uint16_t*>(p.scratch + (size_t)g.slab * g.spad);
    const bool wide = g.spad > 1024;
    const int word = wide ? 8 : 4;
    const int nwords = (g.spad + 8 * word - 1) / (8 * word);
    const size_t tables = (size_t)g.spad * (sizeof(float) + sizeof(uint16_t));
    // a whole number of values per thread, as nearly equal as warps allow
    const int rank_passes = ceil_div(g.spad, 512);
    const int rank_threads = ceil_div(ceil_div(g.spad, rank_passes), 32) * 32;

    PnrSlide s{};
    PnrGrow w{};
    size_t smem = 0;
    auto slide = wide ? k_pnr_slide<uint64_t> : k_pnr_slide<uint32_t>;
    auto grow = wide ? k_pnr_grow<uint64_t> : k_pnr_grow<uint32_t>;
    if (plan.grow) {
        w.first = p.first;
        w.items = items;
        w.nwords = nwords;
        w.out = p.out;
        smem = tables + (size_t)nwords * kGrowTile * word;
        VTA_CUDA_TRY(cudaFuncSetAttribute(grow, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    } else {
        s.first = p.first;
        s.n_combos = p.n_lanes;
        s.lengths = p.lengths;
        s.pfrac = p.pfrac;
        s.out = p.out;
        s.nwords = nwords;
        smem = tables + (size_t)nwords * kSwThreads * word + (size_t)kSwThreads * (kSwStage + 1) * sizeof(float);
        VTA_CUDA_TRY(cudaFuncSetAttribute(slide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, slide, kSwThreads, smem) != cudaSuccess ||
            per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        // few combos: split the tile's times until the threads fill the GPU
        const long long room = (long long)num_sms * per_sm * kSwThreads;
        s.nsub = 1;
        while (g.T / (2 * s.nsub) >= 2 * kSwStage && g.tiles * p.n_lanes * s.nsub * 2 <= room) s.nsub *= 2;
        s.Q = g.T / s.nsub;
        const long long groups = ceil_div((size_t)p.n_lanes * s.nsub, kSwThreads);
        if (groups * g.slab > INT32_MAX) return fail(VTA_ERR_LAUNCH_CONFIG_TOO_LARGE, "percentile: too many combos");
        s.groups = (int)groups;
    }
    ktimer_begin(st);
    for (long long t0 = 0; t0 < g.tiles; t0 += g.slab) {
        const unsigned m = (unsigned)std::min(g.slab, g.tiles - t0);
        t.tile0 = (int)t0;
        k_pnr_ranks<<<m, rank_threads, (size_t)g.spad * sizeof(float), st>>>(t);
        VTA_TRY(check_launch("k_pnr_ranks"));
        s.t = w.t = t;
        if (plan.grow) {
            for (size_t r = 0; r < plan.runs.size(); r += kMaxGridY) {
                w.runs = runs + r;
                grow<<<dim3(m, (unsigned)std::min(kMaxGridY, plan.runs.size() - r)), kGrowTile, smem, st>>>(w);
                VTA_TRY(check_launch("k_pnr_grow"));
            }
        } else {
            slide<<<s.groups * m, kSwThreads, smem, st>>>(s);
            VTA_TRY(check_launch("k_pnr_slide"));
        }
    }
    ktimer_end(st);
    return VTA_OK;
}

}  // namespace vta
