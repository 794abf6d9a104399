// Time-chunked single-series sweeps of ADX and SuperTrend (batch layout:
// one series, lane = parameter combo).
//
// The sequential kernels (k_hlc.cu) run one lane per combo over the whole
// series, so a sweep of a few hundred combos keeps a few warps busy for the
// series' full length.  Here the combos of a 32-combo group are also cut into
// time chunks with the verified warm restart of the many-series plans: a
// chunk that starts past the seeding phase first runs `warm` steps from a
// guessed state (the state decays by (1 - 1/p) per step), records the state
// it reaches at its start and at its end, and k_hlc_chunk_fixup recomputes,
// per combo and in chunk order, every chunk whose recorded start state differs
// (bit for bit) from its predecessor's end state.  Results are therefore
// bit-identical to the sequential kernels.
//
// A warp owns one (group, chunk) item.  What a step takes from the bars alone
// (TR, +DM, -DM; TR, (high + low) / 2, close) is the same for every combo, so
// each lane forms it for one bar of a 32-step tile and the warp reads it back
// from shared memory, four steps per 16-byte broadcast load; the next tile's
// bars are on their way meanwhile.  Outputs are staged per warp in shared
// memory and written as 32 rows x 128 bytes, unrolled.  Seeding steps are
// selects, no branches: a 400-period seeding run is 900 of them in one chain.
// Bound by the chain of one or two warps per scheduler (about 16 instructions
// a step): ADX periods 2..97 on 1M bars 361 -> 177 us with these four.
#include <algorithm>

#include "hlc_item.cuh"
#include "vta_internal.h"

namespace vta {
namespace {

using hlc::In1;
using hlc::store_state;

constexpr int kCW = 4;  // warps per block

template <class Op>
__global__ void __launch_bounds__(kCW * 32) k_hlc_chunk(HlcChunkArgs a) {
    __shared__ hlc::ItemSmem<Op> sm[kCW];
    const int warp = threadIdx.x >> 5;
    const int item = blockIdx.x * kCW + warp;
    if (item < a.n_items) hlc::run_item<Op>(a, item, sm[warp]);
}

__device__ __forceinline__ bool same_state(const float* x, const float* y) {
    const uint4* p = reinterpret_cast<const uint4*>(x);
    const uint4* q = reinterpret_cast<const uint4*>(y);
    const uint4 a0 = p[0], a1 = p[1], b0 = q[0], b1 = q[1];
    return a0.x == b0.x && a0.y == b0.y && a0.z == b0.z && a0.w == b0.w && a1.x == b1.x && a1.y == b1.y &&
           a1.z == b1.z && a1.w == b1.w;
}

// All (chunk, combo) pairs in parallel: count, per combo, the warm-restarted
// chunks whose start state differs from the end state the kernel left before
// them.  Combos with none need no sequential pass.
__global__ void k_hlc_mismatch(HlcChunkArgs a) {
    const int li = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y + 1;
    if (li >= a.n_combos) return;
    if ((long long)k * a.group_chunk[li >> 5] >= a.n) return;
    const size_t sidx = (size_t)k * a.n_combos + li;
    if (a.exact[sidx]) return;
    if (!same_state(a.st_start + sidx * 8, a.st_end + (sidx - a.n_combos) * 8)) atomicAdd(&a.need[li], 1);
}

// Per combo with a mismatch, chunks in order: a warm-restarted chunk whose
// start state is not its predecessor's end state is recomputed from that end
// state (which may itself have been recomputed just before).
template <class Op>
__global__ void k_hlc_chunk_fixup(HlcChunkArgs a) {
    const int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= a.n_combos || a.need[li] == 0) return;
    const int chunk = a.group_chunk[li >> 5];
    const In1 in{a.h, a.l, a.c};
    for (int k = 1; (long long)k * chunk < a.n; ++k) {
        const size_t sidx = (size_t)k * a.n_combos + li, pidx = sidx - a.n_combos;
        if (a.exact[sidx]) continue;
        if (same_state(a.st_start + sidx * 8, a.st_end + pidx * 8)) continue;
        const int c0 = k * chunk, c1 = min(c0 + chunk, a.n);
        Op op;
        op.init(a.periods[li], a.factors ? a.factors[li] : 0.f, a.first);
        float w[8];
        for (int i = 0; i < 8; ++i) w[i] = a.st_end[pidx * 8 + i];
        op.load(w, in, c0);
        for (int t = c0; t < c1; ++t) {
            float o1;
            const float o0 = op.step(in, t, o1);
            a.out0[(size_t)li * a.n + t] = o0;
            if (Op::kTwo) a.out1[(size_t)li * a.n + t] = o1;
        }
        op.save(w);
        store_state(a.st_end + sidx * 8, w);
        atomicAdd(a.fixups, 1);
    }
}

}  // namespace

vta_status launch_hlc_fixup(const HlcChunkArgs& a, cudaStream_t st) {
    if (a.max_chunks <= 1) return VTA_OK;
    const unsigned fix_blocks = ceil_div(a.n_combos, 128);
    const dim3 mm_grid(fix_blocks, (unsigned)(a.max_chunks - 1));
    k_hlc_mismatch<<<mm_grid, 128, 0, st>>>(a);
    VTA_TRY(check_launch("k_hlc_mismatch"));
    if (a.kind == 0) k_hlc_chunk_fixup<hlc::PAdx><<<fix_blocks, 128, 0, st>>>(a);
    else k_hlc_chunk_fixup<hlc::PSuperTrend><<<fix_blocks, 128, 0, st>>>(a);
    return check_launch("k_hlc_chunk_fixup");
}

vta_status launch_hlc_chunk(const HlcChunkArgs& a, cudaStream_t st) {
    const unsigned blocks = ceil_div(a.n_items, kCW);
    ktimer_begin(st);
    if (a.kind == 0) k_hlc_chunk<hlc::PAdx><<<blocks, kCW * 32, 0, st>>>(a);
    else k_hlc_chunk<hlc::PSuperTrend><<<blocks, kCW * 32, 0, st>>>(a);
    VTA_TRY(check_launch("k_hlc_chunk"));
    VTA_TRY(launch_hlc_fixup(a, st));
    ktimer_end(st);
    return VTA_OK;
}

}  // namespace vta
