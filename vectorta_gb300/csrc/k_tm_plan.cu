// Many-series work-list kernels: several indicators over one set of ragged
// time-major OHLC series in one persistent launch.
//
// Work items are (job, time chunk, up to 32 of the series that reach the
// chunk).  A warp takes items from a global counter; its lanes own consecutive
// entries of the chunk's list of series, which are adjacent series as long as
// all of them reach it (every load and store of a time step is then one
// 128-byte row segment) and skip the ones that have ended after that: with
// lengths spread over [1,000, 20,000] fixed tiles of 32 series left half the
// lanes idle.  Series of uneven length stop at their own length: cells past it
// are neither read nor written.
//
// Recurrent jobs (ATR, ADX, SuperTrend) are cut into time chunks with a
// verified warm restart.  Chunk k (c0 = k * chunk) that starts past the
// indicator's seeding phase runs `warm` steps before c0 from a state guessed
// from the inputs; since every state component decays by (1 - 1/p) per step
// the guess is forgotten, and the state it reaches at c0 is recorded.  Every
// chunk also records its state at its end.  k_tm_fixup then walks each
// series' chunks in order and compares (bit for bit) the recorded start state
// of chunk k with the end state of chunk k - 1; where they differ it recomputes
// chunk k from that exact end state.  The outputs are therefore bit-identical
// to one sequential pass over the series, whatever the chunk and warm lengths.
// The percentile job is exact per chunk by construction (its window is
// rebuilt from the `length` inputs before c0).
#include <cfloat>
#include <climits>

#include "vta_internal.h"
#include "vta_plan.h"
#include "hlc_ops.cuh"
#include "pnr_ops.cuh"

namespace vta {
namespace {

__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

struct TmIn {
    const float *h, *l, *c;
    size_t cols, s;
    __device__ float H(int t) const { return __ldg(h + (size_t)t * cols + s); }
    __device__ float L(int t) const { return __ldg(l + (size_t)t * cols + s); }
    __device__ float C(int t) const { return __ldg(c + (size_t)t * cols + s); }
};

using hlc::PAtr;
using hlc::PAdx;
using hlc::PSuperTrend;

// ------------------------------------------------ nearest-rank percentile ---
// (the sorted register window of pnr_ops.cuh)
using pnr::pick;
using pnr::rank;

// ------------------------------------------------ chunk runners -------------
// Inputs are staged per warp in shared memory: a ring of kPS blocks of kPB
// steps x {high, low, close} x 32 lanes, filled with cp.async (4 bytes per lane
// and value, so each step of a warp is one 128-byte row segment when its
// series are adjacent).  Each lane copies and reads only its own column, so no
// cross-lane synchronisation is needed; kPS - 1 blocks are in flight while one
// is computed (the recurrences take about 20 issue slots a step, far less than
// a memory round trip per block).
constexpr int kPB = 8;
constexpr int kPS = 4;
constexpr int kStageFloats = kPS * 3 * kPB * 32;  // per warp
constexpr size_t kPlanSmem = (size_t)kPlanWarps * kStageFloats * sizeof(float);

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct Stage {
    float* base;  // this warp's [kPS][3][kPB][32]
    int lane;
    __device__ __forceinline__ float* at(int buf, int arr, int j) const {
        return base + ((buf * 3 + arr) * kPB + j) * 32 + lane;
    }
};

// A lane's seeding: its state at run_from() and the outputs of the step before
// it (every op's first ones).  rf: run_from(), or kNever for a series too short
// to be seeded, whose outputs are all NaN.
constexpr int kNever = INT_MAX;
struct Seed {
    int rf;
    float y0, y1;
};

// Runs the seeding steps [f, run_from()) of every lane of the warp, each on
// rows of its own: the step index relative to f is the warp's, so the lanes
// pass the op's phases together whatever their first valid rows are.
template <class Op>
__device__ Seed run_seed(Op& op, const TmIn& in, int f, int L) {
    const int n = op.run_from() - f;  // (the same for all lanes)
    const bool ok = f < L && n <= L - f;
    Seed sd{ok ? f + n : kNever, qnan(), qnan()};
    op.start_exact();
    for (int r = 0; r < n; r += kPB) {
        float hv[kPB], lv[kPB], cv[kPB];
#pragma unroll
        for (int j = 0; j < kPB; ++j) {
            const int t = ok ? f + min(r + j, n - 1) : 0;
            hv[j] = in.H(t);
            lv[j] = in.L(t);
            cv[j] = in.C(t);
        }
#pragma unroll
        for (int j = 0; j < kPB; ++j)
            if (r + j < n) sd.y0 = op.stepv(f + r + j, hv[j], lv[j], cv[j], sd.y1);
    }
    return sd;
}

// Steps t in [t, tend) of each lane; EMIT writes the outputs of each step.  t
// is the same for the lanes of `mask` (all call); they run in step to the
// latest tend.  A lane takes part from its sd.rf on, and past its own tend
// computes on without storing (its state is not read again: tend is either the
// warp's or the end of the lane's series).
template <bool EMIT, class Op>
__device__ void run_span(Op& op, const TmIn& in, const Stage& sg, unsigned mask, const Seed& sd, int t, int tend,
                         float* out0, float* out1) {
    const int te = __reduce_max_sync(mask, tend);
    const int rf = __reduce_max_sync(mask, sd.rf == kNever ? INT_MIN : sd.rf);
    if (t >= te) return;
    const size_t row0 = (size_t)t * in.cols + in.s;
    const float *gh = in.h + row0, *gl = in.l + row0, *gc = in.c + row0;  // next row to load
    int tl = t;
    auto load = [&](int buf) {  // (an empty group past the end keeps the count)
#pragma unroll
        for (int j = 0; j < kPB; ++j) {
            if (tl + j < tend) {
                cp_async4(sg.at(buf, 0, j), gh + (size_t)j * in.cols);
                cp_async4(sg.at(buf, 1, j), gl + (size_t)j * in.cols);
                cp_async4(sg.at(buf, 2, j), gc + (size_t)j * in.cols);
            }
        }
        tl += kPB;
        gh += kPB * in.cols;
        gl += kPB * in.cols;
        gc += kPB * in.cols;
        cp_async_commit();
    };
#pragma unroll
    for (int q = 0; q < kPS - 1; ++q) load(q);
    float* o0 = out0 + row0;
    float* o1 = Op::kTwo ? out1 + row0 : nullptr;
    int buf = 0;
    for (int tb = t; tb < te; tb += kPB, buf = (buf + 1) & (kPS - 1)) {
        load((buf + kPS - 1) & (kPS - 1));
        cp_async_wait<kPS - 1>();
        float hv[kPB], lv[kPB], cv[kPB];
#pragma unroll
        for (int j = 0; j < kPB; ++j) {
            hv[j] = *sg.at(buf, 0, j);
            lv[j] = *sg.at(buf, 1, j);
            cv[j] = *sg.at(buf, 2, j);
        }
        auto put = [&](int j, float y0, float y1) {
            if (EMIT && tb + j < tend) {
                o0[(size_t)j * in.cols] = y0;
                if (Op::kTwo) o1[(size_t)j * in.cols] = y1;
            }
        };
        const bool never = sd.rf == kNever;
        if (tb >= rf && tb + kPB <= te) {
#pragma unroll
            for (int j = 0; j < kPB; ++j) {
                float y1 = qnan();
                const float y0 = op.step_run(hv[j], lv[j], cv[j], y1);
                put(j, never ? qnan() : y0, never ? qnan() : y1);
            }
        } else {
#pragma unroll
            for (int j = 0; j < kPB; ++j) {
                const int tt = tb + j;
                if (tt >= te) break;
                float y0 = qnan(), y1 = qnan();
                if (tt >= sd.rf) {
                    y0 = op.step_run(hv[j], lv[j], cv[j], y1);
                } else if (tt == sd.rf - 1) {
                    y0 = sd.y0;
                    y1 = sd.y1;
                }
                put(j, y0, y1);
            }
        }
        o0 += kPB * in.cols;
        if (Op::kTwo) o1 += kPB * in.cols;
    }
}

// Percentile chunk [c0, c1) of each lane.  All lanes of the warp run one
// time loop over [c0 - len + 1, max c1) in step: each step removes the value
// leaving the window and inserts the one entering (NaN values are never in
// the window, which also covers the NaN lead), and writes its output when
// the step is inside the lane's own chunk.  A lane whose series has ended
// follows along without inserting or writing.  Keeping the lanes on one
// loop (instead of each running its own window build and loop) keeps the
// warp converged.
template <int W>
__device__ void pnr_chunk(const TmIn& in, const Stage& sg, unsigned mask, int f, int L, int len, double pf, int c0,
                          int c1, float* out) {
    const int tend = __reduce_max_sync(mask, c1);
    if (tend <= c0) return;  // warp-uniform
    const int tbeg = max(0, c0 - len + 1);
    const int start = f + len - 1;
    const int kfull = rank(pf, len);
    float w[W];
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = __int_as_float(0x7f800000);
    int wl = 0;
    // staged arrays: 0 = entering x[u], 1 = leaving x[u - len]
    auto load = [&](int buf, int ub) {
        for (int j = 0; j < kPB && ub + j < tend; ++j) {
            const int u = ub + j, uo = u - len;
            if (u < L) cp_async4(sg.at(buf, 0, j), in.c + (size_t)u * in.cols + in.s);
            if (uo >= tbeg && uo < L) cp_async4(sg.at(buf, 1, j), in.c + (size_t)uo * in.cols + in.s);
        }
        cp_async_commit();
    };
    load(0, tbeg);
    int buf = 0;
    for (int ub = tbeg; ub < tend; ub += kPB, buf ^= 1) {
        load(buf ^ 1, ub + kPB);
        cp_async_wait<1>();
        const int ue = min(ub + kPB, tend);
        for (int u = ub; u < ue; ++u) {
            const int j = u - ub, uo = u - len;
            const float vo = (uo >= tbeg && uo < L) ? *sg.at(buf, 1, j) : qnan();
            const float vi = u < L ? *sg.at(buf, 0, j) : qnan();
            pnr::replace(w, vo, vi);
            wl += (isnan(vi) ? 0 : 1) - (isnan(vo) ? 0 : 1);
            if (u >= c0 && u < c1)
                out[(size_t)u * in.cols + in.s] = u < start ? qnan() : pick(w, wl, len, kfull, pf);
        }
    }
    cp_async_wait<0>();
}

// One item of a recurrent job; `mask`: the lanes of the warp working on it
// (all of them call).  The warm restart and the run from the series start give
// the same bits, so one lane that cannot restart (its seeding is too near)
// makes all of them run from their seeds rather than split the warp.
template <class Op>
__device__ void run_chunk(const PlanArgs& a, const PlanJob& J, int s, int k, const Stage& sg, unsigned mask) {
    const int L = a.len[s];
    const int c0 = k * J.chunk;
    const int f = a.first_hlc[s];
    const unsigned live = __ballot_sync(mask, c0 < L);
    if (c0 >= L) return;
    const int c1 = min(c0 + J.chunk, L);
    Op op;
    op.init(J.period, J.param, f);
    const TmIn in{a.h, a.l, a.c, (size_t)a.cols, (size_t)s};
    const size_t sidx = (size_t)k * a.cols + s;
    // (a series without a valid bar has nothing to restart or compute)
    const bool exact = __any_sync(live, k == 0 || (f < L && c0 - J.warm < op.run_from()));
    Seed sd;
    int t;
    if (!exact) {
        t = c0 - J.warm;
        sd = Seed{f < L ? t : kNever, qnan(), qnan()};
        op.start_exact();
        if (f < L) op.start_warm(in, t);
    } else {
        sd = run_seed(op, in, f, L);
        t = __reduce_min_sync(live, min(sd.rf, c0));
    }
    run_span<false>(op, in, sg, live, sd, t, c0, J.out0, J.out1);
    float w[8];
    if (k > 0) {
        op.save(w);
        float4* d = reinterpret_cast<float4*>(J.st_start + sidx * 8);
        d[0] = make_float4(w[0], w[1], w[2], w[3]);
        d[1] = make_float4(w[4], w[5], w[6], w[7]);
        J.exact[sidx] = exact || f >= L ? 1 : 0;
    }
    run_span<true>(op, in, sg, live, sd, c0, c1, J.out0, J.out1);
    op.save(w);
    float4* d = reinterpret_cast<float4*>(J.st_end + sidx * 8);
    d[0] = make_float4(w[0], w[1], w[2], w[3]);
    d[1] = make_float4(w[4], w[5], w[6], w[7]);
}

// `mask`: the lanes of the warp working on this item (all of them call).
__device__ void run_pnr(const PlanArgs& a, const PlanJob& J, int s, int k, const Stage& sg, unsigned mask) {
    const int L = a.len[s];
    const int c0 = k * J.chunk;
    const int c1 = max(c0, min(c0 + J.chunk, L));
    const TmIn in{a.h, a.l, a.c, (size_t)a.cols, (size_t)s};
    const int f = a.first_c[s];
    // window registers: the length rounded up to a multiple of 4
    switch (max(4, (J.period + 3) >> 2)) {
        case 4: pnr_chunk<16>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 5: pnr_chunk<20>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 6: pnr_chunk<24>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 7: pnr_chunk<28>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 8: pnr_chunk<32>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 9: pnr_chunk<36>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 10: pnr_chunk<40>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 11: pnr_chunk<44>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 12: pnr_chunk<48>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 13: pnr_chunk<52>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 14: pnr_chunk<56>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        case 15: pnr_chunk<60>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
        default: pnr_chunk<64>(in, sg, mask, f, L, J.period, J.pfrac, c0, c1, J.out0); break;
    }
}

// Persistent work-list kernel: each warp takes items until the list is done.
// A warp's first item is its rank in the order (warp of the block, block), so a
// list shorter than the grid's warps is spread evenly over the SMs (blocks are
// placed round-robin); the others come from the counter.
__global__ void __launch_bounds__(kPlanWarps * 32) k_tm_plan(PlanArgs a) {
    extern __shared__ float plan_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Stage sg{plan_smem + warp * kStageFloats, lane};
    const int n_warps = gridDim.x * kPlanWarps;
    int it = warp * gridDim.x + blockIdx.x;
    while (it < a.n_items) {
        const int4 w = a.items[it];  // {job, first entry of a.lanes, chunk, lanes}
        const unsigned mask = __ballot_sync(0xffffffffu, lane < w.w);
        if (lane < w.w) {
            const int s = a.lanes[w.y + lane];
            const PlanJob& J = a.jobs[w.x];
            switch (J.kind) {
                case PJ_ATR: run_chunk<PAtr>(a, J, s, w.z, sg, mask); break;
                case PJ_ADX: run_chunk<PAdx>(a, J, s, w.z, sg, mask); break;
                case PJ_SUPERTREND: run_chunk<PSuperTrend>(a, J, s, w.z, sg, mask); break;
                default: run_pnr(a, J, s, w.z, sg, mask); break;
            }
        }
        __syncwarp();
        if (lane == 0) it = n_warps + atomicAdd(a.counter, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
    }
}

// Fix-up of a (recurrent job, 32 series) block: its warps compare, over all
// chunks at once, the recorded start state of each warm-restarted chunk with
// the end state of the chunk before it.  Series with a mismatch (rare) then
// take their chunks in order: one whose start state differs from the end state
// that now stands before it is recomputed from that.
constexpr int kFixWarps = 8;

__device__ __forceinline__ bool same_state(const PlanJob& J, size_t sidx, size_t pidx) {
    const uint4* ps = reinterpret_cast<const uint4*>(J.st_start + sidx * 8);
    const uint4* pe = reinterpret_cast<const uint4*>(J.st_end + pidx * 8);
    const uint4 s0 = ps[0], s1 = ps[1], e0 = pe[0], e1 = pe[1];
    return s0.x == e0.x && s0.y == e0.y && s0.z == e0.z && s0.w == e0.w && s1.x == e1.x && s1.y == e1.y &&
           s1.z == e1.z && s1.w == e1.w;
}

template <class Op>
__device__ void fixup_series(const PlanArgs& a, const PlanJob& J, int s) {
    const int L = a.len[s];
    const TmIn in{a.h, a.l, a.c, (size_t)a.cols, (size_t)s};
    for (int k = 1; k * J.chunk < L; ++k) {
        const size_t sidx = (size_t)k * a.cols + s;
        if (J.exact[sidx]) continue;
        const size_t pidx = sidx - a.cols;
        if (same_state(J, sidx, pidx)) continue;
        const int c0 = k * J.chunk;
        const int c1 = min(c0 + J.chunk, L);
        Op op;
        op.init(J.period, J.param, a.first_hlc[s]);
        const float* we = J.st_end + pidx * 8;
        float w[8];
        for (int i = 0; i < 8; ++i) w[i] = we[i];
        op.load(w, in, c0);
        float o1;
        for (int t = c0; t < c1; ++t) {
            const float o0 = op.step(in, t, o1);
            J.out0[(size_t)t * a.cols + s] = o0;
            if (Op::kTwo) J.out1[(size_t)t * a.cols + s] = o1;
        }
        op.save(w);
        float4* d = reinterpret_cast<float4*>(J.st_end + sidx * 8);
        d[0] = make_float4(w[0], w[1], w[2], w[3]);
        d[1] = make_float4(w[4], w[5], w[6], w[7]);
        atomicAdd(&a.stats[0], 1);
    }
}

__global__ void __launch_bounds__(32 * kFixWarps) k_tm_fixup(PlanArgs a) {
    const PlanJob& J = a.jobs[blockIdx.y];
    if (J.kind == PJ_PERCENTILE) return;
    __shared__ int need[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = blockIdx.x * 32 + lane;
    const int L = s < a.cols ? a.len[s] : 0;
    if (warp == 0) need[lane] = 0;
    __syncthreads();
    for (int k = 1 + warp; (long long)k * J.chunk < L; k += kFixWarps) {
        const size_t sidx = (size_t)k * a.cols + s;
        if (!J.exact[sidx] && !same_state(J, sidx, sidx - a.cols)) need[lane] = 1;
    }
    __syncthreads();
    if (warp != 0 || !need[lane]) return;
    switch (J.kind) {
        case PJ_ATR: fixup_series<PAtr>(a, J, s); break;
        case PJ_ADX: fixup_series<PAdx>(a, J, s); break;
        default: fixup_series<PSuperTrend>(a, J, s); break;
    }
}

}  // namespace

vta_status launch_plan_first(const PlanArgs& a, int* first_hlc, int* first_c, cudaStream_t st) {
    return launch_first_valid_tm_hlc(a.h, a.l, a.c, a.cols, a.rows, first_hlc, st, a.len, first_c);
}

int tm_plan_blocks(int num_sms) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tm_plan, kPlanWarps * 32, kPlanSmem) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    return num_sms * per_sm;
}

vta_status launch_tm_plan(const PlanArgs& a, int blocks, cudaStream_t st) {
    k_tm_plan<<<blocks, kPlanWarps * 32, kPlanSmem, st>>>(a);
    return check_launch("k_tm_plan");
}

vta_status launch_tm_fixup(const PlanArgs& a, cudaStream_t st) {
    k_tm_fixup<<<dim3((a.cols + 31) / 32, a.n_jobs), 32 * kFixWarps, 0, st>>>(a);
    return check_launch("k_tm_fixup");
}

}  // namespace vta
