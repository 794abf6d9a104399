// One (group, chunk) item of the warm-restart sweeps of ADX and SuperTrend by
// one warp (k_hlc_chunk.cu says how they are cut; k_adx_scan.cu runs the same
// items beside its passes).
#pragma once
#include <type_traits>

#include "hlc_ops.cuh"
#include "vta_internal.h"

namespace vta {
namespace hlc {

// ops with a wide-tile step form (hlc_ops.cuh)
template <class Op, class = void> struct HasWide : std::false_type {};
template <class Op> struct HasWide<Op, std::void_t<decltype(Op::kWide)>> : std::true_type {};

struct In1 {
    const float *h, *l, *c;
    __device__ float H(int t) const { return __ldg(h + t); }
    __device__ float L(int t) const { return __ldg(l + t); }
    __device__ float C(int t) const { return __ldg(c + t); }
};

__device__ __forceinline__ void store_state(float* dst, const float (&w)[8]) {
    float4* d = reinterpret_cast<float4*>(dst);
    d[0] = make_float4(w[0], w[1], w[2], w[3]);
    d[1] = make_float4(w[4], w[5], w[6], w[7]);
}

// a warp's shared memory
template <class Op> struct ItemSmem {
    float stage0[32][33];
    float stage1[Op::kTwo ? 32 : 1][33];
    float4 xin[3][8];  // a tile's terms
};

template <class Op>
__device__ __forceinline__ void run_item(const HlcChunkArgs& a, int item, ItemSmem<Op>& sm) {
    const int lane = threadIdx.x & 31;
    const int2 it = a.items[item];
    const int g = it.x, k = it.y;
    const int chunk = a.group_chunk[g];
    const int c0 = k * chunk;
    const int c1 = min(c0 + chunk, a.n);
    const int li = g * 32 + lane;
    const bool valid = li < a.n_combos;
    const int lc = valid ? li : g * 32;  // idle lanes shadow the group's first combo (nothing written)
    Op op;
    op.init(a.periods[lc], a.factors ? a.factors[lc] : 0.f, a.first);
    const In1 in{a.h, a.l, a.c};
    const int W = a.group_warm[g];  // multiple of 32
    const bool warm = k > 0 && __all_sync(0xffffffffu, c0 - W >= op.run_from());
    int t0;
    if (warm) {
        t0 = c0 - W;
        op.start_warm(in, t0);
    } else {
        t0 = min(a.first, c0) & ~31;
        op.start_exact();
    }
    // from rf on every lane of the warp is in its running phase
    const int rf = __reduce_max_sync(0xffffffffu, op.run_from());
    // tiles of 32 steps over [tb0, tend); with `emit` the outputs go to the rows
    // (the next tile's bars are loaded while this one is worked on)
    const int rows = min(32, a.n_combos - g * 32);
    auto tiles = [&](int tb0, int tend, auto emit_tag) {
        constexpr bool emit = decltype(emit_tag)::value;
        float nh = 0.f, nl = 0.f, nc = 0.f;
        auto fetch = [&](int t) {
            if (t < tend) {
                nh = __ldg(a.h + t);
                nl = __ldg(a.l + t);
                nc = __ldg(a.c + t);
            }
        };
        fetch(tb0 + lane);
        // the bar before the tile (unused before the first valid bar)
        float lh = 0.f, ll = 0.f, lcl = 0.f;
        if (tb0 > 0 && tb0 < tend) {
            lh = __ldg(a.h + tb0 - 1);
            ll = __ldg(a.l + tb0 - 1);
            lcl = __ldg(a.c + tb0 - 1);
        }
        for (int tb = tb0; tb < tend; tb += 32) {
            const int nt = min(32, tend - tb);
            const int tj = tb + lane;
            const float xh = nh, xl = nl, xc = nc;
            fetch(tj + 32);
            // each lane forms its bar's terms (the same for every combo); the
            // warp reads them back from shared memory, four steps per 16-byte
            // broadcast load in a running tile
            float ph = __shfl_up_sync(0xffffffffu, xh, 1), pl = __shfl_up_sync(0xffffffffu, xl, 1),
                  pc = __shfl_up_sync(0xffffffffu, xc, 1);
            if (lane == 0) {
                ph = lh;
                pl = ll;
                pc = lcl;
            }
            float u0, u1, u2;
            Op::terms(xh, xl, xc, ph, pl, pc, u0, u1, u2);
            if (Op::kFirstTr && tj == a.first) u0 = xh - xl;
            float* xs = reinterpret_cast<float*>(&sm.xin[0][0]);
            __syncwarp();  // the previous tile's reads are done
            xs[lane] = u0;
            xs[32 + lane] = u1;
            xs[64 + lane] = u2;
            __syncwarp();
            auto put = [&](int j, float o0, float o1) {
                if (!emit) return;
                sm.stage0[lane][j] = o0;
                if (Op::kTwo) sm.stage1[lane][j] = o1;
            };
            if (tb >= rf && nt == 32) {
                bool wide = false;
                if constexpr (HasWide<Op>::value) wide = __all_sync(0xffffffffu, op.wide_ok(xh, xl, xc));
                auto run32 = [&](auto wide_tag) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 a4 = sm.xin[0][q], b4 = sm.xin[1][q], c4 = sm.xin[2][q];
                        const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w},
                                    cv[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            float o1;
                            const float o0 =
                                op.template step_terms<decltype(wide_tag)::value>(av[u], bv[u], cv[u], o1);
                            put(4 * q + u, o0, o1);
                        }
                    }
                };
                if (wide)
                    run32(std::true_type{});
                else
                    run32(std::false_type{});
            } else {
#pragma unroll 4
                for (int j = 0; j < nt; ++j) {
                    float o1;
                    const float o0 = op.seed_terms(tb + j, xs[j], xs[32 + j], xs[64 + j], o1);
                    put(j, o0, o1);
                }
            }
            lh = __shfl_sync(0xffffffffu, xh, nt - 1);
            ll = __shfl_sync(0xffffffffu, xl, nt - 1);
            lcl = __shfl_sync(0xffffffffu, xc, nt - 1);
            op.last_bar(lh, ll, lcl);
            if (emit) {
                __syncwarp();
                const size_t o = (size_t)(g * 32) * a.n + tj;
                if (nt == 32 && rows == 32) {
#pragma unroll
                    for (int r = 0; r < 32; ++r) {
                        a.out0[o + (size_t)r * a.n] = sm.stage0[r][lane];
                        if (Op::kTwo) a.out1[o + (size_t)r * a.n] = sm.stage1[r][lane];
                    }
                } else if (lane < nt) {
                    for (int r = 0; r < rows; ++r) {
                        a.out0[o + (size_t)r * a.n] = sm.stage0[r][lane];
                        if (Op::kTwo) a.out1[o + (size_t)r * a.n] = sm.stage1[r][lane];
                    }
                }
                __syncwarp();
            }
        }
    };
    tiles(t0, c0, std::false_type{});
    float w[8];
    const size_t sidx = (size_t)k * a.n_combos + li;
    if (k > 0 && valid) {
        op.save(w);
        store_state(a.st_start + sidx * 8, w);
        a.exact[sidx] = warm ? 0 : 1;
    }
    tiles(c0, c1, std::true_type{});
    if (valid) {
        op.save(w);
        store_state(a.st_end + sidx * 8, w);
    }
}

}  // namespace hlc
}  // namespace vta
