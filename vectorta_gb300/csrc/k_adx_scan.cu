// Exact chunked scan of batch ADX sweeps with long periods.
//
// Past its seeding phase (t >= f + 2p) ADX is two linear Wilder levels with a
// pointwise function between them:
//   s <- s * omr + u        s = (atr, +DM, -DM) sums, u = (TR, +DM, -DM) of bar t
//   dx = DX(s)              adx_dx (hlc_ops.cuh)
//   adx <- (adx * pm1 + dx) * rp
// (omr = 1 - 1/p, pm1 = p - 1, rp = 1/p, all f32 as in PAdx).  The
// warm-restart chunking of k_hlc_chunk.cu runs 32 p + 64 steps before every
// chunk, which for periods in the thousands is many times the chunk itself.
// Here a 32-combo group's time axis after its seeding is cut into chunks of L
// steps and processed exactly, like the chunked linear recurrences:
//   AGG1   per (group, chunk): the first level from a zero state over the chunk;
//   CARRY1 per lane: chunk-entry first-level states, s_{k+1} = omr^L s_k + a_k
//          (double-single; s_1 is the seeding run's end state);
//   AGG2   per (group, chunk): the first level from its exact entry state, DX,
//          and the second level from a zero state;
//   CARRY2 per lane: chunk-entry ADX, adx_{k+1} = (pm1 rp)^L adx_k + b_k;
//   EMIT   per (group, chunk): both levels from their entry states, outputs.
// The seeding run (chunk 0, up to the group's s0) is the exact chunk-0 item of
// k_hlc_chunk.cu.  AGG1 needs no state, so the seeding items run in its launch;
// the sweep's short-period groups, which depend on nothing here, run beside
// EMIT: their chains leave issue slots that EMIT's stores wait in.  399 ADX
// periods on 1M bars 707 -> 685 us, 101 periods of 100..400 on 200k bars
// 182 -> 164 (own launch before the scan -> beside its passes).
// Outputs differ from one sequential f32 pass by the rounding
// of the composed carries (a few 1e-7 relative); a NaN bar enters the sums
// through the same NaN-skipping max and comparisons as in the sequential
// pass.
#include <algorithm>

#include "hlc_item.cuh"
#include "period_coefs.cuh"
#include "vta_internal.h"

namespace vta {
namespace {

constexpr int kSW = 4;  // warps per block

struct D2s {
    float hi, lo;
};
__device__ __forceinline__ D2s ds_norm(float s, float e) {
    const float hi = s + e;
    return {hi, e - (hi - s)};
}
__device__ __forceinline__ D2s ds_mul(D2s a, D2s b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    return ds_norm(p, e);
}
__device__ __forceinline__ D2s ds_add(D2s a, D2s b) {
    const float s = a.hi + b.hi;
    const float bb = s - a.hi;
    const float e = ((a.hi - (s - bb)) + (b.hi - bb)) + (a.lo + b.lo);
    return ds_norm(s, e);
}
__device__ __forceinline__ D2s ds_pow(D2s b, long long n) {
    D2s r = {1.f, 0.f};
    while (n > 0) {
        if (n & 1) r = ds_mul(r, b);
        b = ds_mul(b, b);
        n >>= 1;
    }
    return r;
}

struct Lane {
    float omr, pm1, rp;
    __device__ void init(int p) {
        rp = coef::wilder(p);
        omr = coef::wilder_keep(p);
        pm1 = (float)p - 1.f;
    }
};

enum { PASS_AGG1 = 0, PASS_AGG2 = 1, PASS_EMIT = 2 };


// A warp's staging: a row per lane, CUT behind 8 columns of the tile before; odd
// row stride, so a row's and a column's accesses both fall in 32 banks.
template <bool CUT> struct ScanSmem {
    static constexpr int kLead = CUT ? 8 : 0;
    float stage[32][kLead + 33];
    float4 xin[3][8];  // a tile's TR, +DM and -DM
};
template <bool CUT> union WarpSmem {
    ScanSmem<CUT> scan;
    hlc::ItemSmem<hlc::PAdx> item;
};

// Stores a staged tile of nt steps: row r at o + r n.  CUT (large outputs whose
// rows do not start at 32-byte sectors): each row from its sector boundary on,
// the last m values of the tile before waiting in the kLead columns; `first`
// and `last` tile of a chunk.
template <bool CUT>
__device__ __forceinline__ void store_tile(float* o, int n, int rows, ScanSmem<CUT>& sm, int nt, bool first,
                                           bool last) {
    constexpr int kLead = ScanSmem<CUT>::kLead;
    auto& stage = sm.stage;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if constexpr (CUT) {
        const int m0 = (int)(reinterpret_cast<uintptr_t>(o) >> 2);
        o += lane;
        if (!first && !last && rows == 32) {
#pragma unroll
            for (int r = 0; r < 32; ++r, o += n) {
                const int m = (int)((unsigned)m0 + (unsigned)r * (unsigned)n) & 7;
                o[-m] = stage[r][kLead + lane - m];
            }
        } else {
#pragma unroll 4
            for (int r = 0; r < rows; ++r, o += n) {
                const int m = (int)((unsigned)m0 + (unsigned)r * (unsigned)n) & 7, e = lane - m;
                if ((!first || e >= 0) && e < nt) o[-m] = stage[r][kLead + e];
                if (last && e + 32 < nt) o[32 - m] = stage[r][kLead + 32 + e];
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 1; i < kLead; ++i) stage[lane][i] = stage[lane][32 + i];
    } else if (nt == 32 && rows == 32) {
        o += lane;
#pragma unroll
        for (int r = 0; r < 32; ++r) o[(size_t)r * n] = stage[r][kLead + lane];
    } else if (lane < nt) {
        for (int r = 0; r < rows; ++r) o[(size_t)r * n + lane] = stage[r][kLead + lane];
    }
    __syncwarp();
}

// One (group, chunk >= 1) item per warp; lane = combo of the group.  A step is
// the three first-level updates plus DX and the second level: the bar's own
// terms come from shared memory (formed once per bar by the lane that loaded
// it), the next tile's bars are loaded ahead, and the output rows are written
// by 32 unrolled 128-byte stores.  320 periods on 1M bars: AGG1 221 -> 74 us,
// AGG2 281 -> 147 (both bound by issue), EMIT 472 -> 243 (1.28 GB written, 5.3
// TB/s).
template <int PASS, bool CUT = false>
__global__ void __launch_bounds__(kSW * 32) k_adx_scan(AdxScanArgs a, HlcChunkArgs c) {
    __shared__ WarpSmem<CUT> smem[kSW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ScanSmem<CUT>& sm = smem[warp].scan;
    int item = blockIdx.x * kSW + warp;
    if (PASS != PASS_AGG2) {  // the pass's warm-restart items first
        if (item < c.n_items) {
            hlc::run_item<hlc::PAdx>(c, item, smem[warp].item);
            return;
        }
        item -= c.n_items;
    }
    if (item >= a.n_items) return;
    const int2 it = a.items[item];
    const int gi = it.x, k = it.y;
    const int g = a.groups[gi];
    const int c0 = a.group_s0[gi] + (k - 1) * a.L;
    const int c1 = min(c0 + a.L, a.n);
    const int ci = g * 32 + lane;  // combo
    const bool valid = ci < a.n_combos;
    const size_t si = (size_t)k * a.n_slots + gi * 32 + lane;  // state slot
    Lane ln;
    ln.init(__ldg(a.periods + (valid ? ci : g * 32)));
    float atr = 0.f, pdm = 0.f, mdm = 0.f, adx = 0.f;
    if (PASS != PASS_AGG1) {
        const float4 s = a.carry1[si];
        atr = s.x;
        pdm = s.y;
        mdm = s.z;
    }
    if (PASS == PASS_EMIT) adx = a.carry2[si];
    // inputs of the bar before the chunk (c0 >= 1)
    float ph = __ldg(a.h + c0 - 1), pl = __ldg(a.l + c0 - 1), pc = __ldg(a.c + c0 - 1);
    const int rows = min(32, a.n_combos - g * 32);
    // the next tile's bars are loaded while this one is worked on
    float nh = 0.f, nl = 0.f, nc = 0.f;
    auto fetch = [&](int t) {
        if (t < c1) {
            nh = __ldg(a.h + t);
            nl = __ldg(a.l + t);
            nc = __ldg(a.c + t);
        }
    };
    fetch(c0 + lane);
    for (int tb = c0; tb < c1; tb += 32) {
        const int nt = min(32, c1 - tb);
        const float xh = nh, xl = nl, xc = nc;
        fetch(tb + 32 + lane);
        // each lane forms its bar's TR, +DM and -DM (the same for every combo);
        // the warp reads them back from shared memory, four steps per 16-byte
        // broadcast load in a full tile
        float h1 = __shfl_up_sync(0xffffffffu, xh, 1), l1 = __shfl_up_sync(0xffffffffu, xl, 1),
              c1p = __shfl_up_sync(0xffffffffu, xc, 1);
        if (lane == 0) {
            h1 = ph;
            l1 = pl;
            c1p = pc;
        }
        // DX by the hardware reciprocal where the sums stay normal over
        // these steps (hlc::adx_wide_ok)
        const bool wide = PASS != PASS_AGG1 &&
                          __all_sync(0xffffffffu, hlc::adx_wide_ok(ln.omr, atr, pdm, mdm, xh, xl, xc, ph, pl, pc));
        float u0, u1, u2;
        hlc::PAdx::terms(xh, xl, xc, h1, l1, c1p, u0, u1, u2);
        float* xs = reinterpret_cast<float*>(&sm.xin[0][0]);
        __syncwarp();  // the previous tile's reads are done
        xs[lane] = u0;
        xs[32 + lane] = u1;
        xs[64 + lane] = u2;
        __syncwarp();
        // one step on a bar's terms: PAdx::step_terms' arithmetic
        auto step = [&](int j, float tr, float dp, float dm, auto wide_tag) {
            constexpr bool WIDE = decltype(wide_tag)::value;
            atr = atr * ln.omr + tr;
            pdm = pdm * ln.omr + dp;
            mdm = mdm * ln.omr + dm;
            if (PASS != PASS_AGG1) {
                const float dx = WIDE ? hlc::adx_dx_wide(pdm, mdm) : hlc::adx_dx(pdm, mdm, atr);
                adx = (adx * ln.pm1 + dx) * ln.rp;
            }
            if (PASS == PASS_EMIT) sm.stage[lane][ScanSmem<CUT>::kLead + j] = adx;
        };
        auto steps = [&](auto wide_tag) {
            if (nt == 32) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 t4 = sm.xin[0][q], p4 = sm.xin[1][q], m4 = sm.xin[2][q];
                    step(4 * q, t4.x, p4.x, m4.x, wide_tag);
                    step(4 * q + 1, t4.y, p4.y, m4.y, wide_tag);
                    step(4 * q + 2, t4.z, p4.z, m4.z, wide_tag);
                    step(4 * q + 3, t4.w, p4.w, m4.w, wide_tag);
                }
            } else {
                for (int j = 0; j < nt; ++j) step(j, xs[j], xs[32 + j], xs[64 + j], wide_tag);
            }
        };
        if (wide)
            steps(std::true_type{});
        else
            steps(std::false_type{});
        ph = __shfl_sync(0xffffffffu, xh, nt - 1);
        pl = __shfl_sync(0xffffffffu, xl, nt - 1);
        pc = __shfl_sync(0xffffffffu, xc, nt - 1);
        if (PASS == PASS_EMIT)
            store_tile<CUT>(a.out + (size_t)(g * 32) * a.n + tb, a.n, rows, sm, nt, tb == c0, tb + nt == c1);
    }
    if (PASS == PASS_AGG1) a.agg1[si] = make_float4(atr, pdm, mdm, 0.f);
    if (PASS == PASS_AGG2) a.agg2[si] = adx;
}

// Chunk-entry states per lane slot, in double-single: one warp per slot.
// LEVEL 1: s_1 = the seeding run's end state, s_{k+1} = m s_k + agg1_k with
// m = omr^L; LEVEL 2: adx_1 likewise with m = (pm1 rp)^L and agg2.  Every
// transition k = 1 .. nch - 2 is over a full chunk, so all share m: the warp
// splits them into 32 consecutive blocks, each thread composes its block into
// one affine map x -> A x + B, the maps are scanned across the warp (five
// shuffle levels), and each thread then walks its block again from its
// entry state, writing the entries.
struct Aff {
    D2s A, B[3];
};
__device__ __forceinline__ D2s ds_shfl_up(D2s v, int o) {
    return {__shfl_up_sync(0xffffffffu, v.hi, o), __shfl_up_sync(0xffffffffu, v.lo, o)};
}
template <int LEVEL>
__global__ void __launch_bounds__(128) k_adx_carry(AdxScanArgs a) {
    constexpr int NC = LEVEL == 1 ? 3 : 1;
    const int slot = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (slot >= a.n_slots) return;  // warp-uniform
    const int gi = slot >> 5;
    const int ci = a.groups[gi] * 32 + (slot & 31);
    if (ci >= a.n_combos) return;  // warp-uniform
    Lane ln;
    ln.init(__ldg(a.periods + ci));
    const int s0 = a.group_s0[gi];
    const int nch = 1 + (a.n - s0 + a.L - 1) / a.L;  // chunks of the group, chunk 0 included
    const float* seed = a.seed_state + (size_t)ci * 8;  // k_hlc_chunk's chunk-0 end state
    const D2s m = LEVEL == 1 ? D2s{ln.omr, 0.f} : ds_mul({ln.pm1, 0.f}, {ln.rp, 0.f});
    const D2s mL = ds_pow(m, a.L);
    auto agg = [&](int k) {
        const size_t si = (size_t)k * a.n_slots + slot;
        return LEVEL == 1 ? __ldg(a.agg1 + si) : make_float4(__ldg(a.agg2 + si), 0.f, 0.f, 0.f);
    };
    auto put = [&](int k, const D2s (&x)[NC]) {
        const size_t si = (size_t)k * a.n_slots + slot;
        if (LEVEL == 1)
            a.carry1[si] = make_float4(x[0].hi + x[0].lo, x[1].hi + x[1].lo, x[2].hi + x[2].lo, 0.f);
        else
            a.carry2[si] = x[0].hi + x[0].lo;
    };
    // transitions 1 .. T, T = nch - 2; this thread's block [k0, k1)
    const int T = nch - 2;
    const int per = T > 0 ? (T + 31) / 32 : 0;
    const int k0 = 1 + min(T, lane * per), k1 = 1 + min(T, (lane + 1) * per);
    Aff f;
    f.A = {1.f, 0.f};
#pragma unroll
    for (int c = 0; c < NC; ++c) f.B[c] = {0.f, 0.f};
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        const float4 g4 = agg(k);
        const float g[3] = {g4.x, g4.y, g4.z};
        f.A = ds_mul(mL, f.A);
#pragma unroll
        for (int c = 0; c < NC; ++c) f.B[c] = ds_add(ds_mul(mL, f.B[c]), {g[c], 0.f});
    }
    // inclusive scan of the maps in lane order: (later) o (earlier)
#pragma unroll 1
    for (int o = 1; o < 32; o <<= 1) {
        Aff e;
        e.A = ds_shfl_up(f.A, o);
#pragma unroll
        for (int c = 0; c < NC; ++c) e.B[c] = ds_shfl_up(f.B[c], o);
        if (lane >= o) {
#pragma unroll
            for (int c = 0; c < NC; ++c) f.B[c] = ds_add(ds_mul(f.A, e.B[c]), f.B[c]);
            f.A = ds_mul(f.A, e.A);
        }
    }
    // exclusive map of this thread: the previous lane's inclusive one
    Aff x;
    x.A = ds_shfl_up(f.A, 1);
#pragma unroll
    for (int c = 0; c < NC; ++c) x.B[c] = ds_shfl_up(f.B[c], 1);
    D2s st[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const D2s sd = {seed[LEVEL == 1 ? c : 3], 0.f};
        st[c] = lane == 0 ? sd : ds_add(ds_mul(x.A, sd), x.B[c]);
    }
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        put(k, st);
        const float4 g4 = agg(k);
        const float g[3] = {g4.x, g4.y, g4.z};
#pragma unroll
        for (int c = 0; c < NC; ++c) st[c] = ds_add(ds_mul(mL, st[c]), {g[c], 0.f});
    }
    // the last chunk's entry (k = nch - 1) from the thread whose block ends there
    if (nch >= 2 && k1 == nch - 1 && (k0 < k1 || lane == 0)) put(nch - 1, st);
}

}  // namespace

vta_status launch_adx_scan(const AdxScanArgs& a, const HlcChunkArgs& c, int n_seed, cudaStream_t st) {
    const unsigned cblocks = ceil_div((size_t)a.n_slots * 32, 128);  // a warp per lane slot
    HlcChunkArgs seed = c, rest = c;
    seed.n_items = n_seed;
    rest.items += n_seed;
    rest.n_items -= n_seed;
    auto blocks = [&](int extra) { return ceil_div((size_t)a.n_items + extra, kSW); };
    ktimer_begin(st);
    k_adx_scan<PASS_AGG1><<<blocks(seed.n_items), kSW * 32, 0, st>>>(a, seed);
    VTA_TRY(check_launch("k_adx_scan<agg1>"));
    k_adx_carry<1><<<cblocks, 128, 0, st>>>(a);
    VTA_TRY(check_launch("k_adx_carry<1>"));
    k_adx_scan<PASS_AGG2><<<blocks(0), kSW * 32, 0, st>>>(a, seed);
    VTA_TRY(check_launch("k_adx_scan<agg2>"));
    k_adx_carry<2><<<cblocks, 128, 0, st>>>(a);
    VTA_TRY(check_launch("k_adx_carry<2>"));
    const auto emit = a.cut ? k_adx_scan<PASS_EMIT, true> : k_adx_scan<PASS_EMIT, false>;
    emit<<<blocks(rest.n_items), kSW * 32, 0, st>>>(a, rest);
    VTA_TRY(check_launch("k_adx_scan<emit>"));
    VTA_TRY(launch_hlc_fixup(c, st));
    ktimer_end(st);
    return VTA_OK;
}

}  // namespace vta
