// Lane-level sequential state machines of ATR, ADX and SuperTrend with the
// state interface that time-chunked runs use (shared by the many-series plans
// and the chunked single-series sweeps).
//
// Op interface (one series, one parameter set per lane):
//   init(period, param, f)       constants; f = first valid index
//   run_from() -> int            first t whose entering state is a running
//                                state (everything before is seeding)
//   start_exact()                state entering t = f
//   start_warm(in, t0)           guessed running state entering t0 >= run_from()
//   load(w, in, t0)              exact running state entering t0 from 8 words
//   save(w)                      running state as 8 words
//   step(in, t, o1) -> o0        process t (any phase), outputs for t
//   stepv(t, h, l, c, o1) -> o0  the same with the inputs of t given
//   step_run(h, l, c, o1) -> o0  stepv for t >= run_from() without phase checks
//   terms, step_terms / seed_terms, last_bar  (ADX, SuperTrend) step_run and stepv
//                                in two parts: what depends on the bars alone,
//                                and the rest
//   (ADX also: wide_ok(h, l, c) and step_run<true> for tiles of up to 32 steps
//   whose sums stay normal, with DX by the hardware reciprocal)
// `In` provides H(t), L(t), C(t).  The arithmetic of each op is that of the
// sequential kernels in k_hlc.cu, so a run that starts at the series start is
// bit-identical to them.
#pragma once

#include "vta_internal.h"

namespace vta {
namespace hlc {

__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

// True range with the crate's NaN-skipping comparisons (atr.rs:352-366).
__device__ __forceinline__ float true_range(float hi, float lo, float pc) {
    float tr = hi - lo;
    const float hc = fabsf(hi - pc);
    if (hc > tr) tr = hc;
    const float lc = fabsf(lo - pc);
    if (lc > tr) tr = lc;
    return tr;
}

// DX from the smoothed DM and TR sums.  The crate forms +DI = 100 pdm / atr and
// -DI = 100 mdm / atr, then DX = 100 |+DI - -DI| / (+DI + -DI); the common
// factor 100 / atr cancels, leaving one division.  atr == 0 gives 0 (both DI
// are 0) and a NaN atr gives NaN, as in the crate.  The ratio |a - b| / (a + b)
// lies in [0, 1] and is taken with the fast reciprocal-multiply divide (2 ulp;
// the ADX sweeps and plans are issue-bound and the IEEE divide was a third of
// a step); every ADX kernel shares this function, so the chunked and the
// sequential kernels stay bit-identical.
// 1 / x by the hardware approximation (relative error within about 2^-23;
// subnormal x is read as zero), one instruction
__device__ __forceinline__ float rcp_approx_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Whether up to 32 running ADX steps from this state keep atr and
// pdm + mdm normal and nonzero, given the inputs of those steps and of the
// bar before them (x*, p*): the sums shrink by at most omr^32 >= 2^-32 from
// period 2 on (period 1 keeps nothing of a bar: its sums may be 0) and
// grow by at most 32 x 2^100 when every price is within 2^98 in magnitude,
// so sums in [2^-60, 2^100] at the start stay within [2^-92, 2^106].  On such
// steps DX = |pdm - mdm| / (pdm + mdm) 100 needs none of adx_dx's guards
// (adx_dx_wide).  NaN prices or sums fail the test.
__device__ __forceinline__ bool adx_wide_ok(float omr, float atr, float pdm, float mdm, float xh, float xl, float xc,
                                            float ph, float pl, float pc) {
    const float s = pdm + mdm;
    const bool in_range = fabsf(xh) <= 0x1p98f && fabsf(xl) <= 0x1p98f && fabsf(xc) <= 0x1p98f &&
                          fabsf(ph) <= 0x1p98f && fabsf(pl) <= 0x1p98f && fabsf(pc) <= 0x1p98f;
    return omr >= 0.5f && in_range && atr >= 0x1p-60f && atr <= 0x1p100f && s >= 0x1p-60f && s <= 0x1p100f;
}
__device__ __forceinline__ float adx_dx_wide(float pdm, float mdm) {
    return fabsf(pdm - mdm) * rcp_approx_ftz(pdm + mdm) * 100.f;
}

// (Selects, no branches: the unrolled steps of a batch then form one block of
// code whose divisions overlap.)
__device__ __forceinline__ float adx_dx(float pdm, float mdm, float atr) {
    const float s = pdm + mdm;
    const float q = __fdividef(fabsf(pdm - mdm), s) * 100.f;
    const float d = atr == atr ? (s != 0.f ? q : 0.f) : qnan();
    return atr == 0.f ? 0.f : d;
}

// ATR: atr_compute_into_scalar (atr.rs:329-460); TR(f) = h - l, seed = mean
// of the first p TRs at s = f + p - 1, then rma = fma(-a, rma, rma) + a * tr.
struct PAtr {
    static constexpr bool kTwo = false;
    int p, f;
    float alpha, rma, pc;
    double tr_sum;
    __device__ void init(int period, float, int first) {
        p = period;
        f = first;
        alpha = (float)(1.0 / (double)p);
    }
    __device__ int run_from() const { return f + p; }
    __device__ void start_exact() { tr_sum = 0.0; rma = 0.f; pc = 0.f; }
    template <class In> __device__ void start_warm(const In& in, int t0) {
        pc = in.C(t0 - 1);
        rma = in.H(t0 - 1) - in.L(t0 - 1);
    }
    template <class In> __device__ void load(const float* w, const In& in, int t0) {
        rma = w[0];
        pc = in.C(t0 - 1);
    }
    __device__ void save(float* w) const {
        w[0] = rma;
        w[1] = w[2] = w[3] = w[4] = w[5] = w[6] = w[7] = 0.f;
    }
    template <class In> __device__ float step(const In& in, int t, float& o1) {
        if (t < f) return qnan();
        return stepv(t, in.H(t), in.L(t), in.C(t), o1);
    }
    __device__ float stepv(int t, float hi, float lo, float cl, float&) {
        if (t < f) return qnan();
        const float tr = (t == f) ? hi - lo : true_range(hi, lo, pc);
        pc = cl;
        const int s = f + p - 1;
        if (t < s) {
            tr_sum += (double)tr;
            return qnan();
        }
        if (t == s) {
            tr_sum += (double)tr;
            rma = (float)(tr_sum / (double)p);
            return rma;
        }
        rma = fmaf(-alpha, rma, rma) + alpha * tr;
        return rma;
    }
    // stepv for t >= run_from(): the running update alone
    template <bool WIDE = false>  // (no division: one form)
    __device__ __forceinline__ float step_run(float hi, float lo, float cl, float&) {
        const float tr = true_range(hi, lo, pc);
        pc = cl;
        rma = fmaf(-alpha, rma, rma) + alpha * tr;
        return rma;
    }
};

// ADX: adx_scalar on the slice from f (adx.rs:299-421): Wilder sums over
// relative indices 1..=p, DX from the smoothed DM/TR, ADX = mean of the
// first p DX, then (adx * (p - 1) + dx) / p; first output at f + 2p - 1.
// The arithmetic is the sequential time-major kernel's (k_adx).
struct PAdx {
    static constexpr bool kTwo = false;
    static constexpr bool kFirstTr = false;
    int p, f;
    float rp, omr, pm1;
    float atr, pdm, mdm, dx_sum, adx, ph, pl, pc;
    __device__ void init(int period, float, int first) {
        p = period;
        f = first;
        rp = (float)(1.0 / (double)p);
        omr = (float)(1.0 - 1.0 / (double)p);
        pm1 = (float)p - 1.f;
    }
    __device__ int run_from() const { return f + 2 * p; }
    __device__ void start_exact() {
        atr = pdm = mdm = dx_sum = adx = ph = pl = pc = 0.f;
    }
    template <class In> __device__ void prev_inputs(const In& in, int t0) {
        ph = in.H(t0 - 1);
        pl = in.L(t0 - 1);
        pc = in.C(t0 - 1);
    }
    template <class In> __device__ void start_warm(const In& in, int t0) {
        prev_inputs(in, t0);
        atr = (float)p * (ph - pl);
        pdm = mdm = 0.f;
        adx = 0.f;
    }
    template <class In> __device__ void load(const float* w, const In& in, int t0) {
        atr = w[0]; pdm = w[1]; mdm = w[2]; adx = w[3];
        prev_inputs(in, t0);
    }
    __device__ void save(float* w) const {
        w[0] = atr; w[1] = pdm; w[2] = mdm; w[3] = adx;
        w[4] = w[5] = w[6] = w[7] = 0.f;
    }
    template <class In> __device__ float step(const In& in, int t, float& o1) {
        if (t < f) return qnan();
        return stepv(t, in.H(t), in.L(t), in.C(t), o1);
    }
    __device__ float stepv(int t, float ch, float cl, float cc, float& o1) {
        if (t < f) return qnan();
        float tr, dp, dm;
        terms(ch, cl, cc, ph, pl, pc, tr, dp, dm);
        last_bar(ch, cl, cc);
        return seed_terms(t, tr, dp, dm, o1);
    }
    // One step of any phase on the bar's terms (selects, see adx_dx: the lanes
    // of a sweep are in different phases).  r counts the bars after the first:
    // sums over r = 1..p, the mean of the DX of r = p..2p-1, then running.
    __device__ __forceinline__ float seed_terms(int t, float tr, float dp, float dm, float&) {
        const int r = t - f;
        const bool live = r > 0;
        const float keep = r <= p ? 1.f : omr;  // x * 1 + y is the plain sum
        atr = fmaf(atr, keep, live ? tr : 0.f);
        pdm = fmaf(pdm, keep, live ? dp : 0.f);
        mdm = fmaf(mdm, keep, live ? dm : 0.f);
        const float dx = adx_dx(pdm, mdm, atr);
        dx_sum = r == p ? dx : dx_sum + dx;  // read at r = 2p - 1 only
        const float run = fmaf(adx, pm1, dx) * rp;
        const bool mean = r == 2 * p - 1 && r > p, late = r >= 2 * p;
        adx = mean ? dx_sum * rp : late ? run : adx;
        return mean || late ? adx : qnan();
    }
    // What a running step takes from the bars alone: TR, +DM, -DM.  They are the
    // same for every combo of a sweep, so a warp of combos forms them once per
    // bar (k_hlc_chunk.cu, k_adx_scan.cu).
    static __device__ __forceinline__ void terms(float ch, float cl, float, float ph, float pl, float pc, float& tr,
                                                 float& dp, float& dm) {
        tr = fmaxf(fmaxf(ch - cl, fabsf(ch - pc)), fabsf(cl - pc));
        const float up = ch - ph, down = pl - cl;
        dp = (up > down && up > 0.f) ? up : 0.f;
        dm = (down > up && down > 0.f) ? down : 0.f;
    }
    // stepv for t >= run_from(): the running update alone; WIDE: the steps
    // of a tile for which wide_ok held on every lane at its start
    template <bool WIDE = false>
    __device__ __forceinline__ float step_terms(float tr, float dp, float dm, float&) {
        atr = atr * omr + tr;
        pdm = pdm * omr + dp;
        mdm = mdm * omr + dm;
        adx = (adx * pm1 + (WIDE ? adx_dx_wide(pdm, mdm) : adx_dx(pdm, mdm, atr))) * rp;
        return adx;
    }
    __device__ __forceinline__ void last_bar(float ch, float cl, float cc) { ph = ch; pl = cl; pc = cc; }
    template <bool WIDE = false>
    __device__ __forceinline__ float step_run(float ch, float cl, float cc, float& o1) {
        float tr, dp, dm;
        terms(ch, cl, cc, ph, pl, pc, tr, dp, dm);
        last_bar(ch, cl, cc);
        return step_terms<WIDE>(tr, dp, dm, o1);
    }
    static constexpr bool kWide = true;
    __device__ bool wide_ok(float xh, float xl, float xc) const {
        return adx_wide_ok(omr, atr, pdm, mdm, xh, xl, xc, ph, pl, pc);
    }
};

// SuperTrend: supertrend_scalar (supertrend.rs:457-550) with the ATR of the
// slice from f computed inline; outputs trend and changed, first at f + p - 1.
// The arithmetic is the sequential time-major kernel's (k_supertrend).
struct PSuperTrend {
    static constexpr bool kTwo = true;
    static constexpr bool kFirstTr = true;  // the first valid bar's TR is high - low
    int p, f;
    float alpha, fac, atr, pub, plb, last_close, pc;
    bool upper;
    double tr_sum;
    __device__ void init(int period, float factor, int first) {
        p = period;
        f = first;
        alpha = (float)(1.0 / (double)p);
        fac = factor;
    }
    __device__ int run_from() const { return f + p; }
    __device__ void start_exact() {
        tr_sum = 0.0;
        atr = pub = plb = last_close = pc = 0.f;
        upper = false;
    }
    template <class In> __device__ void start_warm(const In& in, int t0) {
        const float hi = in.H(t0 - 1), lo = in.L(t0 - 1), cl = in.C(t0 - 1);
        atr = hi - lo;
        const float hl2 = (hi + lo) * 0.5f;
        pub = hl2 + fac * atr;
        plb = hl2 - fac * atr;
        last_close = pc = cl;
        upper = cl <= pub;
    }
    template <class In> __device__ void load(const float* w, const In& in, int t0) {
        atr = w[0]; pub = w[1]; plb = w[2];
        upper = w[3] != 0.f;
        last_close = pc = in.C(t0 - 1);
    }
    __device__ void save(float* w) const {
        w[0] = atr; w[1] = pub; w[2] = plb; w[3] = upper ? 1.f : 0.f;
        w[4] = w[5] = w[6] = w[7] = 0.f;
    }
    template <class In> __device__ float step(const In& in, int t, float& v1) {
        v1 = qnan();
        if (t < f) return qnan();
        return stepv(t, in.H(t), in.L(t), in.C(t), v1);
    }
    __device__ float stepv(int t, float hi, float lo, float cl, float& v1) {
        v1 = qnan();
        if (t < f) return qnan();
        float tr, hl2, c;
        terms(hi, lo, cl, 0.f, 0.f, pc, tr, hl2, c);
        if (t == f) tr = hi - lo;
        last_bar(hi, lo, cl);
        return seed_terms(t, tr, hl2, c, v1);
    }
    // One step of any phase on the bar's terms (tr at the first valid bar is
    // high - low: the caller's)
    __device__ __forceinline__ float seed_terms(int t, float tr, float hl2, float cl, float& v1) {
        const int warm = f + p - 1;
        v1 = qnan();
        if (t < f) return qnan();
        if (t > warm) return step_terms(tr, hl2, cl, v1);
        tr_sum += (double)tr;
        if (t < warm) return qnan();
        atr = (float)(tr_sum / (double)p);
        // (product and sum rounded one by one, as the sequential kernel does)
        const float band = __fmul_rn(fac, atr);
        pub = __fadd_rn(hl2, band);
        plb = __fsub_rn(hl2, band);
        last_close = cl;
        upper = cl <= pub;
        v1 = 0.f;
        return upper ? pub : plb;
    }
    // What a running step takes from the bars alone: TR, (high + low) / 2, close
    static __device__ __forceinline__ void terms(float hi, float lo, float cl, float, float, float pc, float& tr,
                                                 float& hl2, float& c) {
        tr = hi - lo;
        const float hc = fabsf(hi - pc);
        if (hc > tr) tr = hc;
        const float lc = fabsf(lo - pc);
        if (lc > tr) tr = lc;
        hl2 = (hi + lo) * 0.5f;
        c = cl;
    }
    // stepv for t >= run_from(): the running update alone
    template <bool WIDE = false>  // (no division: one form)
    __device__ __forceinline__ float step_terms(float tr, float hl2, float cl, float& v1) {
        atr = fmaf(-alpha, atr, atr) + alpha * tr;
        float cub = fmaf(fac, atr, hl2), clb = fmaf(-fac, atr, hl2);
        if (last_close <= pub) cub = fminf(cub, pub);
        if (last_close >= plb) clb = fmaxf(clb, plb);
        // the band holds or the trend flips to the other one (selects: see adx_dx)
        const bool up = cl <= cub, down = cl >= clb;
        const bool hold = upper ? up : down;
        upper = upper == hold;
        v1 = hold ? 0.f : 1.f;
        pub = cub; plb = clb; last_close = cl;
        return upper ? cub : clb;
    }
    __device__ __forceinline__ void last_bar(float, float, float cl) { pc = cl; }
    template <bool WIDE = false>
    __device__ __forceinline__ float step_run(float hi, float lo, float cl, float& v1) {
        float tr, hl2, c;
        terms(hi, lo, cl, 0.f, 0.f, pc, tr, hl2, c);
        last_bar(hi, lo, cl);
        return step_terms(tr, hl2, c, v1);
    }
};


}  // namespace hlc
}  // namespace vta
