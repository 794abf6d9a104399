// Chunked linear-recurrence scans: EMA, DEMA, TEMA, RSI, Wilders, ATR.
//
// Each indicator is a linear time-invariant recurrence once seeded, so the
// time axis is cut into chunks processed in parallel:
//   pass A (k_recur<.., PASS_AGG>):  per (lane, chunk) run the recurrence from
//       a zero state (or from the exact seed inside the seed chunk) and keep
//       the chunk-end state plus the number of applied steps;
//   pass B (k_recur_carry):          per lane, compose the chunk transforms
//       (closed-form powers of the transition matrix) in double-single
//       arithmetic -> carry-in per chunk;
//   pass C (k_recur<.., PASS_EMIT>): per (lane, chunk) re-run from the carry
//       and write the outputs.
// A "lane" is one parameter combo of a single-series sweep (batch layout:
// every lane reads the same x[t], outputs are staged through shared memory so
// each store instruction writes one contiguous 256-byte row segment) or one
// series of a time-major matrix (coalesced loads and stores directly).
// The warm-up rules (seed index, NaN prefix, running-mean outputs) follow the
// crate's scalar paths cited on each op.
#include <climits>

#include "vta_internal.h"
#include "period_coefs.cuh"

namespace vta {
namespace {

constexpr int kWarps = 4;  // warps per block
__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

// Compensated running sum (float value + float error term, Neumaier): the
// warm-up accumulators of the crate are f64, and GB300's FP64 rate is a
// small fraction of FP32, so the per-step sums are kept in float pairs and
// turned into f64 only once, at the seed.  Sums of up to a few thousand
// terms stay within ~1e-14 relative of the f64 ones.
struct Acc {
    float hi, lo;
    __device__ void zero() { hi = 0.f; lo = 0.f; }
    // error terms of non-finite sums are dropped so that inf / NaN propagate
    // through hi exactly as through an f64 sum
    __device__ void add(float v) {
        const float sum = hi + v;
        const float bb = sum - hi;
        const float e = (hi - (sum - bb)) + (v - bb);
        lo += isfinite(e) ? e : 0.f;
        hi = sum;
    }
    // adds the exact difference a - b
    __device__ void add_diff(float a, float b) {
        const float d = a - b;
        const float bb = d - a;
        const float e = (a - (d - bb)) - (b + bb);
        add(d);
        lo += isfinite(e) ? e : 0.f;
    }
    __device__ float f() const { return hi + lo; }
    __device__ double d() const { return (double)hi + (double)lo; }
    __device__ float mean(int p, float inv) const;  // pair_mean
};

__device__ __noinline__ float f64_mean(float2 sum, int p) { return (float)(((double)sum.x + (double)sum.y) / (double)p); }

// sum / p from a compensated sum as f64 gives it, inv = 1 / p.  The residual of
// the first quotient is exact by FMA, so q + c is the mean up to 2^-45 of it
// (scaled where the residual of a small sum would underflow); where 2^-40 more
// or less rounds alike, so does the mean, and only the others (ties of short
// periods, one seed in 2^15) are divided in f64.  An f64 division in the chain
// of every tile that holds a seed took RSI of 58 periods on 5,003 bars from 51
// to 63 us.
__device__ __forceinline__ float pair_mean(float2 sum, int p, float inv) {
    const bool small = fabsf(sum.x) < 0x1p-40f;
    const float k = small ? 0x1p80f : 1.f, hi = sum.x * k, lo = sum.y * k;
    const float q = hi * inv, c = (fmaf(-q, (float)p, hi) + lo) * inv, eps = fabsf(q) * 0x1p-40f;
    const float a = q + (c + eps), b = q + (c - eps);
    const float m = a * (small ? 0x1p-80f : 1.f);
    const bool sure = a == b && p < coef::kExact && (!small || fabsf(m) >= 0x1p-126f);
    return sure ? m : f64_mean(sum, p);
}

__device__ __forceinline__ float Acc::mean(int p, float inv) const {
    const float h = hi + lo, e = lo - (h - hi);
    return pair_mean(make_float2(h, isfinite(e) ? e : 0.f), p, inv);  // (an infinite sum is its own mean)
}

// ------------------------------------------------------------ inputs -------
struct InBatch {
    const float *x, *h, *l, *c;
    __device__ float X(int t) const { return __ldg(x + t); }
    __device__ float H(int t) const { return __ldg(h + t); }
    __device__ float L(int t) const { return __ldg(l + t); }
    __device__ float C(int t) const { return __ldg(c + t); }
};
struct InTm {
    const float *x, *h, *l, *c;
    size_t cols, s;
    __device__ float X(int t) const { return __ldg(x + (size_t)t * cols + s); }
    __device__ float H(int t) const { return __ldg(h + (size_t)t * cols + s); }
    __device__ float L(int t) const { return __ldg(l + (size_t)t * cols + s); }
    __device__ float C(int t) const { return __ldg(c + (size_t)t * cols + s); }
};

// One 32-step tile of a single shared series held in registers: lane l holds
// x[tb + l]; X(t) is a warp shuffle (t - 1 < tb reads the value before the
// tile).  Used by the batch fast path so each step costs no memory access.
struct InTile {
    float xv, hv, lv, cv;  // this lane's element of the tile
    float xb, cb;          // x[tb-1], c[tb-1]
    int tb;
    float4* xs;  // this warp's 2 x 32-float input scratch in shared memory
    __device__ float X(int t) const {
        const int j = t - tb;
        const float v = __shfl_sync(0xffffffffu, xv, j & 31);
        return j >= 0 ? v : xb;
    }
    __device__ float H(int t) const { return __shfl_sync(0xffffffffu, hv, (t - tb) & 31); }
    __device__ float L(int t) const { return __shfl_sync(0xffffffffu, lv, (t - tb) & 31); }
    __device__ float C(int t) const {
        const int j = t - tb;
        const float v = __shfl_sync(0xffffffffu, cv, j & 31);
        return j >= 0 ? v : cb;
    }
};

// The values of one step t of a single shared series (and of t - 1), for the
// general path: X / C at t or t - 1, H / L at t.
struct InStep {
    int t;
    float x0, x1;  // x[t], x[t-1]  (close for the high/low/close ops)
    float h0, l0;  // h[t], l[t]
    __device__ float X(int u) const { return u == t ? x0 : x1; }
    __device__ float C(int u) const { return u == t ? x0 : x1; }
    __device__ float H(int) const { return h0; }
    __device__ float L(int) const { return l0; }
};

// Double-single numbers for the carry scan and the closed-form chunk
// transitions: value = hi + lo with |lo| <= ulp(hi) / 2, about 2^-44
// relative after a few operations.  GB300 runs FP32 at many times its FP64
// rate (one FP64 warp instruction holds the SM's FP64 pipe for many cycles),
// so the scan works with FP32 error-free transformations (exact products by
// FMA, TwoSum) instead of f64.
struct D2 {
    float hi, lo;
};
__device__ __forceinline__ D2 d2_norm(float s, float e) {
    const float hi = s + e;
    return {hi, e - (hi - s)};
}
__device__ __forceinline__ D2 d2_mul(D2 a, D2 b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    return d2_norm(p, e);
}
__device__ __forceinline__ D2 d2_add(D2 a, D2 b) {
    const float s = a.hi + b.hi;
    const float bb = s - a.hi;
    const float e = ((a.hi - (s - bb)) + (b.hi - bb)) + (a.lo + b.lo);
    return d2_norm(s, e);
}
// a * b + c
__device__ __forceinline__ D2 d2_fma(D2 a, D2 b, D2 c) { return d2_add(d2_mul(a, b), c); }
__device__ __forceinline__ D2 d2_neg(D2 a) { return {-a.hi, -a.lo}; }
// num / den for small positive integers, to double-single accuracy: the
// FP32 quotient plus its exact remainder (FMA) divided again
__device__ __forceinline__ D2 d2_ratio(int num, int den) {
    const float fn = (float)num, fd = (float)den;
    const float q = fn / fd;
    const float r = fmaf(-q, fd, fn);
    return d2_norm(q, r / fd);
}
__device__ __forceinline__ D2 d2_from_ll(long long n) {
    const float hi = (float)n;
    return {hi, (float)(n - (long long)hi)};
}
// b^n for a whole step count n >= 0 by repeated squaring
__device__ __forceinline__ D2 d2_pow(D2 b, long long n) {
    D2 r = {1.f, 0.f};
    while (n > 0) {
        if (n & 1) r = d2_mul(r, b);
        b = d2_mul(b, b);
        n >>= 1;
    }
    return r;
}
__device__ __forceinline__ D2 d2_shfl_up(D2 v, int d) {
    return {__shfl_up_sync(0xffffffffu, v.hi, d), __shfl_up_sync(0xffffffffu, v.lo, d)};
}

// ------------------------------------------------------------ ops ----------
// Common op interface:
//   init(p, f)            lane constants; sets f (first valid), s (seed index),
//                         warm (first non-NaN output index)
//   accum(in, t)          warm-up accumulation for t in [f, s]
//   seed()                running state from the accumulators (at t == s)
//   step(in, t) -> int    running update for t > s; returns 1 if applied
//   value(in, t)          output for t >= s
//   warm_value(t)         output for t in [f, s)
//   zero() / get(i) / set(i, v)   running state access (NS components)
//   propagate(S, n, p)    S <- M^n S in f64 (static)

// EMA: ema.rs:430-469 / 858-893.  Warm-up outputs are the running mean of the
// finite values of [f, t]; NaN prefix is [0, f); non-finite x is skipped.
struct OpEma {
    static constexpr bool kHlc = false;
    static constexpr int NS = 1;
    float alpha, beta, y;
    int f, s, warm;
    Acc wsum;
    int wcnt;
    __device__ void init(int p, int first) {
        alpha = coef::ema(p);
        beta = coef::ema_keep(p);
        f = first; s = first + p - 1; warm = first;
        wsum.zero(); wcnt = 0;
    }
    template <class In> __device__ void accum(const In& in, int t) {
        float v = in.X(t);
        if (t == f || isfinite(v)) { wsum.add(v); wcnt += 1; }
    }
    __device__ float cur_mean() const { return wsum.f() / (float)wcnt; }
    __device__ void seed() { y = cur_mean(); }
    // y <- y + alpha (x - y): the fixed point is x itself whatever the f32
    // rounding of alpha.  The crate's form beta y + alpha x, with alpha and
    // beta = 1 - alpha rounded to f32 separately, has the steady-state gain
    // alpha / (1 - beta) = 1 + O(2^-25 / alpha): a bias of 1.5e-5 at p = 1000.
    template <class In> __device__ int step(const In& in, int t) {
        float v = in.X(t);
        if (isfinite(v)) { y = fmaf(alpha, v - y, y); return 1; }
        return 0;
    }
    template <class In> __device__ float value(const In&, int) const { return y; }
    __device__ float warm_value(int) const { return cur_mean(); }
    __device__ void zero() { y = 0.f; }
    __device__ float get(int) const { return y; }
    __device__ void set(int, float v) { y = v; }
    // running step + output without phase checks; returns applied-step flag
    // FIN: every input of the step is known finite (no skip logic)
    template <bool FIN = false, class In> __device__ float fast(const In& in, int t, int& applied) {
        const float v = in.X(t);
        if (FIN) {
            y = fmaf(alpha, v - y, y);
            ++applied;
            return y;
        }
        const bool ok = isfinite(v);
        y = ok ? fmaf(alpha, v - y, y) : y;
        applied += ok;
        return y;
    }
    // closed-form transition of n steps (double-single): a = 2 / (p + 1),
    // an = (1 - a)^n
    static __device__ void coef(int p, D2& a, D2& b) {
        a = d2_ratio(2, p + 1);
        b = d2_add({1.f, 0.f}, d2_neg(a));
    }
    static __device__ void propagate(D2* S, D2, D2, D2 an, int) { S[0] = d2_mul(S[0], an); }
};

// DEMA: dema.rs:291-354 (x86 mul_add form).  Seed x[f] at f; NaN prefix
// [0, f+p-1); out = 2*e1 - e2.
struct OpDema {
    static constexpr bool kHlc = false;
    static constexpr int NS = 2;
    static constexpr int kShape = 1;
    float alpha, a, e1, e2, xf;
    int f, s, warm;
    __device__ void init(int p, int first) {
        alpha = coef::ema(p);
        a = coef::ema_keep(p);
        f = first; s = first; warm = first + p - 1;
    }
    template <class In> __device__ void accum(const In& in, int t) { xf = in.X(t); }
    __device__ void seed() { e1 = xf; e2 = xf; }
    // gain-exact form of e <- a e + alpha x (see OpEma::step)
    template <class In> __device__ int step(const In& in, int t) {
        float v = in.X(t);
        e1 = fmaf(alpha, v - e1, e1);
        e2 = fmaf(alpha, e1 - e2, e2);
        return 1;
    }
    template <class In> __device__ float value(const In&, int t) const {
        return t < warm ? qnan() : fmaf(e1, 2.f, -e2);
    }
    __device__ float warm_value(int) const { return qnan(); }
    __device__ void zero() { e1 = 0.f; e2 = 0.f; }
    __device__ float get(int i) const { return i == 0 ? e1 : e2; }
    __device__ void set(int i, float v) { if (i == 0) e1 = v; else e2 = v; }
    template <bool FIN = false, class In> __device__ float fast(const In& in, int t, int& applied) {
        const float v = in.X(t);
        e1 = fmaf(alpha, v - e1, e1);
        e2 = fmaf(alpha, e1 - e2, e2);
        ++applied;
        return fmaf(e1, 2.f, -e2);
    }
    static __device__ void coef(int p, D2& a, D2& b) { OpEma::coef(p, a, b); }
    static __device__ void propagate(D2* S, D2 n, D2 al, D2 an, int) {
        const D2 s1 = S[0];
        S[0] = d2_mul(an, s1);
        S[1] = d2_mul(an, d2_fma(d2_mul(n, al), s1, S[1]));
    }
};

// TEMA: tema.rs:228-298.  Three EMAs started at f, f+(p-1), f+2(p-1) exactly
// as the crate staggers them; running from s = f+2(p-1); NaN prefix
// [0, f+3(p-1)); out = 3*e1 - 3*e2 + e3; p == 1 copies x.
struct OpTema {
    static constexpr bool kHlc = false;
    static constexpr int NS = 3;
    static constexpr int kShape = 1;
    float per, per1, e1, e2, e3;
    int f, s, warm, start2, p1;
    __device__ void init(int p, int first) {
        per = coef::ema(p);
        per1 = coef::ema_keep(p);
        p1 = p - 1;
        f = first; start2 = first + p1; s = first + 2 * p1; warm = first + 3 * p1;
        e1 = e2 = e3 = 0.f;
    }
    template <class In> __device__ void accum(const In& in, int t) {
        float v = in.X(t);
        if (p1 == 0) { e1 = v; return; }
        if (t == f) e1 = v;  // ema1 = data[first]; the loop then re-applies it
        // gain-exact form of e <- per1 e + per x (see OpEma::step)
        e1 = fmaf(per, v - e1, e1);
        if (t == start2) { e2 = e1; e2 = fmaf(per, e1 - e2, e2); }
        else if (t > start2) e2 = fmaf(per, e1 - e2, e2);
        if (t == s) { e3 = e2; e3 = fmaf(per, e2 - e3, e3); }
    }
    __device__ void seed() {}
    template <class In> __device__ int step(const In& in, int t) {
        float v = in.X(t);
        if (p1 == 0) { e1 = v; return 1; }
        e1 = fmaf(per, v - e1, e1);
        e2 = fmaf(per, e1 - e2, e2);
        e3 = fmaf(per, e2 - e3, e3);
        return 1;
    }
    template <class In> __device__ float value(const In& in, int t) const {
        if (p1 == 0) return e1;
        return t < warm ? qnan() : 3.f * e1 - 3.f * e2 + e3;
    }
    __device__ float warm_value(int) const { return qnan(); }
    __device__ void zero() { e1 = e2 = e3 = 0.f; }
    template <bool FIN = false, class In> __device__ float fast(const In& in, int t, int& applied) {
        const float v = in.X(t);
        ++applied;
        if (p1 == 0) { e1 = v; return v; }
        e1 = fmaf(per, v - e1, e1);
        e2 = fmaf(per, e1 - e2, e2);
        e3 = fmaf(per, e2 - e3, e3);
        return 3.f * e1 - 3.f * e2 + e3;
    }
    __device__ float get(int i) const { return i == 0 ? e1 : (i == 1 ? e2 : e3); }
    __device__ void set(int i, float v) { if (i == 0) e1 = v; else if (i == 1) e2 = v; else e3 = v; }
    // One general-path step for any t >= f: the arithmetic of accum / step
    // with the phase tests (t == f, start2, s) as selects instead of branches,
    // so the lanes of a warp in different warm-up phases do not diverge.
    static constexpr bool kUni = true;
    template <class In> __device__ float uni(const In& in, int t, int& steps) {
        const float v = in.X(t);
        steps += t > s;
        if (p1 == 0) { e1 = v; return v; }
        const float a1 = t == f ? v : e1;
        e1 = fmaf(per, v - a1, a1);
        const float a2 = t == start2 ? e1 : e2;
        const float n2 = fmaf(per, e1 - a2, a2);
        e2 = t >= start2 ? n2 : e2;
        const float a3 = t == s ? e2 : e3;
        const float n3 = fmaf(per, e2 - a3, a3);
        e3 = t >= s ? n3 : e3;
        return t < warm ? qnan() : 3.f * e1 - 3.f * e2 + e3;
    }
    static __device__ void coef(int p, D2& a, D2& b) { OpEma::coef(p, a, b); }
    static __device__ void propagate(D2* S, D2 n, D2 al, D2 an, int p) {
        if (p == 1) {  // p==1 carries nothing (out = x)
            S[0] = {0.f, 0.f};
            return;
        }
        const D2 s1 = S[0], s2 = S[1], s3 = S[2];
        const D2 nal = d2_mul(n, al);
        // n a^2 + n (n - 1) / 2 a^2 = n (n + 1) / 2 a^2
        const D2 c = d2_mul(d2_mul(d2_mul(n, d2_add(n, {1.f, 0.f})), {0.5f, 0.f}), d2_mul(al, al));
        S[0] = d2_mul(an, s1);
        S[1] = d2_mul(an, d2_fma(nal, s1, s2));
        S[2] = d2_mul(an, d2_fma(c, s1, d2_fma(nal, s2, s3)));
    }
};

// RSI: batch rows follow rsi_batch_inner (rsi.rs:568-697: non-finite deltas
// become NaN gains/losses and poison the row); time-major series follow the
// single-series rsi_compute_into_scalar (rsi.rs:327-414: a NaN delta poisons
// only inside the warm-up, later ones count as 0).  NaN prefix [0, f+p).
template <bool kBatchSem>
struct OpRsi {
    static constexpr bool kHlc = false;
    static constexpr int NS = 2;
    static constexpr int kShape = 2;
    float inv_p, beta, ag, al, xprev, pf;
    float sN, sD;  // the emit tiles' scaled state while sc (run_tile below)
    int f, s, warm;
    Acc sg, sl;
    bool wnan, sc;
    __device__ void init(int p, int first) {
        inv_p = coef::wilder(p);
        pf = (float)p;
        beta = coef::wilder_keep(p);
        f = first; s = first + p; warm = s;
        sg.zero(); sl.zero(); wnan = false; sc = false;
    }
    template <class In> __device__ void accum(const In& in, int t) {
        float v = in.X(t);
        if (t > f && !wnan) {
            // the f64 difference of two floats is exact; its sign is v vs xprev
            if (!(isfinite(v) && isfinite(xprev))) wnan = true;
            else if (v > xprev) sg.add_diff(v, xprev);
            else if (v < xprev) sl.add_diff(xprev, v);
        }
        xprev = v;
    }
    __device__ void seed() {
        if (wnan) { ag = qnan(); al = qnan(); }
        else { ag = (float)(sg.d() * (double)inv_p); al = (float)(sl.d() * (double)inv_p); }
        // the crate multiplies by inv_p = 1/p in f64
    }
    template <class In> __device__ int step(const In& in, int t) {
        float v = in.X(t);
        float xp = (t == 0) ? v : in.X(t - 1);
        float d = v - xp;
        float g, lo;
        if (kBatchSem && !isfinite(d)) { g = qnan(); lo = qnan(); }
        else { g = d > 0.f ? d : 0.f; lo = d < 0.f ? -d : 0.f; }
        ag = fmaf(ag, beta, inv_p * g);
        al = fmaf(al, beta, inv_p * lo);
        return 1;
    }
    template <class In> __device__ float value(const In&, int) const {
        float den = ag + al;
        return den == 0.f ? 50.f : __fdividef(100.f * ag, den);
    }
    __device__ float warm_value(int) const { return qnan(); }
    __device__ void zero() { ag = 0.f; al = 0.f; }
    template <bool FIN = false, class In> __device__ float fast(const In& in, int t, int& applied) {
        const float v = in.X(t);
        const float d = v - in.X(t - 1);
        float g = d > 0.f ? d : 0.f, lo = d < 0.f ? -d : 0.f;
        if (!FIN && kBatchSem && !isfinite(d)) { g = qnan(); lo = qnan(); }
        ag = fmaf(ag, beta, inv_p * g);
        al = fmaf(al, beta, inv_p * lo);
        ++applied;
        const float den = ag + al;
        return den == 0.f ? 50.f : __fdividef(100.f * ag, den);
    }
    // One general-path step for any t >= f (see OpTema::uni): the arithmetic of
    // accum, seed, step and value with the phases as selects.  Many series warm
    // up at different rows, and their diverging phases took about 250
    // instructions a step, this about 60: RSI(14) of 3,000 series x 2,520 rows
    // with leads up to 250 57 -> 49 us, of 500 x 20,000 80 -> 65.
    static constexpr bool kUni = true;
    template <class In> __device__ float uni(const In& in, int t, int& steps) {
        const float v = in.X(t), xp = t > f ? in.X(t - 1) : v;
        const bool warm_up = t > f && t <= s, fin = isfinite(v) && isfinite(xp);
        wnan = wnan || (warm_up && !fin);
        const bool acc = warm_up && !wnan, up = v > xp;
        // the exact |v - xp| as a pair
        const float a = up ? v : xp, b = up ? xp : v;
        const float dd = a - b, bb = dd - a, e0 = (a - (dd - bb)) - (b + bb), e = isfinite(e0) ? e0 : 0.f;
        sg.add(acc && up ? dd : 0.f);
        sg.lo += acc && up ? e : 0.f;
        sl.add(acc && v < xp ? dd : 0.f);
        sl.lo += acc && v < xp ? e : 0.f;
        const float d = v - xp;
        const bool bad = kBatchSem && !isfinite(d);
        const float g = bad ? qnan() : d > 0.f ? d : 0.f, lo = bad ? qnan() : d < 0.f ? -d : 0.f;
        const bool run = t > s;
        ag = run ? fmaf(ag, beta, inv_p * g) : ag;
        al = run ? fmaf(al, beta, inv_p * lo) : al;
        steps += run;
        if (t == s) seed();
        xprev = v;
        return t >= s ? value(in, t) : qnan();
    }
    __device__ float get(int i) const { return i == 0 ? ag : al; }
    __device__ void set(int i, float v) { if (i == 0) ag = v; else al = v; }
    // a = 1 / p, an = (1 - 1/p)^n
    static __device__ void coef(int p, D2& a, D2& b) {
        a = d2_ratio(1, p);
        b = d2_add({1.f, 0.f}, d2_neg(a));
    }
    static __device__ void propagate(D2* S, D2, D2, D2 an, int) {
        S[0] = d2_mul(S[0], an);
        S[1] = d2_mul(S[1], an);
    }
};

// Wilders: wilders.rs:262-322.  Seed = mean of x[f..f+p); y = (x-y)*a + y;
// NaN prefix [0, f+p-1); p == 1 copies x.
struct OpWilders {
    static constexpr bool kHlc = false;
    static constexpr int NS = 1;
    float alpha, y;
    int f, s, warm, p;
    Acc wsum;
    __device__ void init(int p_, int first) {
        p = p_;
        alpha = coef::wilder(p);
        f = first; s = first + p - 1; warm = s;
        wsum.zero();
    }
    template <class In> __device__ void accum(const In& in, int t) { wsum.add(in.X(t)); }
    __device__ void seed() { y = wsum.mean(p, alpha); }
    template <class In> __device__ int step(const In& in, int t) {
        float v = in.X(t);
        y = (p == 1) ? v : fmaf(v - y, alpha, y);
        return 1;
    }
    template <class In> __device__ float value(const In&, int) const { return y; }
    __device__ float warm_value(int) const { return qnan(); }
    __device__ void zero() { y = 0.f; }
    __device__ float get(int) const { return y; }
    __device__ void set(int, float v) { y = v; }
    template <bool FIN = false, class In> __device__ float fast(const In& in, int t, int& applied) {
        const float v = in.X(t);
        y = (p == 1) ? v : fmaf(v - y, alpha, y);
        ++applied;
        return y;
    }
    static __device__ void coef(int p, D2& a, D2& b) { OpRsi<true>::coef(p, a, b); }
    static __device__ void propagate(D2* S, D2, D2, D2 an, int p) {
        S[0] = (p == 1) ? D2{0.f, 0.f} : d2_mul(S[0], an);
    }
};

// True range as the crate computes it (atr.rs:352-366): comparisons skip NaN.
__device__ __forceinline__ float true_range(float hi, float lo, float pc) {
    float tr = hi - lo;
    float hc = fabsf(hi - pc);
    if (hc > tr) tr = hc;
    float lc = fabsf(lo - pc);
    if (lc > tr) tr = lc;
    return tr;
}

// ATR: atr.rs:329-460.  TR(f) = h-l; seed = mean TR over [f, f+L);
// rma = (-a).mul_add(rma, rma) + a*tr; NaN prefix [0, f+L-1).
struct OpAtr {
    static constexpr int NS = 1;
    static constexpr bool kHlc = true;
    float alpha, y;
    int f, s, warm, p;
    Acc wsum;
    __device__ void init(int p_, int first) {
        p = p_;
        alpha = coef::wilder(p);
        f = first; s = first + p - 1; warm = s;
        wsum.zero();
    }
    template <class In> __device__ void accum(const In& in, int t) {
        float hi = in.H(t), lo = in.L(t);
        if (t == f) wsum.add_diff(hi, lo);
        else wsum.add(true_range(hi, lo, in.C(t - 1)));
    }
    __device__ void seed() { y = (float)(wsum.d() / (double)p); }
    template <class In> __device__ int step(const In& in, int t) {
        float tr = true_range(in.H(t), in.L(t), in.C(t - 1));
        y = fmaf(-alpha, y, y) + alpha * tr;
        return 1;
    }
    template <class In> __device__ float value(const In&, int) const { return y; }
    // (see OpRsi::uni; ATR(14) of 300 series x 800 rows 43 -> 38 us)
    static constexpr bool kUni = true;
    template <class In> __device__ float uni(const In& in, int t, int& steps) {
        const float hi = in.H(t), lo = in.L(t);
        const float tr = true_range(hi, lo, t > f ? in.C(t - 1) : hi);
        const float d = hi - lo, bb = d - hi, e = (hi - (d - bb)) - (lo + bb);  // as Acc::add_diff
        wsum.add(t > s ? 0.f : t == f ? d : tr);
        wsum.lo += t == f && isfinite(e) ? e : 0.f;
        const bool run = t > s;
        y = run ? fmaf(-alpha, y, y) + alpha * tr : y;
        steps += run;
        if (t == s) seed();
        return t >= s ? y : qnan();
    }
    __device__ float warm_value(int) const { return qnan(); }
    __device__ void zero() { y = 0.f; }
    __device__ float get(int) const { return y; }
    __device__ void set(int, float v) { y = v; }
    template <bool FIN = false, class In> __device__ float fast(const In& in, int t, int& applied) {
        const float tr = true_range(in.H(t), in.L(t), in.C(t - 1));
        y = fmaf(-alpha, y, y) + alpha * tr;
        ++applied;
        return y;
    }
    static __device__ void coef(int p, D2& a, D2& b) { OpRsi<true>::coef(p, a, b); }
    static __device__ void propagate(D2* S, D2, D2, D2 an, int) { S[0] = d2_mul(S[0], an); }
};

// ------------------------------------------------------------ kernels ------
enum { PASS_AGG = 0, PASS_EMIT = 1 };
constexpr float kBeforeSeed = -2.f, kAbsolute = -1.f;

__device__ __forceinline__ int warp_max(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Staging row write at column j ^ sw (sw = 0 or 1) with no per-step address
// arithmetic once j is a compile-time constant: even columns go to row + sw,
// odd ones to row - sw.
__device__ __forceinline__ void stage_put(float* row, int sw, int j, float v) {
    (j & 1 ? row - sw : row + sw)[j] = v;
}

// One warp = 32 lanes x one time chunk.  Tiles of 32 steps where every lane
// of the warp is past its seed and warm-up take the fast path (no phase
// checks: 2-6 FP ops per step); the few tiles around warm-up take the general
// per-step state machine.
// The 32 steps of one register tile, fully unrolled so every shuffle source
// lane is a constant; EMIT stages the outputs in this lane's row.
template <bool FIN, int PASS, class Op>
__device__ __forceinline__ void run_tile(Op& op, const InTile& ti, float* row, int sw, int& steps) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const float y = op.template fast<FIN>(ti, ti.tb + j, steps);
        if (PASS == PASS_EMIT) stage_put(row, sw, j, y);
    }
}

// 1 / x by the hardware approximation (relative error within about 2^-23;
// subnormal x is read as zero), one instruction
__device__ __forceinline__ float rcp_approx_ftz(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The 32 steps of an RSI emit tile on the scaled state (see run_tile below);
// NORMAL: D stays normal over the tile.
template <bool NORMAL, bool kB>
__device__ __forceinline__ void rsi_emit_steps(OpRsi<kB>& op, const InTile& ti, float* row, int sw) {
    float N = op.sN, D = op.sD;
    const float b = op.beta;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float4 e4 = ti.xs[q], a4 = ti.xs[8 + q];
        const float ev[4] = {e4.x, e4.y, e4.z, e4.w}, av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            N = fmaf(b, N, fmaxf(ev[u], 0.f));
            D = fmaf(b, D, av[u]);
            const float y = NORMAL ? N * rcp_approx_ftz(D) : (D == 0.f ? 50.f : __fdividef(N, D));
            stage_put(row, sw, 4 * q + u, y);
        }
    }
    op.sN = N;
    op.sD = D;
}

// RSI emit tile with finite inputs.  Across consecutive such tiles the state
// is held as
//   N = 100 ag p       (the gain sum, scaled by 100 p)
//   D = (ag + al) p    (the gain + loss sum: its input is |d|)
// so a step is N <- b N + max(100 d, 0), D <- b D + |d| and the output
// 100 ag / (ag + al) = N / D: two FMAs and a max, no per-step scaling.  Each
// lane forms its step's 100 d and |d| once; the warp reads them back from
// shared memory four steps per 16-byte broadcast load.  The state goes back
// to (ag, al) only when the lane leaves these tiles (rsi_fast_exit), so the
// scale factors' roundings do not build up from tile to tile.
template <bool FIN, int PASS, bool kB>
__device__ __forceinline__ void run_tile(OpRsi<kB>& op, const InTile& ti, float* row, int sw, int& steps) {
    if constexpr (!(FIN && PASS == PASS_EMIT)) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float y = op.template fast<FIN>(ti, ti.tb + j, steps);
            if (PASS == PASS_EMIT) stage_put(row, sw, j, y);
        }
    } else {
        const int lane = threadIdx.x & 31;
        float xp = __shfl_up_sync(0xffffffffu, ti.xv, 1);
        if (lane == 0) xp = ti.xb;
        const float d = ti.xv - xp;
        float* xs = reinterpret_cast<float*>(ti.xs);
        __syncwarp();  // the previous tile's reads are done
        xs[lane] = 100.f * d;
        xs[32 + lane] = fabsf(d);
        __syncwarp();
        if (!op.sc) {
            op.sN = op.ag * (100.f * op.pf);  // 100 p is exact
            op.sD = (op.ag + op.al) * op.pf;
            op.sc = true;
        }
        // D never shrinks by more than b^32 >= 2^-32 over a tile (its inputs
        // are >= 0) nor grows past D + 32 max|d|, so a tile entered with D in
        // [2^-60, 2^100] and every |d| <= 2^100 keeps D and 1 / D normal: the
        // output is N times the hardware reciprocal, with no zero guard or
        // subnormal handling
        if (__all_sync(0xffffffffu, op.sD >= 0x1p-60f && op.sD <= 0x1p100f && fabsf(d) <= 0x1p100f))
            rsi_emit_steps<true>(op, ti, row, sw);
        else
            rsi_emit_steps<false>(op, ti, row, sw);
        steps += 32;
    }
}

// (ag, al) from the scaled emit-tile state, before any other step reads them
template <class Op> __device__ __forceinline__ void rsi_fast_exit(Op&) {}
template <bool kB> __device__ __forceinline__ void rsi_fast_exit(OpRsi<kB>& op) {
    if (op.sc) {
        op.ag = (op.sN * 0.01f) * op.inv_p;
        op.al = fmaf(op.sD, op.inv_p, -op.ag);
        op.sc = false;
    }
}

// TEMA emit tile with finite inputs: the three cascaded gain-exact EMA steps
// with shuffle-broadcast inputs and no phase checks; p == 1 copies x.
template <bool FIN, int PASS>
__device__ __forceinline__ void run_tile(OpTema& op, const InTile& ti, float* row, int sw, int& steps) {
    if constexpr (!(FIN && PASS == PASS_EMIT)) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float y = op.template fast<FIN>(ti, ti.tb + j, steps);
            if (PASS == PASS_EMIT) stage_put(row, sw, j, y);
        }
    } else {
        const float a = op.per;
        const bool copy = op.p1 == 0;
        float e1 = op.e1, e2 = op.e2, e3 = op.e3;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float v = __shfl_sync(0xffffffffu, ti.xv, j);
            e1 = fmaf(a, v - e1, e1);
            e2 = fmaf(a, e1 - e2, e2);
            e3 = fmaf(a, e2 - e3, e3);
            stage_put(row, sw, j, copy ? v : fmaf(3.f, e1 - e2, e3));
        }
        op.e1 = e1;  // (a p == 1 lane's state is never read: each step copies x)
        op.e2 = e2;
        op.e3 = e3;
        steps += 32;
    }
}

// Ops with a branch-free general-path step (Op::kUni) use it for t >= f.
template <class Op, class = void> struct HasUni : std::false_type {};
template <class Op> struct HasUni<Op, std::void_t<decltype(Op::kUni)>> : std::true_type {};

// ------------------------------------------------------- fast aggregates ---
// AGG blocks of the chunks in which every combo of a batch sweep is already
// running (EMA, DEMA, TEMA, RSI; chunk >= fast_from).  They share the launch
// with the seed chunk's general-path blocks, so the long per-step seeding run
// of chunk 0 overlaps with this work.  The block stages the chunk's inputs in
// shared memory, kAggTile steps at a time, and reads them back four steps per
// 16-byte broadcast load; each thread advances its combo from a zero state:
//   EMA / DEMA / TEMA  the emit pass's gain-exact steps e <- e + a (in - e)
//                      (a = 2 / (p + 1)), two FP ops per component;
//                      taken kAggBlk at a time (CascadeBlock) on inputs centred
//                      on the chunk's first value, whose own response, in
//                      closed form, is added at the end: the rounding of a
//                      step is then that of the series' movement, not its level;
//   RSI                zg = ag p, zl = al p: zg <- b zg + gain, zl <- b zl + loss
//                      (b = 1 - 1/p), kAggBlk steps at a time as a dot with the
//                      powers of b (as many FMAs, one rounding of zg per block),
//                      scaled back at the chunk end.
// So the entry states they give add no more error than the tensor-core
// contraction's (2-norm of the output errors over the reference, 1e-8, 100,001
// bars, periods 2..201, contraction / step by step / this: RSI 23.1 / 24.4 /
// 23.1, EMA of 5..1000 on 200k 20.1 / 20.8 / 20.1).
// A chunk holding a non-finite input
// (RSI: a non-finite difference) returns false and the block runs the general
// pass, which applies the skip / NaN rules.
enum FastKind { FK_NONE = -1, FK_EMA = 0, FK_DEMA = 1, FK_TEMA = 2, FK_RSI = 3 };
constexpr int kAggTile = 1024;  // steps staged per round (x, or gains + losses)

template <class Op> struct FastKindOf { static constexpr int k = FK_NONE; };
template <> struct FastKindOf<OpEma> { static constexpr int k = FK_EMA; };
template <> struct FastKindOf<OpDema> { static constexpr int k = FK_DEMA; };
template <> struct FastKindOf<OpTema> { static constexpr int k = FK_TEMA; };
template <> struct FastKindOf<OpRsi<true>> { static constexpr int k = FK_RSI; };

// smem: 2 * kAggTile floats, 16-byte aligned (their chunk is shorter by warps).
// The EMA cascades advance kAggBlk steps at a time by their exact block
// transition: after B steps from (e1, e2, e3) with inputs x_0..x_{B-1}
// (a = 2/(p+1), b = 1 - a, j = 0 the oldest),
//   e1' = b^B e1 + sum_j a b^(B-1-j) x_j
//   e2' = b^B e2 + a B b^B e1 + sum_j a^2 (B-j) b^(B-1-j) x_j
//   e3' = b^B e3 + a B b^B e2 + a^2 b^B B(B+1)/2 e1
//         + sum_j a^3 (B-j)(B-j+1)/2 b^(B-1-j) x_j,
// evaluated in the gain-exact form e' = e + sum_i c_i (e_i - e) + (dot - W e)
// (W = the sum of the rounded x-weights; the coefficient of e is b^B in exact
// arithmetic), so a constant input stays fixed whatever the weights'
// rounding.  A block costs one FMA per input per component plus a few for
// the update: about half the work of the per-step form, whose two dependent
// FP ops per step also made each lane's chain latency-bound.
constexpr int kAggBlk = 16;

template <int NZ>
struct CascadeBlock {
    float w[NZ][kAggBlk];  // x-weights, j = 0 the oldest input of the block
    float W[NZ];           // their sums
    float c1, c2;          // a B b^B (e1 -> e2 and e2 -> e3), a^2 b^B B(B+1)/2 (e1 -> e3)
    __device__ void init(float al) {
        // b = 1 - a and its powers in f32: the weights carry relative errors
        // near 1e-6, a perturbation of the filter's time constant (the gain
        // stays exact by the update's form)
        const float be = 1.f - al;
        float pw = 1.f;  // b^(B-1-j), j from B-1 down to 0
#pragma unroll
        for (int q = 0; q < NZ; ++q) W[q] = 0.f;
#pragma unroll
        for (int j = kAggBlk - 1; j >= 0; --j) {
            const float r = (float)(kAggBlk - j);  // B - j
            w[0][j] = al * pw;
            if constexpr (NZ > 1) w[1][j] = al * al * r * pw;
            if constexpr (NZ > 2) w[2][j] = al * al * al * (r * (r + 1.f) * 0.5f) * pw;
            pw *= be;
        }
        // the sums in the order the dots accumulate (oldest first)
#pragma unroll
        for (int j = 0; j < kAggBlk; ++j)
#pragma unroll
            for (int q = 0; q < NZ; ++q) W[q] += w[q][j];
        c1 = al * (float)kAggBlk * pw;
        c2 = al * al * pw * (float)(kAggBlk * (kAggBlk + 1) / 2);
    }
    // one block of inputs x[0..B) (shared-memory broadcast reads, x 16-byte
    // aligned) advancing the first M components (the cascade's later stages
    // not yet started stay as they are)
    template <int M = NZ>
    __device__ __forceinline__ void step(float (&z)[NZ], const float* x) const {
        static_assert(M >= 1 && M <= NZ, "components");
        float d[M][2];
#pragma unroll
        for (int q = 0; q < M; ++q) d[q][0] = d[q][1] = 0.f;
#pragma unroll
        for (int j = 0; j < kAggBlk; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(x + j);
#pragma unroll
            for (int q = 0; q < M; ++q) {
                d[q][0] = fmaf(w[q][j], v.x, d[q][0]);
                d[q][1] = fmaf(w[q][j + 1], v.y, d[q][1]);
                d[q][0] = fmaf(w[q][j + 2], v.z, d[q][0]);
                d[q][1] = fmaf(w[q][j + 3], v.w, d[q][1]);
            }
        }
        const float e1 = z[0];
        z[0] = e1 + fmaf(-W[0], e1, d[0][0] + d[0][1]);
        if constexpr (M > 1) {
            const float e2 = z[1];
            z[1] = fmaf(c1, e1 - e2, e2) + fmaf(-W[1], e2, d[1][0] + d[1][1]);
            if constexpr (M > 2) {
                const float e3 = z[2];
                z[2] = fmaf(c1, e2 - e3, fmaf(c2, e1 - e3, e3)) + fmaf(-W[2], e3, d[2][0] + d[2][1]);
            }
        }
    }
    // steps t in [t0, t1) of the first M components: single gain-exact steps
    // up to a 4-aligned index, blocks of kAggBlk, single steps for the rest
    template <int M>
    __device__ __forceinline__ void run(float (&z)[NZ], const float* xs, int t0, int t1, float al) const {
        auto one = [&](float x) {
            z[0] = fmaf(al, x - z[0], z[0]);
            if constexpr (M > 1) z[1] = fmaf(al, z[0] - z[1], z[1]);
            if constexpr (M > 2) z[2] = fmaf(al, z[1] - z[2], z[2]);
        };
        int t = t0;
        for (; t < t1 && (t & 3); ++t) one(xs[t]);
        for (; t + kAggBlk <= t1; t += kAggBlk) step<M>(z, xs + t);
        for (; t < t1; ++t) one(xs[t]);
    }
};

// RSI's block: powers of b = 1 - 1/p, w[j] = b^(B-1-j), and b^B
struct PowerBlock {
    float w[kAggBlk], bB;
    __device__ void init(int p) {
        static_assert(kAggBlk == 16, "powers up to b^16");
        const D2 b1 = d2_ratio(p - 1, p), b2 = d2_mul(b1, b1), b4 = d2_mul(b2, b2), b8 = d2_mul(b4, b4);
        w[15] = 1.f;
        w[14] = b1.hi;
        w[13] = b2.hi;
        w[12] = b2.hi * b1.hi;
#pragma unroll
        for (int j = 0; j < 4; ++j) w[8 + j] = w[12 + j] * b4.hi;
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = w[8 + j] * b8.hi;
        bB = d2_mul(b8, b8).hi;
    }
    __device__ __forceinline__ float dot(const float* x) const {
        float d0 = 0.f, d1 = 0.f;
#pragma unroll
        for (int j = 0; j < kAggBlk; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(x + j);
            d0 = fmaf(w[j], v.x, d0);
            d1 = fmaf(w[j + 1], v.y, d1);
            d0 = fmaf(w[j + 2], v.z, d0);
            d1 = fmaf(w[j + 3], v.w, d1);
        }
        return d0 + d1;
    }
};

// By a block (its lanes: the block's combos) or by one warp.
template <int K, bool WARP>
__device__ __forceinline__ bool agg_fast(const RecurArgs& a, int li, int c0, int c1, float* smem, float4& g) {
    constexpr int NZ = K == FK_EMA ? 1 : (K == FK_TEMA ? 3 : 2);
    float* s0 = smem;
    float* s1 = smem + kAggTile;
    const int tid = WARP ? threadIdx.x & 31 : threadIdx.x, threads = WARP ? 32 : blockDim.x;
    const int p = li < a.n_lanes ? a.periods[li] : 1;
    const float b = coef::wilder_keep(p);  // RSI
    const float al = coef::ema(p);         // the EMAs
    const float ref = K == FK_RSI ? 0.f : __ldg(a.x + c0);
    float z[NZ];
#pragma unroll
    for (int q = 0; q < NZ; ++q) z[q] = 0.f;
    typename std::conditional<K == FK_RSI, PowerBlock, CascadeBlock<NZ>>::type blk;
    if constexpr (K == FK_RSI) blk.init(p);
    else blk.init(al);
    for (int t0 = c0; t0 < c1; t0 += kAggTile) {
        const int m = min(kAggTile, c1 - t0);
        int bad = 0;
        for (int i = tid; i < m; i += threads) {
            const float v = __ldg(a.x + t0 + i);
            if (K == FK_RSI) {
                const float d = v - __ldg(a.x + t0 + i - 1);  // t0 + i >= c0 > 0
                bad |= !isfinite(d);
                s0[i] = d > 0.f ? d : 0.f;
                s1[i] = d < 0.f ? -d : 0.f;
            } else {
                const float d = v - ref;
                bad |= !isfinite(d);
                s0[i] = d;
            }
        }
        if (WARP) {
            if (__any_sync(0xffffffffu, bad)) return false;
            __syncwarp();
        } else if (__syncthreads_or(bad)) {
            return false;
        }
        const int mb = m - m % kAggBlk;
        if constexpr (K == FK_RSI) {
            for (int i = 0; i < mb; i += kAggBlk) {
                z[0] = fmaf(blk.bB, z[0], blk.dot(s0 + i));
                z[1] = fmaf(blk.bB, z[1], blk.dot(s1 + i));
            }
            for (int i = mb; i < m; ++i) {
                z[0] = fmaf(b, z[0], s0[i]);
                z[1] = fmaf(b, z[1], s1[i]);
            }
        } else {
            for (int i = 0; i < mb; i += kAggBlk) blk.step(z, s0 + i);
            for (int i = mb; i < m; ++i) {  // the gain-exact EMA step of the emit pass (OpEma::step)
                z[0] = fmaf(al, s0[i] - z[0], z[0]);
                if constexpr (NZ > 1) z[1] = fmaf(al, z[0] - z[1], z[1]);
                if constexpr (NZ > 2) z[2] = fmaf(al, z[1] - z[2], z[2]);
            }
        }
        if (WARP) __syncwarp();
        else __syncthreads();
    }
    const int n = c1 - c0;
    g = make_float4(0.f, 0.f, 0.f, (float)n);
    if constexpr (K == FK_RSI) {
        const float ip = (float)(1.0 / p);
        g.x = z[0] * ip;
        g.y = z[1] * ip;
    } else {
        // a constant 1 takes the stages to 1 - u, 1 - u (1 + n a) and
        // 1 - u (1 + n a + n (n + 1) / 2 a^2), u = (1 - a)^n
        const D2 u = d2_pow(d2_ratio(p - 1, p + 1), n), ad = d2_ratio(2, p + 1);
        auto centred = [&](D2 resp, float v) {
            const D2 t = d2_add(d2_mul({ref, 0.f}, resp), {v, 0.f});
            return t.hi + t.lo;
        };
        D2 resp = d2_add({1.f, 0.f}, d2_neg(u));
        g.x = centred(resp, z[0]);
        if constexpr (NZ > 1) {
            const D2 au = d2_mul(ad, u);
            resp = d2_add(resp, d2_neg(d2_mul(au, {(float)n, 0.f})));
            g.y = centred(resp, z[1]);
            if constexpr (NZ > 2) {
                const D2 k = d2_from_ll((long long)n * (n + 1) / 2);
                resp = d2_add(resp, d2_neg(d2_mul(d2_mul(ad, au), k)));
                g.z = centred(resp, z[2]);
            }
        }
    }
    return true;
}

// AGG record of a chunk from the tensor-core contraction's S partial sums
// (k_recur_tc.cu): per component the sum of the partials, times the row and
// column scales, plus the centring term.  One thread per lane.
template <int K>
__device__ void agg_from_partials(const RecurArgs& a, int chunk, int len) {
    constexpr int NZ = K == FK_EMA ? 1 : (K == FK_TEMA ? 3 : 2);
    const RecurTcView& v = a.tc;
    const int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li >= a.n_lanes) return;
    const int j0 = chunk - v.g0;
    float z[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < NZ; ++q) {
        const int r = K == FK_RSI ? li : q * v.mpad + li;
        const int j = K == FK_RSI ? j0 + q * v.nc : j0;
        const float* p = v.part + (size_t)j * v.rows + r;
        const size_t stride = (size_t)v.npad * v.rows;
        // four independent loads in flight, summed in split order
        float acc = 0.f;
        int s = 0;
        for (; s + 4 <= v.S; s += 4) {
            const float p0 = __ldg(p + (size_t)s * stride), p1 = __ldg(p + (size_t)(s + 1) * stride);
            const float p2 = __ldg(p + (size_t)(s + 2) * stride), p3 = __ldg(p + (size_t)(s + 3) * stride);
            acc = (((acc + p0) + p1) + p2) + p3;
        }
        for (; s < v.S; ++s) acc += __ldg(p + (size_t)s * stride);
        z[q] = fmaf(acc, __ldg(v.row_scale + r) * __ldg(v.col_scale + j), __ldg(v.col_ref + j) * __ldg(v.row_sum + r));
    }
    reinterpret_cast<float4*>(a.agg)[(size_t)chunk * a.n_lanes + li] = make_float4(z[0], z[1], z[2], (float)len);
}

// ------------------------------------------------------ seed chunk, AGG ---
// The AGG pass needs only the state at the end of the seed chunk [0, c1).
// When every input in [first, c1) is finite and every lane's seed index lies
// inside the chunk, a lane gets there by plain loops instead of the per-step
// phase logic: the warm-up sum in four independent compensated partial sums
// (a short dependency chain), then the running steps from the seed on.  The
// per-step phase logic made each lane's 1,000-2,000-step walk the critical
// path of the whole AGG launch.
// Pair sum of two (hi, lo) compensated values (TwoSum of the heads).
__device__ __forceinline__ float2 pair_add(float2 a, float2 b) {
    const float s = a.x + b.x;
    const float bb = s - a.x;
    const float e = (a.x - (s - bb)) + (b.x - bb);
    const float lo = a.y + b.y + e;
    const float hi = s + lo;
    return make_float2(hi, lo - (hi - s));
}

// Block-wide sums of the seed chunk's warm-up terms in 32-step segments:
// segment i covers [b0 + 32 i, b0 + 32 i + 32) ∩ [b0, c1) and holds, as
// compensated (hi, lo) pairs, the sum of x (EMA: b0 = first) or of the
// exact gains and losses (RSI: b0 = first + 1; the differences to the
// previous bar).  A lane's warm-up sum over p terms from b0 is then p / 32
// segment sums plus at most 31 single terms, instead of a p-step chain.
// seg: float4 {sum hi, sum lo, loss hi, loss lo} per segment.  Called by the
// whole block; every input in [b0 - 1, c1) is finite.
template <int K>
__device__ void seed_segments(const float* xs, int b0, int c1, float4* seg) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nseg = (c1 - b0 + 31) >> 5;
    for (int i = warp; i < nseg; i += nw) {
        const int t = b0 + 32 * i + lane;
        float2 u = make_float2(0.f, 0.f), v = make_float2(0.f, 0.f);
        if (t < c1) {
            if constexpr (K == FK_RSI) {
                const float x1 = xs[t], x0 = xs[t - 1];
                const float d = x1 - x0;  // exact difference d + e (TwoDiff)
                const float bb = d - x1;
                const float e = (x1 - (d - bb)) - (x0 + bb);
                if (d > 0.f) u = make_float2(d, e);
                else if (d < 0.f) v = make_float2(-d, -e);
            } else {
                u = make_float2(xs[t], 0.f);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            u = pair_add(u, make_float2(__shfl_xor_sync(0xffffffffu, u.x, o), __shfl_xor_sync(0xffffffffu, u.y, o)));
            if constexpr (K == FK_RSI)
                v = pair_add(v, make_float2(__shfl_xor_sync(0xffffffffu, v.x, o),
                                            __shfl_xor_sync(0xffffffffu, v.y, o)));
        }
        if (lane == 0) seg[i] = make_float4(u.x, u.y, v.x, v.y);
    }
}

template <int K>
__device__ bool agg_seed_fast(const RecurArgs& a, float* xs, int c1, int cap) {
    const int f = a.first;
    const int li = blockIdx.x * blockDim.x + threadIdx.x;
    const bool lane_ok = li < a.n_lanes;
    const int p = lane_ok ? a.periods[li] : 1;
    // seed index of the lane (the op's s)
    const int s = K == FK_EMA ? f + p - 1 : K == FK_RSI ? f + p : f + 2 * (p - 1);
    int bad = lane_ok && (p <= 0 || s >= c1);
    for (int t = max(f, 0) + threadIdx.x; t < c1; t += blockDim.x) bad |= !isfinite(xs[t]);
    if (__syncthreads_or(bad)) return false;
    // segment sums of the warm-up terms (EMA, RSI) when they fit beside xs
    const int b0 = K == FK_RSI ? f + 1 : f;
    const int seg_off = (c1 + 3) & ~3;
    const bool use_seg = K != FK_TEMA && f >= 0 && seg_off + 4 * ((c1 - b0 + 31) >> 5) <= cap;
    float4* seg = reinterpret_cast<float4*>(xs + seg_off);
    if (use_seg) {
        seed_segments<K>(xs, b0, c1, seg);
        __syncthreads();
    }
    if (!lane_ok) return true;
    float4 g = make_float4(0.f, 0.f, 0.f, kAbsolute);
    if constexpr (K == FK_EMA) {
        // the op's warm-up mean of x[f..s] (every value finite: count p)
        Acc acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q].zero();
        int t = f;
        if (use_seg) {
            const int full = p >> 5;
            for (int i = 0; i < full; ++i) {
                const float4 sv = seg[i];
                acc[i & 1].add(sv.x);
                acc[i & 1].lo += sv.y;
            }
            t = f + 32 * full;
        }
        for (; t + 3 <= s; t += 4)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q].add(xs[t + q]);
        for (; t <= s; ++t) acc[0].add(xs[t]);
        acc[0].add(acc[1].hi); acc[0].add(acc[1].lo);
        acc[2].add(acc[3].hi); acc[2].add(acc[3].lo);
        acc[0].add(acc[2].hi); acc[0].add(acc[2].lo);
        const float al = coef::ema(p);
        CascadeBlock<1> cb;
        cb.init(al);
        float y[1] = {acc[0].f() / (float)p};
        cb.run<1>(y, xs, s + 1, c1, al);  // the running steps, kAggBlk at a time
        g.x = y[0];
    } else if constexpr (K == FK_RSI) {
        // sums of the gains and losses of the p deltas in (f, s], then the
        // Wilder steps (the op's seed() and step() arithmetic)
        Acc sg[2], sl[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) { sg[q].zero(); sl[q].zero(); }
        int t = f + 1;
        if (use_seg) {
            const int full = p >> 5;
            for (int i = 0; i < full; ++i) {
                const float4 sv = seg[i];
                sg[i & 1].add(sv.x);
                sg[i & 1].lo += sv.y;
                sl[i & 1].add(sv.z);
                sl[i & 1].lo += sv.w;
            }
            t = f + 1 + 32 * full;
        }
        for (; t + 1 <= s; t += 2)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float v = xs[t + q], xp = xs[t + q - 1];
                if (v > xp) sg[q].add_diff(v, xp);
                else if (v < xp) sl[q].add_diff(xp, v);
            }
        for (; t <= s; ++t) {
            const float v = xs[t], xp = xs[t - 1];
            if (v > xp) sg[0].add_diff(v, xp);
            else if (v < xp) sl[0].add_diff(xp, v);
        }
        const float beta = coef::wilder_keep(p), ip = coef::wilder(p);
        const double inv_p = (double)ip;
        float ag = (float)((sg[0].d() + sg[1].d()) * inv_p);
        float al = (float)((sl[0].d() + sl[1].d()) * inv_p);
        for (t = s + 1; t < c1; ++t) {
            const float d = xs[t] - xs[t - 1];
            ag = fmaf(ag, beta, ip * (d > 0.f ? d : 0.f));
            al = fmaf(al, beta, ip * (d < 0.f ? -d : 0.f));
        }
        g.x = ag;
        g.y = al;
    } else {
        // TEMA: e1 from x[f]; e2 joins at f + p - 1 as a copy of e1, e3 at s
        // as a copy of e2 (the op's accum), then all three run (p == 1:
        // the op copies x into e1)
        const float per = coef::ema(p);
        if (p == 1) {
            g.x = xs[c1 - 1];
        } else {
            // the three phases kAggBlk steps at a time (CascadeBlock)
            const int start2 = f + p - 1;
            CascadeBlock<3> cb;
            cb.init(per);
            float z[3] = {xs[f], 0.f, 0.f};
            cb.run<1>(z, xs, f + 1, start2 + 1, per);
            z[1] = z[0];
            cb.run<2>(z, xs, start2 + 1, s + 1, per);
            z[2] = z[1];
            cb.run<3>(z, xs, s + 1, c1, per);
            g.x = z[0];
            g.y = z[1];
            g.z = z[2];
        }
    }
    reinterpret_cast<float4*>(a.agg)[li] = g;  // chunk 0
    return true;
}

// One step of the general (per-step phase) path of one lane: warm-up
// accumulation until the seed index, the seed, then running steps.
template <class Op, class In>
__device__ __forceinline__ float general_step(Op& op, bool active, bool seeded_ever, bool& running, int& steps,
                                              const In& in, int t) {
    float v = qnan();
    if constexpr (HasUni<Op>::value) {
        if (active && t >= op.f) v = op.uni(in, t, steps);
        return v;
    }
    if (active && t >= op.f && seeded_ever) {
        if (running) {
            steps += op.step(in, t);
            v = op.value(in, t);
        } else if (t <= op.s) {
            op.accum(in, t);
            if (t == op.s) {
                op.seed();
                running = true;
                v = op.value(in, t);
            } else {
                v = op.warm_value(t);
            }
        }
    } else if (active && t >= op.f && !seeded_ever) {
        op.accum(in, t);  // never seeded (s >= n): warm-up style outputs only
        v = op.warm_value(t);
    }
    return v;
}

// AGG record of one (lane, chunk): state, and applied steps or a marker for
// a chunk before the seed / holding the seed.
template <class Op>
__device__ __forceinline__ float4 agg_record(const Op& op, bool active, bool seeded_ever, int steps, int c0, int c1) {
    const bool abs_chunk = active && seeded_ever && c0 <= op.s && op.s < c1;
    const bool before = !active || !seeded_ever || c1 <= op.s;
    float4 g;
    g.x = Op::NS > 0 ? op.get(0) : 0.f;
    g.y = Op::NS > 1 ? op.get(1) : 0.f;
    g.z = Op::NS > 2 ? op.get(2) : 0.f;
    g.w = before ? kBeforeSeed : (abs_chunk ? kAbsolute : (float)steps);
    if (before) g.x = g.y = g.z = 0.f;
    return g;
}
__device__ __forceinline__ float4* agg_slot(const RecurArgs& a, int chunk, int li) {
    return reinterpret_cast<float4*>(a.agg) + (size_t)chunk * a.n_lanes + li;
}

// Batch EMIT stages 64 steps per lane (two 32-step tiles) and writes each
// row's 256-byte segment with one float2 store per lane: on GB300 that write
// pattern reaches ~6.9 TB/s where 128-byte row segments reach ~6.2 TB/s.
// Staging rows are 66 floats (8-byte aligned float2 reads); rows 16..31 swap
// the two floats of each pair (column c is stored at c ^ 1), so the per-step
// scalar writes of the 32 lanes fall in 32 distinct banks.  The stores are
// marked evict-first (nothing of the call reads them back): 999 EMAs on 1M bars
// 648 -> 635 us, 399 on 500k 185 -> 177.
//
// Rows that do not all start at a 32-byte sector (n % 8 != 0) are CUT at the
// sectors instead: row r writes [seg0 - m, seg0 + 64 - m), m = its segment's
// offset into a sector, so a chunk has two partial sectors per row, not one or
// two per segment (the L2 merges partial sectors at about half the write
// rate).  The last m values of the segment before wait in kCarry columns in
// front of the row.  Bound by the flush: about twice the
// instructions of the whole-segment form.
constexpr int kSeg = 64, kCarry = 8;
constexpr int kStageW = kSeg + 2, kCutW = kCarry + kStageW;

// ------------------------------------------------------- warm-up tiles ----
// Tiles in which some combos are still warming up.  All combos of a batch
// sweep share the series and its first valid index f, so what their warm-up
// needs is one prefix sum over [f, t] of the op's terms (x, the true ranges,
// or the gains and losses): a lane whose seed index s lies in the tile takes
// its seed from the prefix at s, and EMA's warm-up output, the running mean,
// is the prefix over the count.  The prefix of a 32-step tile is one warp scan
// of compensated pairs, and a step is then the running update under the
// predicate t > s: no accumulators, divisions or branches per lane and step
// (the general path's per-lane phases cost about 150 cycles a step, which made
// the seeding chunk the longest of a sweep: with the shorter first chunks that
// this allows, EMA 2..1000 on 20,000 bars 195 -> 45 us, RSI 225 -> 65).  Used when every input of [f, tile end) is finite;
// otherwise the chunk's warm-up takes the general path.
struct WarmTerm {
    float2 a, b;  // compensated terms of one step (b: RSI's loss)
};

template <class Op> struct WarmOf { static constexpr bool ok = false; };
template <> struct WarmOf<OpEma> { static constexpr bool ok = true, two = false; };
template <> struct WarmOf<OpDema> { static constexpr bool ok = true, two = false; };
template <> struct WarmOf<OpWilders> { static constexpr bool ok = true, two = false; };
template <> struct WarmOf<OpAtr> { static constexpr bool ok = true, two = false; };
template <> struct WarmOf<OpTema> { static constexpr bool ok = true, two = false; };
template <> struct WarmOf<OpRsi<true>> { static constexpr bool ok = true, two = true; };

__device__ __forceinline__ float2 exact_diff(float a, float b) {  // a - b as value and error
    const float d = a - b;
    const float bb = d - a;
    return make_float2(d, (a - (d - bb)) - (b + bb));
}

// finite, and small enough that no sum of a warm-up overflows
__device__ __forceinline__ bool warm_fin(float v) { return fabsf(v) <= 0x1p96f; }

// Inputs of one lane's step t of a tile (x0 / c at t, x1 at t - 1), its term,
// and the value the running step reads (x, the true range, or the difference)
template <class Op>
__device__ __forceinline__ WarmTerm warm_term(int t, int f, float x0, float x1, float h, float l, float& in, bool& fin) {
    WarmTerm w{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if constexpr (std::is_same<Op, OpAtr>::value) {
        in = t == f ? h - l : true_range(h, l, x1);
        fin = t < f || (warm_fin(x0) && warm_fin(in));
        if (t >= f) w.a = t == f ? exact_diff(h, l) : make_float2(in, 0.f);
    } else if constexpr (std::is_same<Op, OpRsi<true>>::value) {
        in = t > f ? x0 - x1 : 0.f;
        fin = t < f || (warm_fin(x0) && warm_fin(in));
        if (t > f) {
            if (x0 > x1) w.a = exact_diff(x0, x1);
            else if (x0 < x1) w.b = exact_diff(x1, x0);
        }
    } else {
        in = x0;
        fin = t < f || warm_fin(x0);
        if (t >= f) w.a = make_float2(x0, 0.f);
    }
    return w;
}

__device__ __forceinline__ float2 pair_scan(float2 v) {  // inclusive over the warp
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float2 u = make_float2(__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o));
        if (lane >= o) v = pair_add(u, v);
    }
    return v;
}
__device__ __forceinline__ float2 pair_shfl(float2 v, int src) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
// The prefix of the terms over [f, c0) and whether every input of [f, tend) is
// finite (whole warp)
template <class Op>
__device__ bool warm_prefix(const InBatch& in, int f, int c0, int tend, WarmTerm& pre) {
    // (TEMA's stages start from values, not sums, and take any input)
    if constexpr (std::is_same<Op, OpTema>::value) return true;
    const int lane = threadIdx.x & 31;
    WarmTerm acc{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    bool ok = true;
#pragma unroll 4
    for (int t = f + lane; t < tend; t += 32) {
        float x0, x1 = 0.f, h = 0.f, l = 0.f, v;
        bool fin;
        if constexpr (Op::kHlc) {
            x0 = in.C(t);
            if (t > f) x1 = in.C(t - 1);
            h = in.H(t);
            l = in.L(t);
        } else {
            x0 = in.X(t);
            if (t > f) x1 = in.X(t - 1);
        }
        const WarmTerm w = warm_term<Op>(t, f, x0, x1, h, l, v, fin);
        ok = ok && fin;
        if (t < c0) {
            acc.a = pair_add(acc.a, w.a);
            if (WarmOf<Op>::two) acc.b = pair_add(acc.b, w.b);
        }
    }
    pre.a = pair_shfl(pair_scan(acc.a), 31);
    pre.b = WarmOf<Op>::two ? pair_shfl(pair_scan(acc.b), 31) : acc.b;
    return __all_sync(0xffffffffu, ok);
}

// Steps [tb, tb + nt) of a warm-up tile; xv .. lv: this lane's step of the tile,
// x1: the step before it; pre: the prefix over [f, tb), updated.
template <int PASS, class Op>
__device__ __forceinline__ void warm_tile(Op& op, int f, int tb, int nt, float xv, float x1, float hv, float lv,
                                          WarmTerm& pre, float* srow, int sw) {
    const int lane = threadIdx.x & 31;
    const int t = tb + lane, s = op.s;  // (f: the sweep's, also for lanes without a combo)
    float in = 0.f;
    bool fin;
    WarmTerm w = warm_term<Op>(lane < nt ? t : f - 1, f, xv, x1, hv, lv, in, fin);
    if (!std::is_same<Op, OpTema>::value && !std::is_same<Op, OpDema>::value) {
        w.a = pair_add(pre.a, pair_scan(w.a));  // the prefix over [f, t]
        pre.a = pair_shfl(w.a, 31);
    }
    if (WarmOf<Op>::two) {
        w.b = pair_add(pre.b, pair_scan(w.b));
        pre.b = pair_shfl(w.b, 31);
    }
    const bool here = s >= tb && s < tb + nt;
    const int sl = here ? s - tb : 0;  // the lane holding this lane's seed step
    if constexpr (std::is_same<Op, OpEma>::value) {
        const float mean = (w.a.x + w.a.y) / (float)(t - f + 1);
        float y = op.y;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            if (j >= nt) break;
            const float x = __shfl_sync(0xffffffffu, in, j), m = __shfl_sync(0xffffffffu, mean, j);
            y = tb + j > s ? fmaf(op.alpha, x - y, y) : m;
            if (PASS == PASS_EMIT) srow[j ^ sw] = tb + j < f ? qnan() : y;
        }
        op.y = y;
    } else if constexpr (std::is_same<Op, OpDema>::value) {
        float e1 = op.e1, e2 = op.e2;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            if (j >= nt) break;
            const float x = __shfl_sync(0xffffffffu, in, j);
            const bool run = tb + j > f;
            e1 = run ? fmaf(op.alpha, x - e1, e1) : x;
            e2 = run ? fmaf(op.alpha, e1 - e2, e2) : x;
            if (PASS == PASS_EMIT) srow[j ^ sw] = tb + j < op.warm ? qnan() : fmaf(e1, 2.f, -e2);
        }
        op.e1 = e1;
        op.e2 = e2;
    } else if constexpr (std::is_same<Op, OpTema>::value) {
        // the three stages join at f, start2 and s as copies of the one before
        // (a stage not yet started holds nothing that is read)
        const float a = op.per;
        const bool copy = op.p1 == 0;
        float e1 = op.e1, e2 = op.e2, e3 = op.e3;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            if (j >= nt) break;
            const float x = __shfl_sync(0xffffffffu, in, j);
            const float b1 = tb + j == f ? x : e1;
            e1 = copy ? x : fmaf(a, x - b1, b1);
            const float b2 = tb + j == op.start2 ? e1 : e2;
            e2 = fmaf(a, e1 - b2, b2);
            const float b3 = tb + j == s ? e2 : e3;
            e3 = fmaf(a, e2 - b3, b3);
            if (PASS == PASS_EMIT) srow[j ^ sw] = tb + j < op.warm ? qnan() : (copy ? x : fmaf(3.f, e1 - e2, e3));
        }
        op.e1 = e1;
        op.e2 = e2;
        op.e3 = e3;
    } else if constexpr (std::is_same<Op, OpRsi<true>>::value) {
        const float2 ga = pair_shfl(w.a, sl), la = pair_shfl(w.b, sl);
        const int p = (int)op.pf;
        const float sg = here ? pair_mean(ga, p, op.inv_p) : 0.f, sl_ = here ? pair_mean(la, p, op.inv_p) : 0.f;
        float ag = op.ag, al = op.al;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            if (j >= nt) break;
            const float d = __shfl_sync(0xffffffffu, in, j);
            const bool run = tb + j > s;
            ag = run ? fmaf(ag, op.beta, op.inv_p * fmaxf(d, 0.f)) : sg;
            al = run ? fmaf(al, op.beta, op.inv_p * fmaxf(-d, 0.f)) : sl_;
            if (PASS == PASS_EMIT) {
                const float den = ag + al;
                const float v = den == 0.f ? 50.f : __fdividef(100.f * ag, den);
                srow[j ^ sw] = tb + j < s ? qnan() : v;
            }
        }
        op.ag = ag;
        op.al = al;
    } else {  // Wilders, ATR
        const float2 sum = pair_shfl(w.a, sl);
        const float seed = here ? pair_mean(sum, op.p, op.alpha) : 0.f;
        const bool copy = std::is_same<Op, OpWilders>::value && op.p == 1;
        float y = op.y;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            if (j >= nt) break;
            const float x = __shfl_sync(0xffffffffu, in, j);
            float n;
            if constexpr (std::is_same<Op, OpWilders>::value) n = copy ? x : fmaf(x - y, op.alpha, y);
            else n = fmaf(-op.alpha, y, y) + op.alpha * x;
            y = tb + j > s ? n : seed;
            if (PASS == PASS_EMIT) srow[j ^ sw] = tb + j < s ? qnan() : y;
        }
        op.y = y;
    }
}

// One warp's 32 lanes (combos 32 group .. 32 group + 31) over [c0, c1): AGG
// returns the lane's record, EMIT starts from the state `cv` where the lane is
// running and writes the outputs.  stage: 32 x (CUT ? kCutW : kStageW) floats,
// xin: 16 float4 of the warp's own (EMIT only).
template <class Op, int PASS, bool CUT>
__device__ __forceinline__ float4 recur_span(const RecurArgs& a, int group, int c0, int c1, const float4 cv,
                                             float* stage, float4* xin) {
    const int lane = threadIdx.x & 31;
    const int li = group * 32 + lane;
    const bool valid = li < a.n_lanes;
    Op op;
    int p = 0, first = a.n;
    if (valid) {
        p = a.periods[li];
        first = a.first;
    }
    op.init(p > 0 ? p : 1, first);
    const bool active = valid && first < a.n && p > 0;
    const bool seeded_ever = active && op.s < a.n;
    const InBatch in{a.x, a.h, a.l, a.c};

    // first time index from which this lane needs no phase checks; lanes that
    // never write (invalid / all-NaN) do not hold the warp back
    const int run_from = (active && seeded_ever) ? max(op.s + 1, op.warm) : (valid ? INT_MAX : INT_MIN);
    const int warp_run_from = warp_max(run_from);
    // warm-up tiles: the prefix at c0, if every input they read is finite
    bool warm_ok = false;
    WarmTerm pre{};
    if constexpr (WarmOf<Op>::ok) {
        if (c0 < warp_run_from && a.first < a.n) {  // up to the end of the last such tile
            const int tend = warp_run_from >= c1 ? c1 : min(c1, c0 + (warp_run_from - c0 + 31) / 32 * 32);
            warm_ok = warm_prefix<Op>(in, a.first, c0, tend, pre);
        }
    }

    // chunk entry state
    bool running = false;
    if (active) {
        if (c0 > op.s && seeded_ever) {
            if (PASS == PASS_AGG) {
                op.zero();
            } else {
                if (Op::NS > 0) op.set(0, cv.x);
                if (Op::NS > 1) op.set(1, cv.y);
                if (Op::NS > 2) op.set(2, cv.z);
            }
            running = true;
        } else if (c0 > op.f && (!warm_ok || std::is_same<Op, OpTema>::value)) {
            // the chunk starts inside the warm-up: accumulate [f, c0) first
            // (TEMA's stages have no closed form in the terms)
            const int end = min(c0, op.s + 1);
#pragma unroll 8
            for (int t = op.f; t < end; ++t) op.accum(in, t);
        }
    }

    int steps = 0;
    // this lane's staging row (batch EMIT): the current 64-step segment starts
    // at seg0, the tile at column off = tb - seg0 (0 or 32), swizzle sw
    const int sw = (lane >> 4) & 1;
    constexpr int W = CUT ? kCutW : kStageW, C0 = CUT ? kCarry : 0;
    const bool vec2 = !CUT && PASS == PASS_EMIT && (a.n & 1) == 0 && (c0 & 1) == 0 &&
                      (reinterpret_cast<uintptr_t>(a.out) & 7) == 0;
    // writes a completed segment of the warp's 32 rows (tile [tb, te))
    auto flush = [&](int seg0, int off, int te) {
        if (PASS != PASS_EMIT || (off != kSeg - 32 && te != c1)) return;
        __syncwarp();
        const int row0 = group * 32;
        const int rows = min(32, a.n_lanes - row0);
        const int len = te - seg0;
        float* ob = a.out + (size_t)row0 * a.n + seg0;
        if (CUT) {
            const int m0 = (int)(reinterpret_cast<uintptr_t>(ob) >> 2);
            const bool first = seg0 == c0, last = te == c1;
            const float* sr = stage + kCarry + lane;
            float* op = ob + lane;
            if (!first && !last && rows == 32) {
                // m repeats every 8 rows
                int m[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) m[k] = (int)((unsigned)m0 + (unsigned)k * (unsigned)a.n) & 7;
                op += lane;
                sr += lane;
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    float2 v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int x = i < 16 ? 0 : m[k] & 1 ? -1 : 1;  // the row's swizzle
                        v[k] = make_float2(sr[(i + k) * W + x - m[k]], sr[(i + k) * W + 1 - x - m[k]]);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k, op += a.n) __stcs(reinterpret_cast<float2*>(op - m[k]), v[k]);
                }
            } else {  // a chunk's first segment has no carry, its last leaves none
#pragma unroll 4
                for (int r = 0; r < rows; ++r, sr += W, op += a.n) {
                    const int m = (int)((unsigned)m0 + (unsigned)r * (unsigned)a.n) & 7, odd = (lane - m) & 1;
                    const int x = (r >> 4) & 1 ? 1 - 2 * odd : 0;
                    const int e = lane - m, lo = first ? 0 : -kCarry, hi = last ? len : kSeg - m;
                    if (e >= lo && e < hi) op[-m] = sr[x - m];
                    if (e + 32 < hi) op[32 - m] = sr[32 + x - m];
                    if (e + 64 < hi) op[64 - m] = sr[64 + x - m];
                }
            }
            __syncwarp();
            if (te != c1) {  // the segment's last columns become the next one's carry
                float2* row = reinterpret_cast<float2*>(stage + lane * W);
#pragma unroll
                for (int i = 0; i < kCarry / 2; ++i) row[i] = row[kSeg / 2 + i];
            }
        } else if (vec2 && len == kSeg) {
            // rows 0..15 as staged, rows 16..31 with each pair swapped back
            const int r16 = min(rows, 16);
            float* op = ob + 2 * lane;
#pragma unroll 4
            for (int r = 0; r < r16; ++r, op += a.n)
                __stcs(reinterpret_cast<float2*>(op), *reinterpret_cast<const float2*>(stage + r * W + 2 * lane));
#pragma unroll 4
            for (int r = 16; r < rows; ++r, op += a.n) {
                const float2 v = *reinterpret_cast<const float2*>(stage + r * W + 2 * lane);
                __stcs(reinterpret_cast<float2*>(op), make_float2(v.y, v.x));
            }
        } else {
            for (int h = lane; h < len; h += 32) {
#pragma unroll 4
                for (int r = 0; r < rows; ++r) ob[(size_t)r * a.n + h] = stage[r * W + (h ^ ((r >> 4) & 1))];
            }
        }
        __syncwarp();
    };
    // two loops, so that nothing of the warm-up's state is live in the second
    int tb = c0;
    for (; tb < c1 && tb < warp_run_from; tb += 32) {
        const int te = min(tb + 32, c1);
        const int seg0 = c0 + ((tb - c0) & ~(kSeg - 1));
        const int off = tb - seg0;
        float* srow = stage + lane * W + C0 + off;
        // ---- general path: per-step phase logic
        rsi_fast_exit(op);  // (a no-op: general tiles come before the fast ones)
        // the tile's inputs in registers (one coalesced load per lane);
        // each step's values are broadcast by shuffles at the top of
        // the warp-uniform step loop, before any per-lane branch
        const int nt = te - tb;
        float xv = 0.f, hv = 0.f, lv = 0.f, pb = 0.f;
        if constexpr (Op::kHlc) {
            if (lane < nt) {
                hv = __ldg(a.h + tb + lane);
                lv = __ldg(a.l + tb + lane);
                xv = __ldg(a.c + tb + lane);
            }
            if (tb > 0) pb = __ldg(a.c + tb - 1);
        } else {
            if (lane < nt) xv = __ldg(a.x + tb + lane);
            if (tb > 0) pb = __ldg(a.x + tb - 1);
        }
        bool done = false;
        if constexpr (WarmOf<Op>::ok) {
            if (warm_ok) {
                float xm = __shfl_up_sync(0xffffffffu, xv, 1);
                if (lane == 0) xm = pb;
                warm_tile<PASS>(op, a.first, tb, nt, xv, xm, hv, lv, pre, srow, sw);
                if (active && seeded_ever) {
                    steps += max(0, te - max(tb, op.s + 1));
                    running = op.s < te;
                }
                done = true;
            }
        }
        for (int j = 0; j < (done ? 0 : nt); ++j) {
            InStep st;
            st.t = tb + j;
            st.x0 = __shfl_sync(0xffffffffu, xv, j);
            const float xm = __shfl_sync(0xffffffffu, xv, (j - 1) & 31);
            st.x1 = j > 0 ? xm : pb;
            if constexpr (Op::kHlc) {
                st.h0 = __shfl_sync(0xffffffffu, hv, j);
                st.l0 = __shfl_sync(0xffffffffu, lv, j);
            }
            const float v = general_step(op, active, seeded_ever, running, steps, st, tb + j);
            if (PASS == PASS_EMIT) srow[j ^ sw] = v;
        }
        flush(seg0, off, te);
    }
    for (; tb < c1; tb += 32) {
        const int te = min(tb + 32, c1);
        const int seg0 = c0 + ((tb - c0) & ~(kSeg - 1));
        const int off = tb - seg0;
        float* srow = stage + lane * W + C0 + off;
        // ---- fast path: every lane running and past warm-up
        if (te - tb == 32) {
            // the tile's inputs in registers, one coalesced load per lane
            InTile ti;
            ti.tb = tb;
            ti.xs = xin;
            if constexpr (Op::kHlc) {
                ti.hv = __ldg(a.h + tb + lane);
                ti.lv = __ldg(a.l + tb + lane);
                ti.cv = __ldg(a.c + tb + lane);
                ti.cb = __ldg(a.c + tb - 1);
                ti.xv = ti.cv;
                ti.xb = ti.cb;
            } else {
                ti.xv = __ldg(a.x + tb + lane);
                ti.xb = __ldg(a.x + tb - 1);
            }
            // a tile whose inputs (and the value before it) are all finite
            // runs without per-step skip / NaN logic
            bool fin;
            if constexpr (Op::kHlc) {
                fin = __all_sync(0xffffffffu, isfinite(ti.hv) && isfinite(ti.lv) && isfinite(ti.cv) &&
                                                  isfinite(ti.cb));
            } else {
                fin = __all_sync(0xffffffffu, isfinite(ti.xv) && isfinite(ti.xb));
            }
            if (fin) {
                run_tile<true, PASS>(op, ti, srow, sw, steps);
            } else {
                rsi_fast_exit(op);
                run_tile<false, PASS>(op, ti, srow, sw, steps);
            }
        } else if (PASS == PASS_EMIT) {
            rsi_fast_exit(op);
#pragma unroll 8
            for (int t = tb; t < te; ++t) srow[(t - tb) ^ sw] = op.fast(in, t, steps);
        } else {
#pragma unroll 8
            for (int t = tb; t < te; ++t) op.fast(in, t, steps);
        }
        flush(seg0, off, te);
    }
    return agg_record(op, active, seeded_ever, steps, c0, c1);
}

template <class Op, int PASS, bool CUT = false>
__global__ void __launch_bounds__(kWarps * 32)
k_recur(RecurArgs a) {
    // (AGG stages the chunk's inputs in it)
    __shared__ __align__(16) float stage[kWarps][32][PASS == PASS_AGG ? 33 : CUT ? kCutW : kStageW];
    // per warp: a fast tile's broadcast inputs (EMIT), 2 x 32 floats
    __shared__ float4 xin[kWarps][PASS == PASS_EMIT ? 16 : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = blockIdx.x * kWarps + warp;
    const int li = group * 32 + lane;
    const bool valid = li < a.n_lanes;
    const int chunk = blockIdx.y;
    int c0, c1;
    recur_chunk_bounds(a, chunk, c0, c1);
    if (c0 >= a.n) return;
    if constexpr (PASS == PASS_AGG && FastKindOf<Op>::k != FK_NONE) {
        // chunks the tensor-core contraction covered: sum its partials
        const RecurTcView& v = a.tc;
        if (v.done && chunk >= v.g0 && chunk < v.g0 + v.nc && v.done[chunk] && *v.err == 0) {
            agg_from_partials<FastKindOf<Op>::k>(a, chunk, c1 - c0);
            return;
        }
        static_assert(sizeof(stage) >= 2 * kAggTile * sizeof(float), "fast AGG staging");
        float4 g;
        if (a.fast_agg && chunk >= a.fast_from &&
            agg_fast<FastKindOf<Op>::k, false>(a, li, c0, c1, &stage[0][0][0], g)) {
            if (valid) *agg_slot(a, chunk, li) = g;
            return;
        }
        __syncthreads();  // the general pass below reuses `stage`
        // a first chunk that holds every combo's seed: each thread runs its
        // combo from the chunk's inputs staged in shared memory
        constexpr int FK = FastKindOf<Op>::k;
        if constexpr (FK == FK_EMA || FK == FK_RSI || FK == FK_TEMA) {
            if (a.fast_agg && chunk == 0 && a.fast_from == 1 && c1 <= (int)(sizeof(stage) / sizeof(float)) &&
                a.first < a.n) {
                float* xs = &stage[0][0][0];
                for (int i = threadIdx.x; i < c1; i += blockDim.x) xs[i] = __ldg(a.x + i);
                __syncthreads();
                if (agg_seed_fast<FK>(a, xs, c1, (int)(sizeof(stage) / sizeof(float)))) return;
                __syncthreads();
            }
        }
    }
    // a warp with no valid lane has nothing to compute (whole warp leaves; no
    // block-wide barrier follows)
    if (group * 32 >= a.n_lanes) return;
    float4 cv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (PASS == PASS_EMIT && valid) cv = __ldg(reinterpret_cast<const float4*>(a.carry) + (size_t)chunk * a.n_lanes + li);
    const float4 g = recur_span<Op, PASS, CUT>(a, group, c0, c1, cv, &stage[warp][0][0], &xin[warp][0]);
    if (PASS == PASS_AGG && valid) *agg_slot(a, chunk, li) = g;
}

// Time-major passes: lane = series (each row of a warp is one 128-byte load or
// store).  The rows' inputs are loaded kTmRows at a time, one batch ahead of
// the steps that use them, in the warm-up as in the running phase, so a warp
// waits for memory once per batch.  Chunks are short (pick_chunk_tm) so that a
// few thousand series fill the GPU.  A call on 3,000 series x 2,520 rows:
// RSI(14) 258 -> 62 us, EMA(20) 215 -> 45, ATR(14) 366 -> 67 (chunks of 256
// rows and loads at their use before).
constexpr int kTmRows = 8;

template <bool HLC>
struct TmBatch {
    float x[kTmRows], h[HLC ? kTmRows : 1], l[HLC ? kTmRows : 1];
    // rows [tb, tb + m), clamped past the last
    __device__ __forceinline__ void load(const InTm& in, int tb, int m) {
#pragma unroll
        for (int j = 0; j < kTmRows; ++j) {
            const int t = tb + min(j, m - 1);
            if constexpr (HLC) {
                x[j] = in.C(t);
                h[j] = in.H(t);
                l[j] = in.L(t);
            } else {
                x[j] = in.X(t);
            }
        }
    }
    __device__ __forceinline__ InStep step(int tb, int j, float before) const {
        return InStep{tb + j, x[j], j > 0 ? x[j > 0 ? j - 1 : 0] : before, h[HLC ? j : 0], l[HLC ? j : 0]};
    }
};

// One warp's 32 series over the rows [c0, c1): AGG returns the lane's record,
// EMIT starts from the state `cv` where the lane is running and writes the
// outputs.
template <class Op, int PASS>
__device__ __forceinline__ float4 tm_span(const RecurArgs& a, int li, int c0, int c1, const float4 cv) {
    const bool valid = li < a.n_lanes;
    const int p = a.period, first = valid ? a.first_tm[li] : a.n;
    Op op;
    op.init(p > 0 ? p : 1, first);
    const bool active = valid && first < a.n && p > 0;
    const bool seeded_ever = active && op.s < a.n;
    const InTm in{a.x, a.h, a.l, a.c, (size_t)a.cols, (size_t)(valid ? li : 0)};
    using Batch = TmBatch<Op::kHlc>;

    // chunk entry state (as in k_recur)
    bool running = false;
    if (active) {
        if (c0 > op.s && seeded_ever) {
            if (PASS == PASS_AGG) {
                op.zero();
            } else {
                op.set(0, cv.x);
                if (Op::NS > 1) op.set(1, cv.y);
                if (Op::NS > 2) op.set(2, cv.z);
            }
            running = true;
        } else if (c0 > op.f) {
            const int end = min(c0, op.s + 1);
            float before = 0.f;
            for (int tb = op.f; tb < end; tb += kTmRows) {
                const int m = min(kTmRows, end - tb);
                Batch b;
                b.load(in, tb, m);
#pragma unroll
                for (int j = 0; j < kTmRows; ++j)
                    if (j < m) op.accum(b.step(tb, j, before), tb + j);
                before = b.x[kTmRows - 1];
            }
        }
    }
    const int run_from = (active && seeded_ever) ? max(op.s + 1, op.warm) : (valid ? INT_MAX : INT_MIN);
    const int warp_run_from = warp_max(run_from);

    int steps = 0;
    float before = 0.f;  // x (close) of the row before the batch
    if (c0 > 0) before = Op::kHlc ? in.C(c0 - 1) : in.X(c0 - 1);
    Batch cur, nxt;
    cur.load(in, c0, c1 - c0);
    float* out = a.out + (valid ? li : 0);
    for (int tb = c0; tb < c1; tb += kTmRows) {
        const int m = min(kTmRows, c1 - tb);
        if (tb + kTmRows < c1) nxt.load(in, tb + kTmRows, c1 - tb - kTmRows);
        if (tb >= warp_run_from && m == kTmRows) {
#pragma unroll
            for (int j = 0; j < kTmRows; ++j) {
                const float v = op.fast(cur.step(tb, j, before), tb + j, steps);
                if (PASS == PASS_EMIT && valid) out[(size_t)(tb + j) * a.cols] = v;
            }
            running = true;
        } else {
#pragma unroll
            for (int j = 0; j < kTmRows; ++j) {
                if (j >= m) break;
                const float v = general_step(op, active, seeded_ever, running, steps, cur.step(tb, j, before), tb + j);
                if (PASS == PASS_EMIT && valid) out[(size_t)(tb + j) * a.cols] = v;
            }
        }
        before = cur.x[kTmRows - 1];
        cur = nxt;
    }
    return agg_record(op, active, seeded_ever, steps, c0, c1);
}

template <class Op, int PASS>
__global__ void __launch_bounds__(kWarps * 32) k_recur_tm(RecurArgs a) {
    const int li = blockIdx.x * (kWarps * 32) + threadIdx.x;
    const int chunk = blockIdx.y;
    int c0, c1;
    recur_chunk_bounds(a, chunk, c0, c1);
    if (c0 >= a.n || (li & ~31) >= a.n_lanes) return;  // (whole warps)
    float4 cv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (PASS == PASS_EMIT && li < a.n_lanes)
        cv = reinterpret_cast<const float4*>(a.carry)[(size_t)chunk * a.n_lanes + li];
    const float4 g = tm_span<Op, PASS>(a, li, c0, c1, cv);
    if (PASS == PASS_AGG && li < a.n_lanes) *agg_slot(a, chunk, li) = g;
}

// Carry-in of every chunk: an exclusive scan, over the chunks of one lane, of
// the affine chunk maps S -> M_k S + b_k.  One warp per lane: each thread
// composes a contiguous run of chunks, a Kogge-Stone scan across the warp
// combines the runs, then each thread re-walks its run writing carries.  The
// maps are N x N with N the op's state size, in double-single arithmetic.
// Structure of an op's transition matrix: every product of such matrices
// keeps it, so the f64 work skips the structural zeros (GB300's FP64 rate
// makes them count).  0 = full, 1 = lower triangular (DEMA, TEMA cascades),
// 2 = diagonal (RSI's independent gain / loss averages).
template <class Op, class = void> struct ShapeOf { static constexpr int v = 0; };
template <class Op> struct ShapeOf<Op, std::void_t<decltype(Op::kShape)>> { static constexpr int v = Op::kShape; };
__host__ __device__ constexpr bool shape_nz(int sh, int r, int c) { return sh == 0 || (sh == 1 ? c <= r : c == r); }

template <int N>
struct AffD {
    D2 m[N][N];
    D2 b[N];
};
template <int N>
__device__ __forceinline__ void affd_identity(AffD<N>& a) {
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
        for (int c = 0; c < N; ++c) a.m[r][c] = {r == c ? 1.f : 0.f, 0.f};
        a.b[r] = {0.f, 0.f};
    }
}
// second o first (apply `first`, then `second`)
template <int N, int SH>
__device__ __forceinline__ AffD<N> affd_then(const AffD<N>& first, const AffD<N>& second) {
    AffD<N> o;
#pragma unroll
    for (int r = 0; r < N; ++r) {
        D2 br = second.b[r];
#pragma unroll
        for (int c = 0; c < N; ++c) {
            D2 mrc = {0.f, 0.f};
            if (shape_nz(SH, r, c)) {
#pragma unroll
                for (int q = 0; q < N; ++q)
                    if (shape_nz(SH, r, q) && shape_nz(SH, q, c)) mrc = d2_fma(second.m[r][q], first.m[q][c], mrc);
                br = d2_fma(second.m[r][c], first.b[c], br);
            }
            o.m[r][c] = mrc;
        }
        o.b[r] = br;
    }
    return o;
}
template <int N, int SH>
__device__ __forceinline__ AffD<N> affd_shfl_up(const AffD<N>& a, int d) {
    AffD<N> o;
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
        for (int c = 0; c < N; ++c) o.m[r][c] = shape_nz(SH, r, c) ? d2_shfl_up(a.m[r][c], d) : D2{0.f, 0.f};
        o.b[r] = d2_shfl_up(a.b[r], d);
    }
    return o;
}

// M^n of the op's transition (n steps), column by column from propagate.
template <class Op>
__device__ void trans_pow(long long n, int p, D2 (&m)[Op::NS][Op::NS]) {
    constexpr int N = Op::NS;
    D2 al, b;
    Op::coef(p, al, b);
    const D2 an = d2_pow(b, n), nd = d2_from_ll(n);
#pragma unroll
    for (int c = 0; c < N; ++c) {
        D2 e[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        e[c] = {1.f, 0.f};
        Op::propagate(e, nd, al, an, p);
#pragma unroll
        for (int r = 0; r < N; ++r) m[r][c] = e[r];
    }
}

// Ops whose state, once infinite, stays infinite (many-series RSI: an infinite
// move; the batch form turns it into NaN).  A product of float pairs would make
// it NaN, so the composition leaves infinite records out and holds, per
// component, whether one has passed.
template <class Op> struct InfHeld { static constexpr bool v = false; };
template <> struct InfHeld<OpRsi<false>> { static constexpr bool v = true; };
__device__ __forceinline__ unsigned take_inf(float4& g) {
    const bool x = isinf(g.x), y = isinf(g.y);
    if (x) g.x = 0.f;
    if (y) g.y = 0.f;
    return (x ? 1u : 0u) | (y ? 2u : 0u);
}
__device__ __forceinline__ void put_inf(float4& cv, unsigned held) {
    if (held & 1u) cv.x = INFINITY;
    if (held & 2u) cv.y = INFINITY;
}

// The map of one chunk from its AGG record (state, applied steps or marker).
template <class Op>
__device__ void chunk_map(const float4 g, int p, int chunk, const D2 (&ml)[Op::NS][Op::NS], AffD<Op::NS>& a) {
    constexpr int N = Op::NS;
    if (g.w == kBeforeSeed) {
        affd_identity(a);
        return;
    }
    if (g.w == kAbsolute) {
#pragma unroll
        for (int r = 0; r < N; ++r)
#pragma unroll
            for (int c = 0; c < N; ++c) a.m[r][c] = {0.f, 0.f};
    } else if (g.w == (float)chunk) {
#pragma unroll
        for (int r = 0; r < N; ++r)
#pragma unroll
            for (int c = 0; c < N; ++c) a.m[r][c] = ml[r][c];
    } else {
        trans_pow<Op>((long long)g.w, p, a.m);
    }
    const float gb[3] = {g.x, g.y, g.z};
#pragma unroll
    for (int r = 0; r < N; ++r) a.b[r] = {gb[r], 0.f};
}

// Carry-in state of every (lane, chunk): one warp per lane, each thread a
// contiguous run of chunks.  Pass 1 composes the thread's chunk maps, a warp
// scan of the compositions gives each thread its entry state, pass 2 applies
// the maps chunk by chunk and writes the carries.  Full chunks share one
// linear part M (the transition of `chunk` steps), so a run of them only
// updates the offset (b <- M b + agg) and its power M^cnt is applied once
// when another map follows or the run ends: the work per chunk is a
// matrix-vector product.
template <class Op>
__global__ void k_recur_carry(RecurArgs a, int n_chunks) {
    constexpr int N = Op::NS;
    constexpr int SH = ShapeOf<Op>::v;
    const int lane = threadIdx.x & 31;
    const int li = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;  // one warp per lane of the scan
    if (li >= a.n_lanes) return;
    const int p = a.layout ? a.period : a.periods[li];
    const float4* agg = reinterpret_cast<const float4*>(a.agg);
    float4* carry = reinterpret_cast<float4*>(a.carry);
    const int per = (n_chunks + 31) / 32;
    const int k0 = min(lane * per, n_chunks), k1 = min(k0 + per, n_chunks);
    const float full = (float)a.chunk;
    D2 ml[N][N], mper[N][N];  // transitions of one and of `per` full chunks
    trans_pow<Op>((long long)a.chunk, p, ml);
    trans_pow<Op>((long long)per * a.chunk, p, mper);
    // v <- M v + g (the map of a full chunk applied to a vector)
    auto full_step = [&](D2 (&v)[N], const float4 g) {
        const float gb[3] = {g.x, g.y, g.z};
        D2 t[N];
#pragma unroll
        for (int r = 0; r < N; ++r) {
            D2 x = {gb[r], 0.f};
#pragma unroll
            for (int c = 0; c < N; ++c)
                if (shape_nz(SH, r, c)) x = d2_fma(ml[r][c], v[c], x);
            t[r] = x;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) v[r] = t[r];
    };
    AffD<N> run;
    affd_identity(run);
    int cnt = 0;          // full chunks whose linear part is not yet in run.m
    bool m_zero = false;  // run.m == 0 (after an absolute chunk): powers leave it 0
    auto flush = [&]() {
        if (cnt == 0 || m_zero) {
            cnt = 0;
            return;
        }
        D2 pw[N][N];
        if (cnt == per) {
#pragma unroll
            for (int r = 0; r < N; ++r)
#pragma unroll
                for (int c = 0; c < N; ++c) pw[r][c] = mper[r][c];
        } else {
            trans_pow<Op>((long long)cnt * a.chunk, p, pw);
        }
        D2 m2[N][N];  // run.m <- M^cnt run.m (the offset is already current)
#pragma unroll
        for (int r = 0; r < N; ++r)
#pragma unroll
            for (int c = 0; c < N; ++c) {
                D2 v = {0.f, 0.f};
                if (shape_nz(SH, r, c))
#pragma unroll
                    for (int q = 0; q < N; ++q)
                        if (shape_nz(SH, r, q) && shape_nz(SH, q, c)) v = d2_fma(pw[r][q], run.m[q][c], v);
                m2[r][c] = v;
            }
#pragma unroll
        for (int r = 0; r < N; ++r)
#pragma unroll
            for (int c = 0; c < N; ++c) run.m[r][c] = m2[r][c];
        cnt = 0;
    };
    // the chunk records in a 4-deep register queue: loads run ahead of the
    // dependent math without an unrolled batch (the scan's double-single code
    // is large, and unrolled copies of it overflowed the instruction cache)
    const float4 kNone = make_float4(0.f, 0.f, 0.f, 0.f);
    auto rec = [&](int k) { return k < k1 ? __ldg(agg + (size_t)k * a.n_lanes + li) : kNone; };
    float4 q0 = rec(k0), q1 = rec(k0 + 1), q2 = rec(k0 + 2), q3 = rec(k0 + 3);
    unsigned held = 0;
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        float4 g = q0;
        q0 = q1;
        q1 = q2;
        q2 = q3;
        q3 = rec(k + 4);
        if (InfHeld<Op>::v) held |= take_inf(g);
        if (g.w == full) {
            full_step(run.b, g);
            ++cnt;
        } else {
            flush();
            AffD<N> ak;
            chunk_map<Op>(g, p, a.chunk, ml, ak);
            run = affd_then<N, SH>(run, ak);
            if (g.w == kAbsolute) m_zero = true;
        }
    }
    flush();
    if (InfHeld<Op>::v) {  // what the threads before this one hold
        const unsigned below = (1u << lane) - 1u;
        const bool x = __ballot_sync(0xffffffffu, held & 1u) & below, y = __ballot_sync(0xffffffffu, held & 2u) & below;
        held = (x ? 1u : 0u) | (y ? 2u : 0u);
    }
#pragma unroll 1
    for (int d = 1; d < 32; d <<= 1) {
        const AffD<N> up = affd_shfl_up<N, SH>(run, d);
        if (lane >= d) run = affd_then<N, SH>(up, run);
    }
    AffD<N> ex = affd_shfl_up<N, SH>(run, 1);
    if (lane == 0) affd_identity(ex);
    D2 S[N];  // state at the start of chunk k0
#pragma unroll
    for (int r = 0; r < N; ++r) S[r] = ex.b[r];
    q0 = rec(k0);
    q1 = rec(k0 + 1);
    q2 = rec(k0 + 2);
    q3 = rec(k0 + 3);
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        float4 g = q0;
        q0 = q1;
        q1 = q2;
        q2 = q3;
        q3 = rec(k + 4);
        {
            float4 cv = make_float4(0.f, 0.f, 0.f, 0.f);
            cv.x = S[0].hi + S[0].lo;
            if (N > 1) cv.y = S[N > 1 ? 1 : 0].hi + S[N > 1 ? 1 : 0].lo;
            if (N > 2) cv.z = S[N > 2 ? 2 : 0].hi + S[N > 2 ? 2 : 0].lo;
            if (InfHeld<Op>::v) {
                put_inf(cv, held);
                held |= take_inf(g);
            }
            carry[(size_t)k * a.n_lanes + li] = cv;
            if (g.w == full) {
                full_step(S, g);
            } else {
                AffD<N> ak;
                chunk_map<Op>(g, p, a.chunk, ml, ak);
                D2 t[N];
#pragma unroll
                for (int r = 0; r < N; ++r) {
                    D2 v = ak.b[r];
#pragma unroll
                    for (int c = 0; c < N; ++c)
                        if (shape_nz(SH, r, c)) v = d2_fma(ak.m[r][c], S[c], v);
                    t[r] = v;
                }
#pragma unroll
                for (int r = 0; r < N; ++r) S[r] = t[r];
            }
        }
    }
}

// Short sweeps in one launch: a block owns 32 combos and cuts the series into
// one chunk per warp.  Every warp aggregates its chunk into shared memory,
// composes the records of the chunks before it (its own carry-in) and emits,
// so nothing waits for a second and third launch.  Up to kOneMax bars, where a
// warp's chunk is still 128 steps; TEMA up to period kOneMaxTemaP (a chunk
// inside its staged start runs from the first bar).  us of a call, three
// launches / one: EMA of 10 periods on 1,001 bars 22.6 / 12.3, RSI 30.8 / 18.5; 200
// periods on 2,001 bars: DEMA 24.7 / 18.5, RSI 41 / 33, on 4,001: 24.7 / 28.8
// and 41 / 51; TEMA of 200 periods on 1,001 bars 39 / 62.
constexpr int kOneWarps = 16;
constexpr int kOneMax = 2048, kOneMaxTemaP = 64;
constexpr size_t kOneSmem = (size_t)kOneWarps * (32 * kStageW * sizeof(float) + 16 * sizeof(float4) + 32 * sizeof(float4));

// The state entering chunk q of a lane, from the block's records (rec[32 k +
// lane]: chunk k's) and the transition ml of a full chunk.
template <class Op>
__device__ __forceinline__ float4 entry_state(const float4* rec, int q, int lane, int p, int chunk,
                                              const D2 (&ml)[Op::NS][Op::NS]) {
    constexpr int N = Op::NS;
    constexpr int SH = ShapeOf<Op>::v;
    D2 S[N];
#pragma unroll
    for (int r = 0; r < N; ++r) S[r] = {0.f, 0.f};
    unsigned held = 0;
#pragma unroll 1
    for (int k = 0; k < q; ++k) {
        float4 e = rec[k * 32 + lane];
        if (e.w == kBeforeSeed) continue;
        if (InfHeld<Op>::v) held |= take_inf(e);
        AffD<N> m;
        chunk_map<Op>(e, p, chunk, ml, m);
        D2 t[N];
#pragma unroll
        for (int r = 0; r < N; ++r) {
            D2 v = m.b[r];
#pragma unroll
            for (int c = 0; c < N; ++c)
                if (shape_nz(SH, r, c)) v = d2_fma(m.m[r][c], S[c], v);
            t[r] = v;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) S[r] = t[r];
    }
    float4 cv = make_float4(0.f, 0.f, 0.f, 0.f);
    cv.x = S[0].hi + S[0].lo;
    if (N > 1) cv.y = S[N > 1 ? 1 : 0].hi + S[N > 1 ? 1 : 0].lo;
    if (N > 2) cv.z = S[N > 2 ? 2 : 0].hi + S[N > 2 ? 2 : 0].lo;
    if (InfHeld<Op>::v) put_inf(cv, held);
    return cv;
}

template <class Op>
__global__ void __launch_bounds__(32 * kOneWarps) k_recur_one(RecurArgs a) {
    extern __shared__ __align__(16) float one_smem[];
    float* stage = one_smem;                                                     // [kOneWarps][32][kStageW]
    float4* xin = reinterpret_cast<float4*>(stage + kOneWarps * 32 * kStageW);  // [kOneWarps][16]
    float4* rec = xin + kOneWarps * 16;                                         // [kOneWarps][32]
    const int group = blockIdx.x, lane = threadIdx.x & 31, q = threadIdx.x >> 5;  // q: this warp's chunk
    const int li = group * 32 + lane;
    const bool valid = li < a.n_lanes;
    const int c0 = min(q * a.chunk, a.n), c1 = min(c0 + a.chunk, a.n);
    float* st = stage + q * 32 * kStageW;
    float4* xi = xin + q * 16;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 g = make_float4(0.f, 0.f, 0.f, kBeforeSeed);
    const int p = valid ? a.periods[li] : 1;
    if (c1 < a.n) {  // (nobody reads the last record)
        bool done = false;
        if constexpr (FastKindOf<Op>::k != FK_NONE) {  // every combo is running (agg_fast, above)
            static_assert(32 * kStageW >= 2 * kAggTile, "fast AGG staging");
            Op op;
            op.init(p, a.first);
            if (__all_sync(0xffffffffu, c0 > op.s))
                done = agg_fast<FastKindOf<Op>::k, true>(a, li, c0, c1, st, g);
        }
        if (!done) g = recur_span<Op, PASS_AGG, false>(a, group, c0, c1, zero, st, xi);
    }
    rec[threadIdx.x] = g;
    // the transition of a full chunk, while other warps still aggregate
    D2 ml[Op::NS][Op::NS];
    trans_pow<Op>((long long)a.chunk, p, ml);
    __syncthreads();
    if (c0 >= a.n) return;
    const float4 cv = entry_state<Op>(rec, q, lane, p, a.chunk, ml);
    recur_span<Op, PASS_EMIT, false>(a, group, c0, c1, cv, st, xi);
}

// The same for many series: a block takes 32 series, a warp of it a chunk of
// their rows.  For short histories, whose call is three launches' latency; longer
// ones need more warps than 32 per 32 series (the caller's rule has the times).
constexpr int kTmOneWarps = 32;

template <class Op>
__global__ void __launch_bounds__(32 * kTmOneWarps) k_recur_tm_one(RecurArgs a) {
    __shared__ float4 rec[kTmOneWarps * 32];
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;  // q: this warp's chunk
    const int li = blockIdx.x * 32 + lane;
    const int c0 = min(q * a.chunk, a.n), c1 = min(c0 + a.chunk, a.n);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 g = make_float4(0.f, 0.f, 0.f, kBeforeSeed);
    if (c1 < a.n) g = tm_span<Op, PASS_AGG>(a, li, c0, c1, zero);  // (nobody reads the last record)
    rec[threadIdx.x] = g;
    D2 ml[Op::NS][Op::NS];
    trans_pow<Op>((long long)a.chunk, a.period, ml);
    __syncthreads();
    if (c0 >= a.n) return;
    tm_span<Op, PASS_EMIT>(a, li, c0, c1, entry_state<Op>(rec, q, lane, a.period, a.chunk, ml));
}

template <class Op>
vta_status run_tm_one(RecurArgs a, cudaStream_t st) {
    a.chunk = a.chunk0 = (a.n + kTmOneWarps * kTmRows - 1) / (kTmOneWarps * kTmRows) * kTmRows;
    ktimer_begin(st);
    k_recur_tm_one<Op><<<ceil_div(a.n_lanes, 32), 32 * kTmOneWarps, 0, st>>>(a);
    ktimer_end(st);
    return check_launch("k_recur_tm_one");
}

template <class Op>
vta_status run_one(RecurArgs a, cudaStream_t st) {
    a.chunk = a.chunk0 = (a.n + 64 * kOneWarps - 1) / (64 * kOneWarps) * 64;
    VTA_CUDA_TRY(cudaFuncSetAttribute(k_recur_one<Op>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOneSmem));
    ktimer_begin(st);
    k_recur_one<Op><<<ceil_div(a.n_lanes, 32), 32 * kOneWarps, kOneSmem, st>>>(a);
    ktimer_end(st);
    return check_launch("k_recur_one");
}

// AGG and CARRY (more than one chunk), then EMIT
template <class Op, bool TM>
vta_status run(const RecurArgs& a, cudaStream_t st) {
    if (a.one_launch) {
        if constexpr (TM)
            return run_tm_one<Op>(a, st);
        else
            return run_one<Op>(a, st);
    }
    const int n_chunks = recur_n_chunks(a.n, a.chunk, a.chunk0);
    const int groups = (int)ceil_div(a.n_lanes, 32);
    dim3 grid(ceil_div(groups, kWarps), n_chunks);
    if (n_chunks > 65535) return fail(VTA_ERR_LAUNCH_CONFIG_TOO_LARGE, "recurrence: too many time chunks");
    void (*agg)(RecurArgs);
    void (*emit)(RecurArgs);
    if constexpr (TM) {
        agg = k_recur_tm<Op, PASS_AGG>;
        emit = k_recur_tm<Op, PASS_EMIT>;
    } else {
        agg = k_recur<Op, PASS_AGG>;
        // Cut stores where the rows do not all start at a 16-byte boundary and
        // the outputs are beyond what the L2 merges before it writes them back.
        // us of a call, as they fall / cut: 399 EMAs on 500,001 bars 367 / 231
        // (185 on 500,000), RSIs 383 / 249 (210), 199 DEMAs on 200,001 102 / 82
        // (70), ATRs on 500,001 249 / 200; 80 MB of RSIs 58.1 / 56.3; 8 MB of
        // EMAs 24.6 / 26.6.  Rows at 16-byte boundaries (n % 8 == 4): EMA 241 /
        // 221, DEMA 80 / 81, ATR 194 / 199.
        const bool cut = (a.n % 4 != 0 || reinterpret_cast<uintptr_t>(a.out) % 16 != 0) &&
                         (size_t)a.n_lanes * a.n * sizeof(float) >= kCutBytes;
        emit = cut ? k_recur<Op, PASS_EMIT, true> : k_recur<Op, PASS_EMIT>;
    }
    if (n_chunks > 1) {
        agg<<<grid, kWarps * 32, 0, st>>>(a);
        VTA_TRY(check_launch("k_recur_agg"));
        k_recur_carry<Op><<<ceil_div((size_t)a.n_lanes * 32, 128), 128, 0, st>>>(a, n_chunks);
        VTA_TRY(check_launch("k_recur_carry"));
    }
    ktimer_begin(st);
    emit<<<grid, kWarps * 32, 0, st>>>(a);
    ktimer_end(st);
    return check_launch("k_recur_emit");
}

}  // namespace

bool recur_one_ok(int kind, int n, int pmax, size_t smem_optin) {
    return n <= kOneMax && smem_optin >= kOneSmem && (kind != RK_TEMA || pmax <= kOneMaxTemaP);
}

int recur_state_dim(int kind) {
    switch (kind) {
        case RK_DEMA: return 2;
        case RK_TEMA: return 3;
        case RK_RSI: return 2;
        default: return 1;
    }
}

vta_status launch_recurrence(const RecurArgs& a, cudaStream_t st) {
    const bool tm = a.layout != 0;
    switch (a.kind) {
        case RK_EMA: return tm ? run<OpEma, true>(a, st) : run<OpEma, false>(a, st);
        case RK_DEMA: return tm ? run<OpDema, true>(a, st) : run<OpDema, false>(a, st);
        case RK_TEMA: return tm ? run<OpTema, true>(a, st) : run<OpTema, false>(a, st);
        case RK_RSI: return tm ? run<OpRsi<false>, true>(a, st) : run<OpRsi<true>, false>(a, st);
        case RK_WILDERS: return tm ? run<OpWilders, true>(a, st) : run<OpWilders, false>(a, st);
        case RK_ATR: return tm ? run<OpAtr, true>(a, st) : run<OpAtr, false>(a, st);
        default: return fail(VTA_ERR_INVALID_INPUT, "unknown recurrence kind");
    }
}

}  // namespace vta
