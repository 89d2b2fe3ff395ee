// wide_rows_kernel: rows whose softmax runs over the whole vocabulary (top-k off).
//
// One row at a time per persistent CTA. Warp w owns one contiguous span of the row (1/W_NW of it, rounded up to whole steps);
// in a step every lane handles eight logits (two 16-byte vectors of f32, one of bf16). Nothing is shared between threads inside
// a pass, so a pass contains no barrier.
//
// This header has no include guard: it is included once per instance, with GS_W_NS naming the
// instance's namespace inside gs and GS_W_NT its threads per CTA.
//   256:  four CTAs per SM. With four rows per SM the load latency and the serial tail of one
//         row hide behind the arithmetic of the others: the instance for batches that fill the GPU.
//   1024: one CTA per SM. A row finishes about a quarter sooner: the instance for batches of at
//         most one row per SM.
//
// Usually a row takes one pass (sample_wide_onepass.cuh). What that does not serve takes two, in this file (vectors loaded
// straight into registers one or two steps ahead, with L2 cache hints):
//   sample                     the first step of every warp: an upper estimate (anchor) of the
//                              row's maximum and its range
//   pass 1 (HBM)               max, min, NaN; with an active top-p cut also the count histogram
//                              over 4096 linear buckets of s - anchor, whose width is the power
//                              of two that covers the estimated range
//   bracket                    count-based lower/upper mass bounds bracket the cut to a zone of
//                              buckets (a maximum above the anchor: pass 2 recounts exactly)
//   pass 3 (L2)                exponentials. Mass of d >= dA (certainly kept) per piece of
//                              eight steps, zone logits (dB <= d < dA) into an exact list
//   tail                       weighted selection inside the zone, prefix over the pieces
// and either way the piece that holds the drawn token is looked at again with the exact rule (wide_draw).
//
// Row semantics: model/generate.go:147-240 (mode A), model/qwen/generate.go:92-153 (mode B).
#include "sample_batch.cuh"   // includes row_stream.cuh

#ifndef GS_W_NS
#define GS_W_NS w256
#define GS_W_NT 256
#endif

namespace gs {
namespace GS_W_NS {

constexpr int W_NT = GS_W_NT;           // threads per CTA
constexpr int W_CTAS = 1024 / W_NT;     // CTAs per SM
constexpr int W_NSUB = W_NT;            // sub-buckets of one weighted-selection round
constexpr int W_NW = W_NT / 32;
constexpr int W_NB = 4096;              // histogram buckets
constexpr int W_ZCAP = 2048;            // exact zone list capacity
constexpr int W_D1 = 2;                 // steps of register prefetch in pass 1
constexpr int W_G = 8;                  // steps per piece (power of two)
constexpr int W_MAX_STEPS = (W_NT >= 512) ? 64 : 128;         // steps per warp and pass; longer rows go to the single-CTA kernel
constexpr int W_MAX_PPW = W_MAX_STEPS / W_G;
constexpr int W_MAX_PIECES = W_NW * W_MAX_PPW;                 // 128 (1024 threads: 256)
constexpr int W_EB_REP = 16;            // copies of a table entry in the conflict-free layout
constexpr int W_EB_REP_ENTRIES = 128;   // entries of that layout: d > -(128-1)/32
constexpr int W_OFF_HIST = 0;
constexpr int W_OFF_ZONE = W_OFF_HIST + W_NB * 4;
constexpr int W_OFF_EB = W_OFF_ZONE + W_ZCAP * 8;              // 1024 entries, or 128 entries x 16 copies
// one pass: the lanes' buffers (of the last four slots only what fills one takes any), the warps' lists and where the pieces
// begin in them, the ring of copies, the selection's buckets
constexpr int W1_SLOTS = 16;
constexpr int W1_WCAP = (W_NT >= 512) ? 256 : 512;
constexpr int W1_RING_BYTES = 2 * W_NT * 32;
constexpr int W1_BINS = W_NT;
constexpr int W1_OFF_LIST = 0;
constexpr int W1_OFF_BUF = W1_OFF_LIST + W_NW * W1_WCAP * 4;
constexpr int W1_OFF_RING = W1_OFF_BUF + W1_SLOTS * W_NT * 4;
constexpr int W1_OFF_TAB = W1_OFF_LIST;                        // without a cut there are no lists: the exponential's table
constexpr int W1_OFF_MASS = W1_OFF_BUF;                        // after the pass: the listed logits' masses
constexpr int W1_OFF_BINS = W1_OFF_RING + W1_RING_BYTES;
constexpr int W1_OFF_FROM = W1_OFF_BINS + W1_BINS * 4;
constexpr int W1_END = W1_OFF_FROM + W_NW * (W_MAX_PPW + 1) * 4;
constexpr int W2_END = W_OFF_EB + W_EB_REP * W_EB_REP_ENTRIES * 8;
constexpr int W_OFF_PART = W1_END > W2_END ? W1_END : W2_END;
constexpr int W_DYN_BYTES = W_OFF_PART + W_MAX_PIECES * 8;     // 51 KB (1024 threads: 167 KB)
static_assert(W_EB_REP * W_EB_REP_ENTRIES >= NB1, "either layout fits");
static_assert(W_NT >= 256 && W_NT <= 1024 && W_MAX_PIECES <= W_NT && W_G * 64 <= 2 * W_NT && W_NSUB * 12 <= W_NB * 4,
              "one piece / two vectors of a piece / one sub-bucket per thread");

// Histogram buckets of width 1/scale (scale a power of two): bucket = round(-d * scale),
// clamped to W_NB - 1. Multiplying by a power of two is exact, so the bucket edges are exact.
__device__ __forceinline__ int bucket_w(float d, float scale, float dclamp) {
  const float f = fmaf(fmaxf(d, dclamp), -scale, 8388608.0f);
  return __float_as_int(f) & 0x1fff;
}
// smallest d whose bucket is <= bmax (the edge is a tie that rounds to even)
__device__ __forceinline__ float bucket_floor_w(int bmax, float scale, float dclamp) {
  if (bmax >= W_NB - 1) return -INFINITY;
  if (bmax < 0) return INFINITY;
  const float t = -(static_cast<float>(2 * bmax + 1) * (0.5f / scale));
  return (bucket_w(t, scale, dclamp) <= bmax) ? t : __uint_as_float(__float_as_uint(t) - 1u);
}

__device__ __forceinline__ double lds_f64(uint32_t addr) {
  double v;
  asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
  return v;
}
// exp(d) for -31.9 < d <= 0 from the table E[b] = exp(-b/32) in shared memory: d = -b/32 + dl with
// |dl| <= 1/64 exactly (f32), exp = E[b] * (1 + w), w = dl + dl^2/2 + ... + dl^5/120 in f32. The one
// rounding of w (at most 2^-31 relative to the result, unbiased) is the error that matters.
// The bits of f are 0x4B000000 + b, so bits * eb_mul + eb_bias is the address of E[b] (mod 2^32)
// with eb_mul = 8 and eb_bias = table - 0x4B000000 * 8 for the plain table. In the conflict-free
// layout (rows whose d stay above -(W_EB_REP_ENTRIES-1)/32) entry b has sixteen copies 8 bytes
// apart and lane l reads copy l mod 16, its own pair of banks: eb_mul = 128, eb_bias = table +
// 8 (l mod 16) - 0x4B000000 * 128.
__device__ __forceinline__ double exp_fast_s(float d, uint32_t eb_mul, uint32_t eb_bias) {
  const float f = fmaf(d, -32.0f, 8388608.0f);
  const float dl = fmaf(f - 8388608.0f, 0.03125f, d);
  float t = fmaf(dl, 8.3333338e-3f, 4.1666668e-2f);
  t = fmaf(t, dl, 1.6666667e-1f);
  t = fmaf(t, dl, 0.5f);
  const float w = fmaf(t, dl * dl, dl);
  const double E = lds_f64(__float_as_uint(f) * eb_mul + eb_bias);
  return fma(E, static_cast<double>(w), E);
}
// Two-wide f32 arithmetic (one issue slot for two results on sm_100).
typedef unsigned long long f32x2_t;
__device__ __forceinline__ f32x2_t pk2(float a, float b) { f32x2_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void upk2(f32x2_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2_t fma2(f32x2_t a, f32x2_t b, f32x2_t c) { f32x2_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2_t add2(f32x2_t a, f32x2_t b) { f32x2_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2_t mul2(f32x2_t a, f32x2_t b) { f32x2_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
// exp_fast_s for two arguments at once (D = the pair of d values)
__device__ __forceinline__ void exp_fast_s2(f32x2_t D, uint32_t eb_mul, uint32_t eb_bias, double& e0, double& e1) {
  const f32x2_t F = fma2(D, pk2(-32.0f, -32.0f), pk2(8388608.0f, 8388608.0f));
  const f32x2_t DL = fma2(add2(F, pk2(-8388608.0f, -8388608.0f)), pk2(0.03125f, 0.03125f), D);
  f32x2_t T = fma2(DL, pk2(8.3333338e-3f, 8.3333338e-3f), pk2(4.1666668e-2f, 4.1666668e-2f));
  T = fma2(T, DL, pk2(1.6666667e-1f, 1.6666667e-1f));
  T = fma2(T, DL, pk2(0.5f, 0.5f));
  const f32x2_t W = fma2(T, mul2(DL, DL), DL);
  float f0, f1, w0, w1;
  upk2(F, f0, f1); upk2(W, w0, w1);
  const double E0 = lds_f64(__float_as_uint(f0) * eb_mul + eb_bias);
  const double E1 = lds_f64(__float_as_uint(f1) * eb_mul + eb_bias);
  e0 = fma(E0, static_cast<double>(w0), E0);
  e1 = fma(E1, static_cast<double>(w1), E1);
}
constexpr double W_EXP_REL_ERR = 6e-10;   // bound of exp_fast_s against the exact exponential

// Steps [st0, st1) of one pass; qa/qb hold the vectors of steps st0 .. st0+D-1 on entry and of
// st1 .. st1+D-1 on exit (D steps of register prefetch). CLEAN runs hold no logit outside the
// row and skip all masking; the others (a warp's step that holds the row's first or last vector,
// or vectors past the end) give every logit outside the row the value -Inf and a clear bit in
// `valid`. body(x, valid, st, gv): eight logits of this lane, validity bits, step, the lane's
// first vector.
template <typename T, int D, bool CLEAN, typename F>
__device__ __forceinline__ void wide_steps(const WSpan& sp, const RowView<T>& rv, unsigned long long pol, int lane,
                                           int st0, int st1, uint4 (&qa)[D], uint4 (&qb)[D], F&& body) {
  constexpr int VEC = Elem<T>::VEC, EPI = 8 / VEC, SV = 32 * EPI;
#pragma unroll 1
  for (int st = st0; st < st1; st++) {
    uint4 na, nb;
    w_load<T>(sp, st + D, pol, na, nb);
    float x[8];
    if (EPI == 2) { Elem<T>::unpack(qa[0], x); Elem<T>::unpack(qb[0], x + 4 * (EPI - 1)); }
    else Elem<T>::unpack(qa[0], x);
#pragma unroll
    for (int k = 0; k + 1 < D; k++) { qa[k] = qa[k + 1]; qb[k] = qb[k + 1]; }
    qa[D - 1] = na; qb[D - 1] = nb;
    const int gv = sp.first + st * SV + lane;
    uint32_t valid = 0xffu;
    if (!CLEAN) {
      valid = 0u;
#pragma unroll
      for (int h = 0; h < EPI; h++) {
        const int g = gv + 32 * h;
        const int i0 = g * VEC - rv.shift;
#pragma unroll
        for (int c = 0; c < VEC; c++) {
          const int i = i0 + c;
          if (g < rv.nvec && i >= 0 && i < rv.V) valid |= 1u << (h * VEC + c);
          else x[h * VEC + c] = -INFINITY;
        }
      }
    }
    body(x, valid, st, gv);
  }
}
// One pass over the warp's span with D steps of prefetch: runs of clean and other steps, in order.
#define GS_WIDE_STREAM(T, D, sp, rv, pol, lane, BODY)                                           \
  do {                                                                                          \
    uint4 qa_[D], qb_[D];                                                                       \
    _Pragma("unroll") for (int s_ = 0; s_ < D; s_++) w_load<T>(sp, s_, pol, qa_[s_], qb_[s_]);  \
    if (sp.clean_lo > 0) wide_steps<T, D, false>(sp, rv, pol, lane, 0, sp.clean_lo, qa_, qb_, BODY(false)); \
    wide_steps<T, D, true>(sp, rv, pol, lane, sp.clean_lo, sp.clean_hi, qa_, qb_, BODY(true));  \
    if (sp.clean_hi < sp.nst) wide_steps<T, D, false>(sp, rv, pol, lane, sp.clean_hi, sp.nst, qa_, qb_, BODY(false)); \
  } while (0)

__device__ __forceinline__ unsigned long long policy_keep() { unsigned long long p; asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p)); return p; }
__device__ __forceinline__ unsigned long long policy_drop() { unsigned long long p; asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p)); return p; }

// pass 1: max, min, NaN flag over the row's logits. With HIST it also counts the logits into the
// histogram of q = s - anchor (an upper estimate of the row's maximum taken from a sample), so that
// rows whose maximum stays below the anchor need no second pass for their histogram.
template <typename T, bool HIST, bool TONE>
__device__ __noinline__ void wide_pass1(const WSpan& sp_in, const RowView<T>& rv_in, int lane,
                                        uint32_t hist_bias, float anchor, float Tm, float scale, float dclamp,
                                        float& xmax, float& xmin, bool& nan_seen) {
  const WSpan sp = sp_in;                // registers, not memory, inside the loop
  const RowView<T> rv = rv_in;
  float vmax = -INFINITY, vmin = INFINITY;   // vmax with NaN-propagating maxima: NaN iff the span held one
#define GS_BODY1(CL) [&](const float* x, uint32_t valid, int, int) {                             \
    if (CL) {                                                                                    \
      vmax = max3nan(vmax, x[0], x[1]); vmax = max3nan(vmax, x[2], x[3]);                        \
      vmax = max3nan(vmax, x[4], x[5]); vmax = max3nan(vmax, x[6], x[7]);                        \
      vmin = min3f(vmin, x[0], x[1]); vmin = min3f(vmin, x[2], x[3]);                            \
      vmin = min3f(vmin, x[4], x[5]); vmin = min3f(vmin, x[6], x[7]);                            \
    }                                                                                            \
    _Pragma("unroll") for (int c = 0; c < 8; c++) {                                              \
      if (!CL) {                                                                                 \
        vmax = maxnan(vmax, x[c]);                           /* masked logits read as -Inf */    \
        vmin = fminf(vmin, ((valid >> c) & 1u) ? x[c] : INFINITY);                               \
      }                                                                                          \
      if (HIST) {                                                                                \
        const float s = TONE ? x[c] : __fdiv_rn(x[c], Tm);                                       \
        /* NaN and anything above the anchor land in bucket 0 or W_NB-1: such rows are redone */ \
        const float f = fmaf(fminf(fmaxf(s - anchor, dclamp), 0.0f), -scale, 8388608.0f);        \
        const uint32_t a = __float_as_uint(f) * 4u + hist_bias;                                  \
        if (CL || ((valid >> c) & 1u)) asm volatile("red.shared.add.u32 [%0], 1;" :: "r"(a) : "memory"); \
      }                                                                                          \
    } }
  const unsigned long long pol = policy_keep();
  GS_WIDE_STREAM(T, W_D1, sp, rv, pol, lane, GS_BODY1);
#undef GS_BODY1
  xmax = vmax; xmin = vmin; nan_seen = (vmax != vmax);
}

// pass 2: count histogram of d (logits outside the row are not counted).
// hist_bias = shared address of the histogram - 0x4B000000 * 4 (mod 2^32): see exp_fast_s.
template <typename T, bool TONE>
__device__ __noinline__ void wide_pass2(const WSpan& sp_in, const RowView<T>& rv_in, int lane,
                                        uint32_t hist_bias, float m, float Tm, float scale, float dclamp) {
  const WSpan sp = sp_in;
  const RowView<T> rv = rv_in;
#define GS_BODY2(CL) [&](const float* x, uint32_t valid, int, int) {                             \
    _Pragma("unroll") for (int c = 0; c < 8; c++) {                                              \
      const float s = TONE ? x[c] : __fdiv_rn(x[c], Tm);                                         \
      const float f = fmaf(fmaxf(s - m, dclamp), -scale, 8388608.0f);                            \
      const uint32_t a = __float_as_uint(f) * 4u + hist_bias;                                    \
      if (CL || ((valid >> c) & 1u)) asm volatile("red.shared.add.u32 [%0], 1;" :: "r"(a) : "memory"); \
    } }
  const unsigned long long pol = policy_keep();
  GS_WIDE_STREAM(T, 1, sp, rv, pol, lane, GS_BODY2);
#undef GS_BODY2
}

// pass 3: exponentials. part[warp * ppw + piece] receives the certainly-kept mass (d >= dA) of
// each piece of W_G steps; zone logits (dB <= d < dA) go to the list zl. The lane-private sum of
// all mass comes back in Ssum, the kept mass of the warp's pieces in lane 0's Ksum.
// FAST: every logit of the row has d > -31.9 (bucket-table exponential, no range check);
// TONE: temperature 1; CUT: a top-p cut is active.
template <typename T, bool FAST, bool TONE, bool CUT>
__device__ __noinline__ void wide_pass3(const WSpan& sp_in, const RowView<T>& rv_in, int lane, int warp,
                                        float m, float Tm, float dA, float dB, uint32_t eb_mul, uint32_t eb_bias, const double* s_tab,
                                        double* part, int ppw, uint2* zl, int* zcnt, double& Ssum, double& Ksum) {
  constexpr int VEC = Elem<T>::VEC;
  const WSpan sp = sp_in;
  const RowView<T> rv = rv_in;
  // |d - dmid| <= dhalf is a superset of the zone dB <= d < dA (infinite ends are clamped)
  const float dAc = fminf(dA, 3.0e38f), dBc = fmaxf(dB, -3.0e38f);
  const float dmid = 0.5f * dAc + 0.5f * dBc;
  const float dhalf = (0.5f * dAc - 0.5f * dBc) * 1.000001f + 1e-30f;
  const bool none_kept = CUT && (dA == INFINITY);
  const float dfloor = (eb_mul == 8u) ? -31.9f : -(W_EB_REP_ENTRIES - 1.5f) / 32.0f;   // keeps masked logits inside the table
  double t0 = 0.0, t1 = 0.0, sub = 0.0;
  double stot = 0.0, ksum = 0.0;
#define GS_BODY3(CL) [&](const float* x, uint32_t valid, int st, int gv) {                       \
    float nearest = INFINITY;                                                                    \
    _Pragma("unroll") for (int c = 0; c < 8; c += 2) {                                           \
      const float s0 = TONE ? x[c] : __fdiv_rn(x[c], Tm);                                        \
      const float s1 = TONE ? x[c + 1] : __fdiv_rn(x[c + 1], Tm);                                \
      const float d0 = s0 - m, d1 = s1 - m;                                                      \
      double e0, e1;                                                                             \
      if (FAST) {                                                                                \
        if (CL) exp_fast_s2(pk2(d0, d1), eb_mul, eb_bias, e0, e1);                               \
        else exp_fast_s2(pk2(fmaxf(d0, dfloor), fmaxf(d1, dfloor)), eb_mul, eb_bias, e0, e1);    \
        if (!CL) {                                                                               \
          const bool v0 = (valid >> c) & 1u, v1 = (valid >> (c + 1)) & 1u;                       \
          e0 = __hiloint2double(v0 ? __double2hiint(e0) : 0, v0 ? __double2loint(e0) : 0);       \
          e1 = __hiloint2double(v1 ? __double2hiint(e1) : 0, v1 ? __double2loint(e1) : 0);       \
        }                                                                                        \
      } else {                                                                                   \
        e0 = exp_safe(d0, s_tab);                            /* exp_safe(-Inf) is exactly 0 */   \
        e1 = exp_safe(d1, s_tab);                                                                \
      }                                                                                          \
      t0 += e0; t1 += e1;                                                                        \
      if (CUT) {                                                                                 \
        sub = fma(e0, __hiloint2double((d0 < dA) ? 0x3ff00000 : 0, 0), sub);                     \
        sub = fma(e1, __hiloint2double((d1 < dA) ? 0x3ff00000 : 0, 0), sub);                     \
        nearest = fminf(nearest, fminf(fabsf(d0 - dmid), fabsf(d1 - dmid)));                     \
      }                                                                                          \
    }                                                                                            \
    if (CUT && nearest <= dhalf) {                           /* rare: a logit of this lane near the zone */ \
      _Pragma("unroll") for (int c = 0; c < 8; c++) {                                            \
        const float s = TONE ? x[c] : __fdiv_rn(x[c], Tm);                                       \
        const float d = s - m;                                                                   \
        if ((CL || ((valid >> c) & 1u)) && d < dA && d >= dB) {                                  \
          const int i = (gv + 32 * (c / VEC)) * VEC - rv.shift + (c % VEC);                      \
          const int slot = atomicAdd(zcnt, 1);                                                   \
          if (slot < W_ZCAP) zl[slot] = make_uint2(__float_as_uint(d), static_cast<uint32_t>(i)); \
        }                                                                                        \
      }                                                                                          \
    }                                                                                            \
    if ((st & (W_G - 1)) == W_G - 1 || st == sp.nst - 1) {   /* end of a piece */                \
      const double tot = t0 + t1;                                                                \
      /* With dA = +Inf nothing is certainly kept (exactly 0); otherwise the subtraction's */    \
      /* rounding is far below the row maximum's own mass. */                                    \
      double kw = none_kept ? 0.0 : tot - sub;                                                   \
      kw = warp_sum_d(kw);                                                                       \
      stot += tot;                                                                               \
      if (lane == 0) { part[warp * ppw + (st / W_G)] = kw; ksum += kw; }                         \
      t0 = t1 = 0.0; sub = 0.0;                                                                  \
    } }
  const unsigned long long pol = policy_drop();
  GS_WIDE_STREAM(T, 1, sp, rv, pol, lane, GS_BODY3);
#undef GS_BODY3
  Ssum = stot; Ksum = ksum;
}

// fn(key, d) for every logit of the warp's span that lies in the zone dB <= d < dA, streamed from
// global memory. Only rows whose zone outgrew the shared list come here (long runs of equal
// logits around the cut), so every step takes the masked form.
template <typename T, typename F>
__device__ __forceinline__ void wide_for_zone(const WSpan& sp, const RowView<T>& rv, unsigned long long pol, int lane,
                                              float m, float Tm, float dA, float dB, int mode, F&& fn) {
  constexpr int VEC = Elem<T>::VEC;
  uint4 qa[1], qb[1];
  w_load<T>(sp, 0, pol, qa[0], qb[0]);
  wide_steps<T, 1, false>(sp, rv, pol, lane, 0, sp.nst, qa, qb, [&](const float* x, uint32_t valid, int, int gv) {
#pragma unroll
    for (int c = 0; c < 8; c++) {
      if ((valid >> c) & 1u) {
        const float s = (Tm == 1.0f) ? x[c] : __fdiv_rn(x[c], Tm);
        const float d = s - m;
        if (d < dA && d >= dB) {
          const int i = (gv + 32 * (c / VEC)) * VEC - rv.shift + (c % VEC);
          fn(zone_key(d, i, mode), d);
        }
      }
    }
  });
}

struct WideShared {
  bu::Scratch sc;
  double tab[256];
  double bcd[4];
  int bc[4];
  int cnt;
  int row, why;
  // one pass: the row, its window, and what the pass and the cut find
  const uint4* vbase;
  int V, shift, nvec;
  int span, ppw;           // vectors of a warp's part of the row, pieces in it
  float as, base;          // what the sums are relative to, in units of x / T: the anchor, or, for exact sums, the base
  float Tm, xA, xB;        // above the window: x >= xA; the window: xB <= x < xA
  int far;                 // a logit lies too far above the anchor
  int placed;              // HOW_LOW: the window reaches down to where no mass is; HOW_OFTEN: the lanes' buffers are emptied more often; HOW_TWICE: twice the sample
  double eps;              // relative error bound of the sums
  double kw[W_NW];         // the mass above the window in each warp's part of the row (all its mass where the window is low),
  double zw[W_NW];         // what the window adds to it,
  double pm[W_MAX_PPW];    // kept mass of one warp's pieces
};

// Why a row takes two passes (reserved[6] of its debug record), and which branches the one-pass form took with it (reserved[7]).
enum { WHY_TEMPERATURE = 1,   // the quick quotient is not exact for it
       WHY_SHORT,             // too short for a sample
       WHY_NOT_FINITE,        // NaN or infinite, where looked at
       WHY_HEAVY,             // a few tokens hold much of the mass: not for a sample to place the cut
       WHY_WINDOW,            // the window holds more than the lists do
       WHY_EMPTY_WINDOW,
       WHY_NAN,               // a NaN in the row, or an infinite maximum
       WHY_LIST,              // a list or a lane's buffer did not hold all
       WHY_ANCHOR,            // the maximum lies too far from the anchor
       WHY_SUM,
       WHY_CUT_ABOVE,         // the window failed: the cut lies above it,
       WHY_CUT_BELOW,         // ... or below, or too close to its end
       WHY_LONG,              // longer than a warp's part can be
       WHY_AGAIN };           // (not a reason: the sample is doubled)
enum { HOW_CUT = 1, HOW_LOW = 2, HOW_ONE_CLASS = 4, HOW_BY_PIECE = 8, HOW_INDEX = 16, HOW_EXACT = 32, HOW_OFTEN = 64, HOW_TWICE = 128 };
// How a row ends, from either form. `path`: 2 two passes, 3 one.
struct WideResult {
  float m;                 // largest x / T
  double S, Re;            // all mass, kept mass
  int path, why, how;
};
__device__ __forceinline__ void wide_write(const KernelArgs& A, int64_t row_id, const WideResult& r, int id, uint32_t flags,
                                           double lo, double hi, int kept) {
  A.out_ids[row_id] = id;
  if (A.out_flags) A.out_flags[row_id] = flags;
  if (A.out_debug) {
    RowDebug d;
    d.sum_exp = r.S; d.resum = r.Re / r.S; d.edge_lo = lo; d.edge_hi = hi; d.kept = kept;
    d.max_scaled = r.m; d.threshold = __int_as_float(0x7fc00000); d.path = r.path;
    for (int q = 0; q < 8; q++) d.reserved[q] = 0;
    d.reserved[6] = static_cast<uint32_t>(r.why);
    d.reserved[7] = static_cast<uint32_t>(r.how);
    A.out_debug[row_id] = d;
  }
}
// A row whose sum is no number (S NaN), or whose mode A cut removed every token (generate.go:221-227 divides by zero): every
// comparison of the walk fails, result n-1 (:239).
__device__ __noinline__ void wide_write_nothing_kept(const KernelArgs& A, int64_t row_id, float m, double S, int path, int why, int how, uint32_t flags) {
  const double QNAN = __longlong_as_double(0x7ff8000000000000ll);
  if (A.out_probs) {
    double* pr = A.out_probs + row_id * static_cast<int64_t>(A.V);
    for (int i = threadIdx.x; i < A.V; i += W_NT) pr[i] = QNAN;
  }
  WideResult r;
  const bool number = S == S && S > 0.0;
  r.m = m; r.S = number ? S : QNAN; r.Re = number ? 0.0 : r.S; r.path = path; r.why = why; r.how = how;
  if (threadIdx.x == 0) wide_write(A, row_id, r, A.V - 1, flags | FLAG_NONFINITE | FLAG_FALLBACK, 0.0, 0.0, 0);
}
// The end of a row: u Re falls into piece `psel` or just behind it (rounding), `before` is the kept mass ahead of it
// (psel 0x7fffffff: behind every piece). kept_mass(x, i): the kept mass of logit i, 0 when it is cut away.
template <typename T, typename F>
__device__ __forceinline__ void wide_draw(const KernelArgs& A, const int64_t row_id, const RowView<T>& rv, const int span, const int ppw,
                                          const int psel, const double before, const double u, const WideResult& r, uint32_t flags,
                                          WideShared& sh, F&& kept_mass) {
  constexpr int VEC = Elem<T>::VEC, SV = 32 * (8 / VEC), PV = W_G * SV;
  constexpr int NV = (PV + W_NT - 1) / W_NT;                 // vectors of a piece per thread
  const int tid = threadIdx.x, lane = tid & 31;
  const int V = rv.V, npiece = W_NW * ppw;
  int kept_n = 0;
  if (A.out_probs || A.out_debug) {                          // parity runs only
    double* pr = A.out_probs ? A.out_probs + row_id * static_cast<int64_t>(V) : nullptr;
    const double rq = r.Re / r.S;
    int kept_loc = 0;
    for (int v = tid; v < rv.nvec; v += W_NT) {
      float x[VEC];
      Elem<T>::unpack(__ldg(rv.vbase + v), x);
      const int i0 = v * VEC - rv.shift;
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        const int i = i0 + c;
        if (i >= 0 && i < V) {
          const double f = (kept_mass(x[c], i) / r.S) / rq;
          kept_loc += (f > 0) ? 1 : 0;
          if (pr) pr[i] = f;
        }
      }
    }
    kept_n = bu::sum_i<W_NW>(kept_loc, sh.sc, tid);
  }
  // draw (generate.go:231-239): u < prefix/Re is tested as u*Re < prefix
  const double tgt = u * r.Re;
  double run_end = before;
  // walk pieces from the selected one (rounding can push the crossing into the next piece)
  for (int pi = psel; pi < npiece; pi++) {                   // uniform; normally one trip
    const int w = pi / ppw;
    const int vb = w * span + (pi - w * ppw) * PV;
    const int vend = min(min(vb + PV, w * span + span), rv.nvec);
    const int j = vb + tid * NV;
    double em[NV * VEC];
    double tsum = 0.0;
    const int i0 = j * VEC - rv.shift;
#pragma unroll
    for (int h = 0; h < NV; h++) {
      const bool in = tid * NV + h < PV && j + h < vend;
      float x[VEC];
      Elem<T>::unpack(__ldg(rv.vbase + (in ? j + h : 0)), x);
#pragma unroll
      for (int c = 0; c < VEC; c++) { em[h * VEC + c] = in ? kept_mass(x[c], i0 + h * VEC + c) : 0.0; tsum += em[h * VEC + c]; }
    }
    if (tid == 0) sh.bc[3] = 0x7fffffff;
    double totc;
    const double ex = bu::scan_excl_d<W_NW>(tsum, totc, sh.sc, tid);
    int pick = 0x7fffffff;
    double run = run_end + ex, lo = 0.0, hi = 0.0;
#pragma unroll
    for (int c = 0; c < NV * VEC; c++) {
      const double b = run;
      run += em[c];
      if (em[c] > 0.0 && tgt < run && pick == 0x7fffffff) { pick = i0 + c; lo = b; hi = run; }
    }
    const int first = __reduce_min_sync(FULL, pick);
    if (lane == 0 && first != 0x7fffffff) atomicMin(&sh.bc[3], first);
    __syncthreads();
    const int id = sh.bc[3];
    if (id != 0x7fffffff) {
      if (pick == id) {
        lo /= r.Re; hi /= r.Re;
        if ((lo > 0.0 && u - lo <= 1e-6) || hi - u <= 1e-6) flags |= FLAG_BOUNDARY;
        wide_write(A, row_id, r, id, flags, lo, hi, kept_n);
      }
      return;
    }
    run_end += totc;
    __syncthreads();
  }
  const double end = run_end / r.Re;
  if (u - end <= 1e-6) flags |= FLAG_BOUNDARY;
  if (tid == 0) wide_write(A, row_id, r, V - 1, flags | FLAG_FALLBACK, end, end, kept_n);   // generate.go:239
}

// The exact cut for a zone that outgrew the shared list (long runs of equal logits around the
// cut): the weighted selection of wide_row, with the row itself as the source of the zone's keys,
// one more pass per round. Adds the kept zone mass to part[]; false: the bracket did not hold.
template <typename T>
__device__ __noinline__ bool wide_big_zone(const WSpan& sp_in, const RowView<T>& rv_in, unsigned long long pol, WideShared& sh,
                                           uint32_t* hist, double* part, const double* s_tab, float m, float Tm, float dA,
                                           float dB, float dlow, int mode, double plim, double S, double Ktot, bool fast_ok,
                                           int span, int ppw, unsigned long long& cut_key_out, int& cut_incl_out, uint32_t& flags) {
  const WSpan sp = sp_in;
  const RowView<T> rv = rv_in;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int PV = W_G * 32 * (8 / Elem<T>::VEC);
  bu::Scratch& sc = sh.sc;
  unsigned long long cut_key = 0ull;
  int cut_incl = 0;
  bool bad = false;
  {
    // every zone key with its d: from the list, or from the row when the list overflowed
    auto each_zone = [&](auto&& fn) { wide_for_zone<T>(sp, rv, pol, lane, m, Tm, dA, dB, mode, fn); };
    // G(c) = Ktot + mass{key <= c} rises along the zone order. Both flavours need the first key c*
    // where G crosses: mode B (first G/S >= p) keeps through c*, mode A (first G/S > 1.5p) keeps
    // everything before it. Narrow [lo, hi] around c* with linear sub-buckets until at most 32
    // keys remain, then one warp finishes.
    auto crossed = [&](double g) -> bool { return mode == 0 ? (g / S > plim) : (g / S >= plim); };
    if (Ktot > 0.0 && crossed(Ktot)) bad = true;             // the bracket was wrong
    double* sm = reinterpret_cast<double*>(hist);            // [W_NSUB] mass per sub-bucket
    int* scn = reinterpret_cast<int*>(hist) + 2 * W_NSUB;    // [W_NSUB] count per sub-bucket
    unsigned long long lo = ~0ull, hi = 0ull;
    int nz_loc = 0;
    each_zone([&](unsigned long long k, float) { lo = k < lo ? k : lo; hi = k > hi ? k : hi; nz_loc++; });
    lo = bu::min_u64<W_NW>(lo, sc, tid);
    hi = bu::max_u64<W_NW>(hi, sc, tid);
    double gbase = Ktot;                                     // Ktot + mass of keys below lo; never crossed
    int inrange = bu::sum_i<W_NW>(nz_loc, sc, tid);
    bool all_in = false;
    for (int iter = 0; iter < 10 && inrange > 32 && !bad && !all_in; iter++) {
      const unsigned long long spn = hi - lo;
      int shf = 0;
      while (shf < 63 && (spn >> shf) >= static_cast<unsigned long long>(W_NSUB)) shf++;
      __syncthreads();
      sm[tid] = 0.0; scn[tid] = 0;                           // W_NT == W_NSUB
      __syncthreads();
      each_zone([&](unsigned long long k, float d) {
        if (k >= lo && k <= hi) {
          const int sb = static_cast<int>((k - lo) >> shf);
          atomicAdd(&sm[sb], exp_safe(d, s_tab));
          atomicAdd(&scn[sb], 1);
        }
      });
      __syncthreads();
      const double mine = sm[tid];
      double totm;
      const double exm = bu::scan_excl_d<W_NW>(mine, totm, sc, tid);
      const int first = (scn[tid] > 0 && crossed(gbase + exm + mine)) ? tid : W_NSUB;
      const int sbx = bu::min_i<W_NW>(first, sc, tid);
      if (sbx == W_NSUB) { all_in = true; break; }
      if (tid == sbx) { sh.bcd[0] = gbase + exm; sh.bc[0] = scn[tid]; }
      __syncthreads();
      gbase = sh.bcd[0];
      inrange = sh.bc[0];
      const unsigned long long nlo = lo + (static_cast<unsigned long long>(sbx) << shf);
      unsigned long long nhi = nlo + ((1ull << shf) - 1ull);
      if (nhi < nlo || nhi > hi) nhi = hi;
      lo = nlo; hi = nhi;
    }
    if (inrange > 32 && !all_in) bad = true;
    double g_at = gbase, g_before = gbase;
    if (!bad && !all_in) {
      unsigned long long* few = reinterpret_cast<unsigned long long*>(hist);   // [32]
      __syncthreads();
      if (tid == 0) sh.cnt = 0;
      __syncthreads();
      each_zone([&](unsigned long long k, float) {
        if (k >= lo && k <= hi) { const int slot = atomicAdd(&sh.cnt, 1); if (slot < 32) few[slot] = k; }
      });
      __syncthreads();
      const int nf = min(32, sh.cnt);
      if (warp == 0) {
        const unsigned long long k = (lane < nf) ? few[lane] : ~0ull;
        const double e = (lane < nf) ? exp_safe(zone_key_d(k), s_tab) : 0.0;
        double g = gbase;                                    // G(k) = gbase + masses of the keys <= k
        for (int l = 0; l < nf; l++) {
          const unsigned long long kl = __shfl_sync(FULL, k, l);
          const double el = __shfl_sync(FULL, e, l);
          if (kl <= k) g += el;
        }
        const bool cr = (lane < nf) && crossed(g);
        unsigned long long candk = cr ? k : ~0ull;           // first crossed key = smallest crossed key
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long tt = __shfl_xor_sync(FULL, candk, o);
          candk = tt < candk ? tt : candk;
        }
        const unsigned who = __ballot_sync(FULL, cr && k == candk);
        if (lane == 0) { sc.u[0] = candk; sh.bc[1] = who ? 1 : 0; }
        if (who && lane == __ffs(who) - 1) { sh.bcd[1] = g; sh.bcd[2] = g - e; }
      }
      __syncthreads();
      if (sh.bc[1]) {
        cut_key = sc.u[0];
        g_at = sh.bcd[1];
        g_before = sh.bcd[2];
        cut_incl = (mode == 0) ? 0 : 1;
      } else {
        all_in = true;                                       // rounding: nothing in the last group crossed
      }
      __syncthreads();
    }
    if (!bad && all_in) {
      cut_key = ~0ull; cut_incl = 1;
      if (mode == 1 && dlow < dB) bad = true;                // logits below the zone exist: the bracket promised a crossing
    }
    if (!bad && !all_in) {
      // the sums carry exp_fast_s's error; in G/S >= p it enters as 2 p (1-p) times that bound
      const double etol = 1e-12 + (fast_ok ? 2.0 * plim * fabs(1.0 - plim) * W_EXP_REL_ERR : 0.0);
      if (fabs(g_at / S - plim) <= etol || fabs(g_before / S - plim) <= etol) flags |= FLAG_TOPP_EDGE;
      if (mode == 1) {
        // a later key with the same d as c*: the cut separates equal probabilities
        int tie = 0;
        each_zone([&](unsigned long long k, float) { tie |= (k > cut_key && (k >> 32) == (cut_key >> 32)) ? 1 : 0; });
        if (bu::max_i<W_NW>(tie, sc, tid)) flags |= FLAG_TIE_CUT;
      }
    }
    if (bad) return false;
    // kept zone entries add their mass to the piece they sit in
    __syncthreads();
    each_zone([&](unsigned long long k, float d) {
      if (k < cut_key || (cut_incl && k == cut_key)) {
        const int v = rv.vec_of(zone_key_index(k, mode));
        const int w = v / span;
        atomicAdd(&part[w * ppw + (v - w * span) / PV], exp_safe(d, s_tab));
      }
    });
    __syncthreads();
  }
  cut_key_out = cut_key; cut_incl_out = cut_incl;
  return true;
}

#include "sample_wide_onepass.cuh"

// Two passes over the row: for what one pass does not serve.
template <typename T>
__device__ __noinline__ void wide_twopass_row(const BatchArgs& BA, unsigned char* dyn, WideShared& sh) {
  const int64_t row_id = sh.row;
  const KernelArgs& A = BA.k;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int V = A.V;
  constexpr int VEC = Elem<T>::VEC;
  constexpr int SV = 32 * (8 / VEC);                         // vectors of one warp-step
  constexpr int PV = W_G * SV;                               // vectors of one piece
  const T* row = static_cast<const T*>(A.logits) + row_id * A.row_stride;
  RowView<T> rv;
  rv.init(row, V);
  bu::Scratch& sc = sh.sc;
  const double* s_tab = sh.tab;
  uint32_t* hist = reinterpret_cast<uint32_t*>(dyn + W_OFF_HIST);
  uint2* zl = reinterpret_cast<uint2*>(dyn + W_OFF_ZONE);
  unsigned long long* zk = reinterpret_cast<unsigned long long*>(dyn + W_OFF_ZONE);
  double* ebs = reinterpret_cast<double*>(dyn + W_OFF_EB);
  double* part = reinterpret_cast<double*>(dyn + W_OFF_PART);   // [warp][piece] kept mass, row order

  const RowCfg cfg = A.cfgs[row_id];
  const float Tm = cfg.temperature;
  const bool topp_on = (cfg.top_p > 0.0f && cfg.top_p < 1.0f);
  const int mode = cfg.topp_mode;
  const double u = A.uniforms[row_id];
  const double plim = (mode == 0) ? static_cast<double>(cfg.top_p) * 1.5 : static_cast<double>(cfg.top_p);
  // mode A prunes only while the mass exceeds 1.5p; the mass starts at 1 up to ~1e-11 of rounding
  // and 1.5*float(p) is never that close to 1
  const bool cut_on = topp_on && !(mode == 0 && plim >= 1.0);
  const bool t_is_one = (Tm == 1.0f);
  uint32_t flags = FLAG_GENERAL_PATH;
  // the warp's span: 1/W_NW of the row, rounded up to whole steps
  const int span = (((rv.nvec + W_NW - 1) / W_NW + SV - 1) / SV) * SV;
  const int steps_max = span / SV;
  if (steps_max > W_MAX_STEPS) {
    if (tid == 0) hand_to_single(BA, row_id);
    return;
  }
  const int ppw = (steps_max + W_G - 1) / W_G;               // pieces per warp
  const int npiece = W_NW * ppw;
  const WSpan sp = make_span<T>(rv, warp * span, span, lane);

  float m = 0.0f, dlow = -INFINITY;
  float dA = -INFINITY, dB = -INFINITY;    // certainly kept: d >= dA; zone: dB <= d < dA; dropped: d < dB
  bool fast_ok = false;
  double S = 0.0, Ktot = 0.0;
  int nz = 0;
  // ---- a sample of the row (every warp's first step) gives an upper estimate of the maximum
  // and the bucket width, so that pass 1 can already count the histogram the cut needs
  bool anchored = false;
  float anchor = 0.0f, scale = 128.0f, width = 0.0078125f, dclamp = -31.99f;
  auto set_scale = [&](float range) {      // power of two (1/128 .. 1/65536) at which `range` just fits
    int jexp = 7;
    const float q = 4094.0f / range;                         // +Inf for range 0, 0 for an infinite range
    if (q >= 65536.0f) jexp = 16; else if (q >= 128.0f) jexp = ilogbf(q);
    scale = __int_as_float((127 + jexp) << 23);
    width = 1.0f / scale;
    dclamp = -4095.4f * width;
  };
  if (cut_on) {
    for (int j = tid; j < W_NB; j += W_NT) hist[j] = 0;
    float smax = -INFINITY, smin = INFINITY;
    bool snan = false;
#pragma unroll
    for (int h = 0; h < 8 / VEC; h++) {
      const int g = sp.first + 32 * h + lane;
      if (sp.nst > 0 && g < rv.nvec) rv.visit(g, [&](float xv, int) { smax = fmaxf(smax, xv); smin = fminf(smin, xv); snan |= (xv != xv); });
    }
    const int bad_sample = bu::max_i<W_NW>(snan ? 1 : 0, sc, tid);
    smax = okey_to_float(static_cast<uint32_t>(bu::max_u64<W_NW>(static_cast<unsigned long long>(okey(smax)), sc, tid)));
    smin = okey_to_float(static_cast<uint32_t>(bu::min_u64<W_NW>(static_cast<unsigned long long>(okey(smin)), sc, tid)));
    const float s_hi = scale_t(smax, Tm), s_lo = scale_t(smin, Tm);
    const float r0 = s_hi - s_lo;
    if (!bad_sample && r0 >= 0.0f && r0 < 1e30f && fabsf(s_hi) < 1e30f) {
      // half the sample's range above its maximum (a maximum beyond that costs an extra pass),
      // a quarter below its minimum (what lies lower shares the last bucket)
      const float margin = fmaxf(0.5f * r0, 1e-3f * fmaxf(1.0f, fabsf(s_hi)));
      anchor = s_hi + margin;
      set_scale(r0 + 1.5f * margin);
      anchored = true;
    }
  }

  // ---- pass 1: max, min, NaN (from HBM; L2 is asked to keep the row)
  float xmax = -INFINITY, xmin = INFINITY;
  bool nan_seen = false;
  {
    const uint32_t hb = smem_addr(hist) - 0x4B000000u * 4u;
    if (!anchored) wide_pass1<T, false, true>(sp, rv, lane, hb, anchor, Tm, scale, dclamp, xmax, xmin, nan_seen);
    else if (t_is_one) wide_pass1<T, true, true>(sp, rv, lane, hb, anchor, Tm, scale, dclamp, xmax, xmin, nan_seen);
    else wide_pass1<T, true, false>(sp, rv, lane, hb, anchor, Tm, scale, dclamp, xmax, xmin, nan_seen);
  }
  __syncthreads();
  const int anynan = bu::max_i<W_NW>(nan_seen ? 1 : 0, sc, tid);
  xmax = okey_to_float(static_cast<uint32_t>(bu::max_u64<W_NW>(static_cast<unsigned long long>(okey(xmax)), sc, tid)));
  xmin = okey_to_float(static_cast<uint32_t>(bu::min_u64<W_NW>(static_cast<unsigned long long>(okey(xmin)), sc, tid)));
  m = scale_t(xmax, Tm);
  // A NaN anywhere, or an infinite maximum, makes the softmax sum NaN upstream
  // (generate.go:173-181): every comparison of the walk fails, result n-1 (:239).
  if (anynan || !(fabsf(m) < INFINITY)) {
    wide_write_nothing_kept(A, row_id, m, -1.0, 2, sh.why, 0, flags);
    return;
  }
  dlow = scale_t(xmin, Tm) - m;                  // smallest d of the row (-Inf with a -Inf logit)
  fast_ok = (dlow > -31.9f);                      // every d inside the bucket table's range

  // ---- bracket of the cut from the count histogram
  if (cut_on) {
    // The histogram of pass 1 counts q = s - anchor; it stands when no logit lies above the anchor.
    // Mass bounds relative to exp(anchor) serve as well as bounds relative to exp(max): only their
    // ratios are used. q and d are each rounded once, so a logit's true mass can differ from
    // exp(q) exp(anchor - max) by the factor exp(+-2^-24 * 64): `slack` covers it.
    double slack = 1e-5;
    if (!(anchored && m <= anchor)) {
      anchored = false;
      slack = 1e-7;
      set_scale(-dlow);
      __syncthreads();
      for (int j = tid; j < W_NB; j += W_NT) hist[j] = 0;
      __syncthreads();
      if (t_is_one) wide_pass2<T, true>(sp, rv, lane, smem_addr(hist) - 0x4B000000u * 4u, m, Tm, scale, dclamp);
      else wide_pass2<T, false>(sp, rv, lane, smem_addr(hist) - 0x4B000000u * 4u, m, Tm, scale, dclamp);
    }
    __syncthreads();
    constexpr int PER = W_NB / W_NT;                         // buckets per thread
    // bucket b holds q (or d) in [-(b+.5) width, -(b-.5) width], the last one everything below.
    // Its members' masses lie between edge(b+1) and edge(b), edge(k) = exp(-(k-.5) width): one
    // exponential per thread, the next edges by the common ratio (rounding far inside `slack`).
    // The walk over the thread's buckets is done twice (sums, then the tests against the scanned
    // sums) rather than kept in registers.
    const double ratio = exp_safe(-width, s_tab);
    const double edge0 = exp_safe(-(tid * PER - 0.5f) * width, s_tab);
    double slo = 0.0, shi = 0.0;
    {
      double edge = edge0;
#pragma unroll 4
      for (int j = 0; j < PER; j++) {
        const int b = tid * PER + j;
        const double c = static_cast<double>(hist[b]);
        const double ehi = fmin(edge, 1.0) * (1.0 + slack);
        edge *= ratio;
        const double elo = (b == W_NB - 1) ? 0.0 : edge * (1.0 - slack);
        slo += c * elo; shi += c * ehi;
      }
    }
    double ex_lo, ex_hi, tot_lo, tot_hi;
    bu::scan_excl_d2<W_NW>(slo, shi, ex_lo, ex_hi, tot_lo, tot_hi, sc, tid);
    int b1 = W_NB - 1, b2 = W_NB - 1;
    const double p_lo = plim * (1.0 - 1e-9), p_hi = plim * (1.0 + 1e-9);
    {
      double edge = edge0, a_lo = ex_lo, a_hi = ex_hi;
#pragma unroll 4
      for (int j = 0; j < PER; j++) {
        const int b = tid * PER + j;
        const double c = static_cast<double>(hist[b]);
        const double ehi = fmin(edge, 1.0) * (1.0 + slack);
        edge *= ratio;
        const double elo = (b == W_NB - 1) ? 0.0 : edge * (1.0 - slack);
        a_lo += c * elo; a_hi += c * ehi;
        // largest / smallest possible mass fraction through bucket b against the limit, as products
        const double den_hi = a_hi + (tot_lo - a_lo), den_lo = a_lo + (tot_hi - a_hi);
        bool c1, c2;
        if (mode == 0) { c1 = a_hi > p_lo * den_hi; c2 = a_lo > p_hi * den_lo; }
        else           { c1 = a_hi >= p_lo * den_hi; c2 = a_lo >= p_hi * den_lo; }
        if (c1 && a_hi > 0.0) b1 = min(b1, b);
        if (c2 && a_lo > 0.0) b2 = min(b2, b);
      }
    }
    bu::min_i2<W_NW>(b1, b2, sc, tid);
    if (b2 < b1) b2 = b1;
    const float qA = bucket_floor_w(b1 - 1, scale, dclamp);  // certainly kept: q >= qA
    const float qB = bucket_floor_w(b2, scale, dclamp);      // certainly dropped: q < qB
    if (!anchored) {
      dA = qA; dB = qB;
    } else {
      // Thresholds on d = rn(s - max) that are at least as cautious as those on q = rn(s - anchor):
      // d >= dA must imply q >= qA, and q >= qB must imply d >= dB. Both roundings are monotone:
      // s - anchor >= qA implies q >= qA, and q >= qB implies s - anchor >= pred(qB).
      if (qA == INFINITY) dA = INFINITY;
      else dA = nextafterf(__double2float_ru(static_cast<double>(anchor) + static_cast<double>(qA) - static_cast<double>(m)), INFINITY);
      if (qB == -INFINITY) dB = -INFINITY;
      else dB = nextafterf(__double2float_rd(static_cast<double>(anchor) + static_cast<double>(nextafterf(qB, -INFINITY)) - static_cast<double>(m)), -INFINITY);
      if (dA > 0.0f) dA = INFINITY;                          // no d reaches it: nothing is certainly kept
    }
  }

  // ---- pass 3: exponentials (last use of the row: evict-first)
  // exponential table: sixteen conflict-free copies of the first 128 entries when the row's range
  // allows it, else the plain 1024 entries
  const bool eb_rep = fast_ok && (dlow > -(W_EB_REP_ENTRIES - 2.0f) / 32.0f);
  if (eb_rep) {
    for (int j = tid; j < W_EB_REP * W_EB_REP_ENTRIES; j += W_NT) ebs[j] = __ldg(BA.eb_table + j / W_EB_REP);
  } else if (fast_ok) {
    for (int j = tid; j < NB1; j += W_NT) ebs[j] = __ldg(BA.eb_table + j);
  }
  if (tid < npiece) part[tid] = 0.0;                         // pieces past the row's end stay empty
  if (tid == 0) sh.cnt = 0;
  __syncthreads();
  double Ssum = 0.0, Ksum = 0.0;
  const uint32_t eb_mul = eb_rep ? 8u * W_EB_REP : 8u;
  const uint32_t eb_bias = smem_addr(ebs) + (eb_rep ? 8u * (lane & (W_EB_REP - 1)) : 0u) - 0x4B000000u * eb_mul;
#define GS_P3(F, O, C) wide_pass3<T, F, O, C>(sp, rv, lane, warp, m, Tm, dA, dB, eb_mul, eb_bias, s_tab, part, ppw, zl, &sh.cnt, Ssum, Ksum)
  if (cut_on) {
    if (fast_ok) { if (t_is_one) GS_P3(true, true, true); else GS_P3(true, false, true); }
    else         { if (t_is_one) GS_P3(false, true, true); else GS_P3(false, false, true); }
  } else {
    if (fast_ok) { if (t_is_one) GS_P3(true, true, false); else GS_P3(true, false, false); }
    else         { if (t_is_one) GS_P3(false, true, false); else GS_P3(false, false, false); }
  }
#undef GS_P3
  __syncthreads();
  if (lane != 0) Ksum = 0.0;                                 // kept mass is already warp-reduced into lane 0
  double unused = 0.0;
  S = Ssum; Ktot = Ksum;
  bu::sum_d3<W_NW>(S, Ktot, unused, sc, tid);
  nz = sh.cnt;
  // A zone that outgrew the list (long runs of equal logits around the cut): the same selection
  // runs over the row itself, one more pass per round.
  const bool big = cut_on && nz > W_ZCAP;

  // ---- exact cut inside the zone by weighted selection
  unsigned long long cut_key = 0ull;       // zone entries are kept when key < cut_key, or == with cut_incl
  int cut_incl = 0;
  bool bad = false;
  if (big) {
    if (!wide_big_zone<T>(sp, rv, policy_keep(), sh, hist, part, s_tab, m, Tm, dA, dB, dlow, mode, plim, S, Ktot, fast_ok,
                          span, ppw, cut_key, cut_incl, flags)) {
      if (tid == 0) hand_to_single(BA, row_id);
      return;
    }
  } else if (cut_on && nz > 0) {
    for (int j = tid; j < nz; j += W_NT) {                   // entries -> keys, in place
      const uint2 e = zl[j];
      zk[j] = zone_key(__uint_as_float(e.x), static_cast<int>(e.y), mode);
    }
    __syncthreads();
    // G(c) = Ktot + mass{key <= c} rises along the zone order. Both flavours need the first key c*
    // where G crosses: mode B (first G/S >= p) keeps through c*, mode A (first G/S > 1.5p) keeps
    // everything before it. Narrow [lo, hi] around c* with linear sub-buckets until at most 32
    // keys remain, then one warp finishes.
    auto crossed = [&](double g) -> bool { return mode == 0 ? (g / S > plim) : (g / S >= plim); };
    if (Ktot > 0.0 && crossed(Ktot)) bad = true;             // the bracket was wrong
    double* sm = reinterpret_cast<double*>(hist);            // [W_NSUB] mass per sub-bucket
    int* scn = reinterpret_cast<int*>(hist) + 2 * W_NSUB;    // [W_NSUB] count per sub-bucket
    unsigned long long lo = ~0ull, hi = 0ull;
    for (int j = tid; j < nz; j += W_NT) { const unsigned long long k = zk[j]; lo = k < lo ? k : lo; hi = k > hi ? k : hi; }
    lo = bu::min_u64<W_NW>(lo, sc, tid);
    hi = bu::max_u64<W_NW>(hi, sc, tid);
    double gbase = Ktot;                                     // Ktot + mass of keys below lo; never crossed
    int inrange = nz;
    bool all_in = false;
    for (int iter = 0; iter < 8 && inrange > 32 && !bad && !all_in; iter++) {
      const unsigned long long spn = hi - lo;
      int shf = 0;
      while (shf < 63 && (spn >> shf) >= static_cast<unsigned long long>(W_NSUB)) shf++;
      __syncthreads();
      sm[tid] = 0.0; scn[tid] = 0;                           // W_NT == W_NSUB
      __syncthreads();
      for (int j = tid; j < nz; j += W_NT) {
        const unsigned long long k = zk[j];
        if (k >= lo && k <= hi) {
          const int sb = static_cast<int>((k - lo) >> shf);
          atomicAdd(&sm[sb], exp_safe(zone_key_d(k), s_tab));
          atomicAdd(&scn[sb], 1);
        }
      }
      __syncthreads();
      const double mine = sm[tid];
      double totm;
      const double exm = bu::scan_excl_d<W_NW>(mine, totm, sc, tid);
      const int first = (scn[tid] > 0 && crossed(gbase + exm + mine)) ? tid : W_NSUB;
      const int sbx = bu::min_i<W_NW>(first, sc, tid);
      if (sbx == W_NSUB) { all_in = true; break; }
      if (tid == sbx) { sh.bcd[0] = gbase + exm; sh.bc[0] = scn[tid]; }
      __syncthreads();
      gbase = sh.bcd[0];
      inrange = sh.bc[0];
      const unsigned long long nlo = lo + (static_cast<unsigned long long>(sbx) << shf);
      unsigned long long nhi = nlo + ((1ull << shf) - 1ull);
      if (nhi < nlo || nhi > hi) nhi = hi;
      lo = nlo; hi = nhi;
    }
    if (inrange > 32 && !all_in) bad = true;
    double g_at = gbase, g_before = gbase;
    if (!bad && !all_in) {
      unsigned long long* few = reinterpret_cast<unsigned long long*>(hist);   // [32]
      __syncthreads();
      if (tid == 0) sh.cnt = 0;
      __syncthreads();
      for (int j = tid; j < nz; j += W_NT) {
        const unsigned long long k = zk[j];
        if (k >= lo && k <= hi) { const int slot = atomicAdd(&sh.cnt, 1); if (slot < 32) few[slot] = k; }
      }
      __syncthreads();
      const int nf = min(32, sh.cnt);
      if (warp == 0) {
        const unsigned long long k = (lane < nf) ? few[lane] : ~0ull;
        const double e = (lane < nf) ? exp_safe(zone_key_d(k), s_tab) : 0.0;
        double g = gbase;                                    // G(k) = gbase + masses of the keys <= k
        for (int l = 0; l < nf; l++) {
          const unsigned long long kl = __shfl_sync(FULL, k, l);
          const double el = __shfl_sync(FULL, e, l);
          if (kl <= k) g += el;
        }
        const bool cr = (lane < nf) && crossed(g);
        unsigned long long candk = cr ? k : ~0ull;           // first crossed key = smallest crossed key
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const unsigned long long tt = __shfl_xor_sync(FULL, candk, o);
          candk = tt < candk ? tt : candk;
        }
        const unsigned who = __ballot_sync(FULL, cr && k == candk);
        if (lane == 0) { sc.u[0] = candk; sh.bc[1] = who ? 1 : 0; }
        if (who && lane == __ffs(who) - 1) { sh.bcd[1] = g; sh.bcd[2] = g - e; }
      }
      __syncthreads();
      if (sh.bc[1]) {
        cut_key = sc.u[0];
        g_at = sh.bcd[1];
        g_before = sh.bcd[2];
        cut_incl = (mode == 0) ? 0 : 1;
      } else {
        all_in = true;                                       // rounding: nothing in the last group crossed
      }
      __syncthreads();
    }
    if (!bad && all_in) {
      cut_key = ~0ull; cut_incl = 1;
      if (mode == 1 && dlow < dB) bad = true;                // logits below the zone exist: the bracket promised a crossing
    }
    if (!bad && !all_in) {
      // the sums carry exp_fast_s's error; in G/S >= p it enters as 2 p (1-p) times that bound
      const double etol = 1e-12 + (fast_ok ? 2.0 * plim * fabs(1.0 - plim) * W_EXP_REL_ERR : 0.0);
      if (fabs(g_at / S - plim) <= etol || fabs(g_before / S - plim) <= etol) flags |= FLAG_TOPP_EDGE;
      if (mode == 1) {
        // a later key with the same d as c*: the cut separates equal probabilities
        int tie = 0;
        for (int j = tid; j < nz; j += W_NT) { const unsigned long long k = zk[j]; tie |= (k > cut_key && (k >> 32) == (cut_key >> 32)) ? 1 : 0; }
        if (bu::max_i<W_NW>(tie, sc, tid)) flags |= FLAG_TIE_CUT;
      }
    }
    if (bad) {
      if (tid == 0) hand_to_single(BA, row_id);
      return;
    }
    // kept zone entries add their mass to the piece they sit in
    __syncthreads();
    for (int j = tid; j < nz; j += W_NT) {
      const unsigned long long k = zk[j];
      if (k < cut_key || (cut_incl && k == cut_key)) {
        const int v = rv.vec_of(zone_key_index(k, mode));
        const int w = v / span;
        atomicAdd(&part[w * ppw + (v - w * span) / PV], exp_safe(zone_key_d(k), s_tab));
      }
    }
    __syncthreads();
  }
  // ---- kept mass and the piece that holds the drawn token: prefix over the pieces in row order
  const double pm = (tid < npiece) ? part[tid] : 0.0;
  WideResult r;
  const double pex = bu::scan_excl_d<W_NW>(pm, r.Re, sc, tid);
  r.m = m; r.S = S; r.path = 2; r.why = sh.why; r.how = 0;
  if (!(S == S) || !(S > 0.0) || !(r.Re > 0.0)) {
    wide_write_nothing_kept(A, row_id, m, S, 2, sh.why, 0, flags);
    return;
  }
  const int psel = bu::min_i<W_NW>((tid < npiece && u * r.Re < pex + pm) ? tid : 0x7fffffff, sc, tid);
  if (tid == psel) sh.bcd[0] = pex;
  __syncthreads();
  const double before = (psel != 0x7fffffff) ? sh.bcd[0] : r.Re;
  // final rule for one logit: its kept mass (0 when cut away)
  auto kept_mass = [&](float xv, int i) -> double {
    if (i < 0 || i >= V) return 0.0;
    const float s = t_is_one ? xv : __fdiv_rn(xv, Tm);
    const float d = s - m;
    if (d < dA) {
      if (!(d >= dB)) return 0.0;
      const unsigned long long k = zone_key(d, i, mode);
      if (!(k < cut_key || (cut_incl && k == cut_key))) return 0.0;
    }
    return exp_safe(d, s_tab);
  };
  wide_draw<T>(A, row_id, rv, span, ppw, psel, before, u, r, flags, sh, kept_mass);
}

template <typename T>
__global__ void __launch_bounds__(W_NT, W_CTAS) wide_rows_kernel(const __grid_constant__ BatchArgs BA) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ WideShared sh;
  if (threadIdx.x < 256) sh.tab[threadIdx.x] = BA.k.exp_table[threadIdx.x];
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      int w;                                                 // next row of this kernel's kind
      for (;;) {
        w = atomicAdd(&BA.hdr[HDR_WIDE], 1);
        if (w >= BA.B) { w = -1; break; }
        if (row_kind(BA.k, w) == 1) break;
      }
      sh.row = w;
    }
    __syncthreads();
    const int row = sh.row;
    if (row < 0) break;
    // The narrow kernel may start: every CTA of this one has a row, or has gone. (Started together, the two kernels'
    // CTAs mix at random, and some SMs end up with more rows of this kind than others.)
    pdl_launch();
    const int why = wide_onepass_row<T>(BA, row, dyn, sh);
    if (why == 0) continue;
    if (threadIdx.x == 0) sh.why = why;
    __syncthreads();
    wide_twopass_row<T>(BA, dyn, sh);
  }
}

}  // namespace GS_W_NS
}  // namespace gs

#undef GS_W_NS
#undef GS_W_NT
