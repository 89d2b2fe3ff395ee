// The end of a top-k row, once its candidates (everything that can be among the kept logits) are in
// shared memory: exact k-th largest with ties kept (model/generate.go:157-164), softmax over the kept
// set, top-p (generate.go:184-228, qwen/generate.go:123-153), draw (generate.go:231-239).
//
// A few hundred candidates are no work for a CTA, so what bounds this part is the length of its chain
// of dependent steps. All threads only meet where there is something to share out: a histogram round
// that leaves little more than top_k candidates (narrow_candidates), then every candidate takes its own
// exponential and counts how many of the others come before it (by value and by index), which replaces
// a radix select and two sorts. Everything after that is done by one warp, without barriers. Masses stay sums of exponentials, and limits are multiplied by their total instead: no
// division per token.
#pragma once

#include "block_util.cuh"
#include "sample_kernel.cuh"

namespace gs {

constexpr int KEEP_MAX = 512;        // largest kept set finished in shared memory
constexpr int SS_WORK_BYTES = 13344; // work arrays of finish_small_set

// Lower edge of a narrow bucket of order keys that holds the r-th largest key of a sample (every thread calls
// f(key) for its keys, the same ones on every call); tmax: the largest of the thread's own keys, tmin: the
// smallest. cnts: NBINS counters. Buckets of equal width are counted until the one of the r-th largest
// holds few.
template <int NT_, int NBINS, typename F>
__device__ __forceinline__ uint32_t sample_threshold(F&& for_each_key, int r, uint32_t tmin, uint32_t tmax, uint32_t* cnts, int* bc,
                                                     bu::Scratch& sc, int tid) {
  constexpr int NW_ = NT_ / 32, PER = NBINS / NT_, LOGB = 31 - __builtin_clz(NBINS);
  const int lane = tid & 31, warp = tid >> 5;
  // r threads hold r largest ones of their own: the smallest of the thread maxima is not above the r-th largest
  // while r <= NT_, and keeps the buckets off the keys that nobody asks for
  uint32_t lo = __reduce_min_sync(FULL, (r <= NT_) ? tmax : tmin), hi = __reduce_max_sync(FULL, tmax);
  for (int b = tid; b < NBINS; b += NT_) cnts[b] = 0u;
  if (lane == 0) { sc.i0[warp] = static_cast<int>(lo); sc.i1[warp] = static_cast<int>(hi); }
  __syncthreads();
  lo = __reduce_min_sync(FULL, static_cast<uint32_t>(sc.i0[lane < NW_ ? lane : 0]));
  hi = __reduce_max_sync(FULL, static_cast<uint32_t>(sc.i1[lane < NW_ ? lane : 0]));
  int need = r;
  for (;;) {                                                   // uniform
    const int sh = max(0, 32 - __clz(hi - lo) - LOGB);
    for_each_key([&](uint32_t key) { if (key - lo <= hi - lo) atomicAdd(&cnts[(hi - key) >> sh], 1u); });
    __syncthreads();
    uint32_t mine = 0u;
#pragma unroll
    for (int q = 0; q < PER; q++) mine += cnts[tid * PER + q];
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += t; }
    if (lane == 31) sc.i0[warp] = static_cast<int>(incl);
    __syncthreads();
    uint32_t before = __reduce_add_sync(FULL, (lane < warp) ? static_cast<uint32_t>(sc.i0[lane]) : 0u) + incl - mine;
    if (before < static_cast<uint32_t>(need) && before + mine >= static_cast<uint32_t>(need)) {   // one thread
      int q = 0;
      while (before + cnts[tid * PER + q] < static_cast<uint32_t>(need)) before += cnts[tid * PER + q++];
      bc[0] = tid * PER + q; bc[1] = static_cast<int>(before); bc[2] = static_cast<int>(cnts[tid * PER + q]);
    }
    __syncthreads();
    const uint32_t top = hi - (static_cast<uint32_t>(bc[0]) << sh), width = (1u << sh) - 1u;
    lo = (top - lo > width) ? top - width : lo;
    hi = top;
    need -= bc[1];
    if (sh == 0 || bc[2] <= max(2, r >> 3)) break;
    __syncthreads();
    for (int b = tid; b < NBINS; b += NT_) cnts[b] = 0u;
    __syncthreads();
  }
  return lo;
}

// Leaves in out[] (KEEP_MAX entries) every candidate whose scaled value is not below that of the
// top_k-th largest, and little more. for_each(f) calls f(entry) for every candidate of the calling thread
// (the same ones on every call), n of them in the block. Every key lies in [lo, hi], except keys below lo that
// are known not to be wanted; 256 buckets between the two are counted until the bucket of the top_k-th
// largest holds few. Returns how many there are; more than KEEP_MAX (then they are not all there) only
// when that many tie with the top_k-th. hist: 256 counters, bc: 3 ints. The caller has cleared hist and s_cnt, with
// a barrier since.
template <int NTHREADS, typename F>
__device__ __forceinline__ int narrow_candidates(F&& for_each, int n, int topk, float Tm, uint32_t lo, uint32_t hi,
                                                 uint2* out, uint32_t* hist, int* bc, int* s_cnt, int tid) {
  uint32_t low = 0u;                                           // the lowest key that may be kept
  if (n > topk) {
    int need = topk, above_all = 0;
    for (;;) {                                                 // uniform
      const int sh = max(0, 24 - __clz(hi - lo));              // 256 buckets
      for_each([&](const uint2& e) {
        const uint32_t key = okey(__uint_as_float(e.x));
        if (key - lo <= hi - lo) atomicAdd(&hist[(hi - key) >> sh], 1u);
      });
      __syncthreads();
      if (tid < 32) {
        int loc[8], s = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) { s += static_cast<int>(hist[tid * 8 + j]); loc[j] = s; }
        int run = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(FULL, run, o); if (tid >= o) run += t; }
        const int before = run - s;
        if (before < need && run >= need) {
          int b = 7, prev = 0, cnt = 0;
#pragma unroll
          for (int j = 7; j >= 0; j--)
            if (before + loc[j] >= need) { b = j; prev = (j > 0) ? loc[j - 1] : 0; cnt = loc[j] - prev; }
          bc[0] = tid * 8 + b; bc[1] = before + prev; bc[2] = cnt;
        }
      }
      __syncthreads();
      const uint32_t top = hi - (static_cast<uint32_t>(bc[0]) << sh), width = (1u << sh) - 1u;
      lo = (top - lo > width) ? top - width : lo;
      hi = top;
      above_all += bc[1];
      need -= bc[1];
      if (sh == 0 || above_all + bc[2] <= topk + 24) break;
      __syncthreads();
      for (int j = tid; j < 256; j += NTHREADS) hist[j] = 0u;
      __syncthreads();
    }
    // Logits that the division by T makes equal to the bucket's lower edge belong to its class: the two keys below
    // it, as long as quotients keep 24 bits; whatever has the same quotient otherwise.
    const float edge = okey_to_float(lo), q = fabsf(scale_t(edge, Tm));
    low = (q > 1e-30f && q < 1e30f) ? lo - 4u : okey(quotient_class_floor(edge, Tm));
  }
  for_each([&](const uint2& e) {
    if (okey(__uint_as_float(e.x)) >= low) { const int slot = atomicAdd(s_cnt, 1); if (slot < KEEP_MAX) out[slot] = e; }
  });
  __syncthreads();
  return *s_cnt;
}
// The same over list[0..n).
template <int NTHREADS>
__device__ __noinline__ int narrow_list(const uint2* list, int n, int topk, float Tm, uint32_t lo, uint32_t hi,
                                                 uint2* out, uint32_t* hist, int* bc, int* s_cnt, int tid) {
  __syncthreads();
  for (int j = tid; j < 256; j += NTHREADS) hist[j] = 0u;
  if (tid == 0) *s_cnt = 0;
  __syncthreads();
  return narrow_candidates<NTHREADS>([&](auto&& f) { for (int j = tid; j < n; j += NTHREADS) f(list[j]); },
                                     n, topk, Tm, lo, hi, out, hist, bc, s_cnt, tid);
}

struct SmallSet {                      // finish_small_set's work arrays
  unsigned long long* ckey;            // [512] value, then index; two per 16-byte load
  double* fi;                          // [512] mass in index order (over ckey)
  double* se;                          // [512 + 1] exponentials, falling; then -1
  float* ss;                           // [512] scaled values, falling
  int* sidx;                           // [512] index, index order
  uint16_t* ip;                        // [512 + 1] place in index order of the t-th largest
  float* kth;                          // [1] the top_k-th largest logit
  __device__ __forceinline__ explicit SmallSet(unsigned char* w)
      : ckey(reinterpret_cast<unsigned long long*>(w)), fi(reinterpret_cast<double*>(w)), se(reinterpret_cast<double*>(w + 4096)),
        ss(reinterpret_cast<float*>(w + 8208)), sidx(reinterpret_cast<int*>(w + 10256)), ip(reinterpret_cast<uint16_t*>(w + 12304)),
        kth(reinterpret_cast<float*>(w + 13340)) {}
};

// The part that one warp does: lane l owns the places [l * per, (l + 1) * per) of either order. D: also the
// diagnostics (probabilities, debug record).
template <bool D>
__device__ __forceinline__ void finish_small_warp(const KernelArgs& A, int64_t row_id, const SmallSet& w, int n, int topk, bool topp_on,
                                                  int mode, double plim, double u, RowDebug* dbg, uint32_t flags) {
  const int lane = threadIdx.x & 31;
  const int lper = (n <= 32) ? 0 : 27 - __clz(n - 1);         // per = 2^lper, 32 * per >= n
  const int t0 = min(lane << lper, n), t1 = min(t0 + (1 << lper), n);
  const float skth = (n > topk) ? w.ss[topk - 1] : -INFINITY;
  int nk = 0;                                                 // the kept ones come first
  int turned = 0;
  double acc = 0.0;
#pragma unroll 2
  for (int t = t0; t < t1; t++) {
    const bool kept = w.ss[t] >= skth;
    const double e = w.se[t];
    // two logits that the division or the subtraction has made equal, in the wrong order of indices
    // (the places behind the last one hold no equal mass: se[n] is -1)
    turned |= (kept && w.se[t + 1] == e && (w.ip[t + 1] < w.ip[t]) != (mode == 0)) ? 1 : 0;
    nk += kept ? 1 : 0;
    acc += kept ? e : 0.0;
  }
  nk = __reduce_add_sync(FULL, nk);
  if (__reduce_or_sync(FULL, turned)) {                       // rare: put such runs in order (their masses are equal)
    if (lane == 0) {
      for (int t = 1; t < nk; t++)
        for (int q = t; q > 0 && w.se[q - 1] == w.se[q] && (w.ip[q] < w.ip[q - 1]) != (mode == 0); q--) {
          const uint16_t x = w.ip[q]; w.ip[q] = w.ip[q - 1]; w.ip[q - 1] = x;
        }
    }
    __syncwarp();
  }
  double incl = warp_scan_incl_d(acc, lane);
  const double S = __shfl_sync(FULL, incl, 31);
  int cutn = nk;                                              // how many of the most probable stay
  double total = S;                                           // their mass
  if (topp_on) {
    // mode A (generate.go:184-228): the longest prefix with mass <= 1.5 p; mode B (qwen/generate.go:123-153): the
    // shortest with mass >= p. Prefixes grow, so counting those below the limit finds either.
    const double lim = plim * S;
    double run = incl - acc;
    int c = 0;
#pragma unroll 2
    for (int t = t0; t < min(t1, nk); t++) {
      run += w.se[t];
      c += ((mode == 0) ? run <= lim : run < lim) ? 1 : 0;
    }
    c = __reduce_add_sync(FULL, c);
    cutn = (mode == 0) ? c : min(c + 1, nk);
    if (cutn == 0) {                                          // mode A, everything removed: 0/0 (generate.go:221-227)
      if (D && A.out_probs) {
        double* pr = A.out_probs + row_id * static_cast<int64_t>(A.V);
        for (int i = lane; i < A.V; i += 32) pr[i] = __longlong_as_double(0x7ff8000000000000ll);
      }
      if (lane == 0) {
        A.out_ids[row_id] = A.V - 1;
        if (A.out_flags) A.out_flags[row_id] = flags | FLAG_NONFINITE | FLAG_FALLBACK;
        if (D && A.out_debug) { dbg->sum_exp = S; dbg->resum = 0.0; A.out_debug[row_id] = *dbg; }
      }
      return;
    }
    run = incl - acc;
    double at = 0.0;
#pragma unroll 2
    for (int t = t0; t < min(t1, cutn); t++) { run += w.se[t]; at = run; }
    total = __shfl_sync(FULL, at, (cutn - 1) >> lper);
    if (A.out_flags) {
      // whether the mass on either side of the decision lies within rounding of the limit (A: kept, and one more;
      // B: kept, and one fewer)
      const double eps = 1e-12 * S;
      const double other = (mode == 0) ? ((cutn < nk) ? total + w.se[cutn] : -S) : ((cutn >= 2) ? total - w.se[cutn - 1] : -S);
      if (fabs(total - lim) <= eps || fabs(other - lim) <= eps) flags |= FLAG_TOPP_EDGE;
      if (mode != 0 && cutn < nk && w.se[cutn] == w.se[cutn - 1]) flags |= FLAG_TIE_CUT;
    }
  }
  if (D && A.out_debug) {
    int kept = 0;
    for (int t = t0; t < min(t1, cutn); t++) kept += (w.se[t] > 0.0) ? 1 : 0;
    dbg->kept = __reduce_add_sync(FULL, kept);
    dbg->threshold = w.ss[nk - 1];
    dbg->sum_exp = S;
    dbg->resum = topp_on ? total / S : 1.0;
  }
  // ---- draw (generate.go:231-239): first index with u < cumulative
  for (int t = t0; t < t1; t++) w.fi[w.ip[t]] = (t < cutn) ? w.se[t] : 0.0;
  __syncwarp();
  acc = 0.0;
#pragma unroll 2
  for (int t = t0; t < t1; t++) acc += w.fi[t];
  if (D && A.out_probs) {
    double* pr = A.out_probs + row_id * static_cast<int64_t>(A.V);
    const double norm = topp_on ? total / S : 1.0;
#pragma unroll 1
    for (int t = t0; t < t1; t++) pr[w.sidx[t]] = (w.fi[t] / S) / norm;
  }
  const double target = u * total;
  incl = warp_scan_incl_d(acc, lane);
  double run = incl - acc;
  int below = 0;                                              // cumulative sums that u is not below
#pragma unroll 2
  for (int t = t0; t < t1; t++) { run += w.fi[t]; below += (target < run) ? 0 : 1; }
  const int best = __reduce_add_sync(FULL, below);
  if (best < n) {
    if (lane == (best >> lper)) {
      run = incl - acc;
      for (int t = t0; t < best; t++) run += w.fi[t];
      A.out_ids[row_id] = w.sidx[best];
      if (D || A.out_flags) {
        const double lo = run / total, hi = (run + w.fi[best]) / total;
        if ((run > 0.0 && u - lo <= 1e-6) || hi - u <= 1e-6) flags |= FLAG_BOUNDARY;
        if (A.out_flags) A.out_flags[row_id] = flags;
        if (D && A.out_debug) { dbg->edge_lo = lo; dbg->edge_hi = hi; A.out_debug[row_id] = *dbg; }
      }
    }
  } else {
    const double tot = __shfl_sync(FULL, incl, 31) / total;
    if (lane == 0) {
      flags |= FLAG_FALLBACK;
      if (u - tot <= 1e-6) flags |= FLAG_BOUNDARY;
      A.out_ids[row_id] = A.V - 1;
      if (A.out_flags) A.out_flags[row_id] = flags;
      if (D && A.out_debug) { dbg->edge_lo = dbg->edge_hi = tot; A.out_debug[row_id] = *dbg; }
    }
  }
}

// Finishes a row from the candidates kp[0..n), n <= KEEP_MAX: those whose scaled value is at least that of
// the top_k-th largest are kept (all of them when n <= topk). m: the row's largest scaled value. min_thr: a
// logit that the kept set may not reach below (-Inf: none); when it would, nothing is written and the first
// warp's threads return false. Every thread of the block calls it. work: SS_WORK_BYTES of shared memory, aligned
// to 16 bytes.
// Not inlined: the kernels that stream rows keep their registers for that. (Their arguments have to be
// __grid_constant__, or A would be copied to every thread's stack.) dbg: with D only.
template <int NTHREADS, bool D>
__device__ __noinline__ bool finish_small_set(const KernelArgs& A, int64_t row_id, const uint2* kp, int n, int topk, float m, float Tm,
                                                 bool topp_on, int mode, double plim, double u, float min_thr, unsigned char* work,
                                                 RowDebug* dbg, uint32_t flags) {
  const int tid = threadIdx.x;
  const SmallSet w(work);
  // ---- every candidate counts those ahead of it: by falling logit (equal ones by ascending index; mode A
  // removes the lowest index first, so there the highest comes first), and by index
  for (int j = tid; j < n; j += NTHREADS) {
    const uint32_t ix = (mode == 0) ? kp[j].y : ~kp[j].y;
    w.ckey[j] = (static_cast<unsigned long long>(okey(__uint_as_float(kp[j].x))) << 32) | ix;
  }
  if (tid == 0) { w.se[n] = -1.0; if (n & 1) w.ckey[n] = 0ull; }   // (n odd: below KEEP_MAX)
  if (D && A.out_probs) {
    double* pr = A.out_probs + row_id * static_cast<int64_t>(A.V);
    for (int i = tid; i < A.V; i += NTHREADS) pr[i] = 0.0;
  }
  __syncthreads();
  for (int j = tid; j < n; j += NTHREADS) {
    const float s = scale_t(__uint_as_float(kp[j].x), Tm);
    const double ex = exp(static_cast<double>(s - m));        // f32 subtract, f64 exp (generate.go:176)
    const unsigned long long mine = w.ckey[j];
    const uint32_t ix = static_cast<uint32_t>(mine);
    int r = 0, rx = 0;
    const ulonglong2* pairs = reinterpret_cast<const ulonglong2*>(w.ckey);
#pragma unroll 4
    for (int l = 0; l < (n + 1) >> 1; l++) {
      const ulonglong2 o = pairs[l];
      r += (o.x > mine) ? 1 : 0;
      r += (o.y > mine) ? 1 : 0;
      rx += (static_cast<uint32_t>(o.x) > ix) ? 1 : 0;
      rx += (static_cast<uint32_t>(o.y) > ix) ? 1 : 0;        // (the padding's 0 is above no index)
    }
    const int ri = (mode == 0) ? n - 1 - rx : rx;
    w.ss[r] = s;
    w.se[r] = ex;
    w.ip[r] = static_cast<uint16_t>(ri);
    w.sidx[ri] = static_cast<int>(kp[j].y);
    if (r == topk - 1) *w.kth = __uint_as_float(kp[j].x);
  }
  __syncthreads();
  if (tid >= 32) return true;
  if (min_thr > -INFINITY && n > topk && !(quotient_class_floor(*w.kth, Tm) >= min_thr)) return false;
  finish_small_warp<D>(A, row_id, w, n, topk, topp_on, mode, plim, u, dbg, flags);
  return true;
}

}  // namespace gs
