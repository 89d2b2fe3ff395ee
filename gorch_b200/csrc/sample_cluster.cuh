// Cluster kernel: one thread-block cluster (1, 2, 4 or 8 CTAs) per logits row.
//
// Each CTA owns a contiguous slice of the row's 16-byte vectors and keeps it in
// shared memory, so HBM is read exactly once per logit; later passes read shared
// memory. Cross-CTA reductions go through distributed shared memory: a peer
// stores into the consumer's shared memory, then a cluster barrier publishes it.
// Every CTA loads its own slice with plain vector loads.
//
// Row semantics: model/generate.go:134-260 (mode A), model/qwen/generate.go:
// 77-181 (mode B). Per row:
//   greedy         slice argmax -> rank 0 picks (max value, lowest index).
//   top-k <= 256   pass A: slice -> smem, row max, one running max per thread.
//                  The bucket of the k-th largest of those 512 per-thread maxima
//                  bounds the k-th largest logit from below, so pass B (shared
//                  memory) collects a few hundred candidates at most; rank 0
//                  merges the CTAs' lists and finishes them (small_set.cuh).
//   top-k off      L: slice -> smem, max and min.  P2 (only with an active
//                  top-p cut): count histogram over 1024 linear buckets of
//                  d = s - max; rank 0 brackets the cut from count-based mass
//                  bounds.  P3: exponentials; certainly-kept / dropped mass goes
//                  to running sums, the bracketed zone to an exact list that
//                  rank 0 cuts by weighted selection.  The CTA whose slice holds
//                  the drawn token rescans one warp's run.
// Rows that take another way (top-k above 256, a zone or a candidate list that
// outgrows its buffer) are done by rank 0's CTA alone, with the single-CTA
// kernel's routine: no work list, and no second launch that finds it empty.
//
// Bound: latency. A batch of a few rows moves a megabyte or two; what counts is
// the number of dependent steps, the first of which (the slice's copies) is under
// way before the row's configuration has been read.
//
// Control flow is uniform across a cluster: every CTA passes the same cluster
// barriers, and nobody touches a peer's shared memory after the last one.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "sample_kernel.cuh"
#include "small_set.cuh"

namespace gs {
namespace cg = cooperative_groups;

constexpr int CL_MAX = 8;            // largest cluster
constexpr int NB1 = 1024;            // buckets of width 1/32 over d in [-32, 0]
constexpr int ZCAP = 2048;           // exact zone list capacity on rank 0 (entries of 8 B)
constexpr int ZLOC = 1024;           // per-CTA zone list capacity
constexpr int UCAP = 2048;           // merged top-k candidate capacity on rank 0 ...
constexpr int WCAP = 4096;           // ... and with the lists in rank 0's slice (fits the smallest one)
constexpr int LCAP = 2048;           // a rank's own candidates (region B)
constexpr int KFAST = 256;           // largest top_k served here
constexpr int NSUB = 1024;           // sub-buckets of one weighted-selection round
constexpr int REGION_A = 16384;      // bytes: zone keys / merged candidates / histogram staging
constexpr int REGION_B = 16384;      // bytes: local lists, bucket table, selection scratch
constexpr int MIN_SLICE_BYTES = 32768;
static_assert(WCAP * 8 <= MIN_SLICE_BYTES && KEEP_MAX * 8 <= REGION_B && SS_WORK_BYTES <= MIN_SLICE_BYTES &&
              POOL_BYTES <= MIN_SLICE_BYTES + REGION_A + REGION_B, "region sizes");

struct ClusterArgs {
  KernelArgs k;
  int32_t slice_bytes;      // shared bytes reserved for the slice region
  const double* eb_table;   // 1024 doubles: exp(-b/32)
};

// Written by peers through distributed shared memory. Every slot has exactly one
// writer, so nothing here needs to be initialised.
struct Xchg {
  unsigned long long u64[CL_MAX];   // packed (key << 32 | payload) per rank
  float mn[CL_MAX];                 // slice minimum per rank
  double K[CL_MAX], D[CL_MAX], Z[CL_MAX];
  int cnt[CL_MAX];
  int giveup[CL_MAX];
  // pushed by rank 0
  float dA, dB;
  int zone_total;
  int verdict;            // 0 owner resolves, 1 poisoned, 2 rank 0 does the row alone, 3 id written by rank 0
  int owner;
  unsigned long long cut_key;   // zone entries are kept when key < cut_key, or == cut_key with cut_incl
  int cut_incl;
  double local_target, base_mass, Re, S;
};

// 1024 buckets of width 1/32: round(-32 d) clamped to 1023. Non-decreasing as d falls.
__device__ __forceinline__ int bucket1(float d) {
  float f = fmaf(fmaxf(d, -31.97f), -32.0f, 8388608.0f);
  return __float_as_int(f) & 0x7ff;
}

// Smallest d (d <= 0) whose bucket is <= bmax. round(-32 d) <= bmax holds down to
// -(bmax + 1/2)/32, a tie that rounds to even.
__device__ __forceinline__ float bucket_floor(int bmax) {
  if (bmax >= NB1 - 1) return -INFINITY;
  if (bmax < 0) return INFINITY;
  float t = -(static_cast<float>(2 * bmax + 1) * 0.015625f);
  return (bucket1(t) <= bmax) ? t : __uint_as_float(__float_as_uint(t) - 1u);
}

// exp(d), d <= 0, via the 256-entry 2^(j/256) table entirely in f64 (about 1 ulp);
// falls back to the library below -700 and for -Inf / NaN.
__device__ __forceinline__ double exp_safe(float d, const double* __restrict__ tab) {
  if (!(d >= -700.0f)) return exp(static_cast<double>(d));
  const double x = static_cast<double>(d);
  double t = fma(x, 369.3299304675746, 6755399441055744.0);
  int ki = __double2loint(t);
  double kd = t - 6755399441055744.0;
  double r = fma(kd, -0x1.62e42fee00000p-9, x);
  r = fma(kd, -0x1.a39ef35793c76p-41, r);
  double q = fma(r, 4.1666666666666664e-02, 1.6666666666666666e-01);
  q = fma(q, r, 0.5);
  q = fma(q, r, 1.0);
  double tj = tab[ki & 255];
  double res = fma(tj, q * r, tj);
  int hi = __double2hiint(res) + ((ki >> 8) << 20);
  return __hiloint2double(hi, __double2loint(res));
}

// exp(d) for -31.9 < d <= 0: d = -b/32 + dl with |dl| <= 1/64 exactly (f32),
// exp = E[b] * (1 + dl + tail(dl)); the tail dl^2/2 + ... + dl^5/120 is below
// 1.3e-4 and is evaluated in f32, which leaves a relative error near 2e-11.
__device__ __forceinline__ double exp_fast(float d, const double* __restrict__ eb) {
  float f = fmaf(d, -32.0f, 8388608.0f);
  int b = __float_as_int(f) & 0x7ff;
  float dl = fmaf(f - 8388608.0f, 0.03125f, d);
  float t = fmaf(dl, 8.3333338e-3f, 4.1666668e-2f);
  t = fmaf(t, dl, 1.6666667e-1f);
  t = fmaf(t, dl, 0.5f);
  float tail = t * (dl * dl);
  double w = static_cast<double>(dl) + static_cast<double>(tail);
  double E = eb[b];
  return fma(E, w, E);
}

template <typename T> struct Neutral;
template <> struct Neutral<float> { static constexpr uint32_t word = 0xff800000u; };      // -Inf
template <> struct Neutral<uint16_t> { static constexpr uint32_t word = 0xff80ff80u; };   // two bf16 -Inf

// Load vector v of the row; lanes outside [0, V) become -Inf. Max, min and the NaN
// flag cover the valid lanes only.
template <typename T>
__device__ __forceinline__ uint4 mask_and_stats(const RowView<T>& rv, int v, uint4 raw, float& vmax, float& vmin, bool& nan_seen) {
  constexpr int VEC = Elem<T>::VEC;
  float x[VEC];
  Elem<T>::unpack(raw, x);
  if (v > 0 && v < rv.nvec - 1) {
#pragma unroll
    for (int c = 0; c < VEC; c++) {
      vmax = fmaxf(vmax, x[c]);
      vmin = fminf(vmin, x[c]);
      nan_seen |= (x[c] != x[c]);
    }
    return raw;
  }
  uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  const int i0 = v * VEC - rv.shift;
#pragma unroll
  for (int c = 0; c < VEC; c++) {
    int i = i0 + c;
    if (i < 0 || i >= rv.V) {
      if (sizeof(T) == 4) w[c] = 0xff800000u;
      else if (c & 1) w[c >> 1] = (w[c >> 1] & 0x0000ffffu) | 0xff800000u;
      else w[c >> 1] = (w[c >> 1] & 0xffff0000u) | 0x0000ff80u;
    } else {
      vmax = fmaxf(vmax, x[c]);
      vmin = fminf(vmin, x[c]);
      nan_seen |= (x[c] != x[c]);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// The same without the statistics.
template <typename T>
__device__ __forceinline__ uint4 mask_edges(const RowView<T>& rv, int v, uint4 raw) {
  if (v > 0 && v < rv.nvec - 1) return raw;
  constexpr int VEC = Elem<T>::VEC;
  uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  const int i0 = v * VEC - rv.shift;
#pragma unroll
  for (int c = 0; c < VEC; c++) {
    const int i = i0 + c;
    if (i < 0 || i >= rv.V) {
      if (sizeof(T) == 4) w[c] = 0xff800000u;
      else if (c & 1) w[c >> 1] = (w[c >> 1] & 0x0000ffffu) | 0xff800000u;
      else w[c >> 1] = (w[c >> 1] & 0xffff0000u) | 0x0000ff80u;
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// NaN-propagating maximum of a vector's logits.
template <typename T> __device__ __forceinline__ float vec_max_nan(const uint4& a);
template <> __device__ __forceinline__ float vec_max_nan<float>(const uint4& a) {
  float m;
  asm("{\n\t.reg .f32 t;\n\tmax.NaN.f32 t, %1, %2, %3;\n\tmax.NaN.f32 %0, t, %4;\n\t}"
      : "=f"(m) : "f"(__uint_as_float(a.x)), "f"(__uint_as_float(a.y)), "f"(__uint_as_float(a.z)), "f"(__uint_as_float(a.w)));
  return m;
}
template <> __device__ __forceinline__ float vec_max_nan<uint16_t>(const uint4& a) {
  uint32_t p;
  asm("{\n\t.reg .b32 t, u;\n\tmax.NaN.bf16x2 t, %1, %2;\n\tmax.NaN.bf16x2 u, %3, %4;\n\tmax.NaN.bf16x2 %0, t, u;\n\t}"
      : "=r"(p) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w));
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(__uint_as_float(p << 16)), "f"(__uint_as_float(p & 0xffff0000u)));
  return m;
}
// Maximum of a vector's logits; a NaN counts as less than anything else.
template <typename T> __device__ __forceinline__ float vec_max(const uint4& a);
template <> __device__ __forceinline__ float vec_max<float>(const uint4& a) {
  return fmaxf(fmaxf(__uint_as_float(a.x), __uint_as_float(a.y)), fmaxf(__uint_as_float(a.z), __uint_as_float(a.w)));
}
template <> __device__ __forceinline__ float vec_max<uint16_t>(const uint4& a) {
  uint32_t p;
  asm("{\n\t.reg .b32 t, u;\n\tmax.bf16x2 t, %1, %2;\n\tmax.bf16x2 u, %3, %4;\n\tmax.bf16x2 %0, t, u;\n\t}"
      : "=r"(p) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w));
  return fmaxf(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ uint4 load_masked(const RowView<T>& rv, int v, float& vmax, float& vmin, bool& nan_seen) {
  return mask_and_stats(rv, v, __ldg(rv.vbase + v), vmax, vmin, nan_seen);
}

__device__ __forceinline__ void block_min_i2(int& a_min, int& b_min, Ctl& c, int tid) {
  a_min = __reduce_min_sync(FULL, a_min);
  b_min = __reduce_min_sync(FULL, b_min);
  __syncthreads();
  if ((tid & 31) == 0) { c.red_i[tid >> 5] = a_min; c.red_u64[tid >> 5] = static_cast<unsigned long long>(static_cast<uint32_t>(b_min)); }
  __syncthreads();
  const int l = tid & (NW - 1);
  a_min = __reduce_min_sync(FULL, c.red_i[l]);
  b_min = __reduce_min_sync(FULL, static_cast<int>(c.red_u64[l]));
}
__device__ __forceinline__ unsigned long long block_min_u64(unsigned long long v, Ctl& c, int tid) {
  return ~block_max_u64(~v, c, tid);
}

// Exclusive prefix over two doubles per thread at once.
__device__ __forceinline__ void block_scan_excl_d2(double a, double b, double& ea, double& eb_, double& ta, double& tb, Ctl& c, int tid) {
  int lane = tid & 31, w = tid >> 5;
  double ia = warp_scan_incl_d(a, lane), ib = warp_scan_incl_d(b, lane);
  __syncthreads();
  if (lane == 31) { c.red_d[w] = ia; c.red_d2[w] = ib; }
  __syncthreads();
  const double va = (lane < NW) ? c.red_d[lane] : 0.0, vb = (lane < NW) ? c.red_d2[lane] : 0.0;
  const double sa = warp_scan_incl_d(va, lane), sb = warp_scan_incl_d(vb, lane);
  ta = __shfl_sync(FULL, sa, NW - 1); tb = __shfl_sync(FULL, sb, NW - 1);
  ea = __shfl_sync(FULL, sa - va, w) + ia - a;
  eb_ = __shfl_sync(FULL, sb - vb, w) + ib - b;
}

// D: with the optional outputs (probabilities, debug records).
template <typename T, bool D>
__global__ void __launch_bounds__(NT, 2) sample_cluster_kernel(const __grid_constant__ ClusterArgs CA) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ Ctl ctl;
  __shared__ Xchg X;
  __shared__ double s_tab[256];
  __shared__ double s_kseg[NW];
  __shared__ double s_zk[CL_MAX];
  __shared__ uint32_t s_sel[256];

  cg::cluster_group cluster = cg::this_cluster();
  pdl_launch();                       // (the next kernel waits for this one's end by itself)
  pdl_wait();                         // whatever fills the inputs
  // a row whose sequence has ended (model/generate.go:82-84) is skipped by its whole cluster, before any barrier
  if (CA.k.row_done && CA.k.row_done[CA.k.row_offset + blockIdx.x / cluster.num_blocks()] != 0) return;
  cluster.barrier_arrive();          // matched by the wait before the first remote store
  const int C = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const KernelArgs& A = CA.k;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row_id = A.row_offset + blockIdx.x / C;
  const int V = A.V;
  constexpr int VEC = Elem<T>::VEC;
  const T* row = static_cast<const T*>(A.logits) + row_id * A.row_stride;
  RowView<T> rv;
  rv.init(row, V);
  const int SV = (rv.nvec + C - 1) / C;                 // vectors per slice
  const int v0 = min(rv.nvec, rank * SV), v1 = min(rv.nvec, v0 + SV);
  const int nv = v1 - v0;

  uint4* slice = reinterpret_cast<uint4*>(dyn);
  unsigned char* regA = dyn + CA.slice_bytes;
  unsigned char* regB = regA + REGION_A;

  // the slice's copies go out before anything else is read; a thread later looks at the vectors it copied itself
  for (int j = tid; j < nv; j += NT)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :: "r"(static_cast<uint32_t>(__cvta_generic_to_shared(slice + j))), "l"(rv.vbase + v0 + j) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");

  RowCfg cfg;
  if (A.force_greedy) { cfg.temperature = 0.f; cfg.top_k = 0; cfg.top_p = 0.f; cfg.topp_mode = 0; }
  else cfg = A.cfgs[row_id];
  const float Tm = cfg.temperature;
  const double u = A.force_greedy ? 0.0 : A.uniforms[row_id];

  if (tid < CL_MAX) s_zk[tid] = 0.0;
  if (tid == 0) { ctl.cand_count = 0; ctl.overflow = 0; }

  Xchg* X0 = cluster.map_shared_rank(&X, 0);
  const double QNAN = __longlong_as_double(0x7ff8000000000000ll);
  auto finish = [&](int id, uint32_t flags, const RowDebug& dbg) {
    if (tid == 0) {
      A.out_ids[row_id] = id;
      if (A.out_flags) A.out_flags[row_id] = flags;
      if (D && A.out_debug) A.out_debug[row_id] = dbg;
    }
  };
  auto fill_probs_slice = [&](double v) {   // this CTA's share of the dense probability row
    if (D && A.out_probs) {
      double* pr = A.out_probs + row_id * static_cast<int64_t>(V);
      int i_lo = max(0, v0 * VEC - rv.shift), i_hi = min(V, v1 * VEC - rv.shift);
      for (int i = i_lo + tid; i < i_hi; i += NT) pr[i] = v;
    }
  };
  auto fill_probs_row = [&](double v) {
    if (D && A.out_probs) {
      double* pr = A.out_probs + row_id * static_cast<int64_t>(V);
      for (int i = tid; i < V; i += NT) pr[i] = v;
    }
  };
  auto alone = [&]() {                      // rank 0, after the cluster's last barrier: the row from global memory
    __syncthreads();
    single_cta_row<T>(A, row_id, dyn);
  };

  RowDebug dbg;
  dbg.sum_exp = 0; dbg.resum = 1.0; dbg.edge_lo = 0; dbg.edge_hi = 0; dbg.kept = 0;
  dbg.max_scaled = 0; dbg.threshold = __int_as_float(0x7fc00000); dbg.path = 0;
  for (int q = 0; q < 8; q++) dbg.reserved[q] = 0;
  long long tprev = D ? clock64() : 0;
  auto stamp = [&](int slot) {
    if (D) { const long long now = clock64(); dbg.reserved[slot] = static_cast<uint32_t>(now - tprev); tprev = now; }
  };

  // ================================================================ greedy
  if (Tm == 0.0f) {
    // per vector a maximum and one compare (a NaN is not seen); the place within the vector at the end
    float top = -INFINITY;
    int tv = 0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    for (int j = tid; j < nv; j += NT) {
      const float x = vec_max<T>(mask_edges(rv, v0 + j, slice[j]));
      if (x > top) { top = x; tv = v0 + j; }
    }
    unsigned long long best = (top > -INFINITY) ? (static_cast<unsigned long long>(okey(top)) << 32) | static_cast<uint32_t>(~static_cast<uint32_t>(tv)) : 0ull;
    best = block_max_u64(best, ctl, tid);
    fill_probs_slice(0.0);
    cluster.barrier_wait();
    if (tid == 0) X0->u64[rank] = best;
    cluster.sync();
    if (rank == 0) {
      unsigned long long b = 0;
      for (int r = 0; r < C; r++) b = X.u64[r] > b ? X.u64[r] : b;
      int id = 0x7fffffff;
      if (b != 0ull)
        rv.visit(static_cast<int>(~static_cast<uint32_t>(b & 0xffffffffull)), [&](float x, int i) { if (okey(x) == static_cast<uint32_t>(b >> 32)) id = min(id, i); });
      if (id == 0x7fffffff) id = 0;                          // nothing above -Inf: no logit beats the first one
      float x0 = 0.f;
      rv.visit(0, [&](float x, int i) { if (i == 0) x0 = x; });
      if (x0 != x0) id = 0;     // generate.go:136: maxVal starts as NaN, nothing is greater
      if (D && A.out_probs && tid == 0) A.out_probs[row_id * static_cast<int64_t>(V) + id] = 1.0;
      dbg.kept = 1;
      finish(id, 0u, dbg);
    }
    return;
  }
  if (!(Tm > 0.0f) || !(Tm < INFINITY)) {
    fill_probs_slice(QNAN);
    if (rank == 0) finish(-1, FLAG_BAD_CFG, dbg);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    cluster.barrier_wait();
    return;
  }

  const int topk = (cfg.top_k > 0 && cfg.top_k < V) ? cfg.top_k : 0;
  const bool topp_on = (cfg.top_p > 0.0f && cfg.top_p < 1.0f);
  const int mode = cfg.topp_mode;
  const double plim = (mode == 0) ? static_cast<double>(cfg.top_p) * 1.5 : static_cast<double>(cfg.top_p);
  const bool cut_on = topp_on && !(mode == 0 && plim >= 1.0);
  const bool t_is_one = (Tm == 1.0f);
  uint32_t flags = 0;

  if (topk > KFAST) {
    // large top-k: the single-CTA kernel's counting select serves it
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    cluster.barrier_wait();
    if (rank == 0) alone();
    return;
  }

  // ---- L / pass A: the slice in shared memory; max, min, NaN, one running max per thread
  // (the tables' words are on their way before they are wanted: a trip to L2 in front of the bracket and one in front of the
  // exponentials otherwise)
  const double tab_me = (topk == 0 && tid < 256) ? A.exp_table[tid] : 0.0;
  const double2 eb_me = (topk == 0) ? __ldg(reinterpret_cast<const double2*>(CA.eb_table) + tid) : make_double2(0.0, 0.0);
  float xmax = -INFINITY, xmin = INFINITY;
  bool nan_seen = false;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (topk > 0) {
    // a top-k row needs the maxima only: a few packed instructions per vector
    for (int j = tid; j < nv; j += NT) {
      const int v = v0 + j;
      uint4 raw = slice[j];
      if (v == 0 || v >= rv.nvec - 1) { raw = mask_edges(rv, v, raw); slice[j] = raw; }
      const float m = vec_max_nan<T>(raw);
      nan_seen |= (m != m);
      xmax = fmaxf(xmax, m);                                 // (a NaN poisons the row: what its vector's maximum would be is no matter)
    }
  } else
  for (int j = tid; j < nv; j += NT) {
    const int v = v0 + j;
    const uint4 raw = slice[j];
    const uint4 masked = mask_and_stats(rv, v, raw, xmax, xmin, nan_seen);
    if (v == 0 || v >= rv.nvec - 1) slice[j] = masked;
  }
  if (topk == 0 && tid < 256) s_tab[tid] = tab_me;

  // ======================================================= top-k, k <= 256
  if (topk > 0) {
    // thr0: a lower bound of the k-th largest logit = lower edge of the bucket (256 of them over the range
    // of the order keys) that holds the k-th largest of the 512 per-thread maxima.
    const uint32_t mykey = okey(xmax);
    uint32_t klo = __reduce_min_sync(FULL, mykey), khi = __reduce_max_sync(FULL, mykey);
    const unsigned nanw = __ballot_sync(FULL, nan_seen);
    if (tid < 256) s_sel[tid] = 0u;
    if (lane == 0) { ctl.red_u64[warp] = (static_cast<unsigned long long>(khi) << 32) | klo; ctl.red_i[warp] = nanw ? 1 : 0; }
    if (tid == 0) ctl.bcast_i[0] = 0;
    __syncthreads();                                         // every slice is complete too
    {
      const unsigned long long w = ctl.red_u64[lane & (NW - 1)];
      klo = __reduce_min_sync(FULL, static_cast<uint32_t>(w));
      khi = __reduce_max_sync(FULL, static_cast<uint32_t>(w >> 32));
    }
    const int anynan_loc = __reduce_max_sync(FULL, ctl.red_i[lane & (NW - 1)]);
    const unsigned long long pmax = static_cast<unsigned long long>(khi) << 32;
    const int bsh = max(0, 24 - __clz(khi - klo));
    atomicAdd(&s_sel[(khi - mykey) >> bsh], 1u);
    __syncthreads();
    if (tid < 32) {
      int loc[8], s = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) { s += static_cast<int>(s_sel[tid * 8 + j]); loc[j] = s; }
      int run = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(FULL, run, o); if (tid >= o) run += t; }
      const int before = run - s;
      if (before < topk && run >= topk) {
        int b = 0;
#pragma unroll
        for (int j = 7; j >= 0; j--) if (before + loc[j] >= topk) b = tid * 8 + j;
        const uint32_t top = khi - (static_cast<uint32_t>(b) << bsh), width = (1u << bsh) - 1u;
        const uint32_t edge = (top - klo > width) ? top - width : klo;
        ctl.thr = (edge > 0x007fffffu) ? quotient_class_floor(okey_to_float(edge), Tm) : -INFINITY;   // at or below -Inf: keep everything
        ctl.bcast_i[0] = 1;
      }
    }
    __syncthreads();
    const float thr0 = ctl.bcast_i[0] ? ctl.thr : -INFINITY;  // (fewer than k groups: keep everything)
    // pass B: candidates >= thr0 from shared memory
    uint2* lc = reinterpret_cast<uint2*>(regB);              // LCAP entries
    for (int j = tid; j < nv; j += NT) {
      const uint4 raw = slice[j];
      if (!(vec_max_nan<T>(raw) >= thr0)) continue;
      float x[VEC];
      Elem<T>::unpack(raw, x);
      const int i0 = (v0 + j) * VEC - rv.shift;
      uint32_t hits = 0u;
#pragma unroll
      for (int c = 0; c < VEC; c++) hits |= (x[c] >= thr0 && static_cast<uint32_t>(i0 + c) < static_cast<uint32_t>(V)) ? 1u << c : 0u;
      int slot = atomicAdd(&ctl.cand_count, __popc(hits));
      const T* src = reinterpret_cast<const T*>(slice + j);
      for (; hits; hits &= hits - 1, slot++) {
        const int c = __ffs(hits) - 1;
        if (slot < LCAP) lc[slot] = make_uint2(__float_as_uint(Elem<T>::to_float(src[c])), static_cast<uint32_t>(i0 + c));
      }
    }
    if (tid < 256) s_sel[tid] = 0u;                          // narrow_candidates wants it cleared (and a count: ctl.overflow still is)
    __syncthreads();
    // Where the lists meet: rank 0's region A while UCAP entries are enough for all ranks; a larger top_k takes
    // rank 0's slice, after one more barrier that says that rank 0 is through with it.
    const bool wide_lists = topk * C > UCAP / 2;             // uniform over the cluster
    const int cap_r = wide_lists ? WCAP / C : UCAP / C;
    int n_loc = ctl.cand_count, n_most = cap_r;              // what this rank has, and may send
    if (n_loc > cap_r && n_loc <= LCAP) {                    // more than this rank's share: only what can be kept
      uint2* few = reinterpret_cast<uint2*>(dyn);            // (the slice has been read; peers may already write to region A)
      n_loc = narrow_list<NT>(lc, n_loc, topk, Tm, okey(thr0), khi, few, s_sel, ctl.bcast_i, &ctl.cand_count, tid);
      n_most = min(cap_r, KEEP_MAX);                         // (a larger count is of ties that are not all there; two CTAs' share is 1024)
      for (int j = tid; j < min(n_loc, KEEP_MAX); j += NT) lc[j] = few[j];
      if (tid < 256) s_sel[tid] = 0u;
      __syncthreads();
    }
    const bool giveup = n_loc > min(n_most, LCAP);
    stamp(1);
    cluster.barrier_wait();
    if (wide_lists) cluster.sync();
    if (tid == 0) {
      X0->u64[rank] = pmax | static_cast<unsigned long long>(anynan_loc);
      X0->cnt[rank] = giveup ? 0 : n_loc;
      X0->giveup[rank] = giveup ? 1 : 0;
    }
    if (!giveup) {
      uint2* dst = cluster.map_shared_rank(reinterpret_cast<uint2*>(wide_lists ? dyn : regA), 0) + rank * cap_r;
      for (int j = tid; j < n_loc; j += NT) dst[j] = lc[j];
    }
    cluster.sync();                                          // B1: the last barrier of this path
    if (rank != 0) return;
    stamp(2);
    // ---------------- rank 0: merge and finish in shared memory
    dbg.path = 1;
    unsigned long long mx = 0;
    int anynan = 0, bad = 0, n = 0;
    for (int r = 0; r < C; r++) {
      mx = X.u64[r] > mx ? X.u64[r] : mx;
      anynan |= static_cast<int>(X.u64[r] & 1ull);
      bad |= X.giveup[r];
      n += X.cnt[r];
    }
    if (bad) { alone(); return; }
    xmax = okey_to_float(static_cast<uint32_t>(mx >> 32));
    const float m = scale_t(xmax, Tm);
    dbg.max_scaled = m;
    if (anynan || !(fabsf(m) < INFINITY)) {
      fill_probs_row(QNAN);
      dbg.sum_exp = QNAN;
      finish(V - 1, flags | FLAG_NONFINITE | FLAG_FALLBACK, dbg);
      return;
    }
    const uint2* lists = reinterpret_cast<const uint2*>(wide_lists ? dyn : regA);
    const int caplog = 31 - __clz(cap_r);                    // a power of two
    constexpr int PER = WCAP / NT;
    uint2 mine[PER];                                         // this thread's entries; (x: NaN) where there is none
#pragma unroll
    for (int q = 0; q < PER; q++) {
      const int j = q * NT + tid;
      const bool there = j < (C << caplog) && (j & (cap_r - 1)) < X.cnt[j >> caplog];
      mine[q] = there ? lists[j] : make_uint2(0x7fc00000u, 0u);
    }
    auto each = [&](auto&& f) {
#pragma unroll
      for (int q = 0; q < PER; q++) if (mine[q].x != 0x7fc00000u) f(mine[q]);
    };
    uint2* kp = reinterpret_cast<uint2*>(regB);               // the local list is done with
    const int nk = narrow_candidates<NT>(each, n, topk, Tm, okey(thr0), static_cast<uint32_t>(mx >> 32), kp, s_sel, ctl.bcast_i,
                                         &ctl.overflow, tid);
    if (nk > KEEP_MAX) { alone(); return; }                  // long run of ties at the threshold
    finish_small_set<NT, D>(A, row_id, kp, nk, topk, m, Tm, topp_on, mode, plim, u, -INFINITY, dyn, D ? &dbg : nullptr, flags);
    return;
  }

  // ============================================================ full row (top-k off)
  dbg.path = 2;
  flags |= FLAG_GENERAL_PATH;
  {
    uint32_t khi = __reduce_max_sync(FULL, okey(xmax)), klo = __reduce_min_sync(FULL, okey(xmin));
    const unsigned nanw = __ballot_sync(FULL, nan_seen);
    if (lane == 0) { ctl.red_u64[warp] = (static_cast<unsigned long long>(khi) << 32) | klo; ctl.red_i[warp] = nanw ? 1 : 0; }
    __syncthreads();                                         // every slice is complete too
    const unsigned long long w = ctl.red_u64[lane & (NW - 1)];
    khi = __reduce_max_sync(FULL, static_cast<uint32_t>(w >> 32));
    klo = __reduce_min_sync(FULL, static_cast<uint32_t>(w));
    const int anynan_loc = __reduce_max_sync(FULL, ctl.red_i[lane & (NW - 1)]);
    stamp(0);
    cluster.barrier_wait();
    if (tid < C) {                                           // one thread per receiver, here and below
      Xchg* xr = cluster.map_shared_rank(&X, tid);
      xr->u64[rank] = (static_cast<unsigned long long>(khi) << 32) | static_cast<unsigned long long>(anynan_loc);
      xr->mn[rank] = okey_to_float(klo);
    }
  }
  cluster.sync();                                            // G1
  stamp(1);
  float row_min = INFINITY;
  int anynan = 0;
  {
    unsigned long long mx = 0;
    for (int r = 0; r < C; r++) {
      mx = X.u64[r] > mx ? X.u64[r] : mx;
      anynan |= static_cast<int>(X.u64[r] & 1ull);
      row_min = fminf(row_min, X.mn[r]);
    }
    xmax = okey_to_float(static_cast<uint32_t>(mx >> 32));
  }
  const float m = scale_t(xmax, Tm);
  dbg.max_scaled = m;
  const bool poisoned_early = anynan || !(fabsf(m) < INFINITY);
  // every element has d > -31.9: the bucket-table exponential applies
  const bool fast_ok = !poisoned_early && (scale_t(row_min, Tm) - m > -31.9f);

  // ---- P2: count histogram + bracket of the top-p cut
  float dA = -INFINITY, dB = -INFINITY;    // certainly kept: d >= dA; zone: dB <= d < dA; dropped: d < dB
  int nzone = 0;
  if (cut_on) {
    uint32_t* hist = (rank == 0) ? reinterpret_cast<uint32_t*>(regA) : reinterpret_cast<uint32_t*>(regB);
    for (int j = tid; j < NB1; j += NT) hist[j] = 0;
    __syncthreads();
    for (int j = tid; j < nv; j += NT) {
      float x[VEC];
      Elem<T>::unpack(slice[j], x);
      if (t_is_one) {
#pragma unroll
        for (int c = 0; c < VEC; c++) atomicAdd(&hist[bucket1(x[c] - m)], 1u);
      } else {
#pragma unroll
        for (int c = 0; c < VEC; c++) atomicAdd(&hist[bucket1(__fdiv_rn(x[c], Tm) - m)], 1u);
      }
    }
    __syncthreads();
    if (rank != 0) {
      // rank 0 stages [C][1024] counters across its regions A and B (32 KB at C = 8)
      uint32_t* dst = cluster.map_shared_rank(reinterpret_cast<uint32_t*>(regA), 0) + rank * NB1;
      for (int j = tid; j < NB1; j += NT) dst[j] = hist[j];
    }
    stamp(2);
    cluster.sync();                                          // G2
    if (rank == 0) {
      const uint32_t* all = reinterpret_cast<const uint32_t*>(regA);
      constexpr int PER = NB1 / NT;                          // 2 buckets per thread: those of eb_me
      static_assert(PER == 2, "eb_me");
      double lo_inc[PER], hi_inc[PER];
      int cb[PER];
      double slo = 0.0, shi = 0.0;
#pragma unroll
      for (int j = 0; j < PER; j++) {
        const int b = tid * PER + j;
        uint32_t cnt = 0;
        for (int r = 0; r < C; r++) cnt += all[r * NB1 + b];
        cb[j] = static_cast<int>(cnt);
        const double c = static_cast<double>(cnt);
        // bucket b holds d in [-(b+.5)/32, -(b-.5)/32]; the last one everything below.
        // Masked lanes (-Inf) are counted there too; their mass bound starts at 0.
        const double eb = (j == 0) ? eb_me.x : eb_me.y;
        const double elo = (b == NB1 - 1) ? 0.0 : eb * 0.98449643700540845 * (1.0 - 1e-7);   // exp(-1/64)
        const double ehi = fmin(1.0, eb * 1.0157477085866857 * (1.0 + 1e-7));                 // exp(+1/64)
        slo += c * elo; shi += c * ehi;
        lo_inc[j] = slo; hi_inc[j] = shi;
      }
      double ex_lo, ex_hi, tot_lo, tot_hi;
      block_scan_excl_d2(slo, shi, ex_lo, ex_hi, tot_lo, tot_hi, ctl, tid);
      int b1 = NB1 - 1, b2 = NB1 - 1;
#pragma unroll
      for (int j = 0; j < PER; j++) {
        const int b = tid * PER + j;
        const double a_lo = ex_lo + lo_inc[j], a_hi = ex_hi + hi_inc[j];
        // largest and smallest possible mass fraction through bucket b, against the limit
        const double l_hi = plim * (1.0 - 1e-9) * (a_hi + (tot_lo - a_lo)), l_lo = plim * (1.0 + 1e-9) * (a_lo + (tot_hi - a_hi));
        const bool c1 = (mode == 0) ? a_hi > l_hi : a_hi >= l_hi, c2 = (mode == 0) ? a_lo > l_lo : a_lo >= l_lo;
        if (c1) b1 = min(b1, b);
        if (c2) b2 = min(b2, b);
      }
      block_min_i2(b1, b2, ctl, tid);
      if (b2 < b1) b2 = b1;
      int nz_part = 0;
#pragma unroll
      for (int j = 0; j < PER; j++) {
        const int b = tid * PER + j;
        if (b >= b1 && b <= b2) nz_part += cb[j];
      }
      const int nz = block_sum_i(nz_part, ctl, tid);
      if (tid < C) {
        Xchg* xr = cluster.map_shared_rank(&X, tid);
        xr->dA = bucket_floor(b1 - 1); xr->dB = bucket_floor(b2); xr->zone_total = nz;
      }
    }
    stamp(3);
    cluster.sync();                                          // G3
    dA = X.dA; dB = X.dB; nzone = X.zone_total;
    if (nzone > NT) {                                        // uniform over the cluster
      // The counts alone leave an uncertain mass of some 3 % around the cut, and in a large or flat vocabulary
      // that is more logits than the list holds. Now the zone's own range of d is cut into 1024 buckets, and the
      // masses on either side of it are summed (f32 exponentials, good to 1e-6; the bounds allow 1e-5): the zone
      // that remains is a few buckets, tens of logits. One more look at the slice (shared memory) and two more
      // barriers, where the row used to be left to the single-CTA routine (151,936 logits, sigma 2, p = 0.9, eight
      // CTAs: 376 us).
      const uint32_t klo = (dA == INFINITY) ? 0u : dkey_of(dA) + 1u, khi = (dB == -INFINITY) ? 0x7f7fffffu : dkey_of(dB);
      const int ksh = max(0, 22 - __clz(khi - klo));         // (khi - klo) >> ksh < 1024
      uint32_t* fine = (rank == 0) ? reinterpret_cast<uint32_t*>(regA) : reinterpret_cast<uint32_t*>(regB);
      __syncthreads();
      for (int j = tid; j < NB1; j += NT) fine[j] = 0;
      __syncthreads();
      float ks = 0.f, zs = 0.f, ds = 0.f;
      for (int j = tid; j < nv; j += NT) {
        float x[VEC];
        Elem<T>::unpack(slice[j], x);
#pragma unroll
        for (int c = 0; c < VEC; c++) {
          const float d = (t_is_one ? x[c] : __fdiv_rn(x[c], Tm)) - m;
          float e;
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(d * 1.44269502162933349609375f));
          if (d >= dA) ks += e;
          else if (d >= dB && d > -INFINITY) { zs += e; atomicAdd(&fine[(dkey_of(d) - klo) >> ksh], 1u); }
          else ds += e;
        }
      }
      const double kw = warp_sum_d(ks), rw = warp_sum_d(static_cast<double>(zs) + ds);
      if (lane == 0) { ctl.red_d[warp] = kw; ctl.red_d2[warp] = rw; }
      __syncthreads();
      if (warp == 0) {
        const double kr = warp_sum_d(lane < NW ? ctl.red_d[lane] : 0.0), sr = warp_sum_d(lane < NW ? ctl.red_d2[lane] : 0.0);
        if (lane == 0) { X0->K[rank] = kr; X0->Z[rank] = sr; }
      }
      if (rank != 0) {
        uint32_t* dst = cluster.map_shared_rank(reinterpret_cast<uint32_t*>(regA), 0) + rank * NB1;
        for (int j = tid; j < NB1; j += NT) dst[j] = fine[j];
      }
      cluster.sync();
      if (rank == 0) {
        const uint32_t* all = reinterpret_cast<const uint32_t*>(regA);
        double K = 0.0, S = 0.0;
        for (int r = 0; r < C; r++) { K += X.K[r]; S += X.K[r] + X.Z[r]; }
        const double lim_lo = plim * S * (1.0 - 1e-5), lim_hi = plim * S * (1.0 + 1e-5);
        constexpr int PER = NB1 / NT;
        double lo_inc[PER], hi_inc[PER], slo = 0.0, shi = 0.0;
        int cb[PER];
        auto key_at = [&](int b) { return klo + (static_cast<uint32_t>(b) << ksh); };
#pragma unroll
        for (int j = 0; j < PER; j++) {
          const int b = tid * PER + j;
          uint32_t cnt = 0;
          for (int r = 0; r < C; r++) cnt += all[r * NB1 + b];
          cb[j] = static_cast<int>(cnt);
          if (cnt) {
            shi += cnt * exp_safe(-__uint_as_float(key_at(b)), s_tab);
            slo += cnt * exp_safe(-__uint_as_float(min(key_at(b + 1) - 1u, khi)), s_tab);
          }
          lo_inc[j] = slo; hi_inc[j] = shi;
        }
        double ex_lo, ex_hi, tot_lo, tot_hi;
        block_scan_excl_d2(slo, shi, ex_lo, ex_hi, tot_lo, tot_hi, ctl, tid);
        int b1 = NB1 - 1, b2 = NB1 - 1;
#pragma unroll
        for (int j = PER - 1; j >= 0; j--) {
          // largest and smallest possible mass through the bucket, against the limit
          const double a_hi = K * (1.0 + 1e-5) + ex_hi + hi_inc[j], a_lo = K * (1.0 - 1e-5) + ex_lo + lo_inc[j];
          const bool c1 = (mode == 0) ? a_hi > lim_lo : a_hi >= lim_lo, c2 = (mode == 0) ? a_lo > lim_hi : a_lo >= lim_hi;
          if (c1) b1 = tid * PER + j;
          if (c2) b2 = tid * PER + j;
        }
        block_min_i2(b1, b2, ctl, tid);
        b2 = max(b1, b2);
        int nz_part = 0;
#pragma unroll
        for (int j = 0; j < PER; j++) if (tid * PER + j >= b1 && tid * PER + j <= b2) nz_part += cb[j];
        const int nz = block_sum_i(nz_part, ctl, tid);
        if (tid < C) {
          const float tA = (key_at(b1) == 0u) ? INFINITY : -__uint_as_float(key_at(b1) - 1u);
          const float tB = (b2 == NB1 - 1 || key_at(b2 + 1) > khi) ? dB : -__uint_as_float(key_at(b2 + 1) - 1u);
          Xchg* xr = cluster.map_shared_rank(&X, tid);
          xr->dA = tA; xr->dB = tB; xr->zone_total = nz;
        }
      }
      cluster.sync();
      dA = X.dA; dB = X.dB; nzone = X.zone_total;
      stamp(7);
    }
  }
  // the zone count includes masked lanes when the zone reaches the last bucket; they are never listed
  const bool zone_ok = nzone <= ZCAP + 2 * VEC;

  // ---- P3: exponentials. Each warp owns a contiguous run of the slice; eight elements in flight.
  double* ebs = reinterpret_cast<double*>(regB + 8192);     // bucket table exp(-b/32), 8 KB
  uint2* lz = reinterpret_cast<uint2*>(regB);               // local zone list (d bits, idx), 1024 entries
  __syncthreads();
  if (fast_ok) reinterpret_cast<double2*>(ebs)[tid] = eb_me;
  if (tid == 0) ctl.cand_count = 0;
  __syncthreads();
  const int wv = (nv + NW - 1) / NW;                        // vectors per warp run
  const int w0 = min(nv, warp * wv), w1 = min(nv, w0 + wv);
  double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0, dsum = 0.0, zsum = 0.0;
  if (zone_ok) {
    auto body = [&](auto fast_tag, auto tone_tag) {
      constexpr bool FAST = decltype(fast_tag)::value;
      constexpr bool TONE = decltype(tone_tag)::value;
      constexpr int U = (VEC == 4) ? 2 : 1;                  // vectors per iteration: 8 elements
      for (int j = w0 + lane; j < w1; j += 32 * U) {
        float x[8];
        uint4 ra = slice[j];
        if (U == 2) {
          uint4 rb = (j + 32 < w1) ? slice[j + 32]
                                   : make_uint4(Neutral<T>::word, Neutral<T>::word, Neutral<T>::word, Neutral<T>::word);
          float xa[VEC], xb[VEC];
          Elem<T>::unpack(ra, xa);
          Elem<T>::unpack(rb, xb);
#pragma unroll
          for (int c = 0; c < 4; c++) { x[c] = xa[c]; x[4 + c] = xb[c]; }
        } else {
          float xa[VEC];
          Elem<T>::unpack(ra, xa);
#pragma unroll
          for (int c = 0; c < 8; c++) x[c] = xa[c % VEC];
        }
        double e[8];
        float d[8];
        float dmin = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const float s = TONE ? x[c] : __fdiv_rn(x[c], Tm);
          d[c] = s - m;
          if (FAST) e[c] = (d[c] > -31.9f) ? exp_fast(d[c], ebs) : 0.0;   // only masked lanes (-Inf) are below
          else      e[c] = exp_safe(d[c], s_tab);
          dmin = fminf(dmin, d[c]);
        }
        t0 += e[0] + e[4]; t1 += e[1] + e[5]; t2 += e[2] + e[6]; t3 += e[3] + e[7];
        if (dmin < dA) {
#pragma unroll
          for (int c = 0; c < 8; c++) {
            if (d[c] < dA) {
              if (d[c] >= dB) {
                const int jj = (U == 2 && c >= 4) ? j + 32 : j;
                const int i = (v0 + jj) * VEC - rv.shift + ((U == 2) ? (c & 3) : c);
                if (jj < w1 && i >= 0 && i < V) {
                  const int slot = atomicAdd(&ctl.cand_count, 1);
                  if (slot < ZLOC) lz[slot] = make_uint2(__float_as_uint(d[c]), static_cast<uint32_t>(i));
                  zsum += e[c];
                }
              } else {
                dsum += e[c];
              }
            }
          }
        }
      }
    };
    if (fast_ok) { if (t_is_one) body(std::true_type{}, std::true_type{}); else body(std::true_type{}, std::false_type{}); }
    else         { if (t_is_one) body(std::false_type{}, std::true_type{}); else body(std::false_type{}, std::false_type{}); }
  }
  const double tot_w = warp_sum_d((t0 + t1) + (t2 + t3));
  dsum = warp_sum_d(dsum); zsum = warp_sum_d(zsum);
  // certainly-kept mass of this warp's run. With dA = +Inf nothing is certainly kept (exactly 0);
  // otherwise the row maximum is, and the subtraction's rounding is far below that mass.
  const double kw = (dA == INFINITY) ? 0.0 : tot_w - dsum - zsum;
  if (lane == 0) { s_kseg[warp] = kw; ctl.red_d[warp] = dsum; ctl.red_d2[warp] = zsum; }
  __syncthreads();
  double Kr = 0.0, Dr = 0.0, Zr = 0.0;                       // the slice's masses, in the first warp
  if (warp == 0) {
    Kr = warp_sum_d(lane < NW ? s_kseg[lane] : 0.0);
    Dr = warp_sum_d(lane < NW ? ctl.red_d[lane] : 0.0);
    Zr = warp_sum_d(lane < NW ? ctl.red_d2[lane] : 0.0);
  }
  const int nz_cta = ctl.cand_count;
  // Rank r owns the sub-range [r*ZCAP/C, (r+1)*ZCAP/C) of rank 0's region A.
  const int zcap_r = ZCAP / C;
  const int zlog = 31 - __clz(zcap_r);
  const bool z_over = nz_cta > min(ZLOC, zcap_r);
  const int nz_loc = z_over ? 0 : nz_cta;
  if (tid == 0) {
    X0->K[rank] = Kr; X0->D[rank] = Dr; X0->Z[rank] = Zr;
    X0->cnt[rank] = nz_loc;
    X0->giveup[rank] = (z_over || !zone_ok) ? 1 : 0;
  }
  {
    unsigned long long* dst = cluster.map_shared_rank(reinterpret_cast<unsigned long long*>(regA), 0) + rank * zcap_r;
    for (int j = tid; j < nz_loc; j += NT) {
      const uint2 e = lz[j];
      dst[j] = zone_key(__uint_as_float(e.x), static_cast<int>(e.y), mode);
    }
  }
  stamp(4);
  cluster.sync();                                            // G4
  stamp(5);

  // ---- rank 0: exact cut inside the zone by weighted selection, then the owner of the draw
  if (rank == 0) {
    double Ktot = 0, Dtot = 0, Ztot = 0;
    int bad = 0, nz = 0;
    for (int r = 0; r < C; r++) { Ktot += X.K[r]; Dtot += X.D[r]; Ztot += X.Z[r]; bad |= X.giveup[r]; nz += X.cnt[r]; }
    const double S = Ktot + Ztot + Dtot;
    dbg.sum_exp = S;
    const bool poisoned = poisoned_early || !(S == S) || !(S > 0.0);
    const unsigned long long* zk = reinterpret_cast<const unsigned long long*>(regA);
    // zone entry t of the staged list is live when it lies inside its rank's filled part
    auto zlive = [&](int t) -> bool { return (t & (zcap_r - 1)) < X.cnt[t >> zlog]; };
    unsigned long long cut_key = 0ull;     // nothing of the zone kept
    int cut_incl = 0;
    if (cut_on && !poisoned && !bad && nz > 0) {
      // G(c) = Ktot + mass{key <= c} rises along the zone order. Both flavours need the first
      // key c* where G "crosses": mode B (first G/S >= p) keeps through c*, mode A (first
      // G/S > 1.5p) keeps everything before it. Narrow [lo, hi] around c* with linear
      // sub-buckets until at most 32 keys remain, then one warp finishes.
      auto crossed = [&](double g) -> bool { return mode == 0 ? (g / S > plim) : (g / S >= plim); };
      if (Ktot > 0.0 && crossed(Ktot)) bad = 1;              // the bracket was wrong
      double* sm = reinterpret_cast<double*>(regB);           // [NSUB] mass per sub-bucket
      int* sc = reinterpret_cast<int*>(regB + 8192);          // [NSUB] count per sub-bucket
      const bool few_keys = nz <= NT;                          // uniform
      unsigned long long lo = ~0ull, hi = 0ull;
      if (!few_keys) {
        for (int t = tid; t < ZCAP; t += NT) {
          if (zlive(t)) { const unsigned long long k = zk[t]; lo = k < lo ? k : lo; hi = k > hi ? k : hi; }
        }
        lo = block_min_u64(lo, ctl, tid);
        hi = block_max_u64(hi, ctl, tid);
      }
      double gbase = Ktot;                                     // Ktot + mass of keys below lo; never crossed
      int inrange = nz;
      bool all_in = false;
      for (int iter = 0; iter < 8 && !few_keys && inrange > 32 && !bad && !all_in; iter++) {
        const unsigned long long span = hi - lo;
        int sh = 0;
        while (sh < 63 && (span >> sh) >= static_cast<unsigned long long>(NSUB)) sh++;
        __syncthreads();
        for (int j = tid; j < NSUB; j += NT) { sm[j] = 0.0; sc[j] = 0; }
        __syncthreads();
        for (int t = tid; t < ZCAP; t += NT) {
          if (zlive(t)) {
            const unsigned long long k = zk[t];
            if (k >= lo && k <= hi) {
              const int sb = static_cast<int>((k - lo) >> sh);
              atomicAdd(&sm[sb], exp_safe(zone_key_d(k), s_tab));
              atomicAdd(&sc[sb], 1);
            }
          }
        }
        __syncthreads();
        constexpr int PER = NSUB / NT;
        double inc[PER];
        double s = 0.0;
#pragma unroll
        for (int j = 0; j < PER; j++) { s += sm[tid * PER + j]; inc[j] = s; }
        double totm;
        const double exm = block_scan_excl_d(s, totm, ctl, tid);
        int first = NSUB;
#pragma unroll
        for (int j = 0; j < PER; j++) {
          if (first == NSUB && sc[tid * PER + j] > 0 && crossed(gbase + exm + inc[j])) first = tid * PER + j;
        }
        const int sbx = block_min_i(first, ctl, tid);
        if (sbx == NSUB) { all_in = true; break; }
        if (tid == sbx / PER) {
          const int j = sbx % PER;
          ctl.bcast_d[0] = gbase + exm + (j > 0 ? inc[j - 1] : 0.0);
          ctl.bcast_i[0] = sc[sbx];
        }
        __syncthreads();
        gbase = ctl.bcast_d[0];
        inrange = ctl.bcast_i[0];
        const unsigned long long nlo = lo + (static_cast<unsigned long long>(sbx) << sh);
        unsigned long long nhi = nlo + ((1ull << sh) - 1ull);
        if (nhi < nlo || nhi > hi) nhi = hi;
        lo = nlo; hi = nhi;
      }
      if (!few_keys && inrange > 32 && !all_in) bad = 1;
      double g_at = gbase;                                     // G(c*) and G just before c*
      double g_before = gbase;
      if (few_keys && !bad) {
        // Every key adds up the masses that come no later than its own, all at once: a few thousand cycles
        // for some hundred keys, where narrowing the range takes several rounds of barriers and f64
        // atomics (151,936 logits, sigma 2, p = 0.9, mode B: 31,000 cycles, 16 us).
        unsigned long long* zkeys = reinterpret_cast<unsigned long long*>(regB);
        double* zmass = reinterpret_cast<double*>(regB + 8 * NT);
        __syncthreads();
        int src = -1;                                          // thread t takes the t-th live entry
        for (int r = 0, off = 0; r < C; r++) { const int c = X.cnt[r]; if (tid >= off && tid < off + c) src = r * zcap_r + tid - off; off += c; }
        unsigned long long k = ~0ull;
        if (src >= 0) { k = zk[src]; zkeys[tid] = k; zmass[tid] = exp_safe(zone_key_d(k), s_tab); }
        __syncthreads();
        double g = 0.0, g2 = 0.0;
        if (tid < nz) {
          int l = 0;
#pragma unroll 2
          for (; l + 1 < nz; l += 2) {
            g += (zkeys[l] <= k) ? zmass[l] : 0.0;
            g2 += (zkeys[l + 1] <= k) ? zmass[l + 1] : 0.0;
          }
          if (l < nz) g += (zkeys[l] <= k) ? zmass[l] : 0.0;
          g = Ktot + (g + g2);
        }
        const bool cr = tid < nz && crossed(g);
        const unsigned long long cstar = block_min_u64(cr ? k : ~0ull, ctl, tid);
        if (cr && k == cstar) { ctl.bcast_d[1] = g; ctl.bcast_d[2] = g - zmass[tid]; }   // keys are distinct
        __syncthreads();
        if (cstar != ~0ull) {
          g_at = ctl.bcast_d[1];
          g_before = ctl.bcast_d[2];
          cut_key = cstar;
          cut_incl = (mode == 0) ? 0 : 1;
        } else {
          all_in = true;                                       // nothing in the zone crosses
        }
      } else if (!bad && !all_in) {
        unsigned long long* few = reinterpret_cast<unsigned long long*>(regB);   // [32]
        __syncthreads();
        if (tid == 0) ctl.cand_count = 0;
        __syncthreads();
        for (int t = tid; t < ZCAP; t += NT) {
          if (zlive(t)) {
            const unsigned long long k = zk[t];
            if (k >= lo && k <= hi) { const int slot = atomicAdd(&ctl.cand_count, 1); if (slot < 32) few[slot] = k; }
          }
        }
        __syncthreads();
        const int nf = min(32, ctl.cand_count);
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
          unsigned long long cand = cr ? k : ~0ull;            // first crossed key = smallest crossed key
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(FULL, cand, o);
            cand = t < cand ? t : cand;
          }
          const unsigned who = __ballot_sync(FULL, cr && k == cand);
          if (lane == 0) { ctl.red_u64[0] = cand; ctl.bcast_i[1] = who ? 1 : 0; }
          if (who && lane == __ffs(who) - 1) { ctl.bcast_d[1] = g; ctl.bcast_d[2] = g - e; }
        }
        __syncthreads();
        if (ctl.bcast_i[1]) {
          const unsigned long long cstar = ctl.red_u64[0];
          g_at = ctl.bcast_d[1];
          g_before = ctl.bcast_d[2];
          cut_key = cstar;
          cut_incl = (mode == 0) ? 0 : 1;
        } else {
          all_in = true;                                       // rounding: nothing in the last group crossed
        }
      }
      if (!bad && all_in) {
        cut_key = ~0ull; cut_incl = 1;
        g_at = g_before = Ktot + Ztot;
        if (mode == 1 && Dtot > 0.0) bad = 1;                  // the bracket promised a crossing
      }
      if (!bad && !all_in) {
        if (fabs(g_at / S - plim) <= 1e-12 || fabs(g_before / S - plim) <= 1e-12) flags |= FLAG_TOPP_EDGE;
        if (mode == 1) {
          // a later key with the same d as c*: the cut separates equal probabilities
          int tie = 0;
          for (int t = tid; t < ZCAP; t += NT) {
            if (zlive(t)) { const unsigned long long k = zk[t]; tie |= (k > cut_key && (k >> 32) == (cut_key >> 32)) ? 1 : 0; }
          }
          if (block_max_i(tie, ctl, tid)) flags |= FLAG_TIE_CUT;
        }
      }
      // kept zone mass per owning rank: rank r's part of the list by NW / C warps (f64 atomics of shared memory on a few
      // addresses took longer than the selection: 16,000 logits, sigma 2, p = 0.9: 19,000 cycles of the step, 10,000 so)
      const int wlog = 31 - __clz(max(1, NW / C)), per_r = 1 << wlog;
      __syncthreads();
      if (!bad) {
        const int r = warp >> wlog;
        double e = 0.0;
        if (r < C) {
          for (int t = (warp & (per_r - 1)) * 32 + lane; t < X.cnt[r]; t += per_r * 32) {
            const unsigned long long k = zk[r * zcap_r + t];
            if (k < cut_key || (cut_incl && k == cut_key)) e += exp_safe(zone_key_d(k), s_tab);
          }
        }
        e = warp_sum_d(e);
        if (lane == 0) ctl.red_d[warp] = e;
        __syncthreads();
        if (tid < C) {
          double z = 0.0;
          for (int q = 0; q < per_r; q++) z += ctl.red_d[(tid << wlog) + q];
          s_zk[tid] = z;
        }
      }
      __syncthreads();
    }
    double Zk = 0.0;
    for (int r = 0; r < C; r++) Zk += s_zk[r];
    const double Re = Ktot + Zk;
    dbg.resum = Re / S;
    int owner = -1;
    int code;                                                // see Xchg::verdict
    if (bad) {
      code = 2;
    } else if (poisoned || !(Re > 0.0)) {
      // NaN/Inf in the row, or mode A removed every token (generate.go:221-227): the walk falls through
      flags |= FLAG_NONFINITE | FLAG_FALLBACK;
      dbg.sum_exp = poisoned ? QNAN : S;
      if (!poisoned) dbg.resum = 0.0;
      finish(V - 1, flags, dbg);
      code = 1;
    } else {
      const double tgt = u * Re;
      double acc = 0.0, base = 0.0;
      for (int r = 0; r < C; r++) {
        const double nxt = acc + X.K[r] + s_zk[r];
        if (tgt < nxt) { owner = r; base = acc; break; }
        acc = nxt;
      }
      code = 0;
      if (owner < 0) {
        flags |= FLAG_FALLBACK;                              // generate.go:239
        dbg.edge_lo = dbg.edge_hi = acc / Re;
        if (u - acc / Re <= 1e-6) flags |= FLAG_BOUNDARY;
        finish(V - 1, flags, dbg);
        code = 3;
      }
      if (tid < C) {
        Xchg* xr = cluster.map_shared_rank(&X, tid);
        xr->local_target = tgt - base;
        xr->base_mass = base;
      }
    }
    stamp(6);
    if (tid < C) {
      Xchg* xr = cluster.map_shared_rank(&X, tid);
      xr->owner = owner;
      xr->cut_key = cut_key; xr->cut_incl = cut_incl;
      xr->Re = Re; xr->S = S;
      xr->verdict = code;
    }
    if (tid == 0) {
      if (code == 0) {                                       // the owner adds the id, the edges and the boundary flag
        if (A.out_flags) A.out_flags[row_id] = flags;
        if (D && A.out_debug) A.out_debug[row_id] = dbg;
      }
    }
  }
  cluster.sync();                                            // G5: last barrier

  const int verdict = X.verdict;
  if (verdict == 2) { if (rank == 0) alone(); return; }
  if (verdict == 1) { fill_probs_slice(QNAN); return; }
  const double Re = X.Re, S = X.S;
  const unsigned long long ckey = X.cut_key;
  const int cincl = X.cut_incl;
  // final rule for one element: its kept mass (0 when cut away)
  auto kept_mass = [&](float xv, int i) -> double {
    if (i < 0 || i >= V) return 0.0;
    const float s = t_is_one ? xv : __fdiv_rn(xv, Tm);
    const float d = s - m;
    if (d < dA) {
      if (!(d >= dB)) return 0.0;
      const unsigned long long k = zone_key(d, i, mode);
      if (!(k < ckey || (cincl && k == ckey))) return 0.0;
    }
    return exp_safe(d, s_tab);
  };

  if (D && (A.out_probs || A.out_debug)) {                          // parity runs only
    double* pr = A.out_probs ? A.out_probs + row_id * static_cast<int64_t>(V) : nullptr;
    const double rq = Re / S;
    int kept_loc = 0;
    for (int j = tid; j < nv; j += NT) {
      float x[VEC];
      Elem<T>::unpack(slice[j], x);
      const int i0 = (v0 + j) * VEC - rv.shift;
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        const int i = i0 + c;
        if (i >= 0 && i < V) {
          const double f = (kept_mass(x[c], i) / S) / rq;
          kept_loc += (f > 0) ? 1 : 0;
          if (pr) pr[i] = f;
        }
      }
    }
    const int kept_cta = block_sum_i(kept_loc, ctl, tid);
    if (D && A.out_debug && tid == 0) atomicAdd(&A.out_debug[row_id].kept, kept_cta);
  }
  if (verdict == 3 || rank != X.owner) return;

  // ---- owner: kept mass per warp run = certain mass + kept zone entries, then one run is rescanned
  __syncthreads();
  if (cut_on) {
    // (rank 0's region B was reused by the selection: it takes its part of the staged list instead)
    const unsigned long long* zk = reinterpret_cast<const unsigned long long*>(regA);
    const int n = (rank == 0) ? X.cnt[0] : nz_loc;
    const int j0 = v0 + warp * wv, j1 = (warp == NW - 1) ? v1 : j0 + wv;   // this warp's run: it adds its own entries, no atomics
    double e = 0.0;
    for (int j = lane; j < n; j += 32) {
      unsigned long long k;
      if (rank == 0) k = zk[j];
      else { const uint2 z = lz[j]; k = zone_key(__uint_as_float(z.x), static_cast<int>(z.y), mode); }
      const int v = rv.vec_of(zone_key_index(k, mode));
      if (v >= j0 && v < j1 && (k < ckey || (cincl && k == ckey))) e += exp_safe(zone_key_d(k), s_tab);
    }
    e = warp_sum_d(e);
    if (lane == 0) s_kseg[warp] += e;
  }
  __syncthreads();
  const double ltgt = X.local_target;
  const double base_mass = X.base_mass;
  int wsel = NW - 1;
  double wbase = 0.0;
  {
    double acc = 0.0;
    bool found = false;
    for (int w = 0; w < NW; w++) {
      const double nxt = acc + s_kseg[w];
      if (!found && ltgt < nxt) { wsel = w; wbase = acc; found = true; }
      acc = nxt;
    }
    if (!found) wbase = acc - s_kseg[NW - 1];
  }
  int id = -1;
  int last_kept = -1;
  double edge_lo = 0.0, edge_hi = 0.0, run_end = wbase;
  for (int w = wsel; w < NW && id < 0; w++) {               // uniform; normally one trip
    const int a0 = min(nv, w * wv), a1 = min(nv, a0 + wv);
    for (int jb = a0; jb < a1 && id < 0; jb += NT) {
      const int j = jb + tid;
      double em[VEC];
      double tsum = 0.0;
#pragma unroll
      for (int c = 0; c < VEC; c++) em[c] = 0.0;
      int i0 = 0;
      if (j < a1) {
        float x[VEC];
        Elem<T>::unpack(slice[j], x);
        i0 = (v0 + j) * VEC - rv.shift;
#pragma unroll
        for (int c = 0; c < VEC; c++) { em[c] = kept_mass(x[c], i0 + c); tsum += em[c]; }
      }
      double totc;
      const double ex = block_scan_excl_d(tsum, totc, ctl, tid);
      int pick_loc = 0x7fffffff;
      int lk = -1;
      double run = run_end + ex, lo = 0.0, hi = 0.0;
#pragma unroll
      for (int c = 0; c < VEC; c++) {
        const double before = run;
        run += em[c];
        if (em[c] > 0.0) {
          lk = i0 + c;
          if (ltgt < run && pick_loc == 0x7fffffff) { pick_loc = i0 + c; lo = before; hi = run; }
        }
      }
      const int pick = block_min_i(pick_loc, ctl, tid);
      last_kept = max(last_kept, block_max_i(lk, ctl, tid));
      if (pick != 0x7fffffff) {
        if (pick_loc == pick) { ctl.bcast_d[1] = lo; ctl.bcast_d[2] = hi; }
        __syncthreads();
        id = pick;
        edge_lo = (base_mass + ctl.bcast_d[1]) / Re;
        edge_hi = (base_mass + ctl.bcast_d[2]) / Re;
      }
      run_end += totc;
    }
  }
  uint32_t oflags = 0;
  if (id < 0) {
    // rounding pushed the crossing past this slice's end: take its last kept token
    id = last_kept >= 0 ? last_kept : V - 1;
    oflags |= FLAG_BOUNDARY;
    edge_lo = edge_hi = (base_mass + run_end) / Re;
  } else if ((edge_lo > 0.0 && u - edge_lo <= 1e-6) || edge_hi - u <= 1e-6) {
    oflags |= FLAG_BOUNDARY;
  }
  if (tid == 0) {
    A.out_ids[row_id] = id;
    if (A.out_flags && oflags) atomicOr(&A.out_flags[row_id], oflags);
    if (D && A.out_debug) { A.out_debug[row_id].edge_lo = edge_lo; A.out_debug[row_id].edge_hi = edge_hi; }
  }
}

}  // namespace gs
