// TopK (index_ops.go:153-190), k <= TKL_MAX_K (the narrow kernel takes small k over many rows): the k largest of each row, descending, equal
// values by ascending index; NaNs last (the reference's comparator leaves them unspecified), -0 and
// +0 equal. The values written are the row's own bits.
//
// One CTA per row at a time, one pass over the row:
//   1. a sample spread over the whole row (64-byte pieces, 8192 to 16384 logits) gives a threshold
//      above which k to k + 10 sigma logits are expected;
//   2. the row is streamed once through a ring of asynchronous copies, logits at or above the
//      threshold go to a candidate list in shared memory;
//   3. the candidates are put into buckets by their order key and every one finds its place among
//      those of its own bucket: that place is the place in the output, so neither an exact k-th
//      value nor a sort is needed.
// A row whose list comes out short or overflows (its k-th value is tied thousands of times, or the
// sample missed it) takes topk_exact_row: a radix select over the row, several passes from L2.
//
// Bound: HBM, one read of the row plus the sample (5 % of it). Instances by k: the list has to hold
// what the threshold lets through, and the smaller the list, the more rows an SM has in flight.
// 512 x 151,936 f32, k = 1000 (B200): 111 us; 964 us as a radix select and a bitonic sort of every row.
#pragma once

#include "sample_batch.cuh"

namespace gs {

constexpr int TKL_MIN_K = 64;           // up to here (f32: half of it) the narrow kernel serves TopK of many rows that are not long
constexpr int TKL_MAX_K = 16384;

struct TopKLargeArgs {
  const void* x;           // [B, row_stride]
  int64_t row_stride;
  int32_t V;
  int32_t k;
  float* out_values;       // [B, k]
  int32_t* out_indices;    // [B, k]
  uint32_t* out_flags;     // [B] or null
  int64_t B;
};

// NT threads, a list of CAP candidates, NBINS buckets, STAGES steps of 32 bytes per thread in the ring
// (which the buckets and their members' places lie over when the stream has ended), a sample of SAMPLE logits.
template <int NT_, int CAP_, int NBINS_, int STAGES_, int SAMPLE_, int MINB_>
struct TklShape {
  static constexpr int NT = NT_, CAP = CAP_, NBINS = NBINS_, STAGES = STAGES_, SAMPLE = SAMPLE_, MINB = MINB_;
  static constexpr int RING_BYTES = STAGES * NT * 32;
  static constexpr int SORT_BYTES = NBINS * 4 + ((CAP * 2 + 15) & ~15);
  static constexpr int DYN_BYTES = CAP * 8 + (RING_BYTES > SORT_BYTES ? RING_BYTES : SORT_BYTES);
};
using TklSmall = TklShape<256, 3328, 2048, 3, 8192, 4>;       // k <= 1024, four rows per SM
using TklFew = TklShape<1024, 3328, 2048, 2, 8192, 1>;        // k <= 1024, at most one row per SM: its latency counts
using TklMid = TklShape<512, 7168, 4096, 2, 16384, 2>;        // k <= 4096
using TklLarge = TklShape<1024, 20000, 4096, 1, 16384, 1>;    // k <= TKL_MAX_K
constexpr int TKL_SMALL_K = 1024, TKL_MID_K = 4096;

// The exact form. keys: shared memory for 8 bytes times the power of two at or above k.
template <typename T, int NT>
__device__ __noinline__ void topk_exact_row(const TopKLargeArgs& A, int64_t row, unsigned long long* keys, bu::Scratch& sc,
                                            uint32_t* hist, int* bc, int* s_cnt) {
  const int tid = threadIdx.x;
  const int V = A.V, k = A.k;
  int P = 1;
  while (P < k) P <<= 1;                                     // sort size
  RowView<T> rv;
  rv.init(static_cast<const T*>(A.x) + row * A.row_stride, V);
  // smallest and largest order key of the row: the select starts at the highest bit in which they
  // differ, so that the keys spread over its bins (the top byte of a float is the same for nearly
  // all logits of a row, and 150,000 shared atomics on one counter would take a millisecond)
  uint32_t kmin = 0xffffffffu, kmax = 0u;
  for (int v = tid; v < rv.nvec; v += NT)
    rv.visit(v, [&](float x, int) { const uint32_t key = okey(x); kmin = min(kmin, key); kmax = max(kmax, key); });
  kmax = static_cast<uint32_t>(bu::max_u64<NT / 32>(kmax, sc, tid));
  kmin = ~static_cast<uint32_t>(bu::max_u64<NT / 32>(~kmin, sc, tid));
  // the k-th largest value (as an order key) ...
  const uint32_t kkey = bu::select_kth_of<NT>([&](auto&& f) {
    for (int v = tid; v < rv.nvec; v += NT) rv.visit(v, [&](float x, int) { f(okey(x)); });
  }, k, kmin, kmax, hist, bc, tid);
  // ... how many logits lie above it, and how many equal it
  int above = 0, ties = 0;
  for (int v = tid; v < rv.nvec; v += NT)
    rv.visit(v, [&](float x, int) { const uint32_t key = okey(x); above += (key > kkey) ? 1 : 0; ties += (key == kkey) ? 1 : 0; });
  above = bu::sum_i<NT / 32>(above, sc, tid);
  ties = bu::sum_i<NT / 32>(ties, sc, tid);
  const int need = k - above;                                // 1 <= need <= ties
  // among equals the lowest indices win: the need-th smallest index of them, when not all are wanted
  uint32_t last_index = 0xffffffffu;
  if (need < ties) {                                         // uniform
    const uint32_t inv = bu::select_kth_of<NT>([&](auto&& f) {
      for (int v = tid; v < rv.nvec; v += NT)
        rv.visit(v, [&](float x, int i) { if (okey(x) == kkey) f(~static_cast<uint32_t>(i)); });
    }, need, ~static_cast<uint32_t>(V - 1), 0xffffffffu, hist, bc, tid);
    last_index = ~inv;
  }
  __syncthreads();
  if (tid == 0) *s_cnt = 0;
  for (int j = tid; j < P; j += NT) keys[j] = 0ull;          // padding sorts last
  __syncthreads();
  for (int v = tid; v < rv.nvec; v += NT) {
    rv.visit(v, [&](float x, int i) {
      const uint32_t key = okey(x);
      if (key > kkey || (key == kkey && static_cast<uint32_t>(i) <= last_index)) {
        const int slot = atomicAdd(s_cnt, 1);
        if (slot < k) keys[slot] = (static_cast<unsigned long long>(key) << 32) | static_cast<uint32_t>(~static_cast<uint32_t>(i));
      }
    });
  }
  __syncthreads();
  // an invariant of the two selects; and a k that is promised an answer only while at most KEEP_MAX logits reach the
  // k-th value (gorch_cuda_topk_dev: k <= KFAST) gets none beyond, whichever kernel serves it
  const bool ok = (*s_cnt == k) && !(k <= KFAST && above + ties > KEEP_MAX);
  // bitonic sort, descending (a larger key first: larger value, then lower index)
  for (int size = 2; size <= P; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = tid; t < (P >> 1); t += NT) {
        const int lo = 2 * t - (t & (stride - 1));
        const int hi = lo + stride;
        const bool desc = ((lo & size) == 0);
        const unsigned long long a = keys[lo], b = keys[hi];
        if ((a < b) == desc) { keys[lo] = b; keys[hi] = a; }
      }
      __syncthreads();
    }
  }
  float* ov = A.out_values + row * static_cast<int64_t>(k);
  int32_t* oi = A.out_indices + row * static_cast<int64_t>(k);
  for (int j = tid; j < k; j += NT) {
    if (ok) {
      const int i = static_cast<int>(~static_cast<uint32_t>(keys[j] & 0xffffffffull));
      float xv = 0.f;
      rv.visit(rv.vec_of(i), [&](float x, int ii) { if (ii == i) xv = x; });
      ov[j] = xv; oi[j] = i;
    } else {
      ov[j] = __int_as_float(0x7fc00000); oi[j] = -1;
    }
  }
  if (tid == 0 && A.out_flags) A.out_flags[row] = ok ? 0u : FLAG_INTERNAL;
}

// The largest of the logits in two vectors; a NaN counts as less than anything else.
template <typename T> __device__ __forceinline__ float tkl_max(const uint4& a, const uint4& b);
template <> __device__ __forceinline__ float tkl_max<float>(const uint4& a, const uint4& b) {
  const float m = fmaxf(fmaxf(__uint_as_float(a.x), __uint_as_float(a.y)), fmaxf(__uint_as_float(a.z), __uint_as_float(a.w)));
  return fmaxf(m, fmaxf(fmaxf(__uint_as_float(b.x), __uint_as_float(b.y)), fmaxf(__uint_as_float(b.z), __uint_as_float(b.w))));
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) { uint32_t d; asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
template <> __device__ __forceinline__ float tkl_max<uint16_t>(const uint4& a, const uint4& b) {
  const uint32_t p = max_bf16x2(max_bf16x2(max_bf16x2(a.x, a.y), max_bf16x2(a.z, a.w)), max_bf16x2(max_bf16x2(b.x, b.y), max_bf16x2(b.z, b.w)));
  return fmaxf(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}

template <typename T, typename SH>
__global__ void __launch_bounds__(SH::NT, SH::MINB) topk_large_kernel(TopKLargeArgs A) {
  constexpr int NT = SH::NT, NW = NT / 32, CAP = SH::CAP, NBINS = SH::NBINS, NQ = SH::STAGES;
  constexpr int VEC = Elem<T>::VEC;
  constexpr int SV = 64;                                     // vectors of a warp-step: two per lane
  constexpr int J = SH::SAMPLE / (NT * VEC);                 // sample vectors per thread
  static_assert(J >= 1 && NBINS % NT == 0 && (NBINS & (NBINS - 1)) == 0 && CAP < 65536, "shape");
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ bu::Scratch sc;
  __shared__ uint32_t hist[256];
  __shared__ int bc[4];
  __shared__ int s_cnt;
  __shared__ int s_notes[NW][64];
  uint2* cand = reinterpret_cast<uint2*>(dyn);               // (logit bits, index)
  uint32_t* bins = reinterpret_cast<uint32_t*>(dyn + CAP * 8);
  uint16_t* perm = reinterpret_cast<uint16_t*>(dyn + CAP * 8 + NBINS * 4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int V = A.V, k = A.k;
  const uint32_t ring_addr = smem_addr(dyn + CAP * 8) + static_cast<uint32_t>(tid * 16);
  const uint4* ring = reinterpret_cast<const uint4*>(dyn + CAP * 8) + tid;
  unsigned long long pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  for (int64_t row = blockIdx.x; row < A.B; row += gridDim.x) {
    RowView<T> rv;
    rv.init(static_cast<const T*>(A.x) + row * A.row_stride, V);
    __syncthreads();
    if (tid == 0) s_cnt = 0;
    if (V <= CAP) {                                          // every logit is a candidate
      __syncthreads();
      for (int v = tid; v < rv.nvec; v += NT)
        rv.visit(v, [&](float x, int i) { cand[i] = make_uint2(__float_as_uint(x), static_cast<uint32_t>(i)); });
      if (tid == 0) s_cnt = V;
      __syncthreads();
    } else {
      // the stream's first copies fly while the sample is read and its threshold found
      const int span = (((rv.nvec + NW - 1) / NW + SV - 1) / SV) * SV;
      const WSpan sp = make_span<T, 2>(rv, warp * span, span, lane);
      auto issue = [&](int q) {
        if (q < sp.nst) {
          const uint32_t dst = ring_addr + static_cast<uint32_t>((q % NQ) * 2 * NT * 16);
          const int o = q * SV;
          asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;"
                       :: "r"(dst), "l"(sp.lane_src + min(o, sp.omax)), "l"(pol) : "memory");
          asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;"
                       :: "r"(dst + NT * 16), "l"(sp.lane_src + min(o + 32, sp.omax)), "l"(pol) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      // ---- sample: NT * J vectors in 64-byte pieces, the pieces spread evenly over the row
      uint4 smp[J];
      int nsv;                                               // vectors that the sample holds
      {
        constexpr int PIECES = NT * J / 4;
        const int have = rv.nvec / 4;                        // whole pieces in the row
        nsv = min(have, PIECES) * 4;
#pragma unroll
        for (int j = 0; j < J; j++) {
          const int p = (j * NT + tid) >> 2;
          const int piece = (have > PIECES) ? static_cast<int>(static_cast<int64_t>(p) * have / PIECES) : p;
          const int v = piece * 4 + (tid & 3);
          smp[j] = make_uint4(Neutral<T>::word, Neutral<T>::word, Neutral<T>::word, Neutral<T>::word);
          float a = 0.f, b = 0.f;
          bool c = false;
          if (p < have) smp[j] = load_masked(rv, v, a, b, c);
        }
      }
#pragma unroll
      for (int q = 0; q < NQ; q++) issue(q);
      // ---- threshold: the r-th largest of the sample. k n / V of the sample's n logits are expected above
      // the k-th largest of the row; five standard deviations more make a list shorter than k a matter of
      // one row in millions, and ten stay within CAP
      float thr = -INFINITY;
      {
        const float f = static_cast<float>(nsv) * VEC / static_cast<float>(V);
        const float e = static_cast<float>(k) * f;
        const int r = static_cast<int>(e + 5.0f * sqrtf(e * fmaxf(1.0f - f, 0.05f))) + 4;
        uint32_t kmin = 0xffffffffu, kmax = 0u;
#pragma unroll
        for (int j = 0; j < J; j++) {
          float x[VEC];
          Elem<T>::unpack(smp[j], x);
#pragma unroll
          for (int c = 0; c < VEC; c++) { const uint32_t key = okey(x[c]); kmin = min(kmin, key); kmax = max(kmax, key); }
        }
        if (r < nsv * VEC) {                                 // uniform
          const uint32_t lo = sample_threshold<NT, NBINS>([&](auto&& g) {
#pragma unroll
            for (int j = 0; j < J; j++) {
              float x[VEC];
              Elem<T>::unpack(smp[j], x);
#pragma unroll
              for (int c = 0; c < VEC; c++) g(okey(x[c]));
            }
          }, r, kmin, kmax, reinterpret_cast<uint32_t*>(dyn), bc, sc, tid);   // counters in the candidate list's memory: empty yet
          if (lo != 0u) thr = okey_to_float(lo);
        }
        __syncthreads();
      }
      // ---- the stream. A lane whose logits hold one at or above the threshold only notes where, in its
      // warp's list (a vote and a store, no branch); when a warp has 32 notes, every lane takes one, reads
      // the two vectors again (from L2: they have just passed) and moves what it finds to the candidate
      // list. Looking at the logits on the spot cost the whole warp some hundred instructions a step.
      int* notes = s_notes[warp];
      int nn = 0;
      auto resolve = [&](int count) {
        __syncwarp();
        uint32_t m = 0u;
        float x[2 * VEC];
        int i0 = 0, i1 = 0;
        if (lane < count) {
          const int g0 = notes[lane], g1 = g0 + 32;
          Elem<T>::unpack(__ldg(rv.vbase + g0), x);
          Elem<T>::unpack(__ldg(rv.vbase + min(g1, rv.nvec - 1)), x + VEC);
          i0 = g0 * VEC - rv.shift; i1 = g1 * VEC - rv.shift;
#pragma unroll
          for (int c = 0; c < 2 * VEC; c++) {
            const int i = (c < VEC) ? i0 + c : i1 + c - VEC;
            if (x[c] >= thr && static_cast<uint32_t>(i) < static_cast<uint32_t>(V)) m |= 1u << c;
          }
        }
        const int mine = __popc(m);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += t; }
        int at = 0;
        if (lane == 31) at = atomicAdd(&s_cnt, incl);
        at = __shfl_sync(FULL, at, 31) + incl - mine;
#pragma unroll
        for (int c = 0; c < 2 * VEC; c++) {
          if (m & (1u << c)) {
            if (at < CAP) cand[at] = make_uint2(__float_as_uint(x[c]), static_cast<uint32_t>((c < VEC) ? i0 + c : i1 + c - VEC));
            at++;
          }
        }
      };
      const uint32_t below = (1u << lane) - 1u;
      const int nst = (thr > -INFINITY) ? sp.nst : 0;        // fewer than r logits of the sample above -Inf: the exact form
#pragma unroll 1
      for (int st = 0; st < nst; st++) {
        asm volatile("cp.async.wait_group %0;" :: "n"(NQ - 1) : "memory");
        const int slot = (st % NQ) * 2 * NT;
        const uint4 ca = ring[slot], cb = ring[slot + NT];
        const int gv = sp.first + st * SV + lane;
        float hi = tkl_max<T>(ca, cb);
        if (st >= sp.clean_hi && gv >= rv.nvec) hi = -INFINITY;   // past the row's end: nothing of it is left in these two vectors
        const uint32_t votes = __ballot_sync(FULL, hi >= thr);
        issue(st + NQ);                                      // into the slot just read
        if (hi >= thr) notes[nn + __popc(votes & below)] = gv;
        nn += __popc(votes);
        if (nn >= 32) {                                      // uniform
          resolve(32);
          nn -= 32;
          const int rest = (lane < nn) ? notes[32 + lane] : 0;
          __syncwarp();
          if (lane < nn) notes[lane] = rest;
        }
      }
      if (nn > 0) resolve(nn);
      asm volatile("cp.async.wait_group 0;" ::: "memory");   // the ring's memory is about to hold the buckets
      __syncthreads();
    }
    const int n = s_cnt;
    bool exact = n < k || n > CAP;
    if (!exact) {
      // ---- buckets: equal widths of the order key between the list's ends, largest keys first
      uint32_t kmin = 0xffffffffu, kmax = 0u;
      for (int j = tid; j < n; j += NT) { const uint32_t key = okey(__uint_as_float(cand[j].x)); kmin = min(kmin, key); kmax = max(kmax, key); }
      for (int b = tid; b < NBINS; b += NT) bins[b] = 0u;
      kmax = static_cast<uint32_t>(bu::max_u64<NW>(kmax, sc, tid));
      kmin = ~static_cast<uint32_t>(bu::max_u64<NW>(~kmin, sc, tid));   // (its barriers also publish the cleared bins)
      constexpr int LOGB = 31 - __builtin_clz(NBINS);
      const int sh = max(0, 32 - __clz(kmax - kmin) - LOGB);
      auto bin_of = [&](uint2 e) { return (kmax - okey(__uint_as_float(e.x))) >> sh; };
      for (int j = tid; j < n; j += NT) atomicAdd(&bins[bin_of(cand[j])], 1u);
      __syncthreads();
      constexpr int PER = NBINS / NT;
      uint32_t loc[PER];
      uint32_t sum = 0u, most = 0u;
#pragma unroll
      for (int q = 0; q < PER; q++) { loc[q] = bins[tid * PER + q]; sum += loc[q]; most = max(most, loc[q]); }
      // exclusive prefix of the bucket sizes
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += t; }
      if (lane == 31) sc.i0[warp] = static_cast<int>(incl);
      most = __reduce_max_sync(FULL, most);
      if (lane == 0) sc.i1[warp] = static_cast<int>(most);
      __syncthreads();
      uint32_t base = (lane < warp && lane < NW) ? static_cast<uint32_t>(sc.i0[lane]) : 0u;
      base = __reduce_add_sync(FULL, base);
      most = __reduce_max_sync(FULL, static_cast<uint32_t>(sc.i1[lane < NW ? lane : 0]));
      uint32_t run = base + incl - sum;
#pragma unroll
      for (int q = 0; q < PER; q++) { bins[tid * PER + q] = run; run += loc[q]; }
      __syncthreads();
      exact = most > (k <= KFAST ? 256u : 512u);             // long runs of near-equal logits: the places within a bucket take its size squared
      if (!exact) {
        for (int j = tid; j < n; j += NT) perm[atomicAdd(&bins[bin_of(cand[j])], 1u)] = static_cast<uint16_t>(j);
        __syncthreads();                                     // bins[b] is now the end of bucket b
        float* ov = A.out_values + row * static_cast<int64_t>(k);
        int32_t* oi = A.out_indices + row * static_cast<int64_t>(k);
        for (int p = tid; p < n; p += NT) {
          const uint2 e = cand[perm[p]];
          const uint32_t b = bin_of(e);
          const int from = b ? static_cast<int>(bins[b - 1]) : 0, to = static_cast<int>(bins[b]);
          if (from >= k) continue;
          const uint32_t key = okey(__uint_as_float(e.x));
          int place = from;
          for (int q = from; q < to; q++) {
            const uint2 o = cand[perm[q]];
            const uint32_t ok = okey(__uint_as_float(o.x));
            place += (ok > key || (ok == key && o.y < e.y)) ? 1 : 0;
          }
          if (place < k) { ov[place] = __uint_as_float(e.x); oi[place] = static_cast<int32_t>(e.y); }
        }
        if (tid == 0 && A.out_flags) A.out_flags[row] = 0u;
      }
    }
    if (exact) {                                             // uniform
      __syncthreads();
      topk_exact_row<T, NT>(A, row, reinterpret_cast<unsigned long long*>(dyn), sc, hist, bc, &s_cnt);
    }
  }
}

}  // namespace gs
