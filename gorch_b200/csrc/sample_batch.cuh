// Large-batch kernels: rows are first sorted by what they need, then two
// persistent kernels pull rows from work lists.
//
//   row_kind               what a row needs, from its config alone: greedy and
//                          top-k <= 256 rows are "narrow", top-k-off rows "wide",
//                          top-k above 256 goes to the single-CTA kernel. Each
//                          persistent kernel walks ALL rows with its own atomic
//                          cursor and takes the rows of its kind, so no separate
//                          classification launch and no per-kind lists exist.
//   narrow_rows_kernel     (sample_narrow.cuh, three instances: 256 threads x five CTAs per SM,
//                          or three with a longer ring, 128 threads x eight). One streaming pass per row: the first
//                          16 logits per thread give a threshold (from the per-thread
//                          maxima: a lower bound of the k-th largest logit, or a tighter
//                          estimate that is checked at the row's end); then every warp
//                          walks its own span of the rest, staged through a ring of
//                          asynchronous copies in shared memory, and only notes where
//                          a logit reaches the threshold; the noted vectors are read
//                          again after the stream, and everything from there on happens
//                          on a few hundred candidates in shared memory.
//   wide_rows_kernel       (sample_wide.cuh) rows whose softmax runs over the
//                          whole vocabulary.
//
// Row semantics: model/generate.go:134-260 (mode A), model/qwen/generate.go:
// 77-181 (mode B). Rows a kernel cannot finish (candidate or zone lists that
// outgrow their buffers) are appended to the single-CTA kernel's list.
#pragma once

#include "block_util.cuh"
#include "row_stream.cuh"
#include "sample_cluster.cuh"

namespace gs {

// Vocab-sharded sampling: what one rank knows about one row of its column slice. cand holds every
// local logit at or above the local k-th largest (global indices); the global kept set is a
// subset of the union of the ranks' lists, because the global k-th largest is at least every
// local one.
constexpr int VS_CAND = 128;
constexpr uint32_t VS_NONFINITE = 1u, VS_BAD_CFG = 2u, VS_OVERFLOW = 4u, VS_UNSUPPORTED = 8u, VS_NAN_AT_0 = 16u,
                   VS_SUMEXP = 32u;   // a row without top-k: cand[0] holds the slice's sum of exponentials (f64 bits)
struct VsRecord {
  float xmax;              // largest local logit (not yet divided by the temperature)
  int32_t n;               // entries in cand
  uint32_t flags;          // VS_*
  int32_t pad;
  uint2 cand[VS_CAND];     // (logit bits, global index)
};
static_assert(sizeof(VsRecord) == 16 + 8 * VS_CAND, "record layout is part of the C ABI");
// Record `row` of an array whose records hold `cand` candidates each (16 + 8 * cand bytes apart).
__device__ __forceinline__ VsRecord& vs_record(void* base, int64_t row, int cand) {
  return *reinterpret_cast<VsRecord*>(static_cast<unsigned char*>(base) + row * (16 + 8 * static_cast<int64_t>(cand)));
}
__device__ __forceinline__ const VsRecord& vs_record(const void* base, int64_t row, int cand) {
  return *reinterpret_cast<const VsRecord*>(static_cast<const unsigned char*>(base) + row * (16 + 8 * static_cast<int64_t>(cand)));
}

// A row's top-p setting cuts nothing: off, or the mode A rule with 1.5 p >= 1 (generate.go:184-228).
__device__ __forceinline__ bool vs_cut_inert(const RowCfg& c) {
  const bool on = c.top_p > 0.0f && c.top_p < 1.0f;
  return !on || (c.topp_mode == 0 && static_cast<double>(c.top_p) * 1.5 >= 1.0);
}
// exp(d), d <= 0, as f64: the table form (2e-11) where it applies, the all-f64 routine elsewhere.
// The local pass and the owner's draw use the same function, so that their sums agree term by term.
__device__ __forceinline__ double vs_exp(float d, const double* __restrict__ eb, const double* __restrict__ tab) {
  return (d > -31.9f) ? exp_fast(d, eb) : exp_safe(d, tab);
}

struct BatchArgs {
  KernelArgs k;
  const double* eb_table;   // 1024 doubles: exp(-b/32)
  int32_t* hdr;             // HDR_NARROW, HDR_WIDE: the kernels' row cursors
  int32_t* list_single;     // [0] = count, [1..] rows for the single-CTA kernel
  int64_t B;
};

// 0: narrow kernel, 1: wide kernel, 2: single-CTA kernel, 3: nobody (the row's sequence has ended)
__device__ __forceinline__ int row_kind(const KernelArgs& A, int64_t b) {
  if (A.row_done && A.row_done[b] != 0) return 3;
  if (A.force_greedy || A.vs_records || A.tk_k > 0) return 0;
  const RowCfg c = A.cfgs[b];
  const float T = c.temperature;
  if (T == 0.0f || !(T > 0.0f) || !(T < INFINITY)) return 0;   // greedy, or a bad temperature (reported by the narrow kernel)
  const int topk = (c.top_k > 0 && c.top_k < A.V) ? c.top_k : 0;
  return (topk == 0) ? 1 : (topk <= KFAST ? 0 : 2);
}

__device__ __forceinline__ void hand_to_single(const BatchArgs& BA, int64_t row_id) {
  BA.list_single[1 + atomicAdd(&BA.list_single[0], 1)] = static_cast<int32_t>(row_id);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// The narrow kernel, compiled three times from one source (sample_narrow.cuh): n256 with 256 threads and
// five CTAs per SM for batches of at most one row per CTA slot (a row is then streamed by eight
// warps), n256d with a longer ring for f32 batches of at most two rows per SM, n128 with 128 threads and eight CTAs per SM beyond that (1184 rows in flight: the phases
// before and after a row's stream then run once per slot instead of twice).
#define GS_N_NS n256
#define GS_N_NT 256
#define GS_N_CTAS 5
#define GS_N_RING 16384
#include "sample_narrow.cuh"
#undef GS_N_NS
#undef GS_N_CTAS
#undef GS_N_RING
#define GS_N_NS n256d
#define GS_N_CTAS 3
#define GS_N_RING 32768
#include "sample_narrow.cuh"
#undef GS_N_NS
#undef GS_N_NT
#undef GS_N_CTAS
#undef GS_N_RING
#define GS_N_NS n128
#define GS_N_NT 128
#define GS_N_CTAS 8
#define GS_N_RING 8192
#include "sample_narrow.cuh"
#undef GS_N_NS
#undef GS_N_NT
#undef GS_N_CTAS
#undef GS_N_RING

}  // namespace gs
