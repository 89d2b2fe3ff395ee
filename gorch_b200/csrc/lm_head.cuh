// LM-head projection with the sampling step's first pass in its epilogue.
//
// logits[b, v] = sum_k x[b, k] * w[v, k]: the last matmul of a decode step, MatMulTransB(last, Embed.Weight)
// in model/qwen/qwen.go:80-85 (nn/gpt.go:119-120 for GPT-2; nn/extembed.go:152-195 is its CPU loop), with
// x [B, K] and w [V, K] in bf16 and f32 accumulation. It is the one dense contraction next to the
// sampling path, and it produces the [B, V] logits that the sampling kernels otherwise read back from
// HBM: here the rows of a batch tile stay in tensor memory until the epilogue has taken what sampling
// needs from them.
//
// A pair of CTAs (a cluster of two, tcgen05 cta_group::2) works on one tile of 256 vocabulary rows x up
// to 256 batch rows; the vocabulary is the M side, so that a TMEM lane is a vocabulary column of the
// output and a warp writes 32 neighbouring logits of a batch row at a time. CTA r of the pair holds
// vocabulary rows 128 r .. of the tile, half of the batch rows, and the accumulator of its own vocabulary
// rows. Per item K is walked in chunks of 128:
//   warp 0      producer (both CTAs): TMA loads (w: 128 x 64, x: N / 2 x 64, 128-byte swizzle; two of each per
//               chunk, so that 256 neighbouring bytes of a row are asked for together: 32 x 1,024 x 151,936 in 51 us,
//               6.1 TB/s of weights; 61 us and 5.1 with one) into a ring of shared-memory stages; the bytes of
//               both CTAs complete on the leader's mbarrier
//   warp 1      issuer (leader): one elected thread issues tcgen05.mma (M = 256, N, K = 16) into one of two
//               accumulators of 256 TMEM columns; tcgen05.commit frees the stage / publishes the
//               accumulator in both CTAs
//   warps 2-9   epilogue (both CTAs): thread = vocabulary row (a TMEM lane), the batch rows' logits by
//               tcgen05.ld; either stores them, or (fused sampling) appends those at or above their batch
//               row's threshold to that row's candidate list
//
// Bound: at 512 rows the L2-to-SM traffic, the tensor pipe and HBM ask for about the same time each. A
// tile of 128 x 128 per CTA moves 2.5 GB from L2 for 512 x 1024 x 151,936 (4.1 ms of it per PFLOP; 10 TB/s
// measured: 250 us); a pair's 256 x 256 moves 1.25 GB. At 64 rows it is HBM, the weights' one read.
// Items are dealt out round by round over the pairs; what the last round would leave to a few pairs is cut
// into 32-row items for all of them.
// Every CTA fetches its own tiles (plain TMA loads), and every tensor map covers this GPU's own memory.
//
// Every wait on an mbarrier is bounded: a wait that runs out sets an abort flag that the CTA's other roles
// see in their own waits (the other CTA's run out by themselves), the kernel reports LMH_ERR_TIMEOUT in its
// status word, frees its tensor memory and returns.
#pragma once

#include <cuda.h>

#include "sample_batch.cuh"

namespace gs {

constexpr int LMH_TILE_V = 256;          // vocabulary rows of a tile (UMMA M over the pair); 128 per CTA
constexpr int LMH_CTA_V = 128;
constexpr int LMH_MAX_N = 256;           // batch rows of an item (UMMA N)
constexpr int LMH_BK = 64;               // K of one TMA box: 64 bf16 = one 128-byte swizzle row
constexpr int LMH_SUB = 2;               // boxes of either operand per stage
constexpr int LMH_EPI = 8;               // epilogue warps: two for each quarter of the TMEM lanes
constexpr int LMH_NT = 64 + 32 * LMH_EPI;   // warp 0 producer, warp 1 issuer, then the epilogue
constexpr int LMH_MAX_STAGES = 12;
constexpr int LMH_RING_BYTES = 208 * 1024;
constexpr int LMH_W_BYTES = LMH_CTA_V * LMH_BK * 2;                 // a box of w: 16 KB
constexpr int LMH_DYN_BYTES = LMH_RING_BYTES + 1024;                // + room to align the swizzled tiles to 1024 bytes
constexpr int LMH_TMEM_COLS = 512;       // two accumulators of 256 f32 columns
constexpr uint32_t LMH_WAIT_LIMIT = 4000000u;

constexpr uint32_t LMH_ERR_TIMEOUT = 1u;

// tcgen05 instruction descriptor (kind::f16): D = F32 (bits 4-5 = 1), A = B = BF16 (bits 7-9, 10-12 = 1),
// both K-major (bits 15, 16 = 0), N / 8 at bits 17-22, M / 16 at bits 24-28.
__host__ __device__ constexpr uint32_t lmh_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(LMH_TILE_V >> 4) << 24);
}

constexpr int LMH_CAND_CAP = 2048;       // candidates per row (entries of 8 bytes)
struct LmhRow {
  int32_t cnt;             // candidates so far (those beyond LMH_CAND_CAP are not stored)
  int32_t nan;             // 1: a NaN in the row; 2: at index 0
};

struct LmHeadArgs {
  CUtensorMap map_x;       // x [B, K] bf16, box 64 x box_n, 128-byte swizzle
  CUtensorMap map_w;       // w [V, K] bf16, box 64 x cta_v, 128-byte swizzle
  int32_t B, V, K;
  int32_t box_n;           // batch rows that one TMA load of x brings: half of the largest item
  int32_t item_n;          // batch rows of a full item, a multiple of 32
  int32_t stages;          // of the ring
  int32_t cta_v;           // vocabulary rows of a tile that each CTA takes, at most LMH_CTA_V
  int32_t tile0, tile_step, ntile;   // vocabulary tiles (of 2 cta_v rows) tile0 + i * tile_step, i < ntile
  float* out_logits;       // [B, ld_out] f32, or null
  int64_t ld_out;
  int32_t compact;         // 1: tile i goes to columns [i * 2 cta_v, ...) of out_logits (the sample of tiles)
  // fused sampling (all null when unused)
  const float* thr;        // [B] candidate threshold per row (raw logit units)
  uint2* cand;             // [B][LMH_CAND_CAP] (logit bits, index)
  LmhRow* rows;            // [B]
  uint32_t* status;        // [1] LMH_ERR_* bits, in host memory
  int32_t clear_status;    // 1: this launch clears it first
  int32_t chained;         // 1: launched as a dependent of the kernel that fills thr, with x and w there before; 0: of any kernel
};

// Work items in the order in which pair p takes them: p, p + npairs, ...: first the whole rounds of full
// items (all batch rows of `full` vocabulary tiles, item_n at a time), then the remaining tiles in items
// of small_n batch rows, at most one round of them.
struct LmhItem { int vt, b0, n; };
struct LmhPlan {
  int nb, full, nfull, nsmall, total, item_n, small_n, B;
  __host__ __device__ LmhPlan(int B_, int ntile, int item_n_, int npairs) {
    B = B_; item_n = item_n_;
    nb = (B + item_n - 1) / item_n;
    full = (ntile * nb / npairs) * npairs / nb;
    nfull = full * nb;
    const int rest = (ntile - full) * nb;
    int s = 1;
    while (rest > 0 && 2 * s * rest <= npairs && item_n / (2 * s) >= 32) s *= 2;
    small_n = (item_n / s + 31) & ~31;
    nsmall = (B + small_n - 1) / small_n;
    total = nfull + (ntile - full) * nsmall;
  }
  __device__ __forceinline__ LmhItem at(int i) const {
    LmhItem it;
    const bool f = i < nfull;
    const int q = f ? i : i - nfull, per = f ? nb : nsmall, n = f ? item_n : small_n;
    it.vt = (f ? 0 : full) + q / per;
    it.b0 = (q % per) * n;
    it.n = min(n, ((B - it.b0) + 31) & ~31);
    return it;
  }
};

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
// Bounded wait for the phase with parity `parity` to complete; false when it ran out or another role gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t it = 0; it < LMH_WAIT_LIMIT; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((it & 63u) == 63u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// The address of this CTA's shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(cluster_addr) : "memory");
}
// A tile into this CTA's shared memory; its bytes complete on a barrier that may be the pair's other CTA's.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, unsigned long long pol) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
               :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "l"(pol) : "memory");
}
// Shared-memory matrix descriptor of a K-major tile of 128-byte rows with the 128-byte swizzle: start
// address / 16, leading byte offset 1 (unused for swizzled K-major), stride byte offset 1024 / 16 (eight
// rows), descriptor version 1 at bit 46, layout type 2 (128-byte swizzle) at bits 61-63.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr_bytes) {
  return static_cast<uint64_t>((smem_addr_bytes & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair when the MMAs issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               :: "r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(LMH_NT, 1) lm_head_kernel(const __grid_constant__ LmHeadArgs A) {
  extern __shared__ __align__(16) unsigned char lmh_dyn[];
  __shared__ __align__(8) unsigned long long full_bar[LMH_MAX_STAGES], empty_bar[LMH_MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  __shared__ __align__(16) float stash_thr[LMH_EPI][32];
  __shared__ uint2 stash[LMH_EPI][64];
  __shared__ int stash_row[LMH_EPI][64];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = blockIdx.x & 1u;                                // in the pair; 0 leads
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const uint32_t ring = (smem_addr(lmh_dyn) + 1023u) & ~1023u;          // the swizzled tiles need 1024-byte alignment
  volatile int* abort_flag = &abort_s;
  const int nk64 = A.K / LMH_BK, nkc = (nk64 + LMH_SUB - 1) / LMH_SUB;  // K boxes and chunks per item
  const int nst = A.stages;
  const uint32_t x_bytes = static_cast<uint32_t>(A.box_n) * LMH_BK * 2, stage_bytes = LMH_SUB * (LMH_W_BYTES + x_bytes);
  const LmhPlan plan(A.B, A.ntile, A.item_n, npairs);
  pdl_launch();
  // What fills x and w, or uses the output. Ahead of the tensor memory, which a kernel that still runs may want, and of the
  // bounded waits. The launch overlaps that kernel's end (us a call, back to back, without | so: 4 x 512 x 1,000: 10.1 | 7.5,
  // 16 x 512 x 4,096: 10.2 | 7.0, 300 x 1,024 x 8,192: 14.5 | 12.4, 512 x 1,024 x 151,936: 180.1 | 178.1).
  if (!A.chained) pdl_wait();

  if (tid == 0) {
    for (int s = 0; s < nst; s++) { mbar_init(smem_addr(&full_bar[s]), 1); mbar_init(smem_addr(&empty_bar[s]), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(smem_addr(&acc_full[b]), 1); mbar_init(smem_addr(&acc_empty[b]), 2 * LMH_EPI); }
    abort_s = 0;
    if (A.clear_status && blockIdx.x == 0) *A.status = 0u;              // (a wait runs out seconds later, if ever)
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {                                                      // one warp of each CTA takes the tensor memory
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(&tmem_base_s)), "r"(LMH_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");   // both CTAs' barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_s;

  if (warp == 0) {
    // ---- producer: this CTA's share of every stage; its bytes complete on the leader's barrier
    if (lane == 0) {
      unsigned long long pol_w, pol_x;                                  // the weights pass once per batch tile, x stays
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol_w));
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol_x));
      if (plan.nb > 1) asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol_w));
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int i = pair; i < plan.total && ok; i += npairs) {
        const LmhItem it = plan.at(i);
        const int v0 = ((A.tile0 + it.vt * A.tile_step) * 2 + static_cast<int>(rank)) * A.cta_v;
        const int xb = it.b0 + static_cast<int>(rank) * (it.n >> 1);
        for (int kc = 0; kc < nkc; kc++) {
          if (!mbar_wait(smem_addr(&empty_bar[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t own = smem_addr(&full_bar[stage]), bar = map_rank(own, 0);
          const uint32_t sw = ring + stage * stage_bytes, sx = sw + LMH_SUB * LMH_W_BYTES;
          const int subs = min(LMH_SUB, nk64 - kc * LMH_SUB);
          if (rank == 0) mbar_expect_tx(own, 2 * subs * (static_cast<uint32_t>(A.cta_v) * LMH_BK * 2 + x_bytes));
          for (int u = 0; u < subs; u++) tma_load_2d_pair(sw + u * LMH_W_BYTES, &A.map_w, bar, (kc * LMH_SUB + u) * LMH_BK, v0, pol_w);
          for (int u = 0; u < subs; u++) tma_load_2d_pair(sx + u * x_bytes, &A.map_x, bar, (kc * LMH_SUB + u) * LMH_BK, xb, pol_x);
          if (++stage == static_cast<uint32_t>(nst)) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- issuer
    if (rank == 0 && lane == 0) {
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = true;
      for (int i = pair; i < plan.total && ok; i += npairs) {
        const uint32_t idesc = lmh_idesc(plan.at(i).n);
        if (!mbar_wait(smem_addr(&acc_empty[acc]), acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d_tmem = tmem_base + acc * LMH_MAX_N;
        for (int kc = 0; kc < nkc; kc++) {
          if (!mbar_wait(smem_addr(&full_bar[stage]), phase, abort_flag)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sw = ring + stage * stage_bytes, sx = sw + LMH_SUB * LMH_W_BYTES;
          const int subs = min(LMH_SUB, nk64 - kc * LMH_SUB);
          for (int u = 0; u < subs; u++) {
#pragma unroll
            for (int k = 0; k < LMH_BK / 16; k++)
              umma_f16_pair(d_tmem, umma_desc(sw + u * LMH_W_BYTES + k * 32), umma_desc(sx + u * x_bytes + k * 32), idesc, (kc > 0 || u > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(smem_addr(&empty_bar[stage]));               // the stage is free once these MMAs have read it
          if (++stage == static_cast<uint32_t>(nst)) { stage = 0; phase ^= 1u; }
        }
        if (ok) umma_commit_pair(smem_addr(&acc_full[acc]));            // the accumulator is complete
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 * (w % 4) .. + 31; thread = vocabulary row
    const int q = warp & 3, half = (warp - 2) >> 2;                     // this warp's lanes, and its share of the columns
    uint32_t acc = 0, acc_phase = 0;
    bool ok = true;
    int nstash = 0;
    auto flush = [&](int count) {                                       // the stash's first `count` entries to their rows' lists
      __syncwarp();
      if (lane < count) {
        const uint2 e = stash[warp - 2][lane];
        const int b = stash_row[warp - 2][lane];
        const float x = __uint_as_float(e.x);
        if (x != x) {
          atomicOr(&A.rows[b].nan, (e.y == 0u) ? 3 : 1);
        } else {
          const int slot = atomicAdd(&A.rows[b].cnt, 1);
          if (slot < LMH_CAND_CAP) A.cand[static_cast<int64_t>(b) * LMH_CAND_CAP + slot] = e;
        }
      }
      __syncwarp();
    };
    if (A.chained) pdl_wait();                                          // the thresholds; tiles and MMAs are under way meanwhile
    for (int i = pair; i < plan.total && ok; i += npairs) {
      const LmhItem it = plan.at(i);
      if (!mbar_wait(smem_addr(&acc_full[acc]), acc_phase, abort_flag)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int in_tile = static_cast<int>(rank) * A.cta_v + q * 32 + lane;
      const int v = (A.tile0 + it.vt * A.tile_step) * 2 * A.cta_v + in_tile;
      const bool live = q * 32 + lane < A.cta_v && v < A.V;
      const int ocol = A.compact ? it.vt * 2 * A.cta_v + in_tile : v;
#pragma unroll 1
      for (int c = half * 32; c < it.n; c += 64) {
        uint32_t r[32];
        tmem_ld32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * LMH_MAX_N + c, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int b0 = it.b0 + c, nb = min(32, A.B - b0);              // batch rows of these columns (uniform)
        if (A.out_logits && live) {
          float* dst = A.out_logits + static_cast<int64_t>(b0) * A.ld_out + ocol;
          if (nb == 32) {
#pragma unroll
            for (int j = 0; j < 32; j++) __stcs(dst + j * A.ld_out, __uint_as_float(r[j]));
          } else {
#pragma unroll
            for (int j = 0; j < 32; j++) if (j < nb) __stcs(dst + j * A.ld_out, __uint_as_float(r[j]));
          }
        }
        if (A.thr) {
          // a batch row's threshold is the same for all lanes, and few lanes hold a logit that reaches it: those go to
          // the warp's stash, and from there, 32 at a time, to their rows' lists (an atomic on a row's count per
          // logit where it is found made every warp wait in nearly every chunk)
          stash_thr[warp - 2][lane] = (lane < nb) ? A.thr[b0 + lane] : INFINITY;
          __syncwarp();
          const float4* t4 = reinterpret_cast<const float4*>(stash_thr[warp - 2]);
          uint32_t m = 0u;                                             // columns of this lane that reach their threshold
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const float4 t = t4[j >> 2];
            const float tj = (j & 3) == 0 ? t.x : (j & 3) == 1 ? t.y : (j & 3) == 2 ? t.z : t.w;
            m |= !(__uint_as_float(r[j]) < tj) ? (1u << j) : 0u;       // (true for a NaN)
          }
          if (!live) m = 0u;
          for (uint32_t votes; (votes = __ballot_sync(FULL, m != 0u)) != 0u;) {   // one hit of every lane that has any
            if (m) {
              const int j = __ffs(m) - 1;
              m &= m - 1;
              uint32_t x = r[0];
#pragma unroll
              for (int jj = 1; jj < 32; jj++) x = (j == jj) ? r[jj] : x;
              const int at = nstash + __popc(votes & ((1u << lane) - 1u));
              stash[warp - 2][at] = make_uint2(x, static_cast<uint32_t>(v));
              stash_row[warp - 2][at] = b0 + j;
            }
            nstash += __popc(votes);
            if (nstash >= 32) {                                        // uniform
              flush(32);
              nstash -= 32;
              const uint2 e = stash[warp - 2][32 + lane];
              const int er = stash_row[warp - 2][32 + lane];
              __syncwarp();
              if (lane < nstash) { stash[warp - 2][lane] = e; stash_row[warp - 2][lane] = er; }
            }
          }
          __syncwarp();
        }
      }
      // the accumulator is free again: one arrival per epilogue warp of either CTA at the leader's barrier
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_rank(smem_addr(&acc_empty[acc]), 0));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
    if (nstash > 0) flush(nstash);
  }
  // ---- teardown
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (abort_s) {
    // a wait ran out: give the copies and MMAs still in flight time to land before the shared and
    // tensor memory they target is given back (bounded: about a millisecond)
    for (int it = 0; it < 1000; it++) __nanosleep(1000);
    if (tid == 0) atomicOr_system(A.status, LMH_ERR_TIMEOUT);
  }
  // neither CTA leaves while the other may still arrive on its barriers or read its tiles
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(LMH_TMEM_COLS) : "memory");
  }
}


// ---- fused sampling on top of the projection (greedy and top-k rows) --------------------------------
//
//   1. the projection over a sample of vocabulary tiles (1/32 of the vocabulary, spread over it)
//      gives each row 1024 to 4096 of its logits;
//   2. lmh_threshold_kernel: the r-th largest of that sample, r chosen so that eight times top_k
//      logits of the whole row (at least 256, at most a third of the list) are expected above it: an
//      estimate, not a bound;
//   3. the projection over all tiles: the epilogue appends every logit at or above the row's
//      threshold to the row's candidate list (no [B, V] logits are written);
//   4. lmh_finish_kernel: the exact top_k-th largest of the candidates with ties kept
//      (model/generate.go:157-164), then softmax / top-p / draw on the kept set exactly as the
//      one-GPU narrow kernel does. A row whose estimate failed (fewer than top_k candidates, or more
//      than the list holds) or whose config the fused path does not serve is counted in nfail; the
//      host then recomputes the batch through the unfused path.
constexpr int LMH_SAMPLE_MIN = 1024, LMH_SAMPLE_MAX = 4096;   // logits of a row's sample
constexpr int LMH_F_NT = 256;
constexpr int LMH_F_DYN_BYTES = LMH_CAND_CAP * 8 + 16384 + KEEP_MAX * 8;

struct LmhSampleArgs {
  KernelArgs k;             // V, cfgs, uniforms, out_ids, out_flags, exp_table (logits unused)
  const float* sample;      // [B, nsample] logits of the sampled tiles
  int32_t nsample;
  int32_t fuse_top_k;       // rows with 0 < top_k <= fuse_top_k (or temperature 0) are served
  float* thr;               // [B]
  const uint2* cand;        // [B, LMH_CAND_CAP]
  LmhRow* rows;             // [B]
  int32_t* nfail;           // [1], in host memory
  int64_t B;
};

__device__ __forceinline__ bool lmh_row_served(const RowCfg& c, int V, int fuse_top_k) {
  const float T = c.temperature;
  if (T == 0.0f) return true;
  if (!(T > 0.0f) || !(T < INFINITY)) return true;            // reported as a bad config by the finish kernel
  const int topk = (c.top_k > 0 && c.top_k < V) ? c.top_k : 0;
  return topk > 0 && topk <= fuse_top_k;
}

__global__ void __launch_bounds__(LMH_F_NT) lmh_threshold_kernel(const __grid_constant__ LmhSampleArgs M) {
  constexpr int PER = LMH_SAMPLE_MAX / LMH_F_NT;              // sample logits per thread
  __shared__ bu::Scratch sc;
  __shared__ uint32_t cnts[1024];
  __shared__ int bc[4];
  const int tid = threadIdx.x;
  pdl_launch();
  const int64_t row = blockIdx.x;
  const RowCfg cfg = M.k.cfgs[row];
  const bool served = lmh_row_served(cfg, M.k.V, M.fuse_top_k);
  pdl_wait();                                                 // the sample's logits
  float thr = served ? -INFINITY : INFINITY;                  // -Inf: a sample too small to say, everything is a candidate
  if (served) {
    const int keff = (cfg.temperature == 0.0f || !(cfg.temperature > 0.0f) || !(cfg.temperature < INFINITY)) ? 1 : cfg.top_k;
    const int n = M.nsample;
    uint32_t key[PER], tmin = 0xffffffffu, tmax = 0u;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const int i = j * LMH_F_NT + tid;
      key[j] = (i < n) ? okey(M.sample[row * n + i]) : 0u;    // (0, a NaN's key, is below every other)
      tmin = min(tmin, key[j]);
      tmax = max(tmax, key[j]);
    }
    // expected logits of the whole row above the threshold: eight times top_k, at least 256, at most a
    // third of the list; the r-th largest of the sample stands for the (r V / n)-th largest of the row
    const long long want = min(max(8ll * keff, 256ll), static_cast<long long>(LMH_CAND_CAP / 3));
    const int r = max(2, static_cast<int>((want * n + M.k.V / 2) / M.k.V));
    if (r < n) {
      const uint32_t lo = sample_threshold<LMH_F_NT, 1024>([&](auto&& g) {
#pragma unroll
        for (int j = 0; j < PER; j++) g(key[j]);
      }, r, tmin, tmax, cnts, bc, sc, tid);
      if (lo > 0x007fffffu) thr = okey_to_float(lo);          // NaNs order lowest: a NaN threshold would collect nothing
    }
  }
  if (tid == 0) { M.thr[row] = thr; M.rows[row].cnt = 0; M.rows[row].nan = 0; }
}

__global__ void __launch_bounds__(LMH_F_NT, 4) lmh_finish_kernel(const __grid_constant__ LmhSampleArgs M) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ bu::Scratch sc;
  __shared__ uint32_t s_sel[256];
  __shared__ int s_bc[4];
  __shared__ int s_cnt;
  uint2* list = reinterpret_cast<uint2*>(dyn);                                       // the row's candidates
  unsigned char* work = dyn + LMH_CAND_CAP * 8;                                       // for finish_small_set
  uint2* kept = reinterpret_cast<uint2*>(dyn + LMH_CAND_CAP * 8 + 16384);            // KEEP_MAX entries
  const KernelArgs& A = M.k;
  const int tid = threadIdx.x;
  constexpr int NW = LMH_F_NT / 32;
  pdl_wait();                                                 // the candidates
  for (int64_t row = blockIdx.x; row < M.B; row += gridDim.x) {
    __syncthreads();
    const RowCfg cfg = A.cfgs[row];
    const float Tm = cfg.temperature;
    auto write_row = [&](int id, uint32_t fl) {
      if (tid == 0) {
        A.out_ids[row] = id;
        if (A.out_flags) A.out_flags[row] = fl;
      }
    };
    auto give_up = [&]() { if (tid == 0) atomicAdd_system(M.nfail, 1); write_row(-1, FLAG_INTERNAL); };
    if (!lmh_row_served(cfg, A.V, M.fuse_top_k)) { give_up(); continue; }
    if (Tm != 0.0f && (!(Tm > 0.0f) || !(Tm < INFINITY))) { write_row(-1, FLAG_BAD_CFG); continue; }
    const int cnt = M.rows[row].cnt, nanb = M.rows[row].nan;
    uint32_t kmax = 0x007fffffu;                                // -Inf
    for (int j = tid; j < min(cnt, LMH_CAND_CAP); j += LMH_F_NT) {
      const uint2 e = M.cand[row * LMH_CAND_CAP + j];
      list[j] = e;
      kmax = max(kmax, okey(__uint_as_float(e.x)));
    }
    kmax = static_cast<uint32_t>(bu::max_u64<NW>(kmax, sc, tid));   // (its barriers publish the list)
    const int keff = (Tm == 0.0f) ? 1 : cfg.top_k;
    if (cnt > LMH_CAND_CAP || (cnt < keff && !(nanb & 1))) { give_up(); continue; }   // the estimate failed for this row
    // ---- greedy (generate.go:134-144): largest logit, lowest index; a NaN at index 0 is never beaten
    if (Tm == 0.0f) {
      unsigned long long best = 0ull;
      for (int j = tid; j < cnt; j += LMH_F_NT) {
        const unsigned long long p = (static_cast<unsigned long long>(okey(__uint_as_float(list[j].x))) << 32) |
                                     static_cast<uint32_t>(~list[j].y);
        best = p > best ? p : best;
      }
      best = bu::max_u64<NW>(best, sc, tid);
      int id = static_cast<int>(~static_cast<uint32_t>(best & 0xffffffffull));
      if ((nanb & 2) || cnt == 0) id = 0;
      write_row(id, 0u);
      continue;
    }
    const float m = scale_t(okey_to_float(kmax), Tm);
    // A NaN anywhere, or an infinite maximum: the walk of generate.go:231-239 falls through
    if ((nanb & 1) || !(fabsf(m) < INFINITY)) { write_row(A.V - 1, FLAG_NONFINITE | FLAG_FALLBACK); continue; }
    // ---- top_k-th largest with ties (generate.go:157-164), then the kept set
    const int topk = cfg.top_k;
    const int nk = narrow_list<LMH_F_NT>(list, cnt, topk, Tm, 0u, kmax, kept, s_sel, s_bc, &s_cnt, tid);
    if (nk > KEEP_MAX || cnt <= topk) { give_up(); continue; }
    const bool topp_on = (cfg.top_p > 0.0f && cfg.top_p < 1.0f);
    const int mode = cfg.topp_mode;
    const double plim = (mode == 0) ? static_cast<double>(cfg.top_p) * 1.5 : static_cast<double>(cfg.top_p);
    // Everything at or above the exact threshold must be on the list: that holds when the exact
    // threshold (the floor of the k-th value's class of equal quotients) is not below the list's own.
    if (!finish_small_set<LMH_F_NT, false>(A, row, kept, nk, topk, m, Tm, topp_on, mode, plim, A.uniforms[row], M.thr[row], work, nullptr, 0u))
      give_up();
  }
}

}  // namespace gs
