// libgorchcuda.so: implementation of include/gorch_cuda_shim.h.
//
// Host-side conventions mirror the reference's Metal shim (metal/shim.m):
// opaque handles, strdup'd error strings, int return codes, a blocking default.
// There is no CPU fallback anywhere in this file: every entry point either
// runs the CUDA kernels or returns an error.

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nccl.h>     // types and prototypes only: the library is loaded at run time, on first use

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <mutex>
#include <new>
#include <vector>

#include "../../include/gorch_cuda_shim.h"
#define GS_W_NS w256
#define GS_W_NT 256
#include "sample_wide.cuh"      // gs::w256: 256 threads, four CTAs per SM (throughput)
#define GS_W_NS w1024
#define GS_W_NT 1024
#include "sample_wide.cuh"      // gs::w1024: 1024 threads, one CTA per SM (latency)
#include "sample_vocab.cuh"
#include "index_ops.cuh"
#include "topk_large.cuh"
#include "generate_control.cuh"
#include "row_softmax.cuh"
#include "lm_head.cuh"

namespace {

// Largest slice kept in shared memory: 109 KB of dynamic shared memory per CTA
// (two CTAs per SM) minus the two 16 KB work regions.
constexpr int64_t kSliceCap = 109 * 1024 - gs::REGION_A - gs::REGION_B;

// Batches go to the sorted-batch kernels (one CTA per row) from this many rows or bytes on; smaller ones to
// the cluster kernel (several CTAs per row), whose latency is lower while the GPU is not full. The rows' kinds are
// on the device, so one line serves them all. us, batch | cluster, calls back to back on inputs that are not in L2, for rows with
// top-k, greedy ones, the two mixed with nucleus rows, plain softmax rows, and rows with a top-p cut (f32):
//   112 x 50,257: 28 | 23, 17 | 12, 35 | 27, 25 | 31, 54 | 72;  256 x 50,257: 31 | 41, 20 | 22, 44 | 49, 31 | 58, 79 | 136
//   32 x 151,936: 36 | 19, 21 | 10, 47 | 23, 35 | 23, 83 | 49;  64: 37 | 27, 23 | 15, 51 | 35, 35 | 40, 85 | 85;  128: 40 | 44, 25 | 26, 55 | 55,
//   39 | 72, 99 | 160
// At 50,257 columns rows without top-k change sides long before the others, and the line stays near theirs. Bytes follow that only roughly: up to 48
// rows of 151,936 f32 the clusters would serve nearly every kind sooner (48: 37 | 22, 22 | 13, 50 | 30, 35 | 36, 83 | 77), and behind the line
// top-k, greedy and mixed rows pay (128 x 50,257: 28 | 24, 17 | 13, 37 | 30, for 25 | 32, 54 | 76).
// Short rows stay with the clusters for longer. Up to four rows per SM of 4,096 logits, two waves of clusters:
//   592 x 4,096: 25 | 20, 15 | 10, 36 | 29, 23 | 24, 45 | 41 (8,000 logits, 512 rows: 28 | 21, 16 | 11, 39 | 29, 23 | 27, 49 | 48)
// Beyond four rows per SM, the wide kernel's slots, the batch kernels start a second round of wide rows (592 x 12,000: 30 | 23, 18 | 13,
// 44 | 33, 27 | 31, 57 | 60; 593: 31 | 30, 19 | 15, 44 | 33, 35 | 38, 81 | 68): up to six rows per SM of 16,384 logits
//   888 x 4,000: 25 | 29, 15 | 15, 47 | 40, 34 | 35, 75 | 60;  768 x 16,000: 35 | 35, 21 | 18, 107 | 44, 40 | 51, 104 | 98
//   889 x 16,384: 37 | 41, 23 | 21, 108 | 49, 43 | 59, 108 | 109
// Mixed batches gain most there, rows with a cut some; top-k rows by themselves give a few us back, plain softmax rows up to a quarter.
// An argmax is one launch of the narrow kernel and keeps the lower line.
constexpr int64_t kBatchModeRows = 384;
constexpr int64_t kBatchModeBytes = 24ll << 20;
inline bool use_batch_mode(int sm_count, int64_t B, int64_t V, int64_t elem_bytes, bool argmax) {
  const bool many_short = B >= kBatchModeRows && !argmax && B <= 6 * sm_count && V <= (B > 4 * sm_count ? 16384 : 4096);
  return !many_short && (B >= kBatchModeRows || (B >= 32 && B * V * elem_bytes >= kBatchModeBytes));
}

// LM head with sampling: up to this many bytes of logits they are written to scratch, where the cluster kernel finds them in
// L2. The fused form saves that traffic and pays for it with two more kernels and a second run over part of the weights
// (us a call with its wait, fused | this: 64 x 50,257, K = 1024: 62 | 51; 96: 66 | 57; 104: 66 | 59; 16 x 151,936, K = 512:
// 67 | 58; 32: 67 | 64; K = 2048, 16: 135 | 123; 16 x 4,096, K = 512: 42 | 31). Beyond it the two meet: 110 x 50,257, K = 1024:
// 64 | 60; 128: 64 | 65; 40 x 151,936, K = 512: 68 | 69.
constexpr int64_t kLmhUnfusedBytes = 20ll << 20, kLmhUnfusedK = 512;

struct Buffer {
  int device;
  void* ptr;
  uint64_t bytes;
  uint64_t block;         // bytes that the pool holds for it (a power of two), or 0: not the pool's
};

// Small device blocks that released buffers leave for the next ones, so that a generation or a call that
// needs a few arrays for a moment does not pay for cudaMalloc and cudaFree (tens of microseconds each, and
// cudaFree waits for the device). At most kPoolBytes per process; given back when the last context goes.
// A block may still be in use by work queued before its buffer was released, on any stream: before a
// block is handed out again that was released after the device was last waited for, the device is waited
// for (as cudaFree would have done), once for all such blocks.
struct BufferPool {
  static constexpr uint64_t kMaxBlock = 1ull << 20, kPoolBytes = 32ull << 20;
  struct Block { int device; void* ptr; uint64_t bytes; bool in_doubt; };
  std::mutex lock;
  std::vector<Block> free_blocks;
  uint64_t held = 0;
  int contexts = 0;

  static uint64_t block_of(uint64_t bytes) {
    uint64_t b = 256;
    while (b < bytes) b <<= 1;
    return b <= kMaxBlock ? b : 0;
  }
  // A block of exactly `bytes`, or null. The device is current.
  void* take(int device, uint64_t bytes) {
    std::lock_guard<std::mutex> g(lock);
    size_t at = free_blocks.size();
    for (size_t i = 0; i < free_blocks.size(); i++) {
      if (free_blocks[i].device == device && free_blocks[i].bytes == bytes && (at == free_blocks.size() || !free_blocks[i].in_doubt)) at = i;
    }
    if (at == free_blocks.size()) return nullptr;
    if (free_blocks[at].in_doubt) {
      if (cudaDeviceSynchronize() != cudaSuccess) return nullptr;
      for (Block& b : free_blocks) if (b.device == device) b.in_doubt = false;
    }
    void* p = free_blocks[at].ptr;
    free_blocks[at] = free_blocks.back();
    free_blocks.pop_back();
    held -= bytes;
    return p;
  }
  bool put(int device, void* ptr, uint64_t bytes) {
    std::lock_guard<std::mutex> g(lock);
    if (contexts == 0 || held + bytes > kPoolBytes) return false;
    free_blocks.push_back(Block{device, ptr, bytes, true});
    held += bytes;
    return true;
  }
  void enter() { std::lock_guard<std::mutex> g(lock); contexts++; }
  void leave() {
    std::lock_guard<std::mutex> g(lock);
    if (--contexts > 0) return;
    for (Block& b : free_blocks) { cudaSetDevice(b.device); cudaFree(b.ptr); }
    free_blocks.clear();
    held = 0;
  }
};
BufferPool g_pool;

// Logits in pageable host memory that go through the context's pinned block, and the piece of them that is copied at a time.
constexpr size_t kStageBytes = 1ull << 20, kStagePiece = 128ull << 10;

struct Scratch {  // grow-only device allocation
  void* ptr = nullptr;
  size_t cap = 0;
};

struct Ctx {
  int device = 0;
  int sm_count = 148;
  int64_t l2_bytes = 126ll << 20;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  double* exp_table = nullptr;
  double* eb_table = nullptr;
  Scratch worklist;        // int32[16 + rows + 1]: header of a sorted batch, rows that its kernels leave to the single-CTA kernel
  Scratch st_logits;       // logits of the host-memory calls
  Scratch pinned;          // host memory: their configurations, uniforms, ids, flags, and logits on their way
  Scratch lmh_scratch;       // thresholds, candidate lists, sample logits of the LM-head path
  uint32_t* host_words = nullptr;   // pinned, written by kernels: [0] LM-head status, [1] rows its fused form handed back
  Scratch lmh_logits;        // [B, V] f32 when rows need the unfused samplers
  Scratch vs_local, vs_all;  // records of the vocab-sharded call: this rank's, and every rank's after the all-gather
  Scratch vs_req;            // [B][3] doubles: what the owner's draw of a row without top-k needs
  Scratch vs_rows, vs_done;  // whole rows [B][V padded] and the mask of rows that do not need them (vocab-sharded rows without top-k that are gathered)
  ncclComm_t comm = nullptr; // set by gorch_cuda_comm_init
  int comm_rank = 0, comm_nranks = 0;
  cudaEvent_t ev_vs[4] = {nullptr, nullptr, nullptr, nullptr};
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t ev_left = nullptr;     // the end of the work on the stream that gorch_cuda_set_stream left ...
  bool left_pending = false;         // ... which no later stream waits for yet
  uint64_t waited_launches = 0;      // counters.kernel_launches when the context was last waited for
  int timing = 0;
  int variant = 0;        // 0: by batch size, 1: single-CTA kernel, 2: narrow/wide kernels, 3: cluster kernel,
                          // 4 / 5: as 2 with the wide kernel's 256- / 1024-thread instance forced,
                          // 6 / 7: as 2 with the narrow kernel's 128- / 256-thread instance forced
  int force_cluster = 0;  // 0: choose from the shape
  GorchCudaCounters counters{};
};

// Work lists for gorch_cuda_sample_dev_static: fixed storage inside the loaded module, so the
// entry point never allocates. Every GPU that loads the library holds one copy (about 16 KB)
// until the process exits. In host code this name is only a handle for cudaGetSymbolAddress;
// the device address is looked up once per device (static_lists_ptr, called by gorch_cuda_create_ctx with
// that device current) and passed to the kernels.
constexpr int64_t kStaticMaxRows = 4096;
static __device__ __align__(256) int32_t g_static_worklists[16 + kStaticMaxRows + 1];
constexpr int kMaxDevices = 64;
int32_t* g_static_ptr[kMaxDevices] = {};

// Device address of g_static_worklists on the CURRENT device (looked up once per device).
int static_lists_ptr(int device, int32_t** out, char** errOut);

void set_err(char** errOut, const char* fmt, ...) {
  if (!errOut) return;
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  *errOut = strdup(buf);
}

#define CUDA_TRY(expr, errOut)                                                   \
  do {                                                                           \
    cudaError_t e__ = (expr);                                                    \
    if (e__ != cudaSuccess) {                                                    \
      set_err(errOut, "%s failed: %s", #expr, cudaGetErrorString(e__));          \
      return GORCH_CUDA_ERR_CUDA;                                                \
    }                                                                            \
  } while (0)

// NCCL, loaded on first use (a process that never shards the vocabulary does not need it). Inside a
// process that already holds a libnccl.so.2 (PyTorch's), the loader hands back that same copy.
struct NcclApi {
  void* handle = nullptr;
  ncclResult_t (*GetUniqueId)(ncclUniqueId*) = nullptr;
  ncclResult_t (*CommInitRank)(ncclComm_t*, int, ncclUniqueId, int) = nullptr;
  ncclResult_t (*CommDestroy)(ncclComm_t) = nullptr;
  ncclResult_t (*AllGather)(const void*, void*, size_t, ncclDataType_t, ncclComm_t, cudaStream_t) = nullptr;
  ncclResult_t (*AllReduce)(const void*, void*, size_t, ncclDataType_t, ncclRedOp_t, ncclComm_t, cudaStream_t) = nullptr;
  const char* (*GetErrorString)(ncclResult_t) = nullptr;
};
NcclApi g_nccl;

int load_nccl(char** errOut) {
  if (g_nccl.handle) return GORCH_CUDA_OK;
  void* h = dlopen("libnccl.so.2", RTLD_NOW | RTLD_GLOBAL);
  if (!h) h = dlopen("libnccl.so", RTLD_NOW | RTLD_GLOBAL);
  if (!h) {
    set_err(errOut, "gorch_cuda: cannot load libnccl.so.2: %s", dlerror());
    return GORCH_CUDA_ERR_NCCL;
  }
  NcclApi a;
  a.handle = h;
  a.GetUniqueId = reinterpret_cast<decltype(a.GetUniqueId)>(dlsym(h, "ncclGetUniqueId"));
  a.CommInitRank = reinterpret_cast<decltype(a.CommInitRank)>(dlsym(h, "ncclCommInitRank"));
  a.CommDestroy = reinterpret_cast<decltype(a.CommDestroy)>(dlsym(h, "ncclCommDestroy"));
  a.AllGather = reinterpret_cast<decltype(a.AllGather)>(dlsym(h, "ncclAllGather"));
  a.AllReduce = reinterpret_cast<decltype(a.AllReduce)>(dlsym(h, "ncclAllReduce"));
  a.GetErrorString = reinterpret_cast<decltype(a.GetErrorString)>(dlsym(h, "ncclGetErrorString"));
  if (!a.GetUniqueId || !a.CommInitRank || !a.CommDestroy || !a.AllGather || !a.AllReduce || !a.GetErrorString) {
    set_err(errOut, "gorch_cuda: libnccl.so.2 lacks a symbol this library needs");
    return GORCH_CUDA_ERR_NCCL;
  }
  g_nccl = a;
  return GORCH_CUDA_OK;
}

#define NCCL_TRY(expr, errOut)                                                   \
  do {                                                                           \
    ncclResult_t r__ = (expr);                                                   \
    if (r__ != ncclSuccess) {                                                    \
      set_err(errOut, "%s failed: %s", #expr, g_nccl.GetErrorString(r__));       \
      return GORCH_CUDA_ERR_NCCL;                                                \
    }                                                                            \
  } while (0)

int static_lists_ptr(int device, int32_t** out, char** errOut) {
  if (device < 0 || device >= kMaxDevices) {
    set_err(errOut, "gorch_cuda: device index %d beyond the static table", device);
    return GORCH_CUDA_ERR_LIMIT;
  }
  if (!g_static_ptr[device]) {
    void* p = nullptr;
    CUDA_TRY(cudaGetSymbolAddress(&p, g_static_worklists), errOut);
    g_static_ptr[device] = static_cast<int32_t*>(p);
  }
  *out = g_static_ptr[device];
  return GORCH_CUDA_OK;
}

int ensure(Scratch& s, size_t bytes, char** errOut) {
  if (bytes <= s.cap) return GORCH_CUDA_OK;
  if (s.ptr) {
    CUDA_TRY(cudaFree(s.ptr), errOut);
    s.ptr = nullptr;
    s.cap = 0;
  }
  size_t want = bytes + (bytes >> 3);
  cudaError_t e = cudaMalloc(&s.ptr, want);
  if (e != cudaSuccess) {
    want = bytes;
    e = cudaMalloc(&s.ptr, want);
  }
  if (e != cudaSuccess) {
    s.ptr = nullptr;
    set_err(errOut, "cudaMalloc(%zu bytes) failed: %s", bytes, cudaGetErrorString(e));
    return GORCH_CUDA_ERR_CUDA;
  }
  s.cap = want;
  return GORCH_CUDA_OK;
}

// Grow-only pinned host memory of the context.
int ensure_pinned(Ctx* c, size_t bytes, char** errOut) {
  Scratch& s = c->pinned;
  if (bytes <= s.cap) return GORCH_CUDA_OK;
  if (s.ptr) {
    CUDA_TRY(cudaFreeHost(s.ptr), errOut);
    s.ptr = nullptr;
    s.cap = 0;
  }
  const size_t want = bytes + (bytes >> 2) + 4096;
  CUDA_TRY(cudaHostAlloc(&s.ptr, want, cudaHostAllocMapped | cudaHostAllocPortable), errOut);
  s.cap = want;
  return GORCH_CUDA_OK;
}

bool is_pinned(const void* p) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return false; }
  return at.type == cudaMemoryTypeHost;
}

// Whether what is queued on the stream runs or goes into a graph; Invalidated where the stream cannot be asked.
cudaStreamCaptureStatus capture_status(cudaStream_t stream) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) { cudaGetLastError(); st = cudaStreamCaptureStatusInvalidated; }
  return st;
}

// Waits for the context's stream.
cudaError_t wait_stream(Ctx* c) {
  const cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) c->waited_launches = c->counters.kernel_launches;
  return e;
}

int check_shape(int dtype, int64_t B, int64_t V, int64_t row_stride, char** errOut) {
  if (dtype != GORCH_CUDA_F32 && dtype != GORCH_CUDA_BF16) {
    set_err(errOut, "gorch_cuda: unknown dtype %d", dtype);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (B < 0 || V < 1 || row_stride < V) {
    set_err(errOut, "gorch_cuda: bad shape B=%lld V=%lld row_stride=%lld", (long long)B,
            (long long)V, (long long)row_stride);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (V > 0x7fffff00ll || B > 0x7fffffffll) {
    set_err(errOut, "gorch_cuda: shape beyond 31-bit row / batch limit");
    return GORCH_CUDA_ERR_LIMIT;
  }
  return GORCH_CUDA_OK;
}

size_t elem_size(int dtype) { return dtype == GORCH_CUDA_BF16 ? 2 : 4; }

// A launch on the context's stream; dependent: it may start while the kernel before it runs, and waits for
// that itself (griddepcontrol.wait) where it needs what it wrote. cluster: CTAs per cluster.
template <typename... P, typename... A>
cudaError_t launch_clusters(Ctx* c, void (*kernel)(P...), unsigned grid, unsigned block, size_t dyn, bool dependent, int cluster, const A&... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(grid);
  lc.blockDim = dim3(block);
  lc.dynamicSmemBytes = dyn;
  lc.stream = c->stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = dependent ? 2 : 1;
  return cudaLaunchKernelEx(&lc, kernel, args...);
}
template <typename... P, typename... A>
cudaError_t launch(Ctx* c, void (*kernel)(P...), unsigned grid, unsigned block, size_t dyn, bool dependent, const A&... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(grid);
  lc.blockDim = dim3(block);
  lc.dynamicSmemBytes = dyn;
  lc.stream = c->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&lc, kernel, args...);
}

// The context's row work lists of a sorted batch: 16 header words, all zero between calls, and B + 1 for the rows.
int batch_lists(Ctx* c, int64_t B, int32_t** base, char** errOut) {
  const size_t had = c->worklist.cap;
  int rc = ensure(c->worklist, (16 + static_cast<size_t>(B) + 1) * sizeof(int32_t), errOut);
  if (rc) return rc;
  *base = static_cast<int32_t*>(c->worklist.ptr);
  if (c->worklist.cap != had) CUDA_TRY(cudaMemsetAsync(*base, 0, 16 * sizeof(int32_t), c->stream), errOut);
  return GORCH_CUDA_OK;
}

// The narrow kernel's instances: 256-thread CTAs (five per SM) while every row gets a CTA slot
// of its own, 128-thread CTAs (eight per SM) beyond that. Variants 6 / 7 force one of them (tests). Where no SM gets more than two rows of
// f32, 256 threads with a longer ring and more registers (n256d). us, n256 | n256d, top-k of 50: 64 x 151,936: 46.1 | 36.0, 148 x 100,003:
// 40.0 | 32.7, 256 x 50,257: 33.0 | 29.3, 296 x 100,003: 46.1 | 40.4; greedy, 148 x 151,936: 36.8 | 27.2, 256 x 100,003: 32.5 | 27.3; mixed, 256 x 50,257: 46.3 | 42.4,
// 148 x 151,936: 70.6 | 58.0. Beyond, the two come together (330 x 151,936: 63.7 | 65.1, 400: 71.5 | 70.2). bf16 rows have four steps on their way in either, and
// mixed batches of them are slower beside the wide kernel (256 x 100,003: 49.4 | 50.6, 330: 51.9 | 54.7).
static cudaError_t launch_narrow(Ctx* c, const gs::BatchArgs& ba, int dtype, int64_t B, bool dependent) {
  const int64_t slots256 = static_cast<int64_t>(gs::n256::N_CTAS_PER_SM) * c->sm_count;
  const bool small_ctas = c->variant == 6 || (c->variant != 7 && B > slots256);
  const bool deep = !small_ctas && c->variant != 7 && dtype == GORCH_CUDA_F32 && B <= 2ll * c->sm_count;
  const int64_t slots = small_ctas ? static_cast<int64_t>(gs::n128::N_CTAS_PER_SM) * c->sm_count : slots256;
  const unsigned g = static_cast<unsigned>(B < slots ? B : slots);
  const bool diag = ba.k.out_probs || ba.k.out_debug;
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kernel, int nt, int bytes) { e = launch(c, kernel, g, nt, bytes, dependent, ba); };
  auto pick = [&](auto type) {
    typedef decltype(type) E;
    if (small_ctas) go(diag ? gs::n128::narrow_rows_kernel<E, true> : gs::n128::narrow_rows_kernel<E, false>, gs::n128::N_NT, gs::n128::N_DYN_BYTES);
    else if (deep) go(diag ? gs::n256d::narrow_rows_kernel<float, true> : gs::n256d::narrow_rows_kernel<float, false>, gs::n256d::N_NT, gs::n256d::N_DYN_BYTES);
    else go(diag ? gs::n256::narrow_rows_kernel<E, true> : gs::n256::narrow_rows_kernel<E, false>, gs::n256::N_NT, gs::n256::N_DYN_BYTES);
  };
  if (dtype == GORCH_CUDA_F32) pick(float()); else pick(uint16_t());
  return e;
}

// 16-byte vectors of a row, at most.
int64_t row_vectors(int64_t V, int dtype) {
  const int vec = dtype == GORCH_CUDA_F32 ? 4 : 8;
  return (V + 2 * (vec - 1)) / vec + 1;
}
int64_t slice_bytes(int64_t V, int dtype, int C) { return ((row_vectors(V, dtype) + C - 1) / C) * 16; }

// CTAs per row of the cluster kernel: the smallest power of two whose slice fits the shared-memory budget, raised for
// small batches so that the whole GPU has work; 0 when no size keeps the row in shared memory.
int cluster_size(const Ctx* c, int64_t B, int64_t V, int dtype) {
  int C = 1;
  while (C < gs::CL_MAX && slice_bytes(V, dtype, C) > kSliceCap) C *= 2;
  // (two CTAs of this kernel fit an SM: stop while all clusters are still resident at once;
  // measured on 64 rows of 50257 f32: 43 us with 4 CTAs per row, 55 us with 8)
  while (C < gs::CL_MAX && B * 2 * C <= 2 * c->sm_count && row_vectors(V, dtype) / (2 * C) >= 64) C *= 2;
  if (c->force_cluster) C = c->force_cluster;
  return (slice_bytes(V, dtype, C) > kSliceCap || B * C > 0x7fffffffll) ? 0 : C;
}

int launch_rows(Ctx* c, const void* logits, int dtype, int64_t B, int64_t V, int64_t row_stride,
                const GorchSampleCfg* cfgs, const double* uniforms, int32_t* out_ids,
                uint32_t* out_flags, double* out_probs, GorchSampleDebug* out_debug,
                int force_greedy, char** errOut, int32_t* fixed_lists = nullptr, const int32_t* row_done = nullptr) {
  // fixed_lists: caller-provided storage for the row work lists (16 + B + 1 words) instead of the
  // context's grow-only allocation; with it nothing in here allocates.
  if (B == 0) return GORCH_CUDA_OK;
  static_assert(sizeof(GorchSampleCfg) == sizeof(gs::RowCfg), "cfg layout");
  static_assert(sizeof(GorchSampleDebug) == sizeof(gs::RowDebug), "debug layout");
  if ((reinterpret_cast<uintptr_t>(logits) % elem_size(dtype)) != 0) {
    set_err(errOut, "gorch_cuda: logits pointer not aligned to its element size");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  gs::KernelArgs a;
  a.logits = logits;
  a.row_stride = row_stride;
  a.V = static_cast<int32_t>(V);
  a.force_greedy = force_greedy;
  a.cfgs = reinterpret_cast<const gs::RowCfg*>(cfgs);
  a.uniforms = uniforms;
  a.out_ids = out_ids;
  a.out_flags = out_flags;
  a.out_probs = out_probs;
  a.out_debug = reinterpret_cast<gs::RowDebug*>(out_debug);
  a.exp_table = c->exp_table;
  a.row_offset = 0;
  a.worklist = nullptr;
  a.batch_hdr = nullptr;
  a.vs_records = nullptr;
  a.vs_col_offset = 0;
  a.vs_cand = gs::VS_CAND;
  a.vs_sumexp = 0;
  a.row_done = row_done;
  a.tk_values = nullptr;
  a.tk_indices = nullptr;
  a.tk_k = 0;
  if (c->timing) CUDA_TRY(cudaEventRecord(c->ev0, c->stream), errOut);
  int klaunch = 1;
  const bool batch_mode = c->variant == 2 || c->variant >= 4 || (c->variant == 0 && use_batch_mode(c->sm_count, B, V, static_cast<int64_t>(elem_size(dtype)), force_greedy != 0));
  if (batch_mode) {
    // wide (top-k off) with narrow (greedy / top-k) beside it, then single-CTA (whatever was handed over): one stream, each
    // launched while the one before it runs (programmatic dependent launch). The wide kernel goes first and lets the
    // narrow one start when its CTAs have their rows; the narrow kernel ends after the wide one; the third waits for that.
    int32_t* base = fixed_lists;
    if (base) CUDA_TRY(cudaMemsetAsync(base, 0, 16 * sizeof(int32_t), c->stream), errOut);   // (shared by the contexts of a device)
    else if (int rc = batch_lists(c, B, &base, errOut)) return rc;
    gs::BatchArgs ba;
    ba.k = a;
    ba.eb_table = c->eb_table;
    ba.hdr = base;
    ba.list_single = base + gs::HDR_COUNT;
    ba.B = B;
    // at most one row per SM: a 1024-thread CTA finishes its row sooner than a 256-thread one, and no SM
    // would have held a second row anyway. Beyond that the 256-thread instance wins (measured), also
    // because a 1024-thread CTA takes the whole register file and keeps the narrow kernel off its SM
    const bool wide_big_ctas = c->variant == 5 || (c->variant != 4 && B <= c->sm_count);
    const int wctas = wide_big_ctas ? gs::w1024::W_CTAS : gs::w256::W_CTAS;
    const unsigned gw = static_cast<unsigned>(B < wctas * c->sm_count ? B : wctas * c->sm_count);
    const unsigned gsgl = static_cast<unsigned>(B < 2 * c->sm_count ? B : 2 * c->sm_count);
    gs::KernelArgs aw = a;
    aw.worklist = ba.list_single;
    aw.batch_hdr = base;
    if (force_greedy) ba.k.batch_hdr = base;
    const bool f32 = dtype == GORCH_CUDA_F32;
    cudaError_t e = cudaSuccess;
    if (!force_greedy) {
      if (wide_big_ctas) e = launch(c, f32 ? gs::w1024::wide_rows_kernel<float> : gs::w1024::wide_rows_kernel<uint16_t>, gw, gs::w1024::W_NT, gs::w1024::W_DYN_BYTES, false, ba);
      else e = launch(c, f32 ? gs::w256::wide_rows_kernel<float> : gs::w256::wide_rows_kernel<uint16_t>, gw, gs::w256::W_NT, gs::w256::W_DYN_BYTES, false, ba);
    }
    if (e == cudaSuccess) e = launch_narrow(c, ba, dtype, B, !force_greedy);
    if (e == cudaSuccess && !force_greedy) e = launch(c, f32 ? gs::sample_rows_kernel<float> : gs::sample_rows_kernel<uint16_t>, gsgl, gs::NT, gs::POOL_BYTES, true, aw);
    if (e != cudaSuccess) { cudaGetLastError(); cudaMemsetAsync(base, 0, 16 * sizeof(int32_t), c->stream); }   // nobody has left the header cleared
    CUDA_TRY(e, errOut);
    klaunch = force_greedy ? 1 : 3;
  } else if (c->variant == 1) {
    dim3 grid(static_cast<unsigned>(B)), block(gs::NT);
    if (dtype == GORCH_CUDA_F32) {
      gs::sample_rows_kernel<float><<<grid, block, gs::POOL_BYTES, c->stream>>>(a);
    } else {
      gs::sample_rows_kernel<uint16_t><<<grid, block, gs::POOL_BYTES, c->stream>>>(a);
    }
    CUDA_TRY(cudaGetLastError(), errOut);
  } else {
    const int C = cluster_size(c, B, V, dtype);
    if (C == 0) {
      // rows too wide to keep in shared memory: the single-CTA kernel reads global memory
      dim3 grid(static_cast<unsigned>(B)), block(gs::NT);
      if (dtype == GORCH_CUDA_F32) {
        gs::sample_rows_kernel<float><<<grid, block, gs::POOL_BYTES, c->stream>>>(a);
      } else {
        gs::sample_rows_kernel<uint16_t><<<grid, block, gs::POOL_BYTES, c->stream>>>(a);
      }
      CUDA_TRY(cudaGetLastError(), errOut);
    } else {
      gs::ClusterArgs ca;
      ca.k = a;
      const int64_t need = slice_bytes(V, dtype, C);
      ca.slice_bytes = static_cast<int32_t>(need > gs::MIN_SLICE_BYTES ? need : gs::MIN_SLICE_BYTES);
      ca.eb_table = c->eb_table;
      const size_t dyn = static_cast<size_t>(ca.slice_bytes) + gs::REGION_A + gs::REGION_B;
      const bool diag = out_probs || out_debug;
      auto* kernel = (dtype == GORCH_CUDA_F32) ? (diag ? gs::sample_cluster_kernel<float, true> : gs::sample_cluster_kernel<float, false>)
                                               : (diag ? gs::sample_cluster_kernel<uint16_t, true> : gs::sample_cluster_kernel<uint16_t, false>);
      CUDA_TRY(launch_clusters(c, kernel, static_cast<unsigned>(B * C), gs::NT, dyn, true, C, ca), errOut);
      CUDA_TRY(cudaGetLastError(), errOut);
    }
  }
  c->counters.kernel_launches += static_cast<uint64_t>(klaunch);
  if (force_greedy) c->counters.argmax_launches++; else c->counters.sample_launches++;
  c->counters.rows += static_cast<uint64_t>(B);
  if (c->timing) {
    CUDA_TRY(cudaEventRecord(c->ev1, c->stream), errOut);
    CUDA_TRY(cudaEventSynchronize(c->ev1), errOut);
    CUDA_TRY(cudaEventElapsedTime(&c->counters.last_kernel_ms, c->ev0, c->ev1), errOut);
  }
  return GORCH_CUDA_OK;
}

int validate_host_cfgs(const GorchSampleCfg* cfgs, int64_t B, char** errOut) {
  for (int64_t b = 0; b < B; b++) {
    float t = cfgs[b].temperature;
    if (!(t >= 0.0f) || !(t < std::numeric_limits<float>::infinity())) {
      set_err(errOut, "gorch_cuda: row %lld temperature %g is negative, NaN or infinite",
              (long long)b, (double)t);
      return GORCH_CUDA_ERR_BAD_ARG;
    }
    if (cfgs[b].topp_mode != GORCH_TOPP_MODE_A && cfgs[b].topp_mode != GORCH_TOPP_MODE_B) {
      set_err(errOut, "gorch_cuda: row %lld unknown topp_mode %d", (long long)b, cfgs[b].topp_mode);
      return GORCH_CUDA_ERR_BAD_ARG;
    }
  }
  return GORCH_CUDA_OK;
}

int host_run(Ctx* c, const void* logits, int dtype, int64_t B, int64_t V, int64_t row_stride,
             const GorchSampleCfg* cfgs, const double* uniforms, int32_t* out_ids,
             uint32_t* out_flags, int force_greedy, char** errOut) {
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits || !out_ids || (!force_greedy && (!cfgs || !uniforms))) {
    set_err(errOut, "gorch_cuda: null pointer argument");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (!force_greedy) {
    rc = validate_host_cfgs(cfgs, B, errOut);
    if (rc) return rc;
  }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  const size_t es = elem_size(dtype);
  const size_t lbytes = (static_cast<size_t>(B - 1) * row_stride + V) * es;
  // Everything that is small goes through one pinned block of the context: the kernels read configurations and
  // uniforms from it and leave ids and flags in it, so no copy but that of the logits is needed, and the
  // call waits once. Logits of up to kStageBytes in pageable memory take the same way, a piece being copied into the block
  // while the one before it crosses the link; larger ones are left to the driver.
  const size_t off_flags = (static_cast<size_t>(B) * sizeof(int32_t) + 255) & ~static_cast<size_t>(255);
  const size_t off_cfgs = (off_flags + static_cast<size_t>(B) * sizeof(uint32_t) + 255) & ~static_cast<size_t>(255);
  const size_t off_uni = off_cfgs + static_cast<size_t>(B) * sizeof(GorchSampleCfg);
  const size_t off_logits = (off_uni + static_cast<size_t>(B) * sizeof(double) + 255) & ~static_cast<size_t>(255);
  const bool staged = lbytes <= kStageBytes && !is_pinned(logits);
  if ((rc = ensure_pinned(c, off_logits + (staged ? lbytes : 0), errOut))) return rc;
  unsigned char* pin = static_cast<unsigned char*>(c->pinned.ptr);
  if ((rc = ensure(c->st_logits, lbytes, errOut))) return rc;
  if (!force_greedy) {
    memcpy(pin + off_cfgs, cfgs, B * sizeof(GorchSampleCfg));
    memcpy(pin + off_uni, uniforms, B * sizeof(double));
    c->counters.h2d_bytes += B * (sizeof(GorchSampleCfg) + sizeof(double));
  }
  const void* dev_logits = c->st_logits.ptr;
  // The cluster kernel reads each logit once: it can do that from the pinned block, over the link (one GPT-2 row: 45 us a
  // call, 53 with a copy to device memory first). Kernels that read a row again, and rows that need one, get the copy.
  bool once = staged && c->variant == 0 && !use_batch_mode(c->sm_count, B, V, static_cast<int64_t>(es), force_greedy != 0) && cluster_size(c, B, V, dtype) > 0;
  if (!force_greedy) for (int64_t b = 0; b < B && once; b++) once = !(cfgs[b].top_k > gs::KFAST && cfgs[b].top_k < V);
  if (once) {
    memcpy(pin + off_logits, logits, lbytes);
    dev_logits = pin + off_logits;
  } else if (staged) {
    for (size_t at = 0; at < lbytes; at += kStagePiece) {
      const size_t n = lbytes - at < kStagePiece ? lbytes - at : kStagePiece;
      memcpy(pin + off_logits + at, static_cast<const unsigned char*>(logits) + at, n);
      CUDA_TRY(cudaMemcpyAsync(static_cast<unsigned char*>(c->st_logits.ptr) + at, pin + off_logits + at, n, cudaMemcpyHostToDevice, c->stream), errOut);
    }
  } else {
    CUDA_TRY(cudaMemcpyAsync(c->st_logits.ptr, logits, lbytes, cudaMemcpyHostToDevice, c->stream), errOut);
  }
  c->counters.h2d_bytes += lbytes;
  int32_t* pin_ids = reinterpret_cast<int32_t*>(pin);
  uint32_t* pin_flags = reinterpret_cast<uint32_t*>(pin + off_flags);
  rc = launch_rows(c, dev_logits, dtype, B, V, row_stride, reinterpret_cast<const GorchSampleCfg*>(pin + off_cfgs),
                   reinterpret_cast<const double*>(pin + off_uni), pin_ids, out_flags ? pin_flags : nullptr, nullptr, nullptr, force_greedy, errOut);
  // (also after an error: the block is the next call's, and copies out of it may be under way)
  const cudaError_t waited = wait_stream(c);
  if (rc) return rc;
  CUDA_TRY(waited, errOut);
  memcpy(out_ids, pin_ids, B * sizeof(int32_t));
  c->counters.d2h_bytes += B * sizeof(int32_t);
  if (out_flags) {
    memcpy(out_flags, pin_flags, B * sizeof(uint32_t));
    c->counters.d2h_bytes += B * sizeof(uint32_t);
  }
  return GORCH_CUDA_OK;
}

// ---- LM-head projection (lm_head.cuh) ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode_tiled = nullptr;

int load_encode_tiled(char** errOut) {
  if (g_encode_tiled) return GORCH_CUDA_OK;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres), errOut);
  if (!fn || qres != cudaDriverEntryPointSuccess) {
    set_err(errOut, "gorch_cuda: the driver does not offer cuTensorMapEncodeTiled");
    return GORCH_CUDA_ERR_CUDA;
  }
  g_encode_tiled = reinterpret_cast<EncodeTiledFn>(fn);
  return GORCH_CUDA_OK;
}

// Tensor map of a row-major [rows, K] bf16 matrix: boxes of 64 columns x box_rows rows, 128-byte swizzle,
// zero fill outside the matrix.
int make_bf16_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t ld, int box_rows, char** errOut) {
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(gs::LMH_BK), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_err(errOut, "gorch_cuda: cuTensorMapEncodeTiled failed with code %d", static_cast<int>(r));
    return GORCH_CUDA_ERR_CUDA;
  }
  return GORCH_CUDA_OK;
}

int check_lm_head(Ctx* c, const void* x, const void* w, int64_t B, int64_t V, int64_t K, int64_t ldx, int64_t ldw, char** errOut) {
  if (B < 0 || V < 1 || K < gs::LMH_BK || (K % gs::LMH_BK) != 0 || ldx < K || ldw < K) {
    set_err(errOut, "gorch_cuda: LM head needs B >= 0, V >= 1 and K a multiple of %d (got B=%lld V=%lld K=%lld)", gs::LMH_BK,
            (long long)B, (long long)V, (long long)K);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (B > 0x7fffffffll || V > 0x7fffff00ll || K > 0x7fffffffll) { set_err(errOut, "gorch_cuda: LM head shape beyond 31 bits"); return GORCH_CUDA_ERR_LIMIT; }
  if (B == 0) return GORCH_CUDA_OK;
  if (!x || !w) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(w) & 15u) || ((ldx * 2) & 15) || ((ldw * 2) & 15)) {
    set_err(errOut, "gorch_cuda: LM head operands must be 16-byte aligned with row pitches that are multiples of 16 bytes");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  (void)c;
  return GORCH_CUDA_OK;
}

// Shapes of a projection: batch rows of a full item, vocabulary rows per CTA, the ring's stages, the tensor maps.
int lm_head_args(const Ctx* c, gs::LmHeadArgs& a, const void* x, int64_t ldx, const void* w, int64_t ldw, int64_t B, int64_t V, int64_t K,
                 bool writes_logits, char** errOut) {
  memset(&a, 0, sizeof a);
  a.B = static_cast<int32_t>(B); a.V = static_cast<int32_t>(V); a.K = static_cast<int32_t>(K);
  a.item_n = B >= gs::LMH_MAX_N ? gs::LMH_MAX_N : static_cast<int32_t>((B + 31) & ~31ll);
  a.box_n = a.item_n / 2;
  // Up to 128 batch rows the weights' read decides: tiles as high as make the rounds over all SMs come out even
  // (151,936 rows on 148 SMs: nine rounds of 115 rows instead of eight of 128 and one for two pairs). Beyond,
  // the tensor pipe does, and a tile with fewer rows costs it as much as a full one.
  a.cta_v = gs::LMH_CTA_V;
  if (B <= 128) {
    const int64_t sms = c->sm_count & ~1, rounds = (V + sms * gs::LMH_CTA_V - 1) / (sms * gs::LMH_CTA_V);
    a.cta_v = static_cast<int32_t>((V + sms * rounds - 1) / (sms * rounds));
    // whole 32-byte sectors of the output, where that is worth a few rows of padding (32 batch rows: 59.2 us with 115
    // vocabulary rows per CTA, 60.4 with 120; 128 batch rows: 83 and 79)
    if (writes_logits && B > 32) a.cta_v = (a.cta_v + 7) & ~7;
  }
  const int stage = gs::LMH_SUB * (gs::LMH_W_BYTES + a.box_n * gs::LMH_BK * 2);
  a.stages = gs::LMH_RING_BYTES / stage;
  if (a.stages > gs::LMH_MAX_STAGES) a.stages = gs::LMH_MAX_STAGES;
  int rc = make_bf16_map(&a.map_x, x, B, K, ldx, a.box_n, errOut);
  if (rc) return rc;
  return make_bf16_map(&a.map_w, w, V, K, ldw, a.cta_v, errOut);
}

// One launch of lm_head_kernel over the vocabulary tiles tile0 + i * step, i < ntile. chained: behind the kernel that fills the
// thresholds. dependent: it may start beside the end of the kernel before it (the first one of a chain does not: the
// chain's second projection reads x and w without waiting for what came before the chain).
int launch_lm_head(Ctx* c, gs::LmHeadArgs& a, char** errOut, bool dependent, bool chained = false) {
  const int64_t ntile_total = (static_cast<int64_t>(a.V) + 2 * a.cta_v - 1) / (2 * a.cta_v);
  if (a.ntile < 1 || a.tile0 + static_cast<int64_t>(a.ntile - 1) * a.tile_step >= ntile_total) {
    set_err(errOut, "gorch_cuda: LM head tile range outside the vocabulary");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  const int most = c->sm_count / 2;
  int npairs = gs::LmhPlan(a.B, a.ntile, a.item_n, most).total;
  if (npairs > most) npairs = most;
  a.status = c->host_words;
  a.chained = chained ? 1 : 0;
  a.clear_status = chained ? 0 : 1;
  CUDA_TRY(launch(c, gs::lm_head_kernel, static_cast<unsigned>(2 * npairs), gs::LMH_NT, gs::LMH_DYN_BYTES, dependent, a), errOut);
  c->counters.kernel_launches += 1;
  return GORCH_CUDA_OK;
}

template <typename SH>
cudaError_t topk_large_attributes() {
  const cudaError_t e = cudaFuncSetAttribute(gs::topk_large_kernel<float, SH>, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::DYN_BYTES);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(gs::topk_large_kernel<uint16_t, SH>, cudaFuncAttributeMaxDynamicSharedMemorySize, SH::DYN_BYTES);
}

}  // namespace

extern "C" {

int gorch_cuda_device_count(int* count, char** errOut) {
  if (!count) { set_err(errOut, "gorch_cuda: null count"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaGetDeviceCount(count), errOut);
  return GORCH_CUDA_OK;
}

GorchCudaCtxRef gorch_cuda_create_ctx(int device, char** errOut) {
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n <= 0) {
    set_err(errOut, "gorch_cuda: no CUDA device (%s)", cudaGetErrorString(e));
    return nullptr;
  }
  if (device < 0 || device >= n) {
    set_err(errOut, "gorch_cuda: device %d out of range [0,%d)", device, n);
    return nullptr;
  }
  Ctx* c = new (std::nothrow) Ctx();
  if (!c) { set_err(errOut, "gorch_cuda: out of host memory"); return nullptr; }
  c->device = device;
  g_pool.enter();
  auto fail = [&](const char* what, cudaError_t err) -> GorchCudaCtxRef {
    set_err(errOut, "gorch_cuda: %s failed: %s", what, cudaGetErrorString(err));
    gorch_cuda_release(c);
    return nullptr;
  };
  if ((e = cudaSetDevice(device)) != cudaSuccess) return fail("cudaSetDevice", e);
  cudaDeviceProp prop;
  if ((e = cudaGetDeviceProperties(&prop, device)) != cudaSuccess) return fail("cudaGetDeviceProperties", e);
  if (prop.major < 10) {
    set_err(errOut, "gorch_cuda: device %d is sm_%d%d; this library is built for sm_100a only",
            device, prop.major, prop.minor);
    gorch_cuda_release(c);
    return nullptr;
  }
  c->sm_count = prop.multiProcessorCount;
  if (prop.l2CacheSize > 0) c->l2_bytes = prop.l2CacheSize;
  if ((e = cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking)) != cudaSuccess) return fail("cudaStreamCreate", e);
  c->stream = c->own_stream;
  if ((e = cudaEventCreate(&c->ev0)) != cudaSuccess) return fail("cudaEventCreate", e);
  if ((e = cudaEventCreate(&c->ev1)) != cudaSuccess) return fail("cudaEventCreate", e);
  if ((e = cudaEventCreateWithFlags(&c->ev_left, cudaEventDisableTiming)) != cudaSuccess) return fail("cudaEventCreate", e);
  {
    // device address of the fixed work-list array of gorch_cuda_sample_dev_static on this device
    int32_t* unused = nullptr;
    char* msg = nullptr;
    if (static_lists_ptr(device, &unused, &msg) != GORCH_CUDA_OK) {
      if (errOut) *errOut = msg; else free(msg);
      gorch_cuda_release(c);
      return nullptr;
    }
  }
  if ((e = cudaHostAlloc(reinterpret_cast<void**>(&c->host_words), 64, cudaHostAllocMapped | cudaHostAllocPortable)) != cudaSuccess) return fail("cudaHostAlloc", e);
  memset(c->host_words, 0, 64);
  double tab[256];
  for (int j = 0; j < 256; j++) tab[j] = static_cast<double>(exp2l(static_cast<long double>(j) / 256.0L));
  if ((e = cudaMalloc(&c->exp_table, sizeof tab)) != cudaSuccess) return fail("cudaMalloc(exp table)", e);
  if ((e = cudaMemcpy(c->exp_table, tab, sizeof tab, cudaMemcpyHostToDevice)) != cudaSuccess) return fail("cudaMemcpy(exp table)", e);
  static double ebt[gs::NB1];
  for (int j = 0; j < gs::NB1; j++) ebt[j] = static_cast<double>(expl(-static_cast<long double>(j) / 32.0L));
  if ((e = cudaMalloc(&c->eb_table, sizeof ebt)) != cudaSuccess) return fail("cudaMalloc(bucket table)", e);
  if ((e = cudaMemcpy(c->eb_table, ebt, sizeof ebt, cudaMemcpyHostToDevice)) != cudaSuccess) return fail("cudaMemcpy(bucket table)", e);
  if ((e = cudaFuncSetAttribute(gs::sample_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::POOL_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::sample_rows_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::POOL_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::sample_cluster_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 109 * 1024)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::sample_cluster_kernel<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 109 * 1024)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::sample_cluster_kernel<uint16_t, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 109 * 1024)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::sample_cluster_kernel<uint16_t, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 109 * 1024)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n256::narrow_rows_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n256::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n256::narrow_rows_kernel<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n256::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n256::narrow_rows_kernel<uint16_t, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n256::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n256::narrow_rows_kernel<uint16_t, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n256::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n256d::narrow_rows_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n256d::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n256d::narrow_rows_kernel<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n256d::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n128::narrow_rows_kernel<float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n128::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n128::narrow_rows_kernel<float, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n128::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n128::narrow_rows_kernel<uint16_t, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n128::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::n128::narrow_rows_kernel<uint16_t, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::n128::N_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::multinomial_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::MN_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = topk_large_attributes<gs::TklSmall>()) != cudaSuccess || (e = topk_large_attributes<gs::TklFew>()) != cudaSuccess ||
      (e = topk_large_attributes<gs::TklMid>()) != cudaSuccess || (e = topk_large_attributes<gs::TklLarge>()) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::vocab_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::VM_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::w256::wide_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::w256::W_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::w1024::wide_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::w1024::W_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::w1024::wide_rows_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::w1024::W_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::lm_head_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::LMH_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::lmh_finish_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::LMH_F_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::row_softmax_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::RS_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::row_softmax_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::RS_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::row_softmax_resident_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::RR_SLICE)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::row_softmax_resident_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::RR_SLICE)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  if ((e = cudaFuncSetAttribute(gs::w256::wide_rows_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs::w256::W_DYN_BYTES)) != cudaSuccess) return fail("cudaFuncSetAttribute", e);
  return c;
}

void gorch_cuda_release(GorchCudaCtxRef ctx) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->own_stream) { cudaStreamSynchronize(c->own_stream); }
  if (c->st_logits.ptr) cudaFree(c->st_logits.ptr);
  if (c->pinned.ptr) cudaFreeHost(c->pinned.ptr);
  if (c->host_words) cudaFreeHost(c->host_words);
  if (c->exp_table) cudaFree(c->exp_table);
  if (c->eb_table) cudaFree(c->eb_table);
  if (c->worklist.ptr) cudaFree(c->worklist.ptr);
  if (c->comm && g_nccl.CommDestroy) g_nccl.CommDestroy(c->comm);
  if (c->lmh_scratch.ptr) cudaFree(c->lmh_scratch.ptr);
  if (c->lmh_logits.ptr) cudaFree(c->lmh_logits.ptr);
  if (c->vs_local.ptr) cudaFree(c->vs_local.ptr);
  if (c->vs_all.ptr) cudaFree(c->vs_all.ptr);
  if (c->vs_req.ptr) cudaFree(c->vs_req.ptr);
  if (c->vs_rows.ptr) cudaFree(c->vs_rows.ptr);
  if (c->vs_done.ptr) cudaFree(c->vs_done.ptr);
  for (cudaEvent_t e : c->ev_vs) if (e) cudaEventDestroy(e);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  if (c->ev_left) cudaEventDestroy(c->ev_left);
  if (c->own_stream) cudaStreamDestroy(c->own_stream);
  g_pool.leave();
  delete c;
}

void gorch_cuda_free_string(char* s) { free(s); }

int gorch_cuda_sync(GorchCudaCtxRef ctx, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(wait_stream(c), errOut);
  return GORCH_CUDA_OK;
}

int gorch_cuda_set_stream(GorchCudaCtxRef ctx, void* stream, int external, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  const cudaStream_t next = external ? static_cast<cudaStream_t>(stream) : c->own_stream;
  if (next == c->stream) return GORCH_CUDA_OK;
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  // Scratch memory and the header of the work lists, which a sorted batch finds cleared and leaves cleared, serve one call
  // at a time: what is queued and was not waited for comes before whatever the next stream gets. A stream that is
  // being recorded takes no part (its work runs when the graph does); the event then waits for the stream after it.
  if (c->counters.kernel_launches != c->waited_launches && capture_status(c->stream) == cudaStreamCaptureStatusNone) {
    if (c->left_pending) CUDA_TRY(cudaStreamWaitEvent(c->stream, c->ev_left, 0), errOut);
    CUDA_TRY(cudaEventRecord(c->ev_left, c->stream), errOut);
    c->left_pending = true;
  }
  c->stream = next;
  if (c->left_pending && capture_status(next) == cudaStreamCaptureStatusNone) {
    CUDA_TRY(cudaStreamWaitEvent(next, c->ev_left, 0), errOut);
    c->left_pending = false;
  }
  return GORCH_CUDA_OK;
}

int gorch_cuda_set_timing(GorchCudaCtxRef ctx, int on) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) return GORCH_CUDA_ERR_BAD_ARG;
  c->timing = on ? 1 : 0;
  return GORCH_CUDA_OK;
}

int gorch_cuda_set_kernel_variant(GorchCudaCtxRef ctx, int variant, int cluster_size, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  if ((variant < 0 || variant > 7) ||
      !(cluster_size == 0 || cluster_size == 1 || cluster_size == 2 || cluster_size == 4 || cluster_size == 8)) {
    set_err(errOut, "gorch_cuda: variant must be 0..7, cluster_size 0, 1, 2, 4 or 8");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  c->variant = variant;
  c->force_cluster = cluster_size;
  return GORCH_CUDA_OK;
}

int gorch_cuda_get_counters(GorchCudaCtxRef ctx, GorchCudaCounters* out) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c || !out) return GORCH_CUDA_ERR_BAD_ARG;
  *out = c->counters;
  return GORCH_CUDA_OK;
}

GorchCudaBufferRef gorch_cuda_buffer_alloc(GorchCudaCtxRef ctx, uint64_t bytes, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return nullptr; }
  Buffer* b = new (std::nothrow) Buffer{c->device, nullptr, bytes, BufferPool::block_of(bytes)};
  if (!b) { set_err(errOut, "gorch_cuda: out of host memory"); return nullptr; }
  cudaError_t e = cudaSetDevice(c->device);
  if (e == cudaSuccess && b->block) b->ptr = g_pool.take(c->device, b->block);
  if (e == cudaSuccess && !b->ptr) e = cudaMalloc(&b->ptr, b->block ? b->block : bytes);
  if (e != cudaSuccess) {
    set_err(errOut, "gorch_cuda: cudaMalloc(%llu) failed: %s", (unsigned long long)bytes, cudaGetErrorString(e));
    delete b;
    return nullptr;
  }
  return b;
}

void gorch_cuda_buffer_free(GorchCudaBufferRef buf) {
  Buffer* b = static_cast<Buffer*>(buf);
  if (!b) return;
  if (!b->block || !g_pool.put(b->device, b->ptr, b->block)) {
    cudaSetDevice(b->device);
    cudaFree(b->ptr);
  }
  delete b;
}

uint64_t gorch_cuda_buffer_length(GorchCudaBufferRef buf) {
  Buffer* b = static_cast<Buffer*>(buf);
  return b ? b->bytes : 0;
}

void* gorch_cuda_buffer_device_ptr(GorchCudaBufferRef buf) {
  Buffer* b = static_cast<Buffer*>(buf);
  return b ? b->ptr : nullptr;
}

int gorch_cuda_buffer_upload(GorchCudaBufferRef buf, uint64_t offset, const void* host,
                             uint64_t bytes, char** errOut) {
  Buffer* b = static_cast<Buffer*>(buf);
  if (!b || (!host && bytes) || offset > b->bytes || bytes > b->bytes - offset) {
    set_err(errOut, "gorch_cuda: upload out of range");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  CUDA_TRY(cudaSetDevice(b->device), errOut);
  CUDA_TRY(cudaMemcpy(static_cast<char*>(b->ptr) + offset, host, bytes, cudaMemcpyHostToDevice), errOut);
  return GORCH_CUDA_OK;
}

int gorch_cuda_buffer_download(GorchCudaBufferRef buf, uint64_t offset, void* host,
                               uint64_t bytes, char** errOut) {
  Buffer* b = static_cast<Buffer*>(buf);
  if (!b || (!host && bytes) || offset > b->bytes || bytes > b->bytes - offset) {
    set_err(errOut, "gorch_cuda: download out of range");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  CUDA_TRY(cudaSetDevice(b->device), errOut);
  CUDA_TRY(cudaMemcpy(host, static_cast<char*>(b->ptr) + offset, bytes, cudaMemcpyDeviceToHost), errOut);
  return GORCH_CUDA_OK;
}

int gorch_cuda_sample_host(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                           int64_t V, int64_t row_stride, const GorchSampleCfg* cfgs,
                           const double* uniforms, int32_t* out_ids, uint32_t* out_flags,
                           char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  return host_run(c, logits, dtype, B, V, row_stride, cfgs, uniforms, out_ids, out_flags, 0, errOut);
}

int gorch_cuda_sample_dev(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                          int64_t V, int64_t row_stride, const GorchSampleCfg* cfgs,
                          const double* uniforms, int32_t* out_ids, uint32_t* out_flags,
                          double* out_probs, GorchSampleDebug* out_debug, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits || !cfgs || !uniforms || !out_ids) {
    set_err(errOut, "gorch_cuda: null pointer argument");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  return launch_rows(c, logits, dtype, B, V, row_stride, cfgs, uniforms, out_ids, out_flags,
                     out_probs, out_debug, 0, errOut);
}

static int vocab_local_launch(Ctx* c, const void* logits, int dtype, int64_t B, int64_t Vslice, int64_t row_stride,
                              int64_t col_offset, const GorchSampleCfg* cfgs, void* records, int cand, char** errOut,
                              bool sumexp_rows = true) {
  int rc = check_shape(dtype, B, Vslice, row_stride, errOut);
  if (rc) return rc;
  static_assert(sizeof(gs::VsRecord) == GORCH_VS_RECORD_BYTES, "record layout");
  if (col_offset < 0 || col_offset + Vslice > 0x7fffff00ll) {
    set_err(errOut, "gorch_cuda: column offset %lld out of range", (long long)col_offset);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (cand < 1 || cand > gs::VS_CAND) {
    set_err(errOut, "gorch_cuda: %d candidates per record outside 1..%d", cand, gs::VS_CAND);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits || !cfgs || !records) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(logits) % elem_size(dtype)) != 0) {
    set_err(errOut, "gorch_cuda: logits pointer not aligned to its element size");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  // every row goes through the narrow kernel (row_kind says so when vs_records is set)
  int32_t* base = nullptr;
  if ((rc = batch_lists(c, B, &base, errOut))) return rc;
  gs::BatchArgs ba;
  ba.k.logits = logits; ba.k.row_stride = row_stride; ba.k.V = static_cast<int32_t>(Vslice);
  ba.k.force_greedy = 0; ba.k.cfgs = reinterpret_cast<const gs::RowCfg*>(cfgs); ba.k.uniforms = nullptr;
  ba.k.out_ids = nullptr; ba.k.out_flags = nullptr; ba.k.out_probs = nullptr; ba.k.out_debug = nullptr;
  ba.k.exp_table = c->exp_table; ba.k.row_offset = 0; ba.k.worklist = nullptr; ba.k.batch_hdr = base;
  ba.k.vs_records = records; ba.k.vs_col_offset = static_cast<int32_t>(col_offset); ba.k.vs_cand = cand;
  ba.k.vs_sumexp = sumexp_rows ? 1 : 0;
  ba.k.tk_values = nullptr; ba.k.tk_indices = nullptr; ba.k.tk_k = 0; ba.k.row_done = nullptr;
  ba.eb_table = c->eb_table;
  ba.hdr = base; ba.list_single = base + gs::HDR_COUNT;
  ba.B = B;
  CUDA_TRY(launch_narrow(c, ba, dtype, B, false), errOut);
  c->counters.kernel_launches += 1;
  if (sumexp_rows) {                                         // the records of rows without top-k: disjoint rows, same stream
    const unsigned g = static_cast<unsigned>(B < 4 * c->sm_count ? B : 4 * c->sm_count);
    if (dtype == GORCH_CUDA_F32) gs::vocab_sumexp_kernel<float><<<g, gs::VD_NT, 0, c->stream>>>(ba.k, c->eb_table, B);
    else gs::vocab_sumexp_kernel<uint16_t><<<g, gs::VD_NT, 0, c->stream>>>(ba.k, c->eb_table, B);
    c->counters.kernel_launches += 1;
  }
  CUDA_TRY(cudaGetLastError(), errOut);
  return GORCH_CUDA_OK;
}

static int vocab_merge_launch(Ctx* c, const void* all_records, int nranks, int cand, int64_t B, int64_t V,
                              const GorchSampleCfg* cfgs, const double* uniforms, int32_t* out_ids,
                              uint32_t* out_flags, char** errOut, int my_rank = -1, double* draw_req = nullptr) {
  if (nranks < 1 || nranks > gs::VM_MAX_RANKS) {
    set_err(errOut, "gorch_cuda: vocab merge takes 1..%d ranks, got %d", gs::VM_MAX_RANKS, nranks);
    return GORCH_CUDA_ERR_LIMIT;
  }
  int rc = check_shape(GORCH_CUDA_F32, B, V, V, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!all_records || !cfgs || !uniforms || !out_ids) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  gs::MergeArgs m;
  m.k.logits = nullptr; m.k.row_stride = V; m.k.V = static_cast<int32_t>(V); m.k.force_greedy = 0;
  m.k.cfgs = reinterpret_cast<const gs::RowCfg*>(cfgs); m.k.uniforms = uniforms;
  m.k.out_ids = out_ids; m.k.out_flags = out_flags; m.k.out_probs = nullptr; m.k.out_debug = nullptr;
  m.k.exp_table = c->exp_table; m.k.row_offset = 0; m.k.worklist = nullptr; m.k.batch_hdr = nullptr; m.k.vs_records = nullptr; m.k.vs_col_offset = 0;
  m.k.vs_cand = cand;
  m.k.vs_sumexp = 0;
  m.k.tk_values = nullptr; m.k.tk_indices = nullptr; m.k.tk_k = 0; m.k.row_done = nullptr;
  m.records = all_records;
  m.nranks = nranks;
  m.cand = cand;
  m.B = B;
  m.my_rank = my_rank;
  m.draw_req = draw_req;
  const unsigned g = static_cast<unsigned>(B < 8 * c->sm_count ? B : 8 * c->sm_count);
  gs::vocab_merge_kernel<<<g, gs::VM_NT, gs::vm_dyn_bytes(nranks, cand), c->stream>>>(m);
  CUDA_TRY(cudaGetLastError(), errOut);
  c->counters.kernel_launches += 1;
  c->counters.sample_launches += 1;
  c->counters.rows += B;
  return GORCH_CUDA_OK;
}

int gorch_cuda_vocab_local_dev(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                               int64_t Vslice, int64_t row_stride, int64_t col_offset,
                               const GorchSampleCfg* cfgs, void* records, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  return vocab_local_launch(c, logits, dtype, B, Vslice, row_stride, col_offset, cfgs, records, gs::VS_CAND, errOut);
}

int gorch_cuda_vocab_merge_dev(GorchCudaCtxRef ctx, const void* all_records, int nranks, int64_t B,
                               int64_t V, const GorchSampleCfg* cfgs, const double* uniforms,
                               int32_t* out_ids, uint32_t* out_flags, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  return vocab_merge_launch(c, all_records, nranks, gs::VS_CAND, B, V, cfgs, uniforms, out_ids, out_flags, errOut);
}

int gorch_cuda_vocab_merge_owner_dev(GorchCudaCtxRef ctx, const void* all_records, int nranks, int my_rank, int64_t B,
                                     int64_t V, const GorchSampleCfg* cfgs, const double* uniforms,
                                     int32_t* out_ids, uint32_t* out_flags, double* draw_req, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (my_rank < 0 || my_rank >= nranks || !draw_req) { set_err(errOut, "gorch_cuda: bad rank or null draw request buffer"); return GORCH_CUDA_ERR_BAD_ARG; }
  return vocab_merge_launch(c, all_records, nranks, gs::VS_CAND, B, V, cfgs, uniforms, out_ids, out_flags, errOut, my_rank, draw_req);
}

static int vocab_draw_launch(Ctx* c, const void* logits_slice, int dtype, int64_t B, int64_t Vslice, int64_t row_stride,
                             int64_t col_offset, const GorchSampleCfg* cfgs, const double* draw_req, int32_t* out_ids,
                             uint32_t* out_flags, char** errOut) {
  int rc = check_shape(dtype, B, Vslice, row_stride, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits_slice || !cfgs || !draw_req || !out_ids) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  gs::DrawArgs d;
  d.logits = logits_slice; d.row_stride = row_stride; d.V = static_cast<int32_t>(Vslice);
  d.col_offset = static_cast<int32_t>(col_offset);
  d.cfgs = reinterpret_cast<const gs::RowCfg*>(cfgs); d.draw_req = draw_req;
  d.eb_table = c->eb_table; d.exp_table = c->exp_table;
  d.out_ids = out_ids; d.out_flags = out_flags; d.B = B;
  const unsigned g = static_cast<unsigned>(B < 4 * c->sm_count ? B : 4 * c->sm_count);
  if (dtype == GORCH_CUDA_F32) gs::vocab_draw_kernel<float><<<g, gs::VD_NT, 0, c->stream>>>(d);
  else gs::vocab_draw_kernel<uint16_t><<<g, gs::VD_NT, 0, c->stream>>>(d);
  CUDA_TRY(cudaGetLastError(), errOut);
  c->counters.kernel_launches += 1;
  return GORCH_CUDA_OK;
}

int gorch_cuda_vocab_draw_dev(GorchCudaCtxRef ctx, const void* logits_slice, int dtype, int64_t B, int64_t Vslice,
                              int64_t row_stride, int64_t col_offset, const GorchSampleCfg* cfgs,
                              const double* draw_req, int32_t* out_ids, uint32_t* out_flags, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  return vocab_draw_launch(c, logits_slice, dtype, B, Vslice, row_stride, col_offset, cfgs, draw_req, out_ids, out_flags, errOut);
}

int gorch_cuda_comm_unique_id(void* id_bytes, char** errOut) {
  static_assert(sizeof(ncclUniqueId) == GORCH_CUDA_UNIQUE_ID_BYTES, "unique id size");
  if (!id_bytes) { set_err(errOut, "gorch_cuda: null unique-id buffer"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = load_nccl(errOut);
  if (rc) return rc;
  ncclUniqueId id;
  NCCL_TRY(g_nccl.GetUniqueId(&id), errOut);
  memcpy(id_bytes, &id, sizeof id);
  return GORCH_CUDA_OK;
}

int gorch_cuda_comm_init(GorchCudaCtxRef ctx, int rank, int nranks, const void* unique_id_bytes, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (!unique_id_bytes || nranks < 1 || nranks > gs::VM_MAX_RANKS || rank < 0 || rank >= nranks) {
    set_err(errOut, "gorch_cuda: comm_init needs a unique id and 0 <= rank < nranks <= %d (got rank %d of %d)",
            gs::VM_MAX_RANKS, rank, nranks);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (c->comm) { set_err(errOut, "gorch_cuda: the context already has a communicator"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = load_nccl(errOut);
  if (rc) return rc;
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  ncclUniqueId id;
  memcpy(&id, unique_id_bytes, sizeof id);
  ncclComm_t comm = nullptr;
  NCCL_TRY(g_nccl.CommInitRank(&comm, nranks, id, rank), errOut);
  for (int i = 0; i < 4; i++) {
    if (!c->ev_vs[i]) CUDA_TRY(cudaEventCreate(&c->ev_vs[i]), errOut);
  }
  c->comm = comm;
  c->comm_rank = rank;
  c->comm_nranks = nranks;
  return GORCH_CUDA_OK;
}

int gorch_cuda_comm_release(GorchCudaCtxRef ctx, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (!c->comm) return GORCH_CUDA_OK;
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  CUDA_TRY(wait_stream(c), errOut);
  ncclComm_t comm = c->comm;
  c->comm = nullptr;
  c->comm_nranks = 0;
  NCCL_TRY(g_nccl.CommDestroy(comm), errOut);
  return GORCH_CUDA_OK;
}

static int sample_vocab_sharded(GorchCudaCtxRef ctx, const void* logits_slice, int dtype, int64_t B,
                                int64_t Vslice, int64_t row_stride, int64_t col_offset, int64_t V,
                                int max_top_k, int rows_without_top_k, const GorchSampleCfg* cfgs, const double* uniforms,
                                int32_t* out_ids, uint32_t* out_flags, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (!c->comm) { set_err(errOut, "gorch_cuda: no communicator: call gorch_cuda_comm_init first"); return GORCH_CUDA_ERR_NCCL; }
  if (V < 1 || col_offset < 0 || col_offset + Vslice > V) {
    set_err(errOut, "gorch_cuda: slice [%lld, %lld) outside the vocabulary of %lld", (long long)col_offset,
            (long long)(col_offset + Vslice), (long long)V);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  // candidates per record: the largest top_k of the batch plus room for ties at the local threshold,
  // in steps of eight (0: the full record)
  int cand = gs::VS_CAND;
  if (max_top_k > 0 && max_top_k <= gs::VS_CAND) cand = ((max_top_k + max_top_k / 4 + 8 + 7) / 8) * 8;
  if (cand > gs::VS_CAND) cand = gs::VS_CAND;
  if (B == 0) return GORCH_CUDA_OK;
  const size_t rec_bytes = 16 + 8 * static_cast<size_t>(cand);
  int rc = ensure(c->vs_local, static_cast<size_t>(B) * rec_bytes, errOut);
  if (rc) return rc;
  rc = ensure(c->vs_all, static_cast<size_t>(B) * rec_bytes * static_cast<size_t>(c->comm_nranks), errOut);
  if (rc) return rc;
  if (c->timing) CUDA_TRY(cudaEventRecord(c->ev_vs[0], c->stream), errOut);
  rc = vocab_local_launch(c, logits_slice, dtype, B, Vslice, row_stride, col_offset, cfgs, c->vs_local.ptr, cand, errOut,
                          (rows_without_top_k & 1) != 0);
  if (rc) return rc;
  if (c->timing) CUDA_TRY(cudaEventRecord(c->ev_vs[1], c->stream), errOut);
  // ONE collective: every rank's records to every rank, in rank order, on the context's stream
  NCCL_TRY(g_nccl.AllGather(c->vs_local.ptr, c->vs_all.ptr, static_cast<size_t>(B) * rec_bytes, ncclUint8, c->comm, c->stream), errOut);
  if (c->timing) CUDA_TRY(cudaEventRecord(c->ev_vs[2], c->stream), errOut);
  if (rows_without_top_k & 1) {
    // Rows without top-k: the merge names each such row's owner (the rank in whose slice u * S
    // falls), the owner finds the token in its slice, and an all-reduce (max) of ids and flags
    // hands it to every rank (the others wrote -1 and 0; rows with a top-k agree on every rank).
    if (!out_flags) { set_err(errOut, "gorch_cuda: rows without top-k need out_flags"); return GORCH_CUDA_ERR_BAD_ARG; }
    rc = ensure(c->vs_req, static_cast<size_t>(B) * 3 * sizeof(double), errOut);
    if (rc) return rc;
    double* req = static_cast<double*>(c->vs_req.ptr);
    rc = vocab_merge_launch(c, c->vs_all.ptr, c->comm_nranks, cand, B, V, cfgs, uniforms, out_ids, out_flags, errOut, c->comm_rank, req);
    if (rc) return rc;
    rc = vocab_draw_launch(c, logits_slice, dtype, B, Vslice, row_stride, col_offset, cfgs, req, out_ids, out_flags, errOut);
    if (rc) return rc;
    NCCL_TRY(g_nccl.AllReduce(out_ids, out_ids, static_cast<size_t>(B), ncclInt32, ncclMax, c->comm, c->stream), errOut);
    NCCL_TRY(g_nccl.AllReduce(out_flags, out_flags, static_cast<size_t>(B), ncclUint32, ncclMax, c->comm, c->stream), errOut);
  } else {
    rc = vocab_merge_launch(c, c->vs_all.ptr, c->comm_nranks, cand, B, V, cfgs, uniforms, out_ids, out_flags, errOut);
    if (rc) return rc;
  }
  if (rows_without_top_k & 2) {
    // Rows without top-k that the records cannot serve (a top-p cut over the whole vocabulary; with
    // bit 0 clear every row without top-k): the rows themselves are brought together — every rank
    // puts its slice into a zeroed [B, V] buffer and an all-reduce (sum) fills in the others' (x + 0
    // is x in any order; a -0 may come out as +0, which no comparison or exponential tells apart) —
    // and the ordinary kernels sample those rows on every rank, all others masked out. Correct, not
    // fast: V * B elements cross the links twice.
    if (!out_flags) { set_err(errOut, "gorch_cuda: gathered rows need out_flags"); return GORCH_CUDA_ERR_BAD_ARG; }
    const size_t es = elem_size(dtype);
    const int64_t ldv = (V + 15) & ~15ll;
    rc = ensure(c->vs_rows, static_cast<size_t>(B) * ldv * es, errOut);
    if (rc) return rc;
    rc = ensure(c->vs_done, static_cast<size_t>(B) * sizeof(int32_t), errOut);
    if (rc) return rc;
    CUDA_TRY(cudaMemsetAsync(c->vs_rows.ptr, 0, static_cast<size_t>(B) * ldv * es, c->stream), errOut);
    CUDA_TRY(cudaMemcpy2DAsync(static_cast<unsigned char*>(c->vs_rows.ptr) + static_cast<size_t>(col_offset) * es, ldv * es,
                               logits_slice, static_cast<size_t>(row_stride) * es, static_cast<size_t>(Vslice) * es,
                               static_cast<size_t>(B), cudaMemcpyDeviceToDevice, c->stream), errOut);
    const ncclDataType_t nt = dtype == GORCH_CUDA_F32 ? ncclFloat32 : static_cast<ncclDataType_t>(9);   // 9: ncclBfloat16
    NCCL_TRY(g_nccl.AllReduce(c->vs_rows.ptr, c->vs_rows.ptr, static_cast<size_t>(B) * ldv, nt, ncclSum, c->comm, c->stream), errOut);
    const unsigned gm = static_cast<unsigned>((B + 255) / 256);
    gs::vocab_gather_mask_kernel<<<gm, 256, 0, c->stream>>>(reinterpret_cast<const gs::RowCfg*>(cfgs), static_cast<int32_t>(V), B,
                                                            (rows_without_top_k & 1) != 0, static_cast<int32_t*>(c->vs_done.ptr));
    CUDA_TRY(cudaGetLastError(), errOut);
    c->counters.kernel_launches += 1;
    rc = launch_rows(c, c->vs_rows.ptr, dtype, B, V, ldv, cfgs, uniforms, out_ids, out_flags, nullptr, nullptr, 0, errOut, nullptr,
                     static_cast<const int32_t*>(c->vs_done.ptr));
    if (rc) return rc;
  }
  if (c->timing) {
    CUDA_TRY(cudaEventRecord(c->ev_vs[3], c->stream), errOut);
    CUDA_TRY(cudaEventSynchronize(c->ev_vs[3]), errOut);
    CUDA_TRY(cudaEventElapsedTime(&c->counters.vs_local_ms, c->ev_vs[0], c->ev_vs[1]), errOut);
    CUDA_TRY(cudaEventElapsedTime(&c->counters.vs_gather_ms, c->ev_vs[1], c->ev_vs[2]), errOut);
    CUDA_TRY(cudaEventElapsedTime(&c->counters.vs_merge_ms, c->ev_vs[2], c->ev_vs[3]), errOut);
    CUDA_TRY(cudaEventElapsedTime(&c->counters.last_kernel_ms, c->ev_vs[0], c->ev_vs[3]), errOut);
  }
  return GORCH_CUDA_OK;
}

int gorch_cuda_sample_vocab_sharded_dev(GorchCudaCtxRef ctx, const void* logits_slice, int dtype, int64_t B,
                                        int64_t Vslice, int64_t row_stride, int64_t col_offset, int64_t V,
                                        int max_top_k, const GorchSampleCfg* cfgs, const double* uniforms,
                                        int32_t* out_ids, uint32_t* out_flags, char** errOut) {
  return sample_vocab_sharded(ctx, logits_slice, dtype, B, Vslice, row_stride, col_offset, V, max_top_k, 0, cfgs, uniforms,
                              out_ids, out_flags, errOut);
}

int gorch_cuda_sample_vocab_sharded_ex_dev(GorchCudaCtxRef ctx, const void* logits_slice, int dtype, int64_t B,
                                           int64_t Vslice, int64_t row_stride, int64_t col_offset, int64_t V,
                                           int max_top_k, int rows_without_top_k, const GorchSampleCfg* cfgs,
                                           const double* uniforms, int32_t* out_ids, uint32_t* out_flags, char** errOut) {
  return sample_vocab_sharded(ctx, logits_slice, dtype, B, Vslice, row_stride, col_offset, V, max_top_k, rows_without_top_k,
                              cfgs, uniforms, out_ids, out_flags, errOut);
}

}  // extern "C"
template <typename SH>
static void launch_topk_large(Ctx* c, const gs::TopKLargeArgs& ta, int dtype) {
  const int64_t slots = static_cast<int64_t>(SH::MINB) * c->sm_count;
  const unsigned g = static_cast<unsigned>(ta.B < slots ? ta.B : slots);
  if (dtype == GORCH_CUDA_F32) gs::topk_large_kernel<float, SH><<<g, SH::NT, SH::DYN_BYTES, c->stream>>>(ta);
  else gs::topk_large_kernel<uint16_t, SH><<<g, SH::NT, SH::DYN_BYTES, c->stream>>>(ta);
}
extern "C" {

int gorch_cuda_topk_dev(GorchCudaCtxRef ctx, const void* x, int dtype, int64_t B, int64_t V,
                        int64_t row_stride, int64_t k, float* out_values, int32_t* out_indices,
                        uint32_t* out_flags, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (k < 1 || k > V) {                                    // the reference panics here (index_ops.go:160-162)
    set_err(errOut, "gorch_cuda: TopK k=%lld out of range [1, %lld]", (long long)k, (long long)V);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (k > gs::TKL_MAX_K) {
    set_err(errOut, "gorch_cuda: TopK supports k <= %d, got %lld", gs::TKL_MAX_K, (long long)k);
    return GORCH_CUDA_ERR_LIMIT;
  }
  if (B == 0) return GORCH_CUDA_OK;
  if (!x || !out_values || !out_indices) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  // The narrow kernel (a row per CTA, phases that grow with k) for small k over rows that are not long: us, narrow | the
  // other, 512 rows: 50,257 f32, k = 16: 47 | 53; 40: 53 | 53; 64: 57 | 53; bf16, k = 64: 43 | 47; 151,936 f32, k = 4: 92 | 86.
  // Up to one row per SM the other one wins for every k: all of an SM's threads read the row (us, narrow | this, f32,
  // k = 40: 32 x 4,000: 23 | 14; 32 x 50,257: 33 | 20; 8 x 151,936: 45 | 25; 128 x 151,936: 49 | 31).
  const int64_t min_k = V * static_cast<int64_t>(elem_size(dtype)) >= (400 << 10) ? 0 : (dtype == GORCH_CUDA_F32 ? gs::TKL_MIN_K / 2 : gs::TKL_MIN_K);
  if (k > min_k || B <= c->sm_count) {
    gs::TopKLargeArgs ta;
    ta.x = x; ta.row_stride = row_stride; ta.V = static_cast<int32_t>(V); ta.k = static_cast<int32_t>(k);
    ta.out_values = out_values; ta.out_indices = out_indices; ta.out_flags = out_flags; ta.B = B;
    // by the list that k needs; up to one row per SM a row gets all of an SM's threads
    if (k > gs::TKL_MID_K) launch_topk_large<gs::TklLarge>(c, ta, dtype);
    else if (k > gs::TKL_SMALL_K) launch_topk_large<gs::TklMid>(c, ta, dtype);
    else if (B <= c->sm_count) launch_topk_large<gs::TklFew>(c, ta, dtype);
    else launch_topk_large<gs::TklSmall>(c, ta, dtype);
    CUDA_TRY(cudaGetLastError(), errOut);
    c->counters.kernel_launches += 1;
    return GORCH_CUDA_OK;
  }
  int32_t* base = nullptr;
  if ((rc = batch_lists(c, B, &base, errOut))) return rc;
  gs::BatchArgs ba;
  ba.k.logits = x; ba.k.row_stride = row_stride; ba.k.V = static_cast<int32_t>(V);
  ba.k.force_greedy = 0; ba.k.cfgs = nullptr; ba.k.uniforms = nullptr;
  ba.k.out_ids = nullptr; ba.k.out_flags = out_flags; ba.k.out_probs = nullptr; ba.k.out_debug = nullptr;
  ba.k.exp_table = c->exp_table; ba.k.row_offset = 0; ba.k.worklist = nullptr; ba.k.batch_hdr = base;
  ba.k.vs_records = nullptr; ba.k.vs_col_offset = 0; ba.k.vs_sumexp = 0;
  ba.k.tk_values = out_values; ba.k.tk_indices = out_indices; ba.k.tk_k = static_cast<int32_t>(k); ba.k.row_done = nullptr;
  ba.eb_table = c->eb_table;
  ba.hdr = base; ba.list_single = base + gs::HDR_COUNT;
  ba.B = B;
  CUDA_TRY(launch_narrow(c, ba, dtype, B, false), errOut);
  CUDA_TRY(cudaGetLastError(), errOut);
  c->counters.kernel_launches += 1;
  return GORCH_CUDA_OK;
}

int gorch_cuda_multinomial_dev(GorchCudaCtxRef ctx, const float* probs, int64_t B, int64_t V,
                               int64_t row_stride, const double* uniforms, int32_t* out_ids,
                               uint32_t* out_flags, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(GORCH_CUDA_F32, B, V, row_stride, errOut);
  if (rc) return rc;
  if (V > 8ll * gs::MN_MAX_STEPS * 256 - 64) {
    set_err(errOut, "gorch_cuda: Multinomial supports rows up to %d probabilities", 8 * gs::MN_MAX_STEPS * 256 - 64);
    return GORCH_CUDA_ERR_LIMIT;
  }
  if (B == 0) return GORCH_CUDA_OK;
  if (!probs || !uniforms || !out_ids) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(probs) % 4) != 0) { set_err(errOut, "gorch_cuda: probs pointer not aligned"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  gs::MultinomialArgs m;
  m.probs = probs; m.row_stride = row_stride; m.V = static_cast<int32_t>(V);
  m.uniforms = uniforms; m.out_ids = out_ids; m.out_flags = out_flags; m.B = B;
  // CTAs per row: more while the batch still fits the GPU at two CTAs per SM and a thread keeps four vectors (us, one CTA |
  // so: 8 x 151,936: 34 | 12; 64 x 151,936: 35 | 23; 8 x 50,257: 15 | 9).
  const int64_t slots = 4 * c->sm_count;
  int C = 1;
  while (C < gs::MN_MAX_C && B * 2 * C <= 2 * c->sm_count && V / (2 * C) >= 4 * 4 * gs::MN_NT) C *= 2;
  // Long rows of larger batches go by halves where that saves half a round over the SMs: where at most half the SMs would get one
  // row more than the others. us, one CTA | two, 151,936: 297 rows 62 | 54, 370: 62 | 56, 512: 78 | 73, 666: 95 | 90, and
  // without that half round 371: 62 | 63, 444: 62 | 64, 592: 78 | 82, 1024: 125 | 135. Shorter rows leave less to gain than the
  // pair's exchange costs, and half a round is less of more rounds: 100,000: 297 rows 43 | 39, 512: 55 | 53, 666: 66 | 66, but 800:
  // 76 | 78; 70,000: 512: 41 | 42. Beyond five rounds, 151,936: 800 rows 111 | 109, 960: 125 | 127, 1200: 170 | 162, 2400: 322 | 310.
  const int64_t odd = B % c->sm_count;
  if (V >= (B <= 5 * c->sm_count ? 100000 : 150000) && B > 2 * c->sm_count && odd > 0 && 2 * odd <= c->sm_count) C = 2;
  const int64_t clusters = (C > 1 || B < slots) ? B : slots;
  // (not beside the end of the kernel before it: its CTAs would crowd on the SMs that are free first. 64 x 151,936 behind a
  // softmax: 105 us instead of 60)
  CUDA_TRY(launch_clusters(c, gs::multinomial_rows_kernel, static_cast<unsigned>(clusters * C), gs::MN_NT, gs::MN_DYN_BYTES, false, C, m), errOut);
  c->counters.kernel_launches += 1;
  return GORCH_CUDA_OK;
}

static int launch_generate_control(Ctx* c, const int32_t* ids, const uint32_t* flags,
                                   const GorchGenControl* gc, int64_t B, char** errOut) {
  static_assert(GORCH_GEN_MAX_STOPS == gs::GC_MAX_STOPS && GORCH_GEN_STOP == gs::GC_STOP &&
                GORCH_GEN_MAX_NEW == gs::GC_MAX_NEW && GORCH_GEN_MAX_SEQ == gs::GC_MAX_SEQ &&
                GORCH_GEN_ERROR == gs::GC_ERROR, "generate-control codes");
  if (!gc) { set_err(errOut, "gorch_cuda: null generate-control record"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (B < 0 || B > 0x7fffffffll) { set_err(errOut, "gorch_cuda: bad batch size %lld", (long long)B); return GORCH_CUDA_ERR_BAD_ARG; }
  if (gc->n_stop < 0 || gc->n_stop > GORCH_GEN_MAX_STOPS) {
    set_err(errOut, "gorch_cuda: n_stop %d outside 0..%d", gc->n_stop, GORCH_GEN_MAX_STOPS);
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if (gc->capacity < 0 || gc->max_seq < 0) { set_err(errOut, "gorch_cuda: negative capacity or max_seq"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (B == 0) return GORCH_CUDA_OK;
  if (!ids || !gc->tokens || !gc->lengths || !gc->n_new || !gc->done || !gc->next_input || !gc->live_count ||
      (gc->cached && !gc->cache_len)) {
    set_err(errOut, "gorch_cuda: null pointer in the generate-control record");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  gs::GenControlArgs a;
  a.ids = ids; a.flags = flags;
  a.tokens = gc->tokens; a.capacity = gc->capacity; a.lengths = gc->lengths; a.n_new = gc->n_new;
  a.cache_len = gc->cache_len; a.done = gc->done; a.next_input = gc->next_input;
  a.window_start = gc->window_start; a.live_count = gc->live_count;
  for (int i = 0; i < GORCH_GEN_MAX_STOPS; i++) a.stops[i] = (i < gc->n_stop && gc->stop_tokens[i] >= 0) ? gc->stop_tokens[i] : -1;
  a.n_stop = gc->n_stop; a.max_new = gc->max_new; a.max_seq = gc->max_seq; a.cached = gc->cached ? 1 : 0;
  a.bad_flags = GORCH_FLAG_INTERNAL | GORCH_FLAG_BAD_CFG;
  a.B = static_cast<int>(B);
  CUDA_TRY(launch(c, gs::generate_control_kernel, 1, gs::GC_NT, 0, true, a), errOut);
  c->counters.kernel_launches += 1;
  return GORCH_CUDA_OK;
}

int gorch_cuda_generate_control_dev(GorchCudaCtxRef ctx, const int32_t* ids, const uint32_t* flags,
                                    const GorchGenControl* gc, int64_t B, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  return launch_generate_control(c, ids, flags, gc, B, errOut);
}

int gorch_cuda_generate_step_dev(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                                 int64_t V, int64_t row_stride, const GorchSampleCfg* cfgs,
                                 const double* uniforms, int32_t* out_ids, uint32_t* out_flags,
                                 const GorchGenControl* gc, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  if (!gc) { set_err(errOut, "gorch_cuda: null generate-control record"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (B > 0) {
    if (!logits || !cfgs || !uniforms || !out_ids || !gc->done) {
      set_err(errOut, "gorch_cuda: null pointer argument");
      return GORCH_CUDA_ERR_BAD_ARG;
    }
    CUDA_TRY(cudaSetDevice(c->device), errOut);
    // rows whose sequence has ended are skipped by the sampling kernels (the reference leaves its loop,
    // model/generate.go:82-84); their out_ids / out_flags entries keep what they held
    rc = launch_rows(c, logits, dtype, B, V, row_stride, cfgs, uniforms, out_ids, out_flags, nullptr, nullptr, 0, errOut,
                     nullptr, gc->done);
    if (rc) return rc;
  }
  return launch_generate_control(c, out_ids, out_flags, gc, B, errOut);
}

// CTAs per row of the resident softmax: as few as leave room for two slices per SM (any number up to eight), twice as many
// while the whole batch is resident at once; 0 when eight are too few.
static int softmax_cluster(const Ctx* c, int64_t B, int64_t V, int dtype) {
  const int64_t nvec = row_vectors(V, dtype);
  int C = 1;
  while (C < gs::RR_MAX_C && gs::rr_per(nvec, C) * 16 > gs::RR_SLICE) C++;
  while (2 * C <= gs::RR_MAX_C && B * 2 * C <= 2 * c->sm_count && nvec / (2 * C) >= 2 * gs::RR_NT) C *= 2;
  if (gs::rr_per(nvec, C) * 16 > gs::RR_SLICE || B * C > 0x7fffffffll) return 0;
  // Rows that need three CTAs and more leave slots of a GPC empty; the two-pass kernel then wins (us, two-pass | this)
  // between one wave of clusters and one row per SM (64 x 151,936 f32: 27 | 29; 128 x 100,000: 32 | 33; beyond: 256 x 151,936:
  // 84 | 78, 512 x 100,000: 102 | 92), and for bf16, whose rows are half as long, throughout (256 x 151,936: 50 | 55).
  if (C >= 3 && B * C > 2 * c->sm_count && (B <= c->sm_count || dtype == GORCH_CUDA_BF16)) return 0;
  return C;
}

static int launch_row_softmax(Ctx* c, int dtype, const gs::RowSoftmaxArgs& a, char** errOut) {
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  // A pair of CTAs per row where it was measured to pay: the two-pass ops when one row per SM in
  // flight would not fit in half of L2 (each pass-2 read then came from HBM again), and the
  // cross-entropy backward (no exchange, only finer work units) for rows of 256 KB and more. The
  // cross-entropy forward is one pass: the pair's barrier per row only costs there.
  const int64_t row_bytes = static_cast<int64_t>(a.V) * static_cast<int64_t>(elem_size(dtype));
  bool pair = false;
  if (a.mode == gs::RS_SOFTMAX || a.mode == gs::RS_LOG_SOFTMAX) pair = row_bytes * c->sm_count > (static_cast<int64_t>(c->l2_bytes) / 2);
  else if (a.mode == gs::RS_CE_BWD) pair = row_bytes >= 262144;
  if (a.mode != gs::RS_CE_BWD) {
    // Cross-entropy forward writes nothing, and the persistent kernel then has the next row's copies in flight: the
    // clusters win where a row fits one CTA (us: 1500 x 16,000 f32: 52 | 34; 1500 x 50,257 bf16: 75 | 55) or the whole batch
    // is resident (16 x 151,936 f32: 24 | 17), and lose beyond (256 x 151,936: 48 | 58).
    const int RC = softmax_cluster(c, a.B, a.V, dtype);
    if (RC == 1 || (RC > 1 && (a.mode != gs::RS_CE_FWD || a.B * RC <= 2 * c->sm_count))) {
      auto* kernel = (dtype == GORCH_CUDA_F32) ? gs::row_softmax_resident_kernel<float> : gs::row_softmax_resident_kernel<uint16_t>;
      CUDA_TRY(launch_clusters(c, kernel, static_cast<unsigned>(a.B * RC), gs::RR_NT, static_cast<size_t>(gs::rr_per(row_vectors(a.V, dtype), RC)) * 16,
                               false, RC, a), errOut);
      c->counters.kernel_launches += 1;
      return GORCH_CUDA_OK;
    }
  }
  int C = (pair && c->sm_count >= 2) ? 2 : 1;
  const bool bwd = a.mode == gs::RS_CE_BWD;
  if (bwd)                                                   // few rows: more CTAs each, while they fit at once (16 x 151,936 f32: 17 us by pairs, 14 by eights)
    while (C < gs::RR_MAX_C && a.B * 2 * C <= c->sm_count && row_bytes / (2 * C) >= 16 * gs::RS_NT) C *= 2;
  const int64_t clusters = a.B < c->sm_count / C ? a.B : c->sm_count / C;
  auto* kernel = (dtype == GORCH_CUDA_F32) ? gs::row_softmax_kernel<float> : gs::row_softmax_kernel<uint16_t>;
  CUDA_TRY(launch_clusters(c, kernel, static_cast<unsigned>(clusters * C), gs::RS_NT, gs::RS_DYN_BYTES, bwd, C, a), errOut);
  c->counters.kernel_launches += 1;
  return GORCH_CUDA_OK;
}

int gorch_cuda_softmax_dev(GorchCudaCtxRef ctx, const void* x, int dtype, int64_t B, int64_t V,
                           int64_t row_stride, void* out, int64_t out_stride, int log_softmax,
                           char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (out_stride < V) { set_err(errOut, "gorch_cuda: out_stride %lld below V", (long long)out_stride); return GORCH_CUDA_ERR_BAD_ARG; }
  if (B == 0) return GORCH_CUDA_OK;
  if (!x || !out) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  const size_t es = elem_size(dtype);
  if ((reinterpret_cast<uintptr_t>(x) % es) != 0 || (reinterpret_cast<uintptr_t>(out) % es) != 0) {
    set_err(errOut, "gorch_cuda: pointer not aligned to its element type");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  gs::RowSoftmaxArgs a{};
  a.x = x; a.row_stride = row_stride; a.V = static_cast<int32_t>(V); a.B = B;
  a.mode = log_softmax ? gs::RS_LOG_SOFTMAX : gs::RS_SOFTMAX;
  a.out = out; a.out_stride = out_stride;
  return launch_row_softmax(c, dtype, a, errOut);
}

int gorch_cuda_cross_entropy_fwd_dev(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                                     int64_t V, int64_t row_stride, const int32_t* targets,
                                     float* row_loss, float* row_lse, float* mean_loss,
                                     char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits || !targets || !row_loss || !row_lse) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(logits) % elem_size(dtype)) != 0) {
    set_err(errOut, "gorch_cuda: pointer not aligned to its element type");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  gs::RowSoftmaxArgs a{};
  a.x = logits; a.row_stride = row_stride; a.V = static_cast<int32_t>(V); a.B = B;
  a.mode = gs::RS_CE_FWD; a.targets = targets; a.row_loss = row_loss; a.row_lse = row_lse;
  rc = launch_row_softmax(c, dtype, a, errOut);
  if (rc) return rc;
  if (mean_loss) {
    CUDA_TRY(launch(c, gs::mean_loss_kernel, 1, 256, 0, true, static_cast<const float*>(row_loss), B, mean_loss), errOut);
    c->counters.kernel_launches += 1;
  }
  return GORCH_CUDA_OK;
}

int gorch_cuda_cross_entropy_bwd_dev(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                                     int64_t V, int64_t row_stride, const int32_t* targets,
                                     const float* row_lse, float scale, float* dx,
                                     int64_t dx_stride, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (dx_stride < V) { set_err(errOut, "gorch_cuda: dx_stride %lld below V", (long long)dx_stride); return GORCH_CUDA_ERR_BAD_ARG; }
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits || !targets || !row_lse || !dx) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  if ((reinterpret_cast<uintptr_t>(logits) % elem_size(dtype)) != 0 || (reinterpret_cast<uintptr_t>(dx) % 4) != 0) {
    set_err(errOut, "gorch_cuda: pointer not aligned to its element type");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  gs::RowSoftmaxArgs a{};
  a.x = logits; a.row_stride = row_stride; a.V = static_cast<int32_t>(V); a.B = B;
  a.mode = gs::RS_CE_BWD; a.targets = targets; a.row_lse = const_cast<float*>(row_lse);
  a.scale = scale; a.out = dx; a.out_stride = dx_stride;
  return launch_row_softmax(c, dtype, a, errOut);
}

int64_t gorch_cuda_sample_row(GorchCudaCtxRef ctx, const float* logits, int64_t n,
                              float temperature, int64_t top_k, float top_p, int topp_mode,
                              double uniform, uint32_t* out_flag, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return -1; }
  GorchSampleCfg cfg;
  cfg.temperature = temperature;
  // the reference takes a Go int; anything outside (0, n) disables top-k (generate.go:157)
  cfg.top_k = (top_k > 0 && top_k < n) ? static_cast<int32_t>(top_k) : 0;
  cfg.top_p = top_p;
  cfg.topp_mode = topp_mode;
  int32_t id = -1;
  uint32_t flag = 0;
  int rc = host_run(c, logits, GORCH_CUDA_F32, 1, n, n, &cfg, &uniform, &id, &flag, 0, errOut);
  if (rc) return -1;
  if (out_flag) *out_flag = flag;
  return id;
}

int gorch_cuda_argmax_host(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                           int64_t V, int64_t row_stride, int32_t* out_ids, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  return host_run(c, logits, dtype, B, V, row_stride, nullptr, nullptr, out_ids, nullptr, 1, errOut);
}

int gorch_cuda_argmax_dev(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                          int64_t V, int64_t row_stride, int32_t* out_ids, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!logits || !out_ids) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  return launch_rows(c, logits, dtype, B, V, row_stride, nullptr, nullptr, out_ids, nullptr,
                     nullptr, nullptr, 1, errOut);
}

int gorch_cuda_lm_head_logits_dev(GorchCudaCtxRef ctx, const void* x, int64_t ldx, const void* w, int64_t ldw, int64_t B,
                                  int64_t V, int64_t K, float* out_logits, int64_t ld_out, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_lm_head(c, x, w, B, V, K, ldx, ldw, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!out_logits || ld_out < V) { set_err(errOut, "gorch_cuda: LM head output missing or its pitch below V"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  if ((rc = load_encode_tiled(errOut))) return rc;
  gs::LmHeadArgs a;
  if ((rc = lm_head_args(c, a, x, ldx, w, ldw, B, V, K, true, errOut))) return rc;
  a.tile0 = 0; a.tile_step = 1; a.ntile = static_cast<int32_t>((V + 2 * a.cta_v - 1) / (2 * a.cta_v));
  a.out_logits = out_logits; a.ld_out = ld_out; a.compact = 0;
  return launch_lm_head(c, a, errOut, true);
}

int gorch_cuda_lm_head_sample_dev(GorchCudaCtxRef ctx, const void* x, int64_t ldx, const void* w, int64_t ldw, int64_t B,
                                  int64_t V, int64_t K, int fuse_top_k, const GorchSampleCfg* cfgs, const double* uniforms,
                                  int32_t* out_ids, uint32_t* out_flags, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_lm_head(c, x, w, B, V, K, ldx, ldw, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (!cfgs || !uniforms || !out_ids) { set_err(errOut, "gorch_cuda: null pointer argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  if ((rc = load_encode_tiled(errOut))) return rc;
  gs::LmHeadArgs a;
  if ((rc = lm_head_args(c, a, x, ldx, w, ldw, B, V, K, false, errOut))) return rc;
  const int ntile = static_cast<int>((V + 2 * a.cta_v - 1) / (2 * a.cta_v));
  // the unfused form: logits to scratch, then the ordinary sampling kernels
  auto unfused = [&]() -> int {
    const int64_t ld = (V + 31) & ~31ll;
    int r2 = ensure(c->lmh_logits, static_cast<size_t>(B) * ld * sizeof(float), errOut);
    if (r2) return r2;
    gs::LmHeadArgs u;
    if ((r2 = lm_head_args(c, u, x, ldx, w, ldw, B, V, K, true, errOut))) return r2;
    u.tile0 = 0; u.tile_step = 1; u.ntile = static_cast<int32_t>((V + 2 * u.cta_v - 1) / (2 * u.cta_v));
    u.out_logits = static_cast<float*>(c->lmh_logits.ptr); u.ld_out = ld; u.compact = 0;
    if ((r2 = launch_lm_head(c, u, errOut, true))) return r2;
    return launch_rows(c, c->lmh_logits.ptr, GORCH_CUDA_F32, B, V, ld, cfgs, uniforms, out_ids, out_flags, nullptr, nullptr, 0, errOut);
  };
  if (fuse_top_k < 1 || fuse_top_k > gs::KFAST || V < 4096 || B > 4096) return unfused();
  // From here on the call returns when the ids are there, whichever form serves it, and reports a projection that gave up.
  auto ids_there = [&]() -> int {
    CUDA_TRY(wait_stream(c), errOut);
    const uint32_t status = *static_cast<const volatile uint32_t*>(c->host_words);
    if (status != 0) {
      set_err(errOut, "gorch_cuda: the LM-head kernel gave up a bounded wait (status %u)", status);
      return GORCH_CUDA_ERR_CUDA;
    }
    return GORCH_CUDA_OK;
  };
  if (K >= kLmhUnfusedK && B * V * 4 <= kLmhUnfusedBytes && !use_batch_mode(c->sm_count, B, V, 4, false)) {
    rc = unfused();
    return (rc || capture_status(c->stream) == cudaStreamCaptureStatusActive) ? rc : ids_there();   // (recorded into a graph: nothing runs that could be waited for)
  }
  // the sample: 1/32 of the vocabulary, but 1024 to 4096 logits, in whole tiles
  int64_t want = V / 32;
  if (want < gs::LMH_SAMPLE_MIN) want = gs::LMH_SAMPLE_MIN;
  if (want > gs::LMH_SAMPLE_MAX) want = gs::LMH_SAMPLE_MAX;
  const int stiles = static_cast<int>(want / (2 * a.cta_v) > 1 ? want / (2 * a.cta_v) : 1);

  // ---- the fused form: scratch = [row state | thresholds | sample logits | candidates]; every kernel starts while the
  // one before it runs: the projection's first tiles are under way before the thresholds are there
  const int nsample = stiles * 2 * a.cta_v;
  const size_t off_rows = 0, off_thr = off_rows + sizeof(gs::LmhRow) * static_cast<size_t>(B);
  const size_t off_smp = (off_thr + 4 * static_cast<size_t>(B) + 255) & ~static_cast<size_t>(255);
  const size_t off_cand = (off_smp + sizeof(float) * static_cast<size_t>(B) * nsample + 255) & ~static_cast<size_t>(255);
  const size_t total = off_cand + sizeof(uint2) * static_cast<size_t>(B) * gs::LMH_CAND_CAP;
  if ((rc = ensure(c->lmh_scratch, total, errOut))) return rc;
  unsigned char* base = static_cast<unsigned char*>(c->lmh_scratch.ptr);
  c->host_words[1] = 0u;                                                     // (written by finish kernels only, whose calls waited for them; the projections clear [0])
  // 1. a sample of the vocabulary's tiles (all of them full tiles)
  gs::LmHeadArgs sa = a;
  sa.tile0 = 0; sa.tile_step = (ntile - 1) / stiles; sa.ntile = stiles;
  sa.out_logits = reinterpret_cast<float*>(base + off_smp); sa.ld_out = nsample; sa.compact = 1;
  if ((rc = launch_lm_head(c, sa, errOut, false))) return rc;
  // 2. thresholds
  gs::LmhSampleArgs fa;
  memset(&fa, 0, sizeof fa);
  fa.k.V = static_cast<int32_t>(V); fa.k.row_stride = V;
  fa.k.cfgs = reinterpret_cast<const gs::RowCfg*>(cfgs); fa.k.uniforms = uniforms;
  fa.k.out_ids = out_ids; fa.k.out_flags = out_flags; fa.k.exp_table = c->exp_table; fa.k.vs_cand = gs::VS_CAND; fa.k.vs_sumexp = 0;
  fa.sample = reinterpret_cast<const float*>(base + off_smp); fa.nsample = nsample; fa.fuse_top_k = fuse_top_k;
  fa.thr = reinterpret_cast<float*>(base + off_thr);
  fa.cand = reinterpret_cast<const uint2*>(base + off_cand);
  fa.rows = reinterpret_cast<gs::LmhRow*>(base + off_rows);
  fa.nfail = reinterpret_cast<int32_t*>(c->host_words + 1);
  fa.B = B;
  const unsigned g = static_cast<unsigned>(B < 4 * c->sm_count ? B : 4 * c->sm_count);
  CUDA_TRY(launch(c, gs::lmh_threshold_kernel, static_cast<unsigned>(B), gs::LMH_F_NT, 0, true, fa), errOut);
  // 3. the whole vocabulary, candidates out of the epilogue
  gs::LmHeadArgs ma = a;
  ma.tile0 = 0; ma.tile_step = 1; ma.ntile = ntile;
  ma.out_logits = nullptr; ma.ld_out = 0; ma.compact = 0;
  ma.thr = fa.thr; ma.cand = reinterpret_cast<uint2*>(base + off_cand); ma.rows = fa.rows;
  if ((rc = launch_lm_head(c, ma, errOut, true, true))) return rc;
  // 4. finish every row from its candidates
  CUDA_TRY(launch(c, gs::lmh_finish_kernel, g, gs::LMH_F_NT, gs::LMH_F_DYN_BYTES, true, fa), errOut);
  c->counters.kernel_launches += 2;
  c->counters.sample_launches += 1;
  c->counters.rows += static_cast<uint64_t>(B);
  // rows the fused form could not finish (their estimate failed, or their config is not served): the
  // count comes back to the host, which then recomputes the batch through the unfused form
  if ((rc = ids_there())) return rc;
  const uint32_t refused = *static_cast<const volatile uint32_t*>(c->host_words + 1);
  if (refused > 0) {
    c->counters.lm_head_refused_rows += static_cast<uint64_t>(refused);
    rc = unfused();
    return rc ? rc : ids_there();
  }
  return GORCH_CUDA_OK;
}

int gorch_cuda_lm_head_status(GorchCudaCtxRef ctx, uint32_t* status, char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c || !status) { set_err(errOut, "gorch_cuda: null argument"); return GORCH_CUDA_ERR_BAD_ARG; }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  CUDA_TRY(wait_stream(c), errOut);
  *status = *static_cast<const volatile uint32_t*>(c->host_words);
  return GORCH_CUDA_OK;
}

int gorch_cuda_sample_dev_static(GorchCudaCtxRef ctx, const void* logits, int dtype, int64_t B,
                                 int64_t V, int64_t row_stride, const GorchSampleCfg* cfgs,
                                 const double* uniforms, int32_t* out_ids, uint32_t* out_flags,
                                 char** errOut) {
  Ctx* c = static_cast<Ctx*>(ctx);
  if (!c) { set_err(errOut, "gorch_cuda: null context"); return GORCH_CUDA_ERR_BAD_ARG; }
  int rc = check_shape(dtype, B, V, row_stride, errOut);
  if (rc) return rc;
  if (B == 0) return GORCH_CUDA_OK;
  if (B > kStaticMaxRows) {
    set_err(errOut, "gorch_cuda: gorch_cuda_sample_dev_static serves at most %lld rows per call, got %lld",
            (long long)kStaticMaxRows, (long long)B);
    return GORCH_CUDA_ERR_LIMIT;
  }
  if (!logits || !cfgs || !uniforms || !out_ids) {
    set_err(errOut, "gorch_cuda: null pointer argument");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  if ((reinterpret_cast<uintptr_t>(logits) % elem_size(dtype)) != 0) {
    set_err(errOut, "gorch_cuda: logits pointer not aligned to its element size");
    return GORCH_CUDA_ERR_BAD_ARG;
  }
  CUDA_TRY(cudaSetDevice(c->device), errOut);
  int32_t* base = nullptr;
  if ((rc = static_lists_ptr(c->device, &base, errOut))) return rc;   // looked up when the context was created
  // the same dispatch as gorch_cuda_sample_dev, with the work lists in the fixed array (it keeps the
  // previous call's contents: the dispatch clears the cursors and counts it uses before every launch)
  return launch_rows(c, logits, dtype, B, V, row_stride, cfgs, uniforms, out_ids, out_flags, nullptr, nullptr, 0,
                     errOut, base);
}

}  // extern "C"
