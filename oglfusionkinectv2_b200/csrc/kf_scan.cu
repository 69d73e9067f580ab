// kf_scan.cu — exclusive prefix sum of uint32 (one pass, any length).
//
// Reference: shaders/prefixSum.cs:28-197 (Blelloch work-efficient scan, 2048 elements
// per work group, one level of group sums, so n <= 2048 * 2048 = 4,194,304 (Q17)) driven
// by MCubes::prefixSum (src/mcubes.cpp:136-204), which returns the total as lastElement +
// lastScanElement.  Same result (exclusive scan, uint32 wrap-around, total = sum of the
// input) for any n < 2^32.
//
// B200 design: one pass, each value read and written once (8 bytes an element; a reduction
// before the scan reads the input twice).  Persistent blocks take tiles of the input in turn;
// a tile's prefix is the sum of the tiles before it, which its block finds by looking back over
// the sums that the other blocks have published, to the nearest tile whose own prefix is known
// (the decoupled look-back of Merrill and Garland, 2016).  What bounds this on 148 SMs is the
// hand-over, not the scan: with a block per tile some 600 blocks polled the words of their 256
// predecessors and a tile waited 13 us for its prefix (100 M elements in 283 us at best, the
// reduction and scan before it in 223).  So few blocks hold large tiles, and each works on
// three of them: one on its way into shared memory (16-byte asynchronous copies), one whose sum
// is published, and one that is finished; the sums that a block looks up were published
// a whole tile's time ago.  A block takes tiles in rising order, so the holder of the lowest
// unpublished tile never waits for a higher one; every wait is bounded all the same.
// 100 M elements: 223 us (reduction 77, scan 146; 5.4 TB/s of its 12 bytes an element) -> 172 us
// (4.7 TB/s of 8 bytes); a block per SM with 1,024 threads and 64 KB tiles 172-178, two with 32 KB
// tiles 238; a warp of its own for the look-back 238, because the sums it then meets are newer.
#include <cuda.h>

#include <mutex>

#include "kf_internal.cuh"

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kRounds = 4;  // of four values per thread
constexpr int kTile = kThreads * kRounds * 4;
constexpr int kLooks = 5;   // tiles per lane and look: more than there are blocks
constexpr int kPerSm = 1;   // blocks
constexpr int kStages = 3;  // tiles of a block in shared memory
constexpr uint32_t kMaxLooks = 1u << 18;  // some 0.2 s

// The scratch: the result (total, whether a wait gave up), the ticket counter, a spare word,
// then a status per tile: kSum or kPrefix in the high word, the value in the low one.
constexpr size_t kHeadWords = 4;
constexpr unsigned long long kSum = 1ull << 32, kPrefix = 2ull << 32;

__device__ __forceinline__ void put_status(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long get_status(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Sum of all tiles before `tile`, by one warp.  Bounded: after max_looks looks that found nothing
// new, or when another wait gave up, *gave_up is set.
__device__ __forceinline__ uint32_t look_back(const unsigned long long* status, uint32_t tile, int lane, uint32_t* gave_up,
                                              uint32_t max_looks) {
  uint32_t sum = 0, looks = 0;
  for (int64_t last = (int64_t)tile - 1;;) {  // the nearest tile that is not yet in the sum
    unsigned long long st[kLooks];
#pragma unroll
    for (int k = 0; k < kLooks; ++k) {
      const int64_t t = last - (k * 32 + lane);
      st[k] = t >= 0 ? get_status(status + t) : kPrefix;  // before the first tile: a prefix of 0
    }
    uint32_t part = 0;
    int taken = 0;  // whole groups of 32 in `part`
    bool done = false;
#pragma unroll
    for (int k = 0; k < kLooks; ++k) {
      if (done || taken < k) continue;
      const unsigned empty = __ballot_sync(0xffffffffu, st[k] < kSum);
      const unsigned prefix = __ballot_sync(0xffffffffu, st[k] >= kPrefix);
      const int p = __ffs(prefix) - 1, e = __ffs(empty) - 1;  // nearest of each, -1: none
      if (p >= 0 && (e < 0 || p < e)) {
        if (lane <= p) part += (uint32_t)st[k];
        done = true;
      } else if (e < 0) {
        part += (uint32_t)st[k];
        taken = k + 1;
      }
    }
    sum += part;
    last -= 32 * taken;
    if (done) break;
    if (!taken) {
      // a wait that gave up (the words were overwritten) ends the others as well
      const bool over = *reinterpret_cast<volatile uint32_t*>(gave_up) != 0;
      if (++looks > max_looks || __any_sync(0xffffffffu, over)) {
        if (lane == 0) atomicExch(gave_up, 1u);
        break;
      }
      __nanosleep(20);
    }
  }
  return __reduce_add_sync(0xffffffffu, sum);
}

// A thread's groups of four into its own places of a stage.  Positions are counted from `shift`
// values before in[0], where the address is a multiple of 16 bytes, so that only the first and
// the last group can be partial.  One group of copies per call, empty or not.
__device__ __forceinline__ void load_tile(uint4* stage, const uint32_t* in, uint64_t at, uint32_t shift, uint64_t end) {
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const uint64_t p = at + r * 128;
    uint4* dst = stage + r * 32;
    if (p >= shift && p + 4 <= end) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                   "l"(in + (p - shift))
                   : "memory");
    } else {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (p + 0 >= shift && p + 0 < end) v.x = in[p - shift];
      if (p + 1 >= shift && p + 1 < end) v.y = in[p + 1 - shift];
      if (p + 2 >= shift && p + 2 < end) v.z = in[p + 2 - shift];
      if (p + 3 >= shift && p + 3 < end) v.w = in[p + 3 - shift];
      *dst = v;
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Exclusive scan.  A warp's part of a tile is contiguous, round r of it 32 groups of four; a
// thread loads, adds and stores the same groups.  VEC: out has the same shift.  `in` may equal
// `out`: a tile is in shared memory before it is stored.
template <bool VEC>
__global__ void __launch_bounds__(kThreads, kPerSm)
    scan_kernel(const uint32_t* in, uint32_t* out, uint64_t n, uint32_t shift, uint32_t ntiles, uint32_t* scratch) {
  extern __shared__ uint4 s_data[];
  __shared__ uint32_t s_sum[kWarps];
  __shared__ uint32_t s_pre[2][kWarps];  // of each warp's part within its tile
  __shared__ uint32_t s_base, s_tile[4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long* status = reinterpret_cast<unsigned long long*>(scratch + kHeadWords);
  const uint64_t end = n + shift;
  const uint32_t mine = (uint32_t)(warp * kRounds * 128 + lane * 4);
  uint4* data = s_data + warp * kRounds * 32 + lane;

  auto load = [&](uint32_t k) {
    const uint32_t t = s_tile[k & 3];
    if (t < ntiles)
      load_tile(data + (size_t)(k % kStages) * (kTile / 4), in, (uint64_t)t * kTile + mine, shift, end);
    else
      asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // one ticket after the other: a block's first tiles have to lie a grid apart
  for (uint32_t k = 0; k < 2; ++k) {
    if (threadIdx.x == 0) s_tile[k] = ntiles > 1 ? atomicAdd(scratch + 2, 1u) : k;
    __syncthreads();
    load(k);
  }

  uint32_t pre[kRounds], sum = 0;  // of the tile to be finished next
  for (uint32_t k = 0;; ++k) {  // publishes its k-th tile's sum, finishes its (k - 1)-th tile
    const uint32_t tile = s_tile[k & 3], prev = k ? s_tile[(k - 1) & 3] : ntiles;
    if (tile >= ntiles && prev >= ntiles) break;
    uint32_t next_pre[kRounds], run = 0;
    if (tile < ntiles) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      const uint4* st = data + (size_t)(k % kStages) * (kTile / 4);
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const uint4 v = st[r * 32];
        const uint32_t four = v.x + v.y + v.z + v.w;
        const uint32_t inc = warp_incl_scan(four, lane);
        next_pre[r] = run + inc - four;
        run += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) s_sum[warp] = run;
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t ticket = 0;
      if (lane == 0) ticket = ntiles > 1 ? atomicAdd(scratch + 2, 1u) : ntiles;
      uint32_t next_sum = 0;
      if (tile < ntiles) {
        const uint32_t w = lane < kWarps ? s_sum[lane] : 0u;
        const uint32_t inc = warp_incl_scan(w, lane);
        next_sum = __shfl_sync(0xffffffffu, inc, 31);
        if (lane == 0 && ntiles > 1) put_status(status + tile, (tile ? kSum : kPrefix) | next_sum);
        if (lane < kWarps) s_pre[k & 1][lane] = inc - w;
      }
      if (prev < ntiles) {
        const uint32_t base = prev ? look_back(status, prev, lane, scratch + 1, kMaxLooks) : 0u;
        if (lane == 0) {
          if (prev) put_status(status + prev, kPrefix | (uint32_t)(base + sum));
          s_base = base;
          if (prev == ntiles - 1) {
            scratch[0] = base + sum;
            if (ntiles == 1) scratch[1] = 0;
          }
        }
      }
      sum = next_sum;
      if (lane == 0) s_tile[(k + 2) & 3] = ticket;
    }
    __syncthreads();
    if (prev < ntiles) {
      const uint32_t base = s_base + s_pre[(k - 1) & 1][warp];
      const uint4* st = data + (size_t)((k - 1) % kStages) * (kTile / 4);
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const uint64_t p = (uint64_t)prev * kTile + mine + r * 128;
        const uint4 v = st[r * 32];
        uint4 o;
        o.x = base + pre[r];
        o.y = o.x + v.x;
        o.z = o.y + v.y;
        o.w = o.z + v.z;
        if (VEC && p >= shift && p + 4 <= end) {
          *reinterpret_cast<uint4*>(out + (p - shift)) = o;
        } else {
          if (p + 0 >= shift && p + 0 < end) out[p - shift] = o.x;
          if (p + 1 >= shift && p + 1 < end) out[p + 1 - shift] = o.y;
          if (p + 2 >= shift && p + 2 < end) out[p + 2 - shift] = o.z;
          if (p + 3 >= shift && p + 3 < end) out[p + 3 - shift] = o.w;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRounds; ++r) pre[r] = next_pre[r];
    load(k + 2);  // with three stages, into the one just finished
  }
}

// Self-test: the look-back of the second tile, whose first is never published (*status is 0).
__global__ void look_back_selftest_kernel(const unsigned long long* status, uint32_t* gave_up, uint32_t max_looks) {
  look_back(status, 1u, threadIdx.x, gave_up, max_looks);
}

uint64_t tiles(uint64_t n) { return (n + kTile - 1) / kTile; }

}  // namespace

size_t kf_scan_scratch_words(uint64_t n) { return 2 + kHeadWords + 2 * (size_t)tiles(n + 3); }

int kf_scan_u32(const uint32_t* d_in, uint32_t* d_out, uint64_t n, cudaStream_t stream, uint32_t* d_scratch,
                size_t scratch_words, const uint32_t** result) {
  const uint32_t shift = (uint32_t)(reinterpret_cast<uintptr_t>(d_in) >> 2 & 3u);
  const uint64_t nt = std::max<uint64_t>(1, tiles(n + shift));
  uint32_t* w = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(d_scratch) + 7) & ~(uintptr_t)7);
  if ((size_t)(w - d_scratch) + kHeadWords + 2 * nt > scratch_words) return KF_ERR_CAPACITY;
  *result = w;
  if (nt > 1 && cudaMemsetAsync(w, 0, (kHeadWords + 2 * nt) * 4, stream) != cudaSuccess) return KF_ERR_CUDA;
  const bool vec = shift == (uint32_t)(reinterpret_cast<uintptr_t>(d_out) >> 2 & 3u);
  auto kernel = vec ? scan_kernel<true> : scan_kernel<false>;
  static_assert(kStages == 3, "the tile on its way takes the finished one's place");
  const int smem = (nt > 1 ? kStages : 1) * kTile * 4;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return KF_ERR_CUDA;
  // the limit belongs to the kernel in the whole context, so every call sets the same one: a
  // smaller limit for one tile would refuse the launch that another thread is about to make
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * kTile * 4) != cudaSuccess)
    return KF_ERR_CUDA;
  const unsigned grid = (unsigned)std::min<uint64_t>(nt, (uint64_t)kPerSm * sms);
  kernel<<<grid, kThreads, smem, stream>>>(d_in, d_out, n, shift, (uint32_t)nt, w);
  return cudaGetLastError() == cudaSuccess ? KF_OK : KF_ERR_CUDA;
}

int kf_launch_scan_wait_selftest(const unsigned long long* zero, uint32_t* gave_up, uint32_t max_looks, cudaStream_t stream) {
  look_back_selftest_kernel<<<1, 32, 0, stream>>>(zero, gave_up, std::min(max_looks, kMaxLooks));
  return cudaGetLastError() == cudaSuccess ? KF_OK : KF_ERR_CUDA;
}

// ---- scratch without allocations --------------------------------------------------------
// An allocation per call costs 0.4-0.9 ms: the driver's pool gives its memory back at every
// synchronisation.  So both entry points keep their scratch in arrays compiled into the library,
// of KF_SCAN_WORDS words, which KF_NOALLOC_SCAN_MAX_ELEMENTS elements need (2^28 make 16,385
// tiles: 32,776 words):
//  - kf_prefix_sum_u32_noalloc has one array (131,136 bytes), shared by all its calls on a device;
//  - kf_prefix_sum_u32 waits for its result, so a call borrows one of a few slots and returns
//    it at the end; when none is free, the input is larger or the stream is being captured, the
//    scratch is allocated.
// Every GPU that loads this library holds the arrays (0.66 MB) until the process exits.
#define KF_NOALLOC_SCAN_MAX_ELEMENTS (1ull << 28)
#define KF_SCAN_WORDS 32784
#define KF_SCAN_SLOTS 4
static __device__ __align__(256) uint32_t g_noalloc_scan_scratch[KF_SCAN_WORDS];
static __device__ __align__(256) uint32_t g_scan_slots[KF_SCAN_SLOTS * KF_SCAN_WORDS];

namespace {
std::mutex g_scratch_mu;
// The arrays' device addresses per CUDA context, keyed by the context's process-unique id
// (cuCtxGetId): a context created later (a new primary context after cudaDeviceReset, or a
// context a host framework made with cuCtxCreate) never reuses an entry of an earlier one.
struct ScratchEntry {
  unsigned long long ctx_id;
  uint32_t* noalloc;
  uint32_t* slots;
  unsigned busy;  // a bit per borrowed slot
};
constexpr int kMaxEntries = 64;
ScratchEntry g_entries[kMaxEntries];
int g_entry_count = 0;
typedef CUresult (*PFN_ctx_get_current)(CUcontext*);
typedef CUresult (*PFN_ctx_get_id)(CUcontext, unsigned long long*);
PFN_ctx_get_current g_ctx_get_current = nullptr;
PFN_ctx_get_id g_ctx_get_id = nullptr;

// The current context's id through the driver entry points (the library links only the
// CUDA runtime); false when there is no current context.
bool current_ctx_id(unsigned long long* id) {
  if (!g_ctx_get_current || !g_ctx_get_id) {
    void* f0 = nullptr;
    void* f1 = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f0, cudaEnableDefault) != cudaSuccess ||
        cudaGetDriverEntryPoint("cuCtxGetId", &f1, cudaEnableDefault) != cudaSuccess || !f0 || !f1) {
      cudaGetLastError();
      return false;
    }
    g_ctx_get_current = reinterpret_cast<PFN_ctx_get_current>(f0);
    g_ctx_get_id = reinterpret_cast<PFN_ctx_get_id>(f1);
  }
  CUcontext ctx = nullptr;
  if (g_ctx_get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
  return g_ctx_get_id(ctx, id) == CUDA_SUCCESS;
}

ScratchEntry* find_entry(unsigned long long id) {
  for (int k = 0; k < g_entry_count; ++k)
    if (g_entries[k].ctx_id == id) return &g_entries[k];
  return nullptr;
}

// In host code the arrays only name the symbols; their device addresses are looked up with
// cudaGetSymbolAddress once per CUDA context (the first call in a context, which also makes the
// runtime's primary context current when none is) and cached by context id.  With g_scratch_mu
// held.  *entry: the cached entry, null when there is no id or no room for one.
int scratch_arrays(uint32_t** noalloc, ScratchEntry** entry) {
  *entry = nullptr;
  unsigned long long id = 0;
  bool have_id = current_ctx_id(&id);
  if (have_id) *entry = find_entry(id);
  if (*entry) {
    *noalloc = (*entry)->noalloc;
    return KF_OK;
  }
  void* p = nullptr;
  void* q = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scan_scratch);
  if (e == cudaSuccess) e = cudaGetSymbolAddress(&q, g_scan_slots);
  if (e != cudaSuccess || !p || !q) {
    cudaGetLastError();
    return e == cudaErrorNoDevice ? KF_ERR_NO_DEVICE : KF_ERR_CUDA;
  }
  *noalloc = static_cast<uint32_t*>(p);
  if (!have_id) have_id = current_ctx_id(&id);  // the lookup initialised the primary context
  if (!have_id) return KF_OK;
  int k = g_entry_count;
  if (k == kMaxEntries) {  // an entry with borrowed slots stays: its slots come back to it
    for (k = 0; k < kMaxEntries && g_entries[k].busy; ++k) {
    }
    if (k == kMaxEntries) return KF_OK;
  } else {
    ++g_entry_count;
  }
  g_entries[k] = ScratchEntry{id, *noalloc, static_cast<uint32_t*>(q), 0u};
  *entry = &g_entries[k];
  return KF_OK;
}

// A free slot of the current context's; null: none.
uint32_t* borrow_slot(unsigned long long* ctx_id, int* slot) {
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  uint32_t* noalloc = nullptr;
  ScratchEntry* e = nullptr;
  if (scratch_arrays(&noalloc, &e) != KF_OK || !e) return nullptr;
  for (int k = 0; k < KF_SCAN_SLOTS; ++k)
    if (!(e->busy & 1u << k)) {
      e->busy |= 1u << k;
      *ctx_id = e->ctx_id;
      *slot = k;
      return e->slots + (size_t)k * KF_SCAN_WORDS;
    }
  return nullptr;
}

void return_slot(unsigned long long ctx_id, int slot) {
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (ScratchEntry* e = find_entry(ctx_id)) e->busy &= ~(1u << slot);
}
}  // namespace

extern "C" int kf_prefix_sum_u32(const uint32_t* d_in, uint32_t* d_out, uint64_t n, uint32_t* total,
                                 void* cuda_stream) {
  if ((!d_in || !d_out) && n) return KF_ERR_INVALID_ARGUMENT;
  if (n >= (1ull << 32)) return KF_ERR_INVALID_ARGUMENT;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  const size_t words = kf_scan_scratch_words(n);
  uint32_t* scratch = nullptr;
  unsigned long long ctx_id = 0;
  int slot = -1;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (words <= KF_SCAN_WORDS && cudaStreamIsCapturing(st, &capture) == cudaSuccess &&
      capture == cudaStreamCaptureStatusNone)
    scratch = borrow_slot(&ctx_id, &slot);
  if (!scratch && cudaMallocAsync((void**)&scratch, words * sizeof(uint32_t), st) != cudaSuccess) {
    cudaGetLastError();
    return KF_ERR_OUT_OF_MEMORY;
  }
  const uint32_t* result = nullptr;
  int rc = kf_scan_u32(d_in, d_out, n, st, scratch, words, &result);
  uint32_t h[2] = {0, 0};
  if (!rc && cudaMemcpyAsync(h, result, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess) rc = KF_ERR_CUDA;
  if (slot < 0) cudaFreeAsync(scratch, st);
  if (cudaStreamSynchronize(st) != cudaSuccess)
    rc = KF_ERR_CUDA;  // the slot may still be in use and stays borrowed
  else if (slot >= 0)
    return_slot(ctx_id, slot);
  if (!rc && h[1]) rc = KF_ERR_CUDA;
  if (!rc && total) *total = h[0];
  return rc;
}

extern "C" int kf_prefix_sum_u32_noalloc(const uint32_t* d_in, uint32_t* d_out, uint64_t n, uint32_t* total,
                                         void* cuda_stream) {
  if ((!d_in || !d_out) && n) return KF_ERR_INVALID_ARGUMENT;
  if (n > KF_NOALLOC_SCAN_MAX_ELEMENTS) return KF_ERR_CAPACITY;
  uint32_t* scratch = nullptr;
  int rc;
  {
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    ScratchEntry* e = nullptr;
    rc = scratch_arrays(&scratch, &e);
  }
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)cuda_stream;
  const uint32_t* result = nullptr;
  rc = kf_scan_u32(d_in, d_out, n, st, scratch, KF_SCAN_WORDS, &result);
  if (rc || !total) return rc;
  uint32_t h[2] = {0, 0};
  if (cudaMemcpyAsync(h, result, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess) {
    cudaGetLastError();
    return KF_ERR_CUDA;
  }
  if (h[1]) return KF_ERR_CUDA;
  *total = h[0];
  return KF_OK;
}
