// Device recount of labelings: objective f, cluster sizes and G = A*Z for a batch of labelings of one graph.
// This is the GPU form of the reference's post-solve recount ObjectiveBitwise (src/cc_pbils_cpu.cpp:25-53,
// run by the CLI at include/cc_cli.hpp:337-343) and of State::Rebuild (src/cc_pbils_cpu.cpp:74-95).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>
#include <unordered_map>

#include "ccb.h"
#include "ccb_device.cuh"
#include "ccb_error.h"
#include "ccb_util.h"

namespace ccb {
namespace {

constexpr int kEvalThreads = 256;
constexpr int kEvalWarps = kEvalThreads / kWarp;

// Three launches per call, each over the whole chip whatever the count (one block per labeling left all but one SM idle
// for the recount of a single solution: n = 20000, k = 16 took 15 ms, now about 0.1):
//   k_eval_masks   one bit mask per cluster by warp ballots into `masks` ([labeling][k][words], scratch), f zeroed;
//   k_eval_rows    G = popc(row & mask), a warp per kRows rows and kChunk clusters, so that a mask word loaded serves
//                  kRows rows; each block adds its rows' own-cluster counts to f;
//   k_eval_finish  sizes from the masks, f = edges + sum_c C(size_c, 2) - (the sum so far).  A label outside [0, k) is
//                  in no mask: the sizes then sum to less than n and f is -1.
// What bounds it (B200, n = 20000, k = 16, one labeling: 131 us a call, k_eval_rows 108 of them, 120 with cold caches): POPC
// (8 clocks a warp, n k ceil(n / 32) of them) would take 43 us.  Its pipe is busy 48 % of the time and issue 47 %: 128
// registers leave two blocks an SM, 16 warps, to cover 20 dependent rounds of loads a warp, and 625 blocks are 2.1 waves of
// 296.  The masks take 5 us, sizes and f 10 by one block a labeling.
__global__ void __launch_bounds__(kEvalThreads)
    k_eval_masks(const int32_t* __restrict__ all_labels, int n, int words, int k, uint32_t* __restrict__ masks,
                 int64_t* __restrict__ f_out) {
  const int sol = blockIdx.x;
  const int lane = threadIdx.x % kWarp;
  const int32_t* labels = all_labels + static_cast<size_t>(sol) * n;
  uint32_t* my_masks = masks + static_cast<size_t>(sol) * k * words;
  if (blockIdx.y == 0 && threadIdx.x == 0) f_out[sol] = 0;
  for (int w = blockIdx.y * kEvalWarps + threadIdx.x / kWarp; w < words; w += gridDim.y * kEvalWarps) {
    const int v = w * kWarp + lane;
    const int l = v < n ? labels[v] : -1;
    for (int c = 0; c < k; ++c) {
      const uint32_t m = __ballot_sync(kAllLanes, l == c);
      if (lane == (c % kWarp)) my_masks[static_cast<size_t>(c) * words + w] = m;
    }
  }
}

template <int kChunk, int kRows>
__global__ void __launch_bounds__(kEvalThreads)
    k_eval_rows(const uint32_t* __restrict__ bits, int n, int words, int pitch, int k,
                const int32_t* __restrict__ all_labels, const uint32_t* __restrict__ masks, int64_t* __restrict__ f_out,
                int32_t* __restrict__ g_out) {
  __shared__ long long s_sum[kEvalWarps];
  const int sol = blockIdx.x;
  const int lane = threadIdx.x % kWarp;
  const int v0 = (blockIdx.y * kEvalWarps + threadIdx.x / kWarp) * kRows;
  const int32_t* labels = all_labels + static_cast<size_t>(sol) * n;
  const uint32_t* my_masks = masks + static_cast<size_t>(sol) * k * words;
  long long own_sum = 0;
  if (v0 < n) {
    const int rows = min(kRows, n - v0);
    const int own = lane < rows ? labels[v0 + lane] : -1;
    for (int c0 = 0; c0 < k; c0 += kChunk) {
      int acc[kRows][kChunk];
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
#pragma unroll
        for (int i = 0; i < kChunk; ++i) acc[r][i] = 0;
      }
      for (int w = lane; w < words; w += kWarp) {
        uint32_t m[kChunk];
#pragma unroll
        for (int i = 0; i < kChunk; ++i) m[i] = c0 + i < k ? my_masks[static_cast<size_t>(c0 + i) * words + w] : 0u;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const uint32_t a = r < rows ? __ldg(bits + static_cast<size_t>(v0 + r) * pitch + w) : 0u;
#pragma unroll
          for (int i = 0; i < kChunk; ++i) acc[r][i] += __popc(a & m[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < kChunk; ++i) {
        if (c0 + i >= k) break;
        int mine = 0;  // lane r: row r's count
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const int total = __reduce_add_sync(kAllLanes, acc[r][i]);
          mine = lane == r ? total : mine;
        }
        if (lane < rows) {
          if (g_out != nullptr) g_out[(static_cast<size_t>(sol) * k + c0 + i) * n + v0 + lane] = mine;
          if (own == c0 + i) own_sum += mine;
        }
      }
    }
  }
  const long long sum = BlockSum<kEvalWarps>(own_sum, s_sum);
  if (threadIdx.x == 0 && sum != 0) {
    atomicAdd(reinterpret_cast<unsigned long long*>(f_out + sol), static_cast<unsigned long long>(sum));
  }
}

__global__ void __launch_bounds__(kEvalThreads)
    k_eval_finish(const uint32_t* __restrict__ masks, int n, int words, int k, long long edges,
                  int64_t* __restrict__ f_out, int32_t* __restrict__ sizes_out) {
  __shared__ int s_sizes[kMaxK];
  const int sol = blockIdx.x;
  const int lane = threadIdx.x % kWarp;
  const uint32_t* my_masks = masks + static_cast<size_t>(sol) * k * words;
  for (int c = threadIdx.x / kWarp; c < k; c += kEvalWarps) {  // a warp per cluster
    int size = 0;
    for (int w = lane; w < words; w += kWarp) size += __popc(my_masks[static_cast<size_t>(c) * words + w]);
    size = __reduce_add_sync(kAllLanes, size);
    if (lane == 0) s_sizes[c] = size;
  }
  __syncthreads();
  if (sizes_out != nullptr) {
    for (int c = threadIdx.x; c < k; c += kEvalThreads) sizes_out[static_cast<size_t>(sol) * k + c] = s_sizes[c];
  }
  if (threadIdx.x == 0) {
    long long pairs = 0, placed = 0;
    for (int c = 0; c < k; ++c) {
      pairs += static_cast<long long>(s_sizes[c]) * (s_sizes[c] - 1) / 2;
      placed += s_sizes[c];
    }
    f_out[sol] = placed < n ? -1 : edges + pairs - f_out[sol];
  }
}

template <int kChunk, int kRows>
void LaunchEvalRows(const uint32_t* bits, int n, int words, int pitch, int k, int count, const int32_t* labels,
                    const uint32_t* masks, int64_t* f_out, int32_t* g_out, cudaStream_t st) {
  const dim3 grid(count, (n + kEvalWarps * kRows - 1) / (kEvalWarps * kRows));  // <= 32768 for n <= 2^20
  k_eval_rows<kChunk, kRows><<<grid, kEvalThreads, 0, st>>>(bits, n, words, pitch, k, labels, masks, f_out, g_out);
}

cudaError_t LaunchEvaluate(const uint32_t* bits, int n, int pitch, uint64_t edges, int k, int count,
                           const int32_t* labels, uint32_t* masks, int64_t* f_out, int32_t* sizes_out, int32_t* g_out,
                           cudaStream_t st) {
  const int words = (n + 31) / 32;
  const int parts = std::max(1, std::min((words + kEvalWarps - 1) / kEvalWarps, (256 + count - 1) / count));
  k_eval_masks<<<dim3(count, parts), kEvalThreads, 0, st>>>(labels, n, words, k, masks, f_out);
  if (n > 0) {
    // kChunk * kRows counters a thread: as many rows as the clusters leave
    if (k <= 4) {
      LaunchEvalRows<4, 16>(bits, n, words, pitch, k, count, labels, masks, f_out, g_out, st);
    } else if (k <= 8) {
      LaunchEvalRows<8, 8>(bits, n, words, pitch, k, count, labels, masks, f_out, g_out, st);
    } else {
      LaunchEvalRows<16, 4>(bits, n, words, pitch, k, count, labels, masks, f_out, g_out, st);
    }
  }
  k_eval_finish<<<count, kEvalThreads, 0, st>>>(masks, n, words, k, (long long)edges, f_out, sizes_out);
  return cudaGetLastError();
}

const char* CheckEvaluateArgs(const uint32_t* bits, uint32_t n, uint32_t words_per_row, int32_t k, int32_t count,
                              const int32_t* labels, const int64_t* f_out) {
  if (k < 1 || k > CCB_MAX_CLUSTERS) return "k must be in [1, 64]";
  if (count < 0) return "count must be >= 0";
  if (n > (uint32_t)CCB_MAX_VERTICES_WIDE) return "n exceeds 1048576, the range of the packed move";
  if (n > 0 && words_per_row < (n + 31) / 32) return "words_per_row < ceil(n / 32)";
  if (count > 0 && n > 0 && (bits == nullptr || labels == nullptr)) return "null bitset or labels";
  if (count > 0 && f_out == nullptr) return "null f_out";
  return nullptr;
}

int Report(int status, const char* message) {
  SetLastError(message);
  return status;
}

// Whether a recount is faster as the tensor-core contraction (ccb_evaluate_labelings_tensor, the same integers), by what
// both were measured to take (B200): popcount 4.2 M row-word intersections a us, the contraction 1.25 us a K step of 128
// vertices and wave of CTAs (256 vertices x 256 columns each), 10 us more of set-up.  n = 20000, k = 16: 106 us against
// 150 for one labeling, 4290 against 480 for 64; n = 4001, k = 64, 32 labelings: 455 against 83.
bool PreferTensorRecount(const uint32_t* bits, int n, int words_per_row, int k, int count) {
  int device = 0, sms = 0;
  if (n < 128 || words_per_row % 4 != 0 || reinterpret_cast<uintptr_t>(bits) % 16 != 0) return false;
  const double words = (n + 31) / 32, columns = (double)count * k;
  if (columns * words * 32 > 1024.0 * 1024 * 1024 || columns > 1 << 24) return false;  // its one-hot scratch
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    return false;
  }
  const double waves = std::ceil(std::ceil(n / 256.0) * std::ceil(columns / 256) / sms);
  return 10 + waves * std::ceil(words / 4) * 1.25 < n * words * columns / 4.2e6;
}

constexpr uint64_t kScratchKept = 64ull << 20;  // bytes a context's pool keeps between calls
std::mutex g_scratch_mutex;
std::unordered_map<unsigned long long, cudaMemPool_t> g_scratch_pools;  // by context

// The current context's id, unique for the life of the process (a device reset ends a context and its pools, and the next
// one has another id); 0 when there is none or the driver cannot tell.
unsigned long long CurrentContext() {
  using GetId = PFN_cuCtxGetId_v12000;
  static const GetId get_id = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    const bool found = cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
                       q == cudaDriverEntryPointSuccess;
    return found ? reinterpret_cast<GetId>(p) : nullptr;
  }();
  unsigned long long id = 0;
  return get_id != nullptr && get_id(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

}  // namespace

// The default pool gives its memory back at every synchronisation, so each recount mapped its scratch anew (0.2 ms, up to
// several on a busy host).  A pool of our own per context keeps up to kScratchKept; ccb_release_cache trims it.  Stream
// ordered and thread safe like the default pool, which serves captures and devices without pool support.
cudaError_t ScratchAlloc(void** out, size_t bytes, cudaStream_t st) {
  int device = 0;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaMemPool_t pool = nullptr;
  unsigned long long context = 0;
  if (cudaGetDevice(&device) == cudaSuccess && cudaStreamIsCapturing(st, &capture) == cudaSuccess &&
      capture == cudaStreamCaptureStatusNone && (context = CurrentContext()) != 0) {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    cudaMemPool_t& kept_pool = g_scratch_pools[context];
    if (kept_pool == nullptr) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.handleTypes = cudaMemHandleTypeNone;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device;
      uint64_t kept = kScratchKept;
      if (cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept) == cudaSuccess) {
          kept_pool = pool;
        } else {
          cudaMemPoolDestroy(pool);
        }
      }
    }
    pool = kept_pool;
  }
  if (pool != nullptr && cudaMallocFromPoolAsync(out, bytes, pool, st) == cudaSuccess) return cudaSuccess;
  cudaGetLastError();  // what failed above is tried again below
  return cudaMallocAsync(out, bytes, st);
}

void ScratchTrim() {
  const unsigned long long context = CurrentContext();
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  const auto it = g_scratch_pools.find(context);
  if (it != g_scratch_pools.end() && it->second != nullptr) cudaMemPoolTrimTo(it->second, 0);
  cudaGetLastError();
}

}  // namespace ccb

using namespace ccb;

extern "C" {

int ccb_evaluate_labelings(const uint32_t* bits, uint32_t n, uint32_t words_per_row, uint64_t edges, int32_t k,
                           int32_t count, const int32_t* labels, int64_t* f_out, int32_t* sizes_out, int32_t* g_out,
                           void* stream) {
  if (const char* why = CheckEvaluateArgs(bits, n, words_per_row, k, count, labels, f_out)) {
    return Report(CCB_ERR_INVALID, why);
  }
  if (count == 0) return Report(CCB_OK, "");
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (PreferTensorRecount(bits, (int)n, (int)words_per_row, k, count)) {
    if (RecountTensor(bits, n, words_per_row, edges, k, count, labels, f_out, sizes_out, g_out, st, true, false) == CCB_OK) {
      return CCB_OK;
    }
    cudaGetLastError();  // not enough memory or no contraction here: by popcount, with an eighth of the scratch
  }
  const int words = (int)((n + 31) / 32);
  const size_t mask_bytes = sizeof(uint32_t) * (size_t)count * k * words;
  uint32_t* masks = nullptr;
  cudaError_t e = cudaSuccess;
  if (mask_bytes > 0) {
    e = ScratchAlloc(reinterpret_cast<void**>(&masks), mask_bytes, st);
    if (e != cudaSuccess) return Report(CCB_ERR_DEVICE_MEMORY, cudaGetErrorString(e));
  }
  e = LaunchEvaluate(bits, (int)n, (int)words_per_row, edges, k, count, labels, masks, f_out, sizes_out, g_out, st);
  if (masks) cudaFreeAsync(masks, st);
  if (e != cudaSuccess) return Report(CCB_ERR_CUDA, cudaGetErrorString(e));
  return Report(CCB_OK, "");
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Allocation-free recount.
//
// Some callers cannot allocate device memory when they call in: a host application whose device
// memory is already reserved by its own pool allocator (a framework that took the free memory up
// front, where cudaMalloc fails or fragments that pool), or a latency-critical loop that must not pay
// cudaMalloc / cudaFree, which can synchronise the whole device.  For them the mask scratch of
// the recount lives in a fixed array in device memory, loaded with the library: every GPU that loads
// libccb.so holds these kNoAllocMaskWords words (4 MiB) until the process exits.
//
// The array's host-side name is only a stand-in, not a device address, so the entry point looks the
// address up with cudaGetSymbolAddress once per device (on its first call on that device, with that
// device current) and passes it to the kernel.  Make that first call before any stream capture.
// Under CUDA's default lazy module loading the array is only allocated when that first call loads this
// module onto the device, so a caller that reserves the device's free memory for its own pool must make
// the first call before it does; a call with count = 0 does exactly this set-up and nothing else.  (With
// CUDA_MODULE_LOADING=EAGER the array is allocated when the library is loaded.)  The address is kept for
// the life of the process: after cudaDeviceReset on a device the module is loaded afresh and may sit
// elsewhere, so the entry point must not be used across a device reset.
// Every call shares the one array and finds the last call's contents there.  The recount writes every
// mask word it later reads, so nothing needs clearing between calls; but two calls whose kernels
// overlap on the GPU (different streams, or different host threads) race on the array, so callers
// must order their calls.
// ------------------------------------------------------------------------------------------------
namespace ccb {
namespace {

constexpr size_t kNoAllocMaskWords = size_t(1) << 20;
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) uint32_t g_noalloc_masks[kNoAllocMaskWords];

std::mutex g_noalloc_mutex;
uint32_t* g_noalloc_address[kNoAllocMaxDevices] = {};

// Device address of g_noalloc_masks on the current device, looked up once per device.
cudaError_t NoAllocScratch(uint32_t** out) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device < 0 || device >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_address[device] == nullptr) {
    void* address = nullptr;
    e = cudaGetSymbolAddress(&address, g_noalloc_masks);
    if (e != cudaSuccess) return e;
    g_noalloc_address[device] = static_cast<uint32_t*>(address);
  }
  *out = g_noalloc_address[device];
  return cudaSuccess;
}

}  // namespace
}  // namespace ccb

extern "C" {

int ccb_evaluate_labelings_noalloc(const uint32_t* bits, uint32_t n, uint32_t words_per_row, uint64_t edges,
                                   int32_t k, int32_t count, const int32_t* labels, int64_t* f_out,
                                   int32_t* sizes_out, int32_t* g_out, void* stream) {
  if (const char* why = CheckEvaluateArgs(bits, n, words_per_row, k, count, labels, f_out)) {
    return Report(CCB_ERR_INVALID, why);
  }
  const size_t words = (n + 31) / 32;
  if ((size_t)count * (size_t)k * words > kNoAllocMaskWords) {
    return Report(CCB_ERR_INVALID,
                  "ccb_evaluate_labelings_noalloc: count * k * ceil(n / 32) exceeds the 1048576 mask words of "
                  "its static scratch; split the batch or use ccb_evaluate_labelings");
  }
  uint32_t* masks = nullptr;
  cudaError_t e = NoAllocScratch(&masks);  // also the whole of a count = 0 call: the per-device set-up
  if (e != cudaSuccess) return Report(CCB_ERR_CUDA, cudaGetErrorString(e));
  if (count == 0) return Report(CCB_OK, "");
  e = LaunchEvaluate(bits, (int)n, (int)words_per_row, edges, k, count, labels, masks, f_out, sizes_out, g_out,
                     static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return Report(CCB_ERR_CUDA, cudaGetErrorString(e));
  return Report(CCB_OK, "");
}

}  // extern "C"
