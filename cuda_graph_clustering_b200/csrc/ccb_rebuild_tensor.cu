// G = A*Z on the tensor cores: the one-hot builder, the tcgen05 contraction kernel, and the recount entry
// point ccb_evaluate_labelings_tensor.  See ccb_rebuild_tensor.h for the data flow.
#include "ccb_rebuild_tensor.h"

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "ccb.h"
#include "ccb_error.h"
#include "ccb_util.h"

namespace ccb {
namespace {

constexpr int kTileK = 128;                         // vertices u per pipeline stage: one 128-byte row
constexpr int kStages = 3;
constexpr int kSubTiles = 2;                        // 128-row accumulators per CTA, sharing each Z stage
constexpr int kMmaK = 32;                           // K of one kind::i8 MMA, in bytes
constexpr int kThreads = 192;                       // warp 0 TMA, warp 1 MMA + TMEM, warps 2..5 expand + epilogue
constexpr int kATileBytes = kTensorTileM * kTileK;  // int8 A sub-tile per stage: 16 KiB
constexpr int kBitsTileBytes = kTensorTileM * 16;   // adjacency words of a sub-tile per stage: 4 per row, 2 KiB
constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // a wait gives up after 2 s ...
constexpr uint32_t kWaitSpinLimit = 1u << 24;               // ... or this many polls

// ---- PTX wrappers ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t SmemAddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void BarInit(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void BarArrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(SmemAddr(bar)) : "memory");
}

__device__ __forceinline__ void BarArriveExpectTx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(SmemAddr(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool BarTryWait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(SmemAddr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits for the phase of `bar` with the given parity.  Gives up (false) after kWaitLimitNs or kWaitSpinLimit
// polls, or as soon as another role of the CTA gave up (*abort, when given).
__device__ __noinline__ bool BarWait(uint64_t* bar, uint32_t parity, volatile int* abort) {
  if (BarTryWait(bar, parity)) return true;
  const unsigned long long t0 = GlobalTimerNs();
  for (uint32_t spin = 1;; ++spin) {
    if (BarTryWait(bar, parity)) return true;
    if ((spin & 63) == 0) {
      if (abort != nullptr && *abort) return false;
      if (spin >= kWaitSpinLimit || GlobalTimerNs() - t0 > kWaitLimitNs) return false;
    }
  }
}

__device__ __forceinline__ void FenceBarrierInit() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Generic-proxy shared-memory writes become visible to the async proxy (the tensor cores' operand reads).
__device__ __forceinline__ void FenceProxyAsyncShared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 2-D tiled TMA load into this CTA's shared memory, completing on `bar` (no multicast).
__device__ __forceinline__ void TmaLoad2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(SmemAddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(SmemAddr(bar))
      : "memory");
}

__device__ __forceinline__ void TmemAlloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(slot)), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void TmemRelinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void TmemDealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void TcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void TcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, unsigned 8-bit operands, int32 accumulators.
__device__ __forceinline__ void MmaI8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                      uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives on `bar` once every MMA this thread issued so far has completed.
__device__ __forceinline__ void MmaCommit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(SmemAddr(bar))
               : "memory");
}

// 16 consecutive 32-bit accumulator columns of this thread's TMEM lane.  Load and wait are one statement: between two, the
// compiler may use a register before its load has landed.
__device__ __forceinline__ void TmemLoad16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Shared-memory matrix descriptor of a K-major operand in the 128-byte swizzled layout: rows of 128 bytes,
// 8-row atoms of 1024 bytes (stride byte offset), 1024-byte aligned tile base.  Fields: start address >> 4
// (bits 0-13), leading byte offset 1 (unused for swizzled K-major), stride byte offset 1024 >> 4 (bits
// 32-45), descriptor version 1 (bits 46-47), base offset 0, layout 2 = 128-byte swizzle (bits 61-63).
// Advancing K by 32 bytes inside the atom adds 2 to the start field.
__device__ __forceinline__ uint64_t Sw128Desc(uint32_t smem_addr) {
  const uint64_t lo = ((smem_addr >> 4) & 0x3FFFu) | (1u << 16);
  const uint64_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return lo | (hi << 32);
}

// Instruction descriptor of kind::i8: int32 accumulator (bits 4-5 = 2), unsigned 8-bit A and B (bits 7-12 =
// 0), both K-major, N >> 3 (bits 17-22), M >> 4 (bits 24-28).
__host__ __device__ constexpr uint32_t IdescI8(int m, int n) {
  return (2u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// Four adjacency bits -> four bytes 0/1 (bit j -> byte j): the multiply places bit j at bit 8j with no carries.
__device__ __forceinline__ uint32_t Spread4(uint32_t nibble) { return (nibble * 0x00204081u) & 0x01010101u; }

struct TensorArgs {
  void* g;             // [col][ld] of GainT, may be null
  int ld;
  int n;               // vertices (labels exist for v < n)
  int n_store;         // rows written per column
  int columns;         // live columns (count * k)
  int k;
  int bn;
  int ktiles;
  int tmem_cols;
  const void* labels;  // [slot][label_ld]
  int label_ld;
  int64_t* intra;      // [slot]
  int32_t* error;
  const Control* stop; // null: always run
};

template <typename LabelT, typename GainT>
__global__ void __launch_bounds__(kThreads, 1)
    k_rebuild_tensor(const __grid_constant__ CUtensorMap bits_map, const __grid_constant__ CUtensorMap z_map,
                     TensorArgs a) {
  if (a.stop != nullptr && a.stop->stop) return;  // uniform: before any barrier or TMEM use
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int bn = a.bn;
  uint8_t* s_a = base;                                        // [stage][sub][128 rows][128 B], swizzled
  uint8_t* s_b = s_a + kStages * kSubTiles * kATileBytes;     // [stage][bn rows][128 B], swizzled by TMA
  uint8_t* s_bits = s_b + kStages * bn * kTileK;              // [stage][sub][128 rows][16 B]
  uint64_t* full = reinterpret_cast<uint64_t*>(s_bits + kStages * kSubTiles * kBitsTileBytes);
  uint64_t* a_ready = full + kStages;
  uint64_t* empty = a_ready + kStages;
  uint64_t* accum = empty + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x / kWarp;
  const int lane = threadIdx.x % kWarp;
  const int m0 = blockIdx.x * kTensorTileM * kSubTiles;
  const int n0 = blockIdx.y * bn;
  const int ktiles = a.ktiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      BarInit(&full[s], 1);
      BarInit(&a_ready[s], 4);
      BarInit(&empty[s], 1);
    }
    BarInit(accum, 1);
    *abort = 0;
    FenceBarrierInit();
  }
  if (warp == 1) {
    TmemAlloc(tmem_slot, a.tmem_cols);
    TmemRelinquish();
  }
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  const uint32_t tmem = *tmem_slot;

  auto give_up = [&]() {
    *abort = 1;
    atomicExch(a.error, kErrorWaitTimeout);
  };

  if (warp == 0) {
    if (lane == 0) {
      // TMA producer: stage s holds the adjacency words of K step kt and the Z block's bytes of it.
      const uint32_t bytes = kSubTiles * kBitsTileBytes + bn * kTileK;
      int issued = 0;
      for (int kt = 0; kt < ktiles; ++kt) {
        const int s = kt % kStages;
        if (kt >= kStages && !BarWait(&empty[s], ((kt / kStages) - 1) & 1, abort)) {
          give_up();
          break;
        }
        BarArriveExpectTx(&full[s], bytes);
#pragma unroll
        for (int sub = 0; sub < kSubTiles; ++sub) {  // a box past the last row reads zeros
          TmaLoad2d(s_bits + (s * kSubTiles + sub) * kBitsTileBytes, &bits_map, kt * 4, m0 + sub * kTensorTileM,
                    &full[s]);
        }
        TmaLoad2d(s_b + s * bn * kTileK, &z_map, kt * kTileK, n0, &full[s]);
        issued = kt + 1;
      }
      // drain: every copy issued has landed before the CTA may exit
      for (int kt = std::max(0, issued - kStages); kt < issued; ++kt) {
        if (!BarWait(&full[kt % kStages], (kt / kStages) & 1, nullptr)) give_up();
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = IdescI8(kTensorTileM, bn);
      const uint32_t a_base = SmemAddr(s_a);
      const uint32_t b_base = SmemAddr(s_b);
      for (int kt = 0; kt < ktiles; ++kt) {
        const int s = kt % kStages;
        const uint32_t par = (kt / kStages) & 1;
        if (!BarWait(&full[s], par, abort) || !BarWait(&a_ready[s], par, abort)) {
          give_up();
          break;
        }
        TcFenceAfter();
        const uint64_t bd = Sw128Desc(b_base + s * bn * kTileK);
#pragma unroll
        for (int sub = 0; sub < kSubTiles; ++sub) {  // accumulator `sub` in TMEM columns [sub * bn, (sub + 1) * bn)
          const uint64_t ad = Sw128Desc(a_base + (s * kSubTiles + sub) * kATileBytes);
#pragma unroll
          for (int j = 0; j < kTileK / kMmaK; ++j) {
            MmaI8(tmem + sub * bn, ad + 2 * j, bd + 2 * j, idesc, (kt > 0 || j > 0) ? 1u : 0u);
          }
        }
        MmaCommit(&empty[s]);  // the stage is free once these MMAs have read it
      }
      MmaCommit(accum);  // every MMA issued has completed: the accumulator is final (or, on abort, idle)
      if (!BarWait(accum, 0, nullptr)) give_up();
    }
    __syncwarp();
  } else {
    // Expansion: thread r turns row r's 128 adjacency bits of the stage into 128 bytes of the A tile, in the
    // 128-byte swizzle (16-byte chunk q of row r at chunk q ^ (r % 8) of its 1024-byte atom).
    const int r = (warp - 2) * kWarp + lane;
    for (int kt = 0; kt < ktiles; ++kt) {
      const int s = kt % kStages;
      if (!__all_sync(kAllLanes, BarWait(&full[s], (kt / kStages) & 1, abort))) {  // warp-uniform outcome
        if (lane == 0) give_up();
        break;
      }
#pragma unroll
      for (int sub = 0; sub < kSubTiles; ++sub) {
        const int t = s * kSubTiles + sub;
        const uint4 w = *reinterpret_cast<const uint4*>(s_bits + t * kBitsTileBytes + r * 16);
        const uint32_t words[4] = {w.x, w.y, w.z, w.w};
        uint8_t* row = s_a + t * kATileBytes + (r >> 3) * 1024 + (r & 7) * kTileK;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t h = (words[q >> 1] >> ((q & 1) * 16)) & 0xFFFFu;
          uint4 out;
          out.x = Spread4(h & 0xFu);
          out.y = Spread4((h >> 4) & 0xFu);
          out.z = Spread4((h >> 8) & 0xFu);
          out.w = Spread4(h >> 12);
          *reinterpret_cast<uint4*>(row + ((q ^ (r & 7)) << 4)) = out;
        }
      }
      FenceProxyAsyncShared();
      __syncwarp();
      if (lane == 0) BarArrive(&a_ready[s]);
    }
    // Epilogue: warp w reads TMEM lanes 32 * (w % 4) .. +31, i.e. vertices m0 + 32 * (w % 4) + lane.
    const bool ok = __all_sync(kAllLanes, BarWait(accum, 0, nullptr));
    if (!ok && lane == 0) give_up();
    TcFenceAfter();
    const int quarter = warp & 3;
    const LabelT* labels = static_cast<const LabelT*>(a.labels);
    GainT* g = static_cast<GainT*>(a.g);
    const bool write = ok && !*abort;
    for (int sub = 0; sub < kSubTiles; ++sub) {
      const int v = m0 + sub * kTensorTileM + quarter * kWarp + lane;
      const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quarter * kWarp) << 16) + sub * bn;
      // columns in order: cluster c of slot; a slot's label of v is loaded a slot ahead
      int slot = n0 / a.k, c = n0 - slot * a.k, part = 0;
      const int slots = a.columns / a.k;
      auto label = [&](int of) {
        return of < slots && v < a.n ? static_cast<int>(labels[static_cast<size_t>(of) * a.label_ld + v]) : -1;
      };
      int own = label(slot), own_next = label(slot + 1);
      auto flush = [&]() {
        const unsigned total = __reduce_add_sync(kAllLanes, static_cast<unsigned>(part));
        if (lane == 0 && write && total != 0) {
          atomicAdd(reinterpret_cast<unsigned long long*>(a.intra + slot), static_cast<unsigned long long>(total));
        }
        part = 0;
      };
      const bool store = write && g != nullptr && v < a.n_store;
      GainT* out = g + static_cast<size_t>(n0) * a.ld + v;
      for (int c0 = 0; c0 < bn; c0 += 16) {
        if (n0 + c0 >= a.columns) break;
        uint32_t acc[16];
        TmemLoad16(lane_addr + c0, acc);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (n0 + c0 + i >= a.columns) break;
          const int val = static_cast<int>(acc[i]);
          if (store) *out = static_cast<GainT>(val);
          out += a.ld;
          part += own == c ? val : 0;
          if (++c == a.k) {
            flush();
            c = 0;
            ++slot;
            own = own_next;
            own_next = label(slot + 1);
          }
        }
      }
      if (c != 0) flush();
    }
  }
  TcFenceBefore();
  __syncthreads();
  if (warp == 1) {
    TcFenceAfter();
    TmemDealloc(tmem, a.tmem_cols);
  }
}

// Z rows, sizes and bad-label flags of the recount's labelings.
__global__ void __launch_bounds__(256)
    k_build_z(const int32_t* __restrict__ labels, int n, int k, int kz, uint8_t* __restrict__ z,
              int32_t* __restrict__ sizes, int kpad, int64_t* __restrict__ intra, int32_t* __restrict__ bad) {
  __shared__ int s_sizes[kMaxK];
  __shared__ int s_bad;
  const int slot = blockIdx.x;
  const int tid = threadIdx.x;
  const int32_t* lab = labels + static_cast<size_t>(slot) * n;
  for (int c = tid; c < k; c += blockDim.x) s_sizes[c] = 0;
  if (tid == 0) s_bad = 0;
  __syncthreads();
  const int words = kz / 4;
  uint32_t* rows = reinterpret_cast<uint32_t*>(z + static_cast<size_t>(slot) * k * kz);
  for (int i = tid; i < words; i += blockDim.x) {
    int l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int u = 4 * i + j;
      l[j] = u < n ? lab[u] : -1;
      if (u < n && (l[j] < 0 || l[j] >= k)) {
        s_bad = 1;
        l[j] = -1;
      }
      if (l[j] >= 0) atomicAdd(&s_sizes[l[j]], 1);
    }
    for (int c = 0; c < k; ++c) {
      rows[static_cast<size_t>(c) * words + i] = static_cast<uint32_t>(l[0] == c) |
                                                 (static_cast<uint32_t>(l[1] == c) << 8) |
                                                 (static_cast<uint32_t>(l[2] == c) << 16) |
                                                 (static_cast<uint32_t>(l[3] == c) << 24);
    }
  }
  __syncthreads();
  for (int c = tid; c < k; c += blockDim.x) sizes[static_cast<size_t>(slot) * kpad + c] = s_sizes[c];
  if (tid == 0) {
    intra[slot] = 0;
    bad[slot] = s_bad;
  }
}

// The labels of a rebuild (GWW copy, perturbation, neighbourhood or as they are: RebuildBody's first phase), their
// cluster sizes and their one-hot rows Z in one pass: a block takes `span` vertices of a slot, a thread four of them
// at a time, whose label bytes and Z words are written whole.
constexpr int kLabelsThreads = 256;

// Whether the iteration that a rebuild belongs to has been stopped.
template <typename GainT>
__device__ __forceinline__ bool RebuildStopped(const RebuildArgs<GainT>& a) {
  return a.ctl != nullptr && (a.mode == kRebuildPerturb || a.mode == kRebuildCopy) && a.ctl->stop;
}

// Cluster sizes zeroed for k_labels_z to add to, where several blocks share a slot.
template <typename GainT>
__global__ void __launch_bounds__(kLabelsThreads) k_clear_sizes(RebuildArgs<GainT> a, int count) {
  const int i = blockIdx.x * kLabelsThreads + threadIdx.x;
  if (i < count && !RebuildStopped(a)) a.cur.sizes[i] = 0;
}

template <typename GainT>
__global__ void __launch_bounds__(kLabelsThreads)
    k_labels_z(RebuildArgs<GainT> a, uint8_t* __restrict__ z, int kz, int span) {
  if (RebuildStopped(a)) return;
  __shared__ int s_sizes[kMaxK];
  const int slot = blockIdx.x;
  const int tid = threadIdx.x;
  const int lane = tid % kWarp;
  const int n = a.gr.n, k = a.k, ld = a.ld;
  for (int c = tid; c < k; c += kLabelsThreads) s_sizes[c] = 0;
  __syncthreads();
  const uint8_t* from = a.cur.labels + static_cast<size_t>(slot) * ld;
  if (a.mode == kRebuildPerturb || a.mode == kRebuildCopy) {
    from = a.next_labels + static_cast<size_t>(a.src_map != nullptr ? a.src_map[slot] : slot) * ld;
  }
  const int center = a.first + slot;
  const uint32_t* center_row = a.gr.bits + static_cast<size_t>(a.mode == kRebuildNeighborhood ? center : 0) * a.gr.pitch;
  uint32_t* to = reinterpret_cast<uint32_t*>(a.cur.labels + static_cast<size_t>(slot) * ld);
  const int words = kz / 4;
  uint32_t* rows = reinterpret_cast<uint32_t*>(z + static_cast<size_t>(slot) * k * kz);
  int size0 = 0, size1 = 0;  // of clusters lane and lane + 32
  const int first = blockIdx.y * span / 4;
  const int last = min(words, first + span / 4);
  for (int i = first + tid; i < last; i += kLabelsThreads) {  // whole warps: span is a multiple of 128
    uint32_t packed = 4 * i < ld && a.mode != kRebuildNeighborhood ? reinterpret_cast<const uint32_t*>(from)[i] : 0u;
    int l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int u = 4 * i + j;
      l[j] = static_cast<int>((packed >> (8 * j)) & 0xffu);
      if (a.mode == kRebuildNeighborhood) {
        l[j] = u < n && !(u == center || Bit(center_row, u)) ? 1 : 0;
      } else if (a.mode == kRebuildPerturb && u < n) {
        l[j] = PerturbLabelOf(a.stream, static_cast<uint64_t>(slot) * n + u, a.iteration, l[j], k, a.probability);
      }
    }
    packed = static_cast<uint32_t>(l[0]) | static_cast<uint32_t>(l[1]) << 8 | static_cast<uint32_t>(l[2]) << 16 |
             static_cast<uint32_t>(l[3]) << 24;
    if (4 * i < n && a.mode != kRebuildInPlace) to[i] = packed;
#pragma unroll
    for (int j = 0; j < 4; ++j) l[j] = 4 * i + j < n ? l[j] : -1;
    for (int c = 0; c < k; ++c) {
      const uint32_t word = static_cast<uint32_t>(l[0] == c) | static_cast<uint32_t>(l[1] == c) << 8 |
                            static_cast<uint32_t>(l[2] == c) << 16 | static_cast<uint32_t>(l[3] == c) << 24;
      rows[static_cast<size_t>(c) * words + i] = word;
      const int total = __reduce_add_sync(kAllLanes, (word * 0x01010101u) >> 24);
      size0 += lane == c ? total : 0;
      size1 += lane + kWarp == c ? total : 0;
    }
  }
  if (lane < k && size0 != 0) atomicAdd(&s_sizes[lane], size0);
  if (lane + kWarp < k && size1 != 0) atomicAdd(&s_sizes[lane + kWarp], size1);
  __syncthreads();
  for (int c = tid; c < k; c += kLabelsThreads) {
    int32_t* size = a.cur.sizes + static_cast<size_t>(slot) * a.kpad + c;
    if (gridDim.y == 1) {
      *size = s_sizes[c];
    } else if (s_sizes[c] != 0) {
      atomicAdd(size, s_sizes[c]);
    }
  }
  if (tid == 0 && blockIdx.y == 0) a.intra[slot] = 0;
}

// What the recount's last step needs to count a labeling again by popcount.
struct RecountArgs {
  const uint32_t* bits;
  int n, words, pitch;
  const int32_t* labels;  // [count][n]
  uint32_t* masks;        // scratch: labeling s at s * mask_step words, [k][words]
  size_t mask_step;
  int32_t* g;             // [count][k][n], may be null
};

// One labeling's intra-cluster sum (each pair twice) and, with a.g, its G, by the whole block: the sum in thread 0.
template <int kThreads>
__device__ long long RecountByPopcount(const RecountArgs& a, int slot, int k) {
  constexpr int kWarps = kThreads / kWarp;
  __shared__ long long s_sum[kWarps];
  const int lane = threadIdx.x % kWarp;
  const int warp = threadIdx.x / kWarp;
  const int32_t* labels = a.labels + static_cast<size_t>(slot) * a.n;
  uint32_t* masks = a.masks + slot * a.mask_step;
  for (int w = warp; w < a.words; w += kWarps) {
    const int v = w * kWarp + lane;
    const int l = v < a.n ? labels[v] : -1;
    for (int c = 0; c < k; ++c) {
      const uint32_t m = __ballot_sync(kAllLanes, l == c);
      if (lane == 0) masks[static_cast<size_t>(c) * a.words + w] = m;
    }
  }
  __syncthreads();
  long long own_sum = 0;
  for (int v = warp; v < a.n; v += kWarps) {
    const uint32_t* row = a.bits + static_cast<size_t>(v) * a.pitch;
    const int own = labels[v];
    for (int c = 0; c < k; ++c) {
      int common = 0;
      for (int w = lane; w < a.words; w += kWarp) common += __popc(row[w] & masks[static_cast<size_t>(c) * a.words + w]);
      common = __reduce_add_sync(kAllLanes, common);
      if (lane == 0) {
        if (a.g != nullptr) a.g[(static_cast<size_t>(slot) * k + c) * a.n + v] = common;
        if (own == c) own_sum += common;
      }
    }
  }
  return BlockSum<kWarps>(own_sum, s_sum);
}

// f = m + sum_c C(size_c, 2) - intra per labeling (the recount's last step); -1 for a bad label.  When the contraction's
// bounded wait gave up: with a.bits null -2, else each block counts its labelings again, slowly, over the one-hot scratch.
constexpr int kFinishThreads = 128;
__global__ void __launch_bounds__(kFinishThreads)
    k_tensor_finish(const int32_t* sizes, int kpad, const int64_t* intra, const int32_t* bad, const int32_t* error, int count,
                    int k, long long edges, int64_t* f_out, RecountArgs a) {
  const int first = blockIdx.x * kFinishThreads;
  const int slot = first + threadIdx.x;
  const auto objective = [&](int s, long long own) {
    long long pairs = 0;
    for (int c = 0; c < k; ++c) {
      const long long sz = sizes[static_cast<size_t>(s) * kpad + c];
      pairs += sz * (sz - 1) / 2;
    }
    return bad[s] ? -1ll : edges + pairs - own;
  };
  if (*error == 0) {
    if (slot < count) f_out[slot] = objective(slot, intra[slot]);
  } else if (a.bits == nullptr) {
    if (slot < count) f_out[slot] = -2;
  } else {
    for (int s = first; s < min(count, first + kFinishThreads); ++s) {
      const long long own = RecountByPopcount<kFinishThreads>(a, s, k);
      if (threadIdx.x == 0) f_out[s] = objective(s, own);
    }
  }
}

using EncodeTiledFn = PFN_cuTensorMapEncodeTiled_v12000;

EncodeTiledFn EncodeTiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  });
  return fn;
}

size_t TensorSmem(int bn) {
  return 1024 + static_cast<size_t>(kStages) * (kSubTiles * (kATileBytes + kBitsTileBytes) + bn * kTileK) +
         (3 * kStages + 1) * sizeof(uint64_t) + 16;
}

}  // namespace

bool PlanTensorRebuild(TensorRebuild& t, int n, int columns, int sms, const char** why) {
  if (n < kTensorTileM) {
    *why = "the tensor-core rebuild needs n >= 128";
    return false;
  }
  if (columns < 1) {
    *why = "no columns";
    return false;
  }
  t.n = n;
  t.words = (n + 31) / 32;
  t.ktiles = (t.words + 3) / 4;
  t.kz = t.ktiles * kTileK;
  t.columns = columns;
  t.m_tiles = (n + kTensorTileM * kSubTiles - 1) / (kTensorTileM * kSubTiles);
  // Columns per CTA: the fewest clocks of the CTAs that one SM runs one after another, by what a CTA was measured to
  // take: 2400 a K step (expanding 256 rows of bits; the MMAs and the Z copy hide behind it up to 256 columns), 80 a
  // column of the epilogue.  Wide blocks win when K is long (n = 65536, pop 128, k = 2: one block of 256 columns),
  // narrow ones fill the SMs when it is short (n = 1000, 2048 columns: 64).
  long long least = -1;
  for (int bn = kTensorMaxN; bn >= 16; bn -= 16) {
    const long long ctas = (long long)t.m_tiles * ((columns + bn - 1) / bn);
    const long long cost = (ctas + sms - 1) / sms * (2400ll * t.ktiles + 80ll * std::min(bn, columns) + 4000);
    if (least < 0 || cost < least) {
      least = cost;
      t.bn = bn;
    }
  }
  t.bn = std::min(t.bn, (columns + 15) / 16 * 16);
  t.n_tiles = (columns + t.bn - 1) / t.bn;
  t.z_rows = t.n_tiles * t.bn;
  t.tmem_cols = 32;
  while (t.tmem_cols < kSubTiles * t.bn) t.tmem_cols *= 2;
  t.smem = TensorSmem(t.bn);
  return true;
}

cudaError_t EncodeTensorRebuild(TensorRebuild& t, const uint32_t* bits, int pitch_words, uint8_t* z) {
  EncodeTiledFn encode = EncodeTiled();
  if (encode == nullptr) return cudaErrorNotSupported;
  t.z = z;
  {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(t.words), static_cast<cuuint64_t>(t.n)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch_words) * 4};
    const cuuint32_t box[2] = {4, kTensorTileM};
    const cuuint32_t estr[2] = {1, 1};
    if (encode(&t.bits_map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint32_t*>(bits), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
      return cudaErrorInvalidValue;
    }
  }
  {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(t.kz), static_cast<cuuint64_t>(t.z_rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(t.kz)};
    const cuuint32_t box[2] = {kTileK, static_cast<cuuint32_t>(t.bn)};
    const cuuint32_t estr[2] = {1, 1};
    if (encode(&t.z_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, z, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
      return cudaErrorInvalidValue;
    }
  }
  return cudaSuccess;
}

template <typename GainT>
cudaError_t LaunchLabelsZ(const TensorRebuild& t, const RebuildArgs<GainT>& a, int count, int sms, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  // about two blocks per SM, each of whole 128-vertex groups; one block per slot writes the sizes itself
  const int groups = t.kz / kTileK;
  const int want = std::max(1, std::min(groups, (2 * sms + count - 1) / count));
  const int span = (groups + want - 1) / want * kTileK;
  const int blocks = (t.kz + span - 1) / span;
  if (blocks > 1) {  // a kernel, not a memset: past a stop the population stays as it is
    const int sizes = count * a.kpad;
    k_clear_sizes<GainT><<<(sizes + kLabelsThreads - 1) / kLabelsThreads, kLabelsThreads, 0, st>>>(a, sizes);
  }
  k_labels_z<GainT><<<dim3(count, blocks), kLabelsThreads, 0, st>>>(a, t.z, t.kz, span);
  return cudaGetLastError();
}

template <typename LabelT, typename GainT>
cudaError_t LaunchTensorRebuild(const TensorRebuild& t, GainT* g, int ld, int n_store, int count, int k,
                                const LabelT* labels, int label_ld, int64_t* intra, int32_t* error, const Control* ctl,
                                cudaStream_t st) {
  const int columns = count * k;
  if (columns <= 0) return cudaSuccess;
  if (columns > t.z_rows) return cudaErrorInvalidValue;
  // one limit for every plan: a smaller one set here could come between another thread's limit and its launch
  const cudaError_t attr = cudaFuncSetAttribute(k_rebuild_tensor<LabelT, GainT>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TensorSmem(kTensorMaxN));
  if (attr != cudaSuccess) return attr;
  TensorArgs a{};
  a.g = g;
  a.ld = ld;
  a.n = t.n;
  a.n_store = n_store;
  a.columns = columns;
  a.k = k;
  a.bn = t.bn;
  a.ktiles = t.ktiles;
  a.tmem_cols = t.tmem_cols;
  a.labels = labels;
  a.label_ld = label_ld;
  a.intra = intra;
  a.error = error;
  a.stop = ctl;
  const dim3 grid(t.m_tiles, (columns + t.bn - 1) / t.bn);
  k_rebuild_tensor<LabelT, GainT><<<grid, kThreads, t.smem, st>>>(t.bits_map, t.z_map, a);
  return cudaGetLastError();
}

template cudaError_t LaunchLabelsZ<int16_t>(const TensorRebuild&, const RebuildArgs<int16_t>&, int, int, cudaStream_t);
template cudaError_t LaunchLabelsZ<int32_t>(const TensorRebuild&, const RebuildArgs<int32_t>&, int, int, cudaStream_t);
template cudaError_t LaunchTensorRebuild<uint8_t, int16_t>(const TensorRebuild&, int16_t*, int, int, int, int,
                                                           const uint8_t*, int, int64_t*, int32_t*, const Control*,
                                                           cudaStream_t);
template cudaError_t LaunchTensorRebuild<uint8_t, int32_t>(const TensorRebuild&, int32_t*, int, int, int, int,
                                                           const uint8_t*, int, int64_t*, int32_t*, const Control*,
                                                           cudaStream_t);

int RecountTensor(const uint32_t* bits, uint32_t n, uint32_t words_per_row, uint64_t edges, int32_t k, int32_t count,
                  const int32_t* labels, int64_t* f_out, int32_t* sizes_out, int32_t* g_out, cudaStream_t st, bool recover,
                  bool gave_up) {
  auto report = [](int status, const std::string& message) {
    SetLastError(message);
    return status;
  };
  if (k < 1 || k > CCB_MAX_CLUSTERS) return report(CCB_ERR_INVALID, "k must be in [1, 64]");
  if (count < 0) return report(CCB_ERR_INVALID, "count must be >= 0");
  if (n > (uint32_t)CCB_MAX_VERTICES_WIDE) return report(CCB_ERR_INVALID, "n exceeds 1048576");
  if (count == 0) return report(CCB_OK, "");
  if (bits == nullptr || labels == nullptr || f_out == nullptr) return report(CCB_ERR_INVALID, "null pointer");
  if (words_per_row < (n + 31) / 32) return report(CCB_ERR_INVALID, "words_per_row < ceil(n / 32)");
  if (words_per_row % 4 != 0 || reinterpret_cast<uintptr_t>(bits) % 16 != 0) {
    return report(CCB_ERR_INVALID, "the tensor-core recount needs 16-byte aligned rows (words_per_row % 4 == 0)");
  }
  if ((long long)count * k > (1 << 24)) return report(CCB_ERR_INVALID, "count * k exceeds 16777216");
  TensorRebuild t;
  const char* why = nullptr;
  int device = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return report(CCB_ERR_CUDA, cudaGetErrorString(e));
  if (!PlanTensorRebuild(t, (int)n, count * k, sms, &why)) return report(CCB_ERR_INVALID, why);
  const int kpad = (k + 3) / 4 * 4;
  const size_t z_bytes = (size_t)t.z_rows * t.kz;
  const size_t sizes_bytes = sizes_out ? 0 : (size_t)count * kpad * 4;
  const size_t scratch = z_bytes + (size_t)count * 8 + (size_t)count * 4 + 16 + sizes_bytes;
  uint8_t* buf = nullptr;
  e = ScratchAlloc(reinterpret_cast<void**>(&buf), scratch, st);
  if (e != cudaSuccess) return report(CCB_ERR_DEVICE_MEMORY, cudaGetErrorString(e));
  uint8_t* z = buf;
  int64_t* intra = reinterpret_cast<int64_t*>(buf + z_bytes);  // z_bytes is a multiple of 128
  int32_t* bad = reinterpret_cast<int32_t*>(intra + count);
  int32_t* error = bad + count;
  int32_t* sizes = sizes_out ? sizes_out : error + 4;
  const int sizes_ld = sizes_out ? k : kpad;
  auto fail = [&](cudaError_t err) {
    cudaFreeAsync(buf, st);
    return report(CCB_ERR_CUDA, cudaGetErrorString(err));
  };
  if ((e = cudaMemsetAsync(z + (size_t)count * k * t.kz, 0, z_bytes - (size_t)count * k * t.kz, st)) != cudaSuccess ||
      (e = cudaMemsetAsync(error, gave_up ? 1 : 0, 4, st)) != cudaSuccess) {
    return fail(e);
  }
  if ((e = EncodeTensorRebuild(t, bits, (int)words_per_row, z)) != cudaSuccess) return fail(e);
  k_build_z<<<count, 256, 0, st>>>(labels, (int)n, k, t.kz, z, sizes, sizes_ld, intra, bad);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
  if ((e = LaunchTensorRebuild<int32_t, int32_t>(t, g_out, (int)n, (int)n, count, k, labels, (int)n, intra, error, nullptr,
                                                 st)) != cudaSuccess) {
    return fail(e);
  }
  // a labeling's k one-hot rows hold its k masks: kz >= 32 words bytes each
  const RecountArgs again{recover ? bits : nullptr, (int)n, t.words, (int)words_per_row, labels,
                          reinterpret_cast<uint32_t*>(z), (size_t)k * t.kz / 4, g_out};
  k_tensor_finish<<<(count + kFinishThreads - 1) / kFinishThreads, kFinishThreads, 0, st>>>(
      sizes, sizes_ld, intra, bad, error, count, k, (long long)edges, f_out, again);
  if ((e = cudaGetLastError()) != cudaSuccess) return fail(e);
  cudaFreeAsync(buf, st);
  return report(CCB_OK, "");
}

}  // namespace ccb

using namespace ccb;

extern "C" {

int ccb_evaluate_labelings_tensor(const uint32_t* bits, uint32_t n, uint32_t words_per_row, uint64_t edges, int32_t k,
                                  int32_t count, const int32_t* labels, int64_t* f_out, int32_t* sizes_out,
                                  int32_t* g_out, void* stream) {
  return RecountTensor(bits, n, words_per_row, edges, k, count, labels, f_out, sizes_out, g_out,
                       static_cast<cudaStream_t>(stream), false, false);
}

// Not in ccb.h: the contraction that ccb_evaluate_labelings takes, with its wait marked as given up from the start, so that
// a test sees the labelings counted again without making a kernel wait.
int ccb_test_recount_gave_up(const uint32_t* bits, uint32_t n, uint32_t words_per_row, uint64_t edges, int32_t k,
                             int32_t count, const int32_t* labels, int64_t* f_out, int32_t* sizes_out, int32_t* g_out,
                             void* stream) {
  return RecountTensor(bits, n, words_per_row, edges, k, count, labels, f_out, sizes_out, g_out,
                       static_cast<cudaStream_t>(stream), true, true);
}

}  // extern "C"
