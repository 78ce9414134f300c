// Steepest descent with the slot state in registers as move keys: compile-time K <= 8, V vertices per thread
// (u = tid + j * T, j < V), n <= V * T.  Same trajectory as k_descent and the reference's BestMove/ApplyMove
// (src/cc_pbils_cpu.cpp:99-139).
//
// For each owned vertex u a thread keeps K 32-bit keys
//     key_c(u) = 16 h_c(u) + c  (+ 2^20 for c = the label of u),   h_c(u) = size_c - 2 G_c(u),
// so the key of moving u to c orders candidates by h, then by the lower cluster: the reference's rule
// (MoveDelta, cc_math.hpp:75-77: the gain of a -> c is h_c - h_a + 1).  A foreign h_c <= n - size_a and the
// own h_a >= 2 - size_a, so foreign minus own h is at most n - 2 < 2^15 on the narrow path; the penalty
// (2^16 in units of h) therefore makes the minimum over the K lanes the best foreign target and the
// maximum the vertex's own cluster: no label, no G, no per-cluster offset is stored.
//
// A move (v: from -> to) shifts, for every vertex u, key_from by +16 if u is a neighbour of v and -16
// otherwise (size_from - 1, and G_from - 1 for neighbours), and key_to by the opposite amount; with the
// per-move coefficients coef_c = [c = from] - [c = to] that is one multiply-add per lane, folded into the
// scan of the next move.  The moved vertex itself (not its own neighbour) also moves its penalty from lane
// `from` to lane `to`.
#pragma once

#include <cstdint>

#include "ccb_device.cuh"

namespace ccb {

constexpr int kRegPenalty = 1 << 20;

// Minimum and maximum of K lanes with three-input min / max (DPX on sm_90 and later).
template <int K>
__device__ __forceinline__ void LanesMinMax(const int* x, int& lo, int& hi) {
  lo = x[0];
  hi = x[0];
  int c = 1;
#pragma unroll
  for (; c + 1 < K; c += 2) {
    lo = __vimin3_s32(lo, x[c], x[c + 1]);
    hi = __vimax3_s32(hi, x[c], x[c + 1]);
  }
  if (c < K) {
    lo = min(lo, x[c]);
    hi = max(hi, x[c]);
  }
}

// ---- compact pairs (n <= 1023) --------------------------------------------------------------------------
// Two vertices share 32-bit registers, a 16-bit lane each.  A vertex's K lanes are
//     foreign c:  8 (h_c + 1024) + c  (below 2^14, |h| <= n)      own a:  the same + 2^15,
// so that over the lanes the minimum is the best foreign target (smaller cluster first) and the maximum the own
// cluster.  Thread t holds the pairs (2 q, 2 q + 1), q = t + p T: their bits lie side by side in one row word.  A move
// (v: from -> to) adds +-8 to lanes `from` and -+8 to lanes `to` of every vertex by adjacency to v: with d the packed
// pair of +-8, one multiply-add of the 32-bit register per lane (no half leaves [0, 2^16), so none carries into the
// other).  The gain field of a vertex is X = (min & ~7) - (max & ~7) + 0xC000 = 8 (gain - 1) + 2^14; its move key
// X << 16 | u << 6 | from << 3 | to orders by gain, then vertex, and carries both clusters.  Lanes of absent vertices
// never move (no adjacency, no -8) and hold a gain that is never chosen.
//
// Bound by issue: 32-bit adds and multiply-adds take two clocks a warp here, 16-bit pair minima one, and every warp
// pays the move's overhead (argmin, decode, row address), so 128 threads hold 8 vertices each.  ns a move of 128 slots
// (B200), with one 32-bit key a lane on 256 threads and now: n = 1000, p = 0.5, k = 5 416, 279 (64 threads x 16: 415,
// 256 x 4: 336); n = 500, k = 8 456, 270; n = 200, k = 4 455, 304.
constexpr int kCompactMaxBits = 10;

template <int K, int T, int V>
__device__ __forceinline__ void DescentRegistersCompact(const DescentArgs<int16_t>& a, int slot, int w,
                                                        const uint32_t* rows, uint32_t* s_records) {
  constexpr int kWarps = T / kWarp;
  constexpr int P = V / 2;
  constexpr uint32_t kClusterBits = 0x00070007u;
  const int tid = threadIdx.x;
  const int lane = tid % kWarp;
  const int n = a.gr.n;
  const int ld = a.ld;

  uint32_t key[P][K];
  uint32_t code[P];  // u << 6 of both vertices
  uint32_t down[P];  // 8 in the half of each present vertex
  {
    const int16_t* g_src = a.cur.g + static_cast<size_t>(w) * K * ld;
    const uint8_t* l_src = a.cur.labels + static_cast<size_t>(w) * ld;
    const int32_t* sizes = a.cur.sizes + static_cast<size_t>(w) * a.kpad;
    int sz[K];
#pragma unroll
    for (int c = 0; c < K; ++c) sz[c] = sizes[c];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      code[p] = 0u;
      down[p] = 0u;
#pragma unroll
      for (int c = 0; c < K; ++c) key[p][c] = 0u;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int u = 2 * (tid + p * T) + half;
        const bool ok = u < n;
        const int own = ok ? l_src[u] : 0;
        code[p] |= static_cast<uint32_t>(ok ? u << 6 : 0) << (16 * half);
        down[p] |= (ok ? 8u : 0u) << (16 * half);
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const int h = ok ? sz[c] - 2 * static_cast<int>(g_src[static_cast<size_t>(c) * ld + u]) : (c == 0 ? -1024 : 1023);
          key[p][c] |= static_cast<uint32_t>(8 * (h + 1024) + c + (c == own ? 0x8000 : 0)) << (16 * half);
        }
      }
    }
  }
  const long long start = a.cur.f[w];
  // every move lowers f, which is at most n (n - 1) / 2 unless the caller's edge count is off by more
  const int move_budget = static_cast<int>(min(start, 0x7fffffffll));
  int gained = 0;
  int applied = 0;
  int from = 0, to = 0;
  int mine = -1;          // the moved vertex's pair among this thread's
  uint32_t bias = 0u;     // the own-cluster bias in the moved vertex's half
  const int shift = 2 * (tid & 15);
  const uint32_t* row = nullptr;

  while (true) {
    if (row != nullptr) {  // fold the last move into the lanes
      uint32_t rw[P];
#pragma unroll
      for (int p = 0; p < P; ++p) rw[p] = 2 * (tid + p * T) < n ? row[(tid + p * T) >> 4] : 0u;
      int coef[K];
#pragma unroll
      for (int c = 0; c < K; ++c) coef[c] = (c == from ? 1 : 0) - (c == to ? 1 : 0);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const uint32_t y = rw[p] >> shift;
        const uint32_t bits = (y & 1u) | ((y << 15) & 0x10000u);
        const int d = static_cast<int>(bits * 16u - down[p] - (mine == p ? bias : 0u));
#pragma unroll
        for (int c = 0; c < K; ++c) key[p][c] += static_cast<uint32_t>(coef[c] * d);
      }
    }
    uint32_t best = ~0u;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      uint32_t lo = key[p][0], hi = key[p][0];
#pragma unroll
      for (int c = 1; c < K; ++c) {
        lo = __vminu2(lo, key[p][c]);
        hi = __vmaxu2(hi, key[p][c]);
      }
      const uint32_t x = (lo & ~kClusterBits) - (hi & ~kClusterBits) + 0xC000C000u;
      const uint32_t low = code[p] | (lo & kClusterBits) | ((hi << 3) & (kClusterBits << 3));
      best = min(best, min(__byte_perm(low, x, 0x5410), __byte_perm(low, x, 0x7632)));
    }
    // the block's best key: each warp's to shared memory (double-buffered), one barrier
    best = WarpMin(best);
    if constexpr (kWarps > 1) {
      uint32_t* rec = s_records + (applied & 1) * kWarps;
      if (lane == 0) rec[tid / kWarp] = best;
      __syncthreads();
      if constexpr (kWarps == 2) {
        const uint2 r = *reinterpret_cast<const uint2*>(rec);
        best = min(r.x, r.y);
      } else if constexpr (kWarps == 4) {
        const uint4 r = *reinterpret_cast<const uint4*>(rec);
        best = min(min(r.x, r.y), min(r.z, r.w));
      } else {
        best = WarpMin(lane < kWarps ? rec[lane] : ~0u);
      }
    }
    if (best >= (16384u - 8u) << 16) break;  // gain >= 0
    const int v = static_cast<int>((best >> 6) & 1023u);
    from = static_cast<int>((best >> 3) & 7u);
    to = static_cast<int>(best & 7u);
    row = rows + v * a.gr.pitch;
    const int q = v >> 1;
    mine = q % T == tid ? q / T : -1;
    bias = 0x8000u << (16 * (v & 1));
    gained += (static_cast<int>(best >> 16) - 16384) / 8 + 1;
    if (++applied > move_budget) {
      if (tid == 0) atomicExch(&a.ctl->error, kErrorMoveBound);
      break;
    }
  }

  uint8_t* dst = a.next.labels + static_cast<size_t>(slot) * ld;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    uint32_t hi = key[p][0];
#pragma unroll
    for (int c = 1; c < K; ++c) hi = __vmaxu2(hi, key[p][c]);
    const int u = 2 * (tid + p * T);
    if (u < n) dst[u] = static_cast<uint8_t>(hi & 7u);
    if (u + 1 < n) dst[u + 1] = static_cast<uint8_t>((hi >> 16) & 7u);
  }
  if (tid == 0) {
    a.next.f[slot] = start + gained;
    if (applied) atomicAdd(&a.ctl->moves, static_cast<unsigned long long>(applied));
  }
}

template <int K, int T, int V, bool kSmemRows>
__device__ __forceinline__ void DescentRegisters(const DescentArgs<int16_t>& a, int slot) {
  constexpr int kWarps = T / kWarp;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_winner;
  __shared__ int s_stop;
  __shared__ __align__(16) MoveRecord<uint32_t> s_records[2 * kWarps];

  const int tid = threadIdx.x;
  const int lane = tid % kWarp;
  const int n = a.gr.n;
  const int ld = a.ld;
  const int bits = a.key_bits;

  if (tid == 0) {
    s_stop = a.ctl->stop;
    if (!s_stop) {
      const int64_t* f = a.cur.f;
      s_winner = a.tournament > 0 ? TournamentWinner(a.select_stream, slot, a.iteration, a.population, a.tournament,
                                                     [f](int i) { return f[i]; })
                                  : slot;
    }
  }
  const uint32_t* rows = a.gr.bits;
  if constexpr (kSmemRows) {
    const size_t row_words = static_cast<size_t>(n) * a.gr.pitch;
    const uint4* src = reinterpret_cast<const uint4*>(a.gr.bits);
    uint4* dst = reinterpret_cast<uint4*>(smem);
    for (size_t i = tid; i < row_words / 4; i += T) dst[i] = __ldg(src + i);
    rows = reinterpret_cast<const uint32_t*>(smem);
  }
  __syncthreads();
  if (s_stop) return;
  const int w = s_winner;
  if constexpr (T * V <= 1024) {
    if (a.key_bits <= kCompactMaxBits) {
      DescentRegistersCompact<K, T, V>(a, slot, w, rows, reinterpret_cast<uint32_t*>(s_records));
      return;
    }
  }

  int key[V][K];
  int ucode[V];  // (2^B << B) | u: adding gain << B gives the block-wide move key
  unsigned valid = 0;
  {
    const int16_t* g_src = a.cur.g + static_cast<size_t>(w) * K * ld;
    const uint8_t* l_src = a.cur.labels + static_cast<size_t>(w) * ld;
    const int32_t* sizes = a.cur.sizes + static_cast<size_t>(w) * a.kpad;
    int s16[K];
#pragma unroll
    for (int c = 0; c < K; ++c) s16[c] = 16 * sizes[c] + c;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int u = tid + j * T;
      const bool ok = u < n;
      valid |= ok ? (1u << j) : 0u;
      const int own = ok ? l_src[u] : 0;
#pragma unroll
      for (int c = 0; c < K; ++c) {
        const int gc = ok ? g_src[static_cast<size_t>(c) * ld + u] : 0;
        key[j][c] = s16[c] - 32 * gc + (c == own ? kRegPenalty : 0);
      }
      ucode[j] = ok ? (((1 << bits) << bits) | u) : (1 << 30);
    }
  }
  long long objective = a.cur.f[w];
  const long long move_budget = objective;

  unsigned long long applied = 0;
  int parity = 0;
  bool pending = false;  // a move still to be folded into the keys
  int coef[K];           // [c = from] - [c = to] of that move
#pragma unroll
  for (int c = 0; c < K; ++c) coef[c] = 0;
  const uint32_t* prev_row = rows;
  const uint32_t lane_bit = 1u << lane;
  const uint32_t no_move = (1u << bits) << bits;

  while (true) {
    uint32_t rw[V];
#pragma unroll
    for (int j = 0; j < V; ++j) rw[j] = (pending && ((valid >> j) & 1)) ? prev_row[(tid + j * T) >> 5] : 0u;
    uint32_t best = KeyTraits<uint32_t>::kNone;
    uint32_t payload = 0;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int d = (rw[j] & lane_bit) ? 16 : -16;
#pragma unroll
      for (int c = 0; c < K; ++c) key[j][c] += coef[c] * d;
      int kmin, kmax;
      LanesMinMax<K>(key[j], kmin, kmax);
      const int gain = (kmin >> 4) - (kmax >> 4) + (kRegPenalty >> 4) + 1;
      // (gain + 2^B) << B | u for every vertex: improving moves sort below 2^(2B), the rest above it
      // (gain <= n - 1), and absent vertices carry 2^31 in ucode.
      const uint32_t mk = static_cast<uint32_t>(gain * (1 << bits)) + static_cast<uint32_t>(ucode[j]);
      if (mk < best) {
        best = mk;
        payload = static_cast<uint32_t>(kmax & 15) | (static_cast<uint32_t>(kmin & 15) << 8);
      }
    }
    const MoveRecord<uint32_t> m = BlockArgMin<uint32_t, kWarps>(best, payload, s_records + parity * kWarps);
    if (m.key >= no_move) break;
    parity ^= 1;

    const int v = MoveVertex(m.key, bits);
    const int from = static_cast<int>(m.payload & 0xff);
    const int to = static_cast<int>(m.payload >> 8);
#pragma unroll
    for (int c = 0; c < K; ++c) coef[c] = (c == from ? 1 : 0) - (c == to ? 1 : 0);
    if (v % T == tid) {
      const int jv = v / T;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        if (j == jv) {
#pragma unroll
          for (int c = 0; c < K; ++c) key[j][c] -= coef[c] * kRegPenalty;
        }
      }
    }
    prev_row = rows + static_cast<size_t>(v) * a.gr.pitch;
    pending = true;
    objective += MoveDelta(m.key, bits);
    ++applied;
    if (static_cast<long long>(applied) > move_budget) {
      if (tid == 0) atomicExch(&a.ctl->error, kErrorMoveBound);
      break;
    }
  }

  uint8_t* dst = a.next.labels + static_cast<size_t>(slot) * ld;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    if ((valid >> j) & 1) {
      int kmin, kmax;
      LanesMinMax<K>(key[j], kmin, kmax);
      dst[tid + j * T] = static_cast<uint8_t>(kmax & 15);
    }
  }
  if (tid == 0) {
    a.next.f[slot] = objective;
    if (applied) atomicAdd(&a.ctl->moves, applied);
  }
}

// One slot per block (plain path).
template <int K, int T, int V, bool kSmemRows>
__global__ void __launch_bounds__(T, 1) k_descent_registers(DescentArgs<int16_t> a) {
  DescentRegisters<K, T, V, kSmemRows>(a, blockIdx.x);
}

}  // namespace ccb
