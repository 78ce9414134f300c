// Steepest descent over a window of moves: exact, with the full scan of the vertices done once per window instead
// of once per move.  Same trajectory as k_descent and the reference's BestMove/ApplyMove
// (src/cc_pbils_cpu.cpp:99-139).
//
// A move (v: from -> to) changes h_c(u) = size_c - 2 G_c(u) of any vertex u by exactly 1 (up or down) for
// c = from and c = to and leaves every other h_c alone.  So the gain of u, min over c != a of h_c - h_a + 1,
// falls by at most m_a + max m_c after a run of moves, with m_c the number of those moves that had c as source or
// target; D, the sum of the two largest m_c, bounds it for every vertex.  A window therefore
//   1. refreshes all vertices: applies the last window's moves to the counters G, recomputes every gain and picks
//      the threshold theta such that at most kCap vertices have a gain below it: the members S;
//   2. makes moves looking at S alone, as long as the best member's gain is below theta - D: every other vertex
//      has a gain of at least theta - D, so the best member is the best vertex (members are kept in vertex order:
//      ties go to the lower vertex as in a full scan).
// When the bound no longer decides, the next window starts.  A window makes at least one move.
//
// The refresh reads each vertex's adjacency to the window's moved vertices as a bit vector x over the moves: a
// warp's lanes load the moved vertices' rows (16 bytes, 128 vertices) and transpose them in registers
// (WarpTranspose32).  With F and T the masks of the moves leaving and entering c, the counter changes by
// popc(x & T) - popc(x & F) = popc((x ^ F) & (F | T)) - popc(F).
//
// Up to n = 16383 (kHalf) the slot's array holds h_c(u) itself in 16 bits, biased by 2^14, with the top bit set in u's own
// cluster: a pair of vertices then takes one multiply-add to update, one 16-bit pair minimum (the best foreign h) and one
// maximum (the own) per cluster, and no label is read.  Above, where h needs 17 bits, it holds the counters G_c(u).
//
// If more than kWindowCap vertices share the best gain g, the members are the kWindowCap lowest of them and theta is g + 1.
// The rest of them keep a gain of at least g - D = theta - 1 - D, and a member that reaches it is the lower vertex; every
// other vertex stays at theta - D or above.  So the same test decides, and noise-free communities, whose vertices all tie
// and whose gains fall by two with every move, get whole windows (with one move a window n = 16000, k = 3 took 8.3 us a
// move, now 0.64; the kernel without windows 4.1).
//
// What bounds it (B200, G(n, p), clocks per move of a slot at 1.965 GHz): the members' moves, about 835 at K = 3 and
// 1060 at K = 8, are issue of 32-bit integer instructions (two warps per scheduler, two clocks each) plus 360 for the
// row of the moved vertex from L2; four members on 256 threads measured best (K = 3: 2 x 512 threads 840 against 785,
// 8 x 128 900; S of 512 or 2048 gives the refresh or the scan more than it takes from the other).  The refresh is one
// pass over all vertices per window of 25 to 35 moves: n = 16000, k = 3 505 a move (620 with counters, keys and labels
// instead of h), n = 32000, k = 8 with its counters in L2 2280 (issue 54 %, L2 3.1 TB/s); the choice of S 75 to 270.  A
// descent of 128 slots with one scan of every vertex per move took, us per move: n = 16000, k = 3: 4.5, now 0.85; n =
// 32000, k = 8: 13.3, now 2.5; n = 9001, k = 24: 11.9, now 2.6.
//
// 512 threads leave 128 registers each and an SM to one slot.  The forms of 16 and 32 keys with their array in global memory
// and the wide form of 4 clusters spill 8 to 72 bytes a thread; the others take 105 to 128 registers and spill nothing.
#pragma once

#include <cstdint>
#include <type_traits>

#include "ccb_descent_incremental.cuh"
#include "ccb_device.cuh"

namespace ccb {

constexpr int kWindowHalfMax = 16383;  // largest n whose h fit 15 bits
constexpr int kWindowMoves = 64;   // most moves of a window (two 32-bit vectors)
constexpr int kWindowBins = 128;   // gains above the lower bound that a threshold can take
constexpr int kWindowThreads = 512;
constexpr int kWindowCap = 1024;         // most members of a window (k <= 8 also runs with more)
constexpr int kWindowPenalty = 1 << 26;  // own-cluster bias of a member's keys (2^20 in units of h)
constexpr int kWindowAbsent = 1 << 25;   // key of a cluster past k: above every foreign key, below every own one

// How the members' moves are made for a cluster bound: with all K keys of a member in registers (`keys` of them, k
// padded to it), or (keys = 0) with its counters in shared memory and its best key cached; and by how many threads,
// for at most `cap` members.
struct WindowForm {
  int keys, threads;
};
__host__ __device__ constexpr WindowForm WindowFormOf(int k, int cap) {
  return k <= 8    ? WindowForm{k, cap > kWindowCap ? 512 : 256}
         : k <= 16 ? WindowForm{16, 256}
         : k <= 32 ? WindowForm{32, 512}
                   : WindowForm{0, 512};
}

// The bound of a cluster count that an instance is compiled for: k itself up to 8, then 16, 32, 64.
__host__ __device__ constexpr int WindowBound(int k) { return k <= 8 ? k : k <= 16 ? 16 : k <= 32 ? 32 : 64; }

// 32 x 32 bit transpose across a warp: lane j holds row j, lane l gets column l (bit j = row j's bit l).
struct WarpTranspose32 {
  uint32_t sel16, sel8, keep4, keep2, keep1;
  int rot4, rot2, rot1;
  __device__ __forceinline__ explicit WarpTranspose32(int lane) {
    sel16 = (lane & 16) ? 0x3276u : 0x5410u;
    sel8 = (lane & 8) ? 0x3715u : 0x6240u;
    keep4 = (lane & 4) ? 0xf0f0f0f0u : 0x0f0f0f0fu;
    keep2 = (lane & 2) ? 0xccccccccu : 0x33333333u;
    keep1 = (lane & 1) ? 0xaaaaaaaau : 0x55555555u;
    rot4 = (lane & 4) ? 28 : 4;
    rot2 = (lane & 2) ? 30 : 2;
    rot1 = (lane & 1) ? 31 : 1;
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(kAllLanes, x, 16), sel16);
    x = __byte_perm(x, __shfl_xor_sync(kAllLanes, x, 8), sel8);
    uint32_t y = __shfl_xor_sync(kAllLanes, x, 4);
    x = (x & keep4) | (__funnelshift_l(y, y, rot4) & ~keep4);
    y = __shfl_xor_sync(kAllLanes, x, 2);
    x = (x & keep2) | (__funnelshift_l(y, y, rot2) & ~keep2);
    y = __shfl_xor_sync(kAllLanes, x, 1);
    return (x & keep1) | (__funnelshift_l(y, y, rot1) & ~keep1);
  }
};

// Leading dimension of the window's counters: whole quads of row words, 128 vertices each.
__host__ __device__ constexpr int WindowLd(int n) { return (n + 127) / 128 * 128; }

// Place of vertex u in the window's counters and distances: a quad's 128 vertices are stored lane-major, so that the
// lane that holds vertices l, 32 + l, 64 + l and 96 + l after the transposes reads and writes them as one 8-byte word.
__device__ __forceinline__ int WindowPlace(int u) { return (u & ~127) | ((u & 31) << 2) | ((u >> 5) & 3); }

// Dynamic shared memory: distances (16 bits a vertex), the counters when they fit, and where the moves need them the
// members' counters (leading dimension cap + 2: a column's entries fall into different banks) and cached keys.
__host__ __device__ constexpr size_t WindowSmem(int n, int k, bool counters, int cap) {
  return static_cast<size_t>(WindowLd(n)) * 2 * (1 + (counters ? k : 0)) +
         (k > 32 ? static_cast<size_t>(k) * (cap + 2) * 2 + static_cast<size_t>(cap) * 12 : 0);
}

// The barrier of the first kThreads threads.
template <int kThreads>
__device__ __forceinline__ void WindowScanBarrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
}

// State of a block's windows in shared memory.
template <int kCap>
struct WindowShared {
  uint4 mask[kMaxK][2];      // per cluster and 32 moves: F | T, F, popc(F), (first entry) 64 size + c
  int off[kMaxK];            // 64 size_c + c
  int hist[kWindowBins];
  int warp_count[kWindowThreads / kWarp];
  int member[kCap];          // vertices of S, ascending except at k <= 8
  int move_v[kWindowMoves];
  int move_ft[kWindowMoves];  // from | to << 8
  uint32_t record[2][kWindowThreads / kWarp];  // each scan warp's best move key
  int winner, stop;
  int moves;      // of the last window
  int low;        // lower bound L of every gain
  int smallest;   // smallest gain of the refresh
  int members;    // |S|
  int bins;       // theta - L
  int partial;    // 1 when S holds only part of the vertices of the best gain
  int finished;
};

// What a window's moves add up to, kept by every scan warp: lane l holds m_c of clusters l and l + 32.
struct WindowBook {
  int count0 = 0, count1 = 0;
  int top1 = 0, top2 = 0;  // the two largest m_c
  int moves = 0;
  __device__ __forceinline__ static void Grow(int before, int& top1, int& top2) {
    const int first = before == top1 ? 1 : 0;
    top2 += before == top2 ? 1 - first : 0;
    top1 += first;
  }
  template <bool kWide>  // more than 32 clusters
  __device__ __forceinline__ void Add(int from, int to) {
    const int lane = threadIdx.x % kWarp;
    const int nf = __shfl_sync(kAllLanes, kWide && from >= kWarp ? count1 : count0, from & 31);
    const int nt = __shfl_sync(kAllLanes, kWide && to >= kWarp ? count1 : count0, to & 31);
    Grow(nf, top1, top2);
    Grow(nt, top1, top2);
    count0 += (lane == from ? 1 : 0) + (lane == to ? 1 : 0);
    if (kWide) count1 += (lane + kWarp == from ? 1 : 0) + (lane + kWarp == to ? 1 : 0);
    ++moves;
  }
  // The window's end, by one thread: `gain` is the best member's.
  template <int kCap>
  __device__ __forceinline__ void Close(WindowShared<kCap>& s, int theta, int gain) const {
    const int bound = theta - s.partial - top1 - top2;  // partial: vertices outside S started at the best gain itself
    s.moves = moves;
    s.finished = gain >= 0 && bound >= 0;
    s.low = min(gain, bound);
  }
};

// Calls f with the compile-time value of c, 0 <= c < kEnd (c the same in the whole block): a tree of branches.
template <int kBegin, int kEnd, typename F>
__device__ __forceinline__ void WithCluster(int c, F&& f) {
  if constexpr (kEnd - kBegin == 1) {
    f(std::integral_constant<int, kBegin>());
  } else {
    constexpr int kMid = (kBegin + kEnd) / 2;
    if (c < kMid) {
      WithCluster<kBegin, kMid>(c, f);
    } else {
      WithCluster<kMid, kEnd>(c, f);
    }
  }
}

// The moves of one window with a member's K keys 64 h_c + c in registers (k <= K clusters; the own key biased by
// kWindowPenalty, so that the minimum of the keys is the best foreign target and the maximum the own cluster), V
// members per thread.  Move keys are field << kField | id << 2 kC | from << kC | to with field = gain - L + kBias,
// clamped, and id the vertex (K <= 8, n <= 65536: the row address comes from the key itself) or the member.  Leaves in s the moves, the new lower bound and whether no vertex can improve.
template <int K, int V, int T, int kCap, bool kHalf>
__device__ __forceinline__ void WindowMovesK(const GraphView& gr, int k, const uint16_t* g, int ldw, uint8_t* lab,
                                             WindowShared<kCap>& s, long long& objective) {
  constexpr int kC = K <= 8 ? 3 : 5;  // bits of a cluster in a move key
  constexpr bool kByVertex = K <= 8;
  constexpr int kIdBits = kByVertex ? 16 : 11;
  constexpr uint32_t kIdMask = ((1u << kIdBits) - 1u) << (2 * kC);
  constexpr int kField = 2 * kC + kIdBits;
  constexpr uint32_t kFieldMax = (1u << ((kByVertex ? 32 : 31) - kField)) - 1u;
  constexpr int kBias = 256;
  constexpr int kClusterMask = (1 << kC) - 1;
  constexpr int kWarps = T / kWarp;
  const int tid = threadIdx.x;
  const int lane = tid % kWarp;
  const int warp = tid / kWarp;
  const int count = s.members;
  const int low = s.low;
  const int theta = low + s.bins;
  int key[V][K];
  int su[V];
  uint32_t code[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = j * T + tid;
    const bool ok = i < count;
    su[j] = s.member[ok ? i : 0];
    code[j] = ok ? static_cast<uint32_t>(kByVertex ? su[j] : i) << (2 * kC) : ~0u;
    const int own = kHalf ? 0 : lab[su[j]];
    const uint16_t* gu = g + WindowPlace(su[j]);
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (kHalf && (K <= 8 || c < k)) {  // h + 2^14 in every key: the gains are the same
        const int x = gu[static_cast<size_t>(c) * ldw];
        key[j][c] = 64 * (x & 0x7fff) + c + (x >= 0x8000 ? kWindowPenalty : 0);
      } else if (K <= 8 || c < k) {
        key[j][c] = s.off[c] - 128 * static_cast<int>(gu[static_cast<size_t>(c) * ldw]) + (c == own ? kWindowPenalty : 0);
      } else {
        key[j][c] = kWindowAbsent;
      }
    }
  }
  const int gain_base = (kWindowPenalty >> 6) + 1 - low + kBias;
  int from = 0, to = 0;
  int coef[K <= 8 ? K : 1];
  int mine = -1;  // the moved vertex's place among this thread's members
  uint32_t rw[V];
  WindowBook book;
  uint32_t best;
  while (true) {
    if (book.moves > 0) {  // the last move: keys of `from` and `to`
      int d[V];
#pragma unroll
      for (int j = 0; j < V; ++j) {  // the moved vertex's bias goes from lane `from` to lane `to`
        d[j] = static_cast<int>((rw[j] >> (su[j] & 31)) & 1u) * 128 - (mine == j ? 64 + kWindowPenalty : 64);
      }
      if constexpr (K <= 8) {
#pragma unroll
        for (int c = 0; c < K; ++c) {
#pragma unroll
          for (int j = 0; j < V; ++j) key[j][c] += coef[c] * d[j];
        }
      } else {
        WithCluster<0, K>(from, [&](auto c) {
#pragma unroll
          for (int j = 0; j < V; ++j) key[j][c.value] += d[j];
        });
        WithCluster<0, K>(to, [&](auto c) {
#pragma unroll
          for (int j = 0; j < V; ++j) key[j][c.value] -= d[j];
        });
      }
    }
    best = ~0u;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      int lo = key[j][0], hi = key[j][0];
      int c = 1;
#pragma unroll
      for (; c + 1 < K; c += 2) {
        lo = __vimin3_s32(lo, key[j][c], key[j][c + 1]);
        hi = __vimax3_s32(hi, key[j][c], key[j][c + 1]);
      }
      if (c < K) {
        lo = min(lo, key[j][c]);
        hi = max(hi, key[j][c]);
      }
      const int field = (lo >> 6) - (hi >> 6) + gain_base;
      const uint32_t mk = (min(static_cast<uint32_t>(field), kFieldMax) << kField) | code[j] |
                          static_cast<uint32_t>((hi & kClusterMask) << kC) | static_cast<uint32_t>(lo & kClusterMask);
      best = min(best, mk);
    }
    uint32_t* rec = s.record[book.moves & 1];
    best = WarpMin(best);
    if (lane == 0) rec[warp] = best;
    WindowScanBarrier<T>();
    best = WarpMin(lane < kWarps ? rec[lane] : ~0u);
    const int gain = static_cast<int>(best >> kField) - kBias + low;
    // below theta - D the best member is the best vertex; a gain of 0 or more is no move
    if (book.moves >= kWindowMoves || gain >= min(theta - book.top1 - book.top2, 0) || (best >> kField) >= kFieldMax) break;
    const int id = static_cast<int>((best & kIdMask) >> (2 * kC));
    const int v = kByVertex ? id : s.member[id];
    const uint32_t* row = gr.bits + static_cast<size_t>(v) * gr.pitch;
#pragma unroll
    for (int j = 0; j < V; ++j) rw[j] = row[su[j] >> 5];
    from = static_cast<int>((best >> kC) & kClusterMask);
    to = static_cast<int>(best & kClusterMask);
    if constexpr (K <= 8) {
#pragma unroll
      for (int c = 0; c < K; ++c) coef[c] = (c == from ? 1 : 0) - (c == to ? 1 : 0);
    }
    objective += gain;
    if constexpr (kByVertex) {
      mine = -1;
#pragma unroll
      for (int j = 0; j < V; ++j) mine = code[j] == (best & kIdMask) ? j : mine;
    } else {
      mine = id % T == tid ? id / T : -1;
    }
    if (mine >= 0) {
      lab[v] = static_cast<uint8_t>(to);
      s.move_v[book.moves] = v;
      s.move_ft[book.moves] = from | to << 8;
    }
    book.Add<false>(from, to);
  }
  if (tid == 0) book.Close(s, theta, static_cast<int>(best >> kField) - kBias + low);
}

// A member's counters and cached keys in shared memory (runtime k).
template <int kCap>
struct WindowMembers {
  static constexpr int kLd = kCap + 2;
  uint16_t* g;  // [k][kLd]
  int* best;    // smallest key over the non-empty foreign clusters
  int* bound;   // and the second smallest
  int* own;     // the own cluster's key
  __device__ void Carve(unsigned char* p, int k) {
    g = reinterpret_cast<uint16_t*>(p);
    best = reinterpret_cast<int*>(p + static_cast<size_t>(k) * kLd * 2);
    bound = best + kCap;
    own = bound + kCap;
  }
  // All threads: the members' counters from g, their keys with them.
  template <int kThreads, bool kHalf>
  __device__ __forceinline__ void Fill(const uint16_t* counters, int ldw, const uint8_t* lab, const int* member,
                                       int count, const int* off, int k) {
    for (int i = threadIdx.x; i < count; i += kThreads) {
      const int u = member[i];
      const int at = WindowPlace(u);
      const int o = lab[u];
      int b1 = 0x7fffffff, b2 = 0x7fffffff, ko = 0;
#pragma unroll 16
      for (int c = 0; c < k; ++c) {
        int x = counters[static_cast<size_t>(c) * ldw + at];
        const int offc = off[c];
        if constexpr (kHalf) x = ((offc >> 6) - (x & 0x7fff) + 0x4000) >> 1;  // G = (size - h) / 2
        g[c * kLd + i] = static_cast<uint16_t>(x);
        const int key = offc - 128 * x;
        if (c == o) {
          ko = key;
        } else if (offc >= 64) {
          b2 = min(b2, max(b1, key));
          b1 = min(b1, key);
        }
      }
      best[i] = b1;
      bound[i] = b2;
      own[i] = ko;
    }
  }
};

// Folds a move (from -> to) into a member's cached keys, given its new keys kf = key_from and kt = key_to: kb the
// smallest key over the non-empty foreign clusters as far as it is known (INT_MAX: not), lb a lower bound on the keys
// of every other non-empty foreign cluster, ko the own cluster's key (label = ko & 63).  kb <= lb means that kb is
// the best; otherwise lb bounds it.
__device__ __forceinline__ void WindowFold(bool moved, int kf, int kt, int from, int to, bool from_empty, int& kb,
                                           int& lb, int& ko) {
  constexpr int kNone = 0x7fffffff;
  const int own = ko & 63;
  const bool of = own == from, ot = own == to;
  const int b = kb & 63;
  const int rest = (b == from || b == to) ? kNone : kb;  // the cached best, where the move left it alone
  if (moved) {  // `to` is its own cluster now, `from` a foreign one
    ko = kt;
    lb = min(lb, min(rest, from_empty ? kNone : kf));
    kb = kNone;
    return;
  }
  ko = of ? kf : (ot ? kt : ko);
  const int cf = (of || from_empty) ? kNone : kf;
  const int ct = ot ? kNone : kt;
  const int lo = min(cf, ct), hi = max(cf, ct);
  kb = min(rest, lo);
  lb = min(lb, min(max(rest, lo), hi));
}

// Smallest and second smallest key over the non-empty clusters c != own of member i, by the whole warp: lane l holds
// off of clusters l and l + 32 (INT_MAX past k) and reads their counters.
__device__ __forceinline__ int2 WindowRescan(const uint16_t* g, int ld, int i, int off0, int off1, int k, int own) {
  constexpr int kNone = 0x7fffffff;
  const int lane = threadIdx.x % kWarp;
  int k1 = kNone, k2 = kNone;
  if (lane < k && lane != own && off0 >= 64) k1 = off0 - 128 * static_cast<int>(g[lane * ld + i]);
  if (lane + kWarp < k && lane + kWarp != own && off1 >= 64) {
    k2 = off1 - 128 * static_cast<int>(g[(lane + kWarp) * ld + i]);
  }
  const int lo = min(k1, k2);
  const int b1 = __reduce_min_sync(kAllLanes, lo);
  const int b2 = __reduce_min_sync(kAllLanes, lo == b1 ? max(k1, k2) : lo);
  return make_int2(b1, b2);
}

// The moves of one window at 32 < k <= 64: the members' counters in shared memory, their cached keys (WindowFold) in
// registers.  A member whose best is only bounded takes part with its bound; it is rescanned by its warp when the
// bound comes near the best key of the block.  Move keys are field << 23 | member << 12 | from << 6 | to with field =
// gain - L + 128, clamped; to = from marks a bound.
template <int V, int T, int kCap>
__device__ __forceinline__ void WindowMovesN(const GraphView& gr, int k, const WindowMembers<kCap>& mem, uint8_t* lab,
                                             WindowShared<kCap>& s, long long& objective) {
  constexpr uint32_t kFieldMax = 511u;
  constexpr int kBias = 128;
  constexpr int kWarps = T / kWarp;
  constexpr int kLd = WindowMembers<kCap>::kLd;
  const int tid = threadIdx.x;
  const int lane = tid % kWarp;
  const int warp = tid / kWarp;
  const int count = s.members;
  const int low = s.low;
  const int theta = low + s.bins;
  // lane l: 64 size + c of clusters l and l + 32
  int off0 = lane < k ? s.off[lane] : 0x3fffffff;
  int off1 = lane + kWarp < k ? s.off[lane + kWarp] : 0x3fffffff;
  int kb[V], lb[V], ko[V], su[V];
  uint32_t code[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = j * T + tid;
    const bool ok = i < count;
    su[j] = s.member[ok ? i : 0];
    code[j] = ok ? static_cast<uint32_t>(i) << 12 : ~0u;
    kb[j] = ok ? mem.best[i] : 0;
    lb[j] = ok ? mem.bound[i] : 0x7fffffff;
    ko[j] = ok ? mem.own[i] : 0;
  }
  auto lowest_empty = [&]() {  // its key is its index for every vertex
    const unsigned lo = __ballot_sync(kAllLanes, off0 == lane);
    const unsigned hi = __ballot_sync(kAllLanes, off1 == lane + kWarp);
    return lo ? __ffs(lo) - 1 : (hi ? 31 + __ffs(hi) : 0x7fffffff);
  };
  int empty_key = lowest_empty();
  int from = 0, to = 0, moved = -1;
  int offf = 0, offt = 0;
  bool fold = false;
  uint32_t near = 0;  // bounds below it are made exact at once
  uint32_t rw[V];
#pragma unroll
  for (int j = 0; j < V; ++j) rw[j] = 0u;
  WindowBook book;
  uint32_t best;
  for (int round = 0;; ++round) {  // one per move, and one more for each best key that was not exact
    if (fold) {
      const bool from_empty = offf == from;
      const uint16_t* gf_row = mem.g + from * kLd;
      const uint16_t* gt_row = mem.g + to * kLd;
      int gf[V], gt[V];
#pragma unroll
      for (int j = 0; j < V; ++j) {
        gf[j] = gf_row[j * T + tid];
        gt[j] = gt_row[j * T + tid];
      }
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const int i = j * T + tid;
        if (i >= count) continue;
        if ((rw[j] >> (su[j] & 31)) & 1u) {
          mem.g[from * kLd + i] = static_cast<uint16_t>(--gf[j]);
          mem.g[to * kLd + i] = static_cast<uint16_t>(++gt[j]);
        }
        WindowFold(i == moved, offf - 128 * gf[j], offt - 128 * gt[j], from, to, from_empty, kb[j], lb[j], ko[j]);
      }
      __syncwarp();  // every lane's counters are visible to the warp's rescans
    }
    best = ~0u;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int i = j * T + tid;
      auto move_key = [&]() {
        const int known = min(kb[j], empty_key);
        const bool sure = known <= lb[j];
        const int kbest = sure ? known : lb[j];
        const int field = (kbest >> 6) - (ko[j] >> 6) + 1 - low + kBias;
        return (min(static_cast<uint32_t>(field), kFieldMax) << 23) | code[j] |
               static_cast<uint32_t>((ko[j] & 63) << 6) | static_cast<uint32_t>((sure ? known : ko[j]) & 63);
      };
      uint32_t mk = move_key();
      unsigned m = __ballot_sync(kAllLanes, ((mk >> 6) & 63u) == (mk & 63u) && mk < near);
      if (m) {
        do {
          const int l = __ffs(m) - 1;
          m &= m - 1;
          const int own_l = __shfl_sync(kAllLanes, ko[j] & 63, l);
          const int2 r = WindowRescan(mem.g, kLd, i - lane + l, off0, off1, k, own_l);
          if (lane == l) {
            kb[j] = r.x;
            lb[j] = r.y;
          }
        } while (m);
        mk = move_key();
      }
      best = min(best, mk);
    }
    uint32_t* rec = s.record[round & 1];
    best = WarpMin(best);
    if (lane == 0) rec[warp] = best;
    WindowScanBarrier<T>();
    best = WarpMin(lane < kWarps ? rec[lane] : ~0u);
    const int gain = static_cast<int>(best >> 23) - kBias + low;
    if (book.moves >= kWindowMoves || gain >= min(theta - book.top1 - book.top2, 0) || (best >> 23) >= kFieldMax) break;
    from = static_cast<int>((best >> 6) & 63u);
    to = static_cast<int>(best & 63u);
    near = (best & ~0x7fffffu) + (3u << 23);
    fold = from != to;
    if (!fold) continue;  // the best key is a bound: made exact in the next round
    moved = static_cast<int>((best >> 12) & 2047u);
    const int v = s.member[moved];
    const uint32_t* row = gr.bits + static_cast<size_t>(v) * gr.pitch;
#pragma unroll
    for (int j = 0; j < V; ++j) rw[j] = row[su[j] >> 5];
    objective += gain;
    if (moved % T == tid) {
      lab[v] = static_cast<uint8_t>(to);
      s.move_v[book.moves] = v;
      s.move_ft[book.moves] = from | to << 8;
    }
    book.Add<true>(from, to);
    const int f0 = lane == from, f1 = lane + kWarp == from, t0 = lane == to, t1 = lane + kWarp == to;
    off0 += 64 * (t0 - f0);
    off1 += 64 * (t1 - f1);
    offf = __shfl_sync(kAllLanes, from < kWarp ? off0 : off1, from & 31);
    offt = __shfl_sync(kAllLanes, to < kWarp ? off0 : off1, to & 31);
    empty_key = lowest_empty();
  }
  if (tid == 0) book.Close(s, theta, static_cast<int>(best >> 23) - kBias + low);
}

// One slot's descent.  K: the cluster count at compile time (2 .. 8), or the bound of a runtime one (16, 32, 64) that
// picks how the moves are made.  kHalf: n <= 16383 (see above).  kSmemG: the counters in shared memory, else
// in the slot's rows of `next` (leading dimension WindowLd(n) either way).  GainT: the population's G.
template <int kBound, int kCap, bool kSmemG, bool kHalf, typename GainT>
__device__ __forceinline__ void DescentWindow(const DescentArgs<GainT>& a, int slot) {
  constexpr int K = kBound <= 8 ? kBound : 0;
  constexpr int T = kWindowThreads;
  constexpr int kWarps = T / kWarp;
  constexpr WindowForm kForm = WindowFormOf(kBound, kCap);
  constexpr int V = kCap / kForm.threads;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ WindowShared<kCap> s;

  const int tid = threadIdx.x;
  const int lane = tid % kWarp;
  const int warp = tid / kWarp;
  const int n = a.gr.n;
  const int k = K > 0 ? K : a.k;
  const int ld = a.ld;
  const int ldw = WindowLd(n);
  const int quads = ldw / 128;
  const int pitch = a.gr.pitch;

  if (tid == 0) {
    s.stop = a.ctl->stop;
    if (!s.stop) {
      const int64_t* f = a.cur.f;
      s.winner = a.tournament > 0 ? TournamentWinner(a.select_stream, slot, a.iteration, a.population, a.tournament,
                                                     [f](int i) { return f[i]; })
                                  : slot;
      s.moves = 0;
      s.low = 1 - n;
      s.finished = 0;
      s.smallest = 0x7fffffff;
    }
  }
  __syncthreads();
  if (s.stop) return;
  const int w = s.winner;

  uint16_t* dist = reinterpret_cast<uint16_t*>(smem);  // gain - L of every vertex, clamped
  uint16_t* g = kSmemG ? dist + ldw
                       : reinterpret_cast<uint16_t*>(a.next.g) + static_cast<size_t>(slot) * k * ldw;
  uint8_t* lab = a.next.labels + static_cast<size_t>(slot) * ld;
  [[maybe_unused]] WindowMembers<kCap> members;
  if constexpr (kForm.keys == 0) members.Carve(smem + static_cast<size_t>(ldw) * 2 * (1 + (kSmemG ? k : 0)), k);
  {
    const GainT* g_src = a.cur.g + static_cast<size_t>(w) * k * ld;
    const uint8_t* lab_src = a.cur.labels + static_cast<size_t>(w) * ld;
    const int32_t* sizes = a.cur.sizes + static_cast<size_t>(w) * a.kpad;
    for (int i = warp; i < k * quads; i += kWarps) {
      const int c = i / quads, quad = i - c * quads;
      uint32_t x[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int u = 128 * quad + 32 * t + lane;
        x[t] = u < ld ? static_cast<uint16_t>(g_src[static_cast<size_t>(c) * ld + u]) : 0u;
        if constexpr (kHalf) {  // places past n are never read back
          const uint32_t own = u < n && lab_src[u] == c ? 0x8000u : 0u;
          x[t] = u < n ? static_cast<uint32_t>(sizes[c] - 2 * static_cast<int>(x[t]) + 0x4000) | own : 0x4000u;
        }
      }
      reinterpret_cast<uint2*>(g + static_cast<size_t>(c) * ldw)[32 * quad + lane] =
          make_uint2(x[0] | x[1] << 16, x[2] | x[3] << 16);
    }
    const uint4* ls = reinterpret_cast<const uint4*>(lab_src);
    uint4* ldst = reinterpret_cast<uint4*>(lab);
    for (int i = tid; i < ld / 16; i += T) ldst[i] = ls[i];
    for (int c = tid; c < k; c += T) s.off[c] = 64 * sizes[c] + c;
  }
  long long objective = a.cur.f[w];
  const long long move_budget = objective;
  unsigned long long applied = 0;
  const WarpTranspose32 transpose(lane);
  const int quads_per_warp = (quads + kWarps - 1) / kWarps;
  const int quad0 = warp * quads_per_warp;
  const int quad1 = min(quads, quad0 + quads_per_warp);
  __syncthreads();

  bool known_low = false;  // L is near the smallest gain
  while (true) {
    // ---- the last window's moves as masks per cluster
    const int moves = s.moves;
    for (int c = warp; c < k; c += kWarps) {
      const int ft0 = lane < moves ? s.move_ft[lane] : 0xffff;
      const int ft1 = lane + kWarp < moves ? s.move_ft[lane + kWarp] : 0xffff;
      const uint32_t f0 = __ballot_sync(kAllLanes, (ft0 & 0xff) == c), t0 = __ballot_sync(kAllLanes, (ft0 >> 8) == c);
      const uint32_t f1 = __ballot_sync(kAllLanes, (ft1 & 0xff) == c), t1 = __ballot_sync(kAllLanes, (ft1 >> 8) == c);
      if (lane == 0) {
        const int left = __popc(f0) + __popc(f1), grown = __popc(t0) + __popc(t1) - left;
        const int off = s.off[c] + 64 * grown;
        s.off[c] = off;
        // kHalf: h changes by grown + 2 left - 2 popc((x ^ F) & (F | T)), of a pair at once
        s.mask[c][0] = make_uint4(f0 | t0, f0, kHalf ? static_cast<uint32_t>(grown + 2 * left) * 0x10001u : __popc(f0),
                                  static_cast<uint32_t>(off));
        s.mask[c][1] = make_uint4(f1 | t1, f1, __popc(f1), 0u);
      }
    }
    if (kHalf && tid < moves) {  // the moved vertices' own-cluster bits (flips: their order does not matter)
      const int place = WindowPlace(s.move_v[tid]);
      const uint32_t bit = 0x8000u << (16 * (place & 1));
      uint32_t* words = reinterpret_cast<uint32_t*>(g) + place / 2;
      atomicXor(words + static_cast<size_t>(s.move_ft[tid] & 0xff) * (ldw / 2), bit);
      atomicXor(words + static_cast<size_t>(s.move_ft[tid] >> 8) * (ldw / 2), bit);
    }
    for (int b = tid; b < kWindowBins; b += T) s.hist[b] = 0;
    __syncthreads();

    // ---- refresh: counters, gains, their distances from L
    {
      const int low = s.low;
      int smallest = 0x7fffffff;
      const uint32_t* row0 = a.gr.bits + static_cast<size_t>(lane < moves ? s.move_v[lane] : 0) * pitch;
      const uint32_t* row1 = a.gr.bits + static_cast<size_t>(lane + kWarp < moves ? s.move_v[lane + kWarp] : 0) * pitch;
      // a quad's adjacency words and labels are read one quad ahead
      uint4 n0 = make_uint4(0u, 0u, 0u, 0u), n1 = n0;
      int next_own[4];
      auto read_ahead = [&](int quad) {
        if (lane < moves) n0 = *reinterpret_cast<const uint4*>(row0 + 4 * quad);
        if (lane + kWarp < moves) n1 = *reinterpret_cast<const uint4*>(row1 + 4 * quad);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int u = 128 * quad + 32 * t + lane;
          next_own[t] = !kHalf && u < n ? lab[u] : 0;
        }
      };
      if (quad0 < quad1) read_ahead(quad0);
      for (int quad = quad0; quad < quad1; ++quad) {
        uint32_t x0[4] = {n0.x, n0.y, n0.z, n0.w}, x1[4] = {n1.x, n1.y, n1.z, n1.w};
        int own[4] = {next_own[0], next_own[1], next_own[2], next_own[3]};
        if (quad + 1 < quad1) read_ahead(quad + 1);
        if (moves > 0) {
#pragma unroll
          for (int t = 0; t < 4; ++t) x0[t] = transpose(x0[t]);
        }
        if (moves > kWarp) {
#pragma unroll
          for (int t = 0; t < 4; ++t) x1[t] = transpose(x1[t]);
        }
        const int u0 = 128 * quad + lane;
        int kmin[4], ko[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          kmin[t] = 0x7fffffff;
          ko[t] = 0;
        }
        uint2* gq = reinterpret_cast<uint2*>(g) + 32 * quad + lane;
        const size_t step = static_cast<size_t>(ldw) / 4;
        constexpr int kGroup = K > 0 ? K : 8;  // clusters whose loads are in flight together
        uint32_t left[4] = {0u, 0u, 0u, 0u};   // compile-time K: minus the changes so far (all changes sum to zero)
        uint2 low2 = make_uint2(~0u, ~0u), high2 = make_uint2(0u, 0u);  // kHalf: smallest and largest h, in pairs
        for (int c0 = 0; c0 < k; c0 += kGroup) {
          uint2 gv[kGroup];
#pragma unroll
          for (int i = 0; i < kGroup; ++i) {
            if (K > 0 || c0 + i < k) gv[i] = gq[(c0 + i) * step];
          }
#pragma unroll
          for (int i = 0; i < kGroup; ++i) {
            const int c = c0 + i;
            if (K == 0 && c >= k) break;
            const uint4 m0 = s.mask[c][0];
            if (K > 0 ? moves > 0 : m0.x != 0u || (moves > kWarp && s.mask[c][1].x != 0u)) {
              const bool last = K > 0 && i == K - 1;
              uint32_t d[4];
              if (!last) {
#pragma unroll
                for (int t = 0; t < 4; ++t) d[t] = __popc((x0[t] ^ m0.y) & m0.x);
                if (moves > kWarp) {
                  const uint4 m1 = s.mask[c][1];
#pragma unroll
                  for (int t = 0; t < 4; ++t) d[t] += __popc((x1[t] ^ m1.y) & m1.x) - (kHalf ? 0u : m1.z);
                }
              }
              if constexpr (kHalf) {
                uint32_t e0 = left[0], e1 = left[1];
                if (!last) {
                  e0 = m0.z - 2u * (d[0] + (d[1] << 16));
                  e1 = m0.z - 2u * (d[2] + (d[3] << 16));
                  left[0] -= e0;
                  left[1] -= e1;
                }
                gv[i].x += e0;
                gv[i].y += e1;
              } else {
#pragma unroll
                for (int t = 0; t < 4; ++t) d[t] = last ? left[t] : d[t] - m0.z;
#pragma unroll
                for (int t = 0; t < 4; ++t) left[t] -= d[t];
                gv[i].x += d[0] + (d[1] << 16);
                gv[i].y += d[2] + (d[3] << 16);
              }
              gq[c * step] = gv[i];
            }
            if constexpr (kHalf) {
              low2.x = __vminu2(low2.x, gv[i].x);
              low2.y = __vminu2(low2.y, gv[i].y);
              high2.x = __vmaxu2(high2.x, gv[i].x);
              high2.y = __vmaxu2(high2.y, gv[i].y);
            } else {
              const int off = static_cast<int>(m0.w);
              const int key[4] = {off - 128 * static_cast<int>(gv[i].x & 0xffffu), off - 128 * static_cast<int>(gv[i].x >> 16),
                                  off - 128 * static_cast<int>(gv[i].y & 0xffffu), off - 128 * static_cast<int>(gv[i].y >> 16)};
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const bool is_own = own[t] == c;
                ko[t] = is_own ? key[t] : ko[t];
                kmin[t] = min(kmin[t], is_own ? 0x7fffffff : key[t]);
              }
            }
          }
        }
        int gains[4];
        if constexpr (kHalf) {
          gains[0] = static_cast<int>(low2.x & 0xffffu) - static_cast<int>(high2.x & 0xffffu) + 0x8001;
          gains[1] = static_cast<int>(low2.x >> 16) - static_cast<int>(high2.x >> 16) + 0x8001;
          gains[2] = static_cast<int>(low2.y & 0xffffu) - static_cast<int>(high2.y & 0xffffu) + 0x8001;
          gains[3] = static_cast<int>(low2.y >> 16) - static_cast<int>(high2.y >> 16) + 0x8001;
        } else {
#pragma unroll
          for (int t = 0; t < 4; ++t) gains[t] = (kmin[t] >> 6) - (ko[t] >> 6) + 1;
        }
        uint32_t d16[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int gain = u0 + 32 * t < n ? gains[t] : 0x3fffffff;
          smallest = min(smallest, gain);
          d16[t] = static_cast<uint32_t>(min(gain - low, 65535));
          if (known_low && d16[t] < kWindowBins) atomicAdd(&s.hist[d16[t]], 1);
        }
        reinterpret_cast<uint2*>(dist)[32 * quad + lane] = make_uint2((d16[0] & 0xffffu) | d16[1] << 16,
                                                                      (d16[2] & 0xffffu) | d16[3] << 16);
      }
      smallest = __reduce_min_sync(kAllLanes, smallest);
      if (lane == 0) atomicMin(&s.smallest, smallest);
    }
    __syncthreads();
    const int smallest = s.smallest;
    if (smallest >= 0) break;
    if (!known_low || smallest - s.low >= kWindowBins) {  // L is too far below: once more from the smallest gain
      __syncthreads();
      if (tid == 0) {
        s.low = smallest;
        s.moves = 0;
        s.smallest = 0x7fffffff;
      }
      known_low = true;
      __syncthreads();
      continue;
    }
    // ---- theta: the most bins that hold at most kCap vertices, at least the smallest gain's
    if (warp == 0) {
      constexpr int kPer = kWindowBins / kWarp;
      int h[kPer];
      int sum = 0;
#pragma unroll
      for (int b = 0; b < kPer; ++b) {
        h[b] = s.hist[lane * kPer + b];
        sum += h[b];
      }
      int incl = sum;
#pragma unroll
      for (int o = 1; o < kWarp; o <<= 1) {
        const int y = __shfl_up_sync(kAllLanes, incl, o);
        if (lane >= o) incl += y;
      }
      int run = incl - sum;
      int bins = 0;
#pragma unroll
      for (int b = 0; b < kPer; ++b) {
        run += h[b];
        if (run <= kCap) bins = lane * kPer + b + 1;
      }
      bins = __reduce_max_sync(kAllLanes, bins);
      if (lane == 0) {
        const int least = smallest - s.low + 1;
        s.partial = bins < least ? 1 : 0;
        s.bins = max(bins, least);
      }
    }
    __syncthreads();
    // ---- S: each warp counts, then writes, the members of its own quads
    {
      const int bins = s.bins;
      auto members_of = [&](int quad) {  // bit t: vertex 32 t + lane of the quad is a member
        const uint2 d = reinterpret_cast<const uint2*>(dist)[32 * quad + lane];
        return (static_cast<int>(d.x & 0xffffu) < bins ? 1u : 0u) | (static_cast<int>(d.x >> 16) < bins ? 2u : 0u) |
               (static_cast<int>(d.y & 0xffffu) < bins ? 4u : 0u) | (static_cast<int>(d.y >> 16) < bins ? 8u : 0u);
      };
      uint32_t mine = 0;
      for (int quad = quad0; quad < quad1; ++quad) {
        const uint32_t in = members_of(quad);
        mine += (in & 1u) + ((in >> 1) & 1u) + ((in >> 2) & 1u) + (in >> 3);
      }
      const uint32_t lane_members = mine;
      mine = __reduce_add_sync(kAllLanes, mine);
      if (lane == 0) s.warp_count[warp] = static_cast<int>(mine);
      __syncthreads();
      const int wc = lane < kWarps ? s.warp_count[lane] : 0;
      int at = __reduce_add_sync(kAllLanes, lane < warp ? wc : 0);
      const int total = __reduce_add_sync(kAllLanes, wc);
      if (kBound <= 8 && !s.partial) {
        // move keys carry the vertex: any order will do, so a lane writes its own vertices one after another (no
        // population counts, which take eight clocks each)
        int incl = static_cast<int>(lane_members);
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
          const int y = __shfl_up_sync(kAllLanes, incl, o);
          if (lane >= o) incl += y;
        }
        int p = at + incl - static_cast<int>(lane_members);
        const int end = at + incl;
        for (int quad = quad0; quad < quad1 && __any_sync(kAllLanes, p < end); ++quad) {
          const uint32_t in = members_of(quad);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if ((in >> t) & 1u) s.member[p++] = 128 * quad + 32 * t + lane;
          }
        }
      } else if (mine > 0) {  // in vertex order: the lowest kCap of them where S cannot hold all
        const unsigned below = (1u << lane) - 1u;
        for (int quad = quad0; quad < quad1; ++quad) {
          const uint32_t in = members_of(quad);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const unsigned b = __ballot_sync(kAllLanes, (in >> t) & 1u);
            if (b == 0u) continue;
            if ((in >> t) & 1u) {
              const int p = at + __popc(b & below);
              if (p < kCap) s.member[p] = 128 * quad + 32 * t + lane;
            }
            at += __popc(b);
          }
        }
      }
      if (tid == 0) {
        s.members = min(total, kCap);
        s.smallest = 0x7fffffff;
      }
    }
    __syncthreads();
    // ---- moves
    if constexpr (kForm.keys > 0) {
      if (tid < kForm.threads) WindowMovesK<kForm.keys, V, kForm.threads, kCap, kHalf>(a.gr, k, g, ldw, lab, s, objective);
    } else {
      members.template Fill<T, kHalf>(g, ldw, lab, s.member, s.members, s.off, k);
      __syncthreads();
      if (tid < kForm.threads) WindowMovesN<V, kForm.threads, kCap>(a.gr, k, members, lab, s, objective);
    }
    __syncthreads();
    applied += static_cast<unsigned long long>(s.moves);
    if (static_cast<long long>(applied) > move_budget) {
      if (tid == 0) atomicExch(&a.ctl->error, kErrorMoveBound);
      break;
    }
    if (s.finished) break;
  }
  if (tid == 0) {
    a.next.f[slot] = objective;
    if (applied) atomicAdd(&a.ctl->moves, applied);
  }
}

// One slot per block (plain path).
template <int kBound, int kCap, bool kSmemG, bool kHalf, typename GainT>
__global__ void __launch_bounds__(kWindowThreads, 1) k_descent_window(DescentArgs<GainT> a) {
  DescentWindow<kBound, kCap, kSmemG, kHalf, GainT>(a, blockIdx.x);
}

}  // namespace ccb
