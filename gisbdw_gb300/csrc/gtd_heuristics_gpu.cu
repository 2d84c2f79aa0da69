// The greedy elimination heuristics of gtd_heuristics.cu as one batched GPU
// launch: the same picks, so the trees are identical to the host's (and so to
// the reference's heuristic chain, Treedepth/src/branch_and_bound/heuristics/).
//
// A step takes the component of the smallest remaining vertex (ComponentCmp,
// elimination_tree.hpp:67-72), picks a vertex of it and eliminates it: its
// parent is the vertex eliminated last in its component. A pick depends on its
// component alone, so the order of the components does not matter: kinds 0, 1
// and 2 take one vertex from every component at once (greedy_rounds), kind 3
// goes step by step (greedy), one warp per graph.
//   kind 1  highest degree inside the component, ties to the smallest id
//           (highest_degree_heuristic.hpp:18-44)
//   kind 2  variance score D / sqrt(gamma + A) + E * #components of C - v,
//           ties to the higher degree, then the smallest id
//           (variance_heuristic.hpp:24-78; A, D, E = 1.0, 0.2, 0.8), in
//           double with the host's operation order
//   kind 0  the better of kinds 1 and 2 (benchmark.cpp:50-55)
//   kind 3  the highest caller score, ties to the smallest id
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "gtd_handle.h"

namespace gtd {
namespace {

constexpr int kHWarps = 4;
constexpr int kHMaxN = 128;

struct HeurGraph {
  int32_t n;
  int32_t off;  // first vertex's (lo, hi) pair in the pool, parent pool offset
};

struct HeurWarp {
  uint64_t alo[kHMaxN], ahi[kHMaxN];
  int16_t owner[kHMaxN];
  uint8_t cdepth[kHMaxN];
};

__device__ __forceinline__ bool hhas(uint64_t lo, uint64_t hi, int v) {
  return v < 64 ? ((lo >> v) & 1ull) : ((hi >> (v - 64)) & 1ull);
}
__device__ __forceinline__ void hclear(uint64_t& lo, uint64_t& hi, int v) {
  if (v < 64)
    lo &= ~(1ull << v);
  else
    hi &= ~(1ull << (v - 64));
}
__device__ __forceinline__ int hfirst(uint64_t lo, uint64_t hi) {
  return lo ? __ffsll(static_cast<long long>(lo)) - 1 : 63 + __ffsll(static_cast<long long>(hi));
}

// Component of S holding v, by one lane (serial BFS).
__device__ void lane_component(const HeurWarp* w, uint64_t Slo, uint64_t Shi, int v, uint64_t& rlo, uint64_t& rhi) {
  rlo = v < 64 ? (1ull << v) : 0ull;
  rhi = v >= 64 ? (1ull << (v - 64)) : 0ull;
  uint64_t flo = rlo, fhi = rhi;
  while (flo | fhi) {
    uint64_t nlo = 0, nhi = 0;
    while (flo | fhi) {
      const int u = hfirst(flo, fhi);
      hclear(flo, fhi, u);
      nlo |= w->alo[u];
      nhi |= w->ahi[u];
    }
    nlo &= Slo & ~rlo;
    nhi &= Shi & ~rhi;
    rlo |= nlo;
    rhi |= nhi;
    flo = nlo;
    fhi = nhi;
  }
}

struct Pick {
  double score;
  int v;
};
// The host's scan order: higher score, then smaller id.
__device__ __forceinline__ bool better(const Pick& a, const Pick& b) {
  if (a.v < 0)
    return false;
  if (b.v < 0)
    return true;
  if (a.score != b.score)
    return a.score > b.score;
  return a.v < b.v;
}

// One greedy elimination of the warp's graph; returns the tree height.
__device__ int greedy(HeurWarp* w, int n, const float* scores, int32_t* parent) {
  const int lane = threadIdx.x & 31;
  for (int u = lane; u < n; u += 32) {
    w->owner[u] = -1;
    w->cdepth[u] = 0;
  }
  __syncwarp();
  uint64_t rem_lo = n >= 64 ? ~0ull : ((1ull << n) - 1);
  uint64_t rem_hi = n > 64 ? (n == 128 ? ~0ull : ((1ull << (n - 64)) - 1)) : 0ull;
  int height = 0;
  while (rem_lo | rem_hi) {
    // component of the smallest remaining vertex (every lane computes it)
    uint64_t Clo, Chi;
    lane_component(w, rem_lo, rem_hi, hfirst(rem_lo, rem_hi), Clo, Chi);
    Pick best{0.0, -1};
    for (int k = 0; k < kHMaxN / 32; ++k) {
      const int u = lane + 32 * k;
      if (u >= n || !hhas(Clo, Chi, u))
        continue;
      const Pick c{static_cast<double>(scores[u]), u};
      if (better(c, best))
        best = c;
    }
    for (int off = 16; off > 0; off >>= 1) {
      Pick o;
      o.score = __shfl_xor_sync(0xffffffffu, best.score, off);
      o.v = __shfl_xor_sync(0xffffffffu, best.v, off);
      if (better(o, best))
        best = o;
    }
    const int v = best.v;
    const int dv = w->cdepth[v];
    if (lane == 0)
      parent[v] = w->owner[v];
    height = max(height, dv + 1);
    __syncwarp();
    for (int k = 0; k < kHMaxN / 32; ++k) {
      const int u = lane + 32 * k;
      if (u < n && u != v && hhas(Clo, Chi, u)) {
        w->owner[u] = static_cast<int16_t>(v);
        w->cdepth[u] = static_cast<uint8_t>(dv + 1);
      }
    }
    hclear(rem_lo, rem_hi, v);
    __syncwarp();
  }
  return height;
}

__global__ void __launch_bounds__(32 * kHWarps) heuristic_kernel(const HeurGraph* graphs, int count,
                                                                 const uint64_t* adj2, const float* scores,
                                                                 int32_t* td_out, int32_t* parent_out) {
  __shared__ HeurWarp wm[kHWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  HeurWarp* w = &wm[warp];
  for (int g = blockIdx.x * kHWarps + warp; g < count; g += gridDim.x * kHWarps) {
    const HeurGraph G = graphs[g];
    for (int u = lane; u < G.n; u += 32) {
      w->alo[u] = adj2[2 * (size_t(G.off) + u)];
      w->ahi[u] = adj2[2 * (size_t(G.off) + u) + 1];
    }
    __syncwarp();
    const int td = greedy(w, G.n, scores + G.off, parent_out + G.off);
    if (lane == 0)
      td_out[g] = td;
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Kinds 0, 1, 2: a thread per vertex, every component at once.
// ---------------------------------------------------------------------------

// A vertex set of W words.
template <int W>
struct Bits {
  uint32_t w[W];
};

template <int W>
__device__ __forceinline__ bool any(const Bits<W>& s) {
  uint32_t x = 0;
#pragma unroll
  for (int i = 0; i < W; ++i)
    x |= s.w[i];
  return x != 0;
}
template <int W>
__device__ __forceinline__ bool has(const Bits<W>& s, int v) {
  uint32_t x = 0;
#pragma unroll
  for (int i = 0; i < W; ++i)
    x = (v >> 5) == i ? s.w[i] : x;
  return (x >> (v & 31)) & 1u;
}
template <int W>
__device__ __forceinline__ void set_bit(Bits<W>& s, int v, bool on) {
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const uint32_t bit = (v >> 5) == i ? 1u << (v & 31) : 0u;
    s.w[i] = on ? s.w[i] | bit : s.w[i] & ~bit;
  }
}
template <int W>
__device__ __forceinline__ int first(const Bits<W>& s) {
  int r = -1;
#pragma unroll
  for (int i = W - 1; i >= 0; --i)
    r = s.w[i] ? 32 * i + __ffs(s.w[i]) - 1 : r;
  return r;
}
template <int W>
__device__ __forceinline__ int size(const Bits<W>& s) {
  int r = 0;
#pragma unroll
  for (int i = 0; i < W; ++i)
    r += __popc(s.w[i]);
  return r;
}

// Adjacency rows of W words; row kHMaxN is empty.
template <int W>
__device__ __forceinline__ Bits<W> row(const uint32_t* adj, int v) {
  Bits<W> r;
  if constexpr (W == 4) {
    const uint4 x = reinterpret_cast<const uint4*>(adj)[v];
    r.w[0] = x.x;
    r.w[1] = x.y;
    r.w[2] = x.z;
    r.w[3] = x.w;
  } else if constexpr (W == 2) {
    const uint2 x = reinterpret_cast<const uint2*>(adj)[v];
    r.w[0] = x.x;
    r.w[1] = x.y;
  } else {
    r.w[0] = adj[v];
  }
  return r;
}

// The components of S by one thread, f(component) for each in the order of
// their lowest vertices. One loop over all of them, up to four vertices a step
// in no particular order, the lowest of every word (and the highest, of one or
// two words): their loads overlap, and lanes with different sets take about as
// many steps, where the levels of a breadth-first search, or components, nested
// in it would wait for the widest of the warp's.
template <int W, class F>
__device__ __forceinline__ void for_components(const uint32_t* adj, Bits<W> S, F&& f) {
  Bits<W> reach = {}, todo = {};
  while (any(S)) {
    if (!any(todo)) {
      set_bit(todo, first(S), true);
      reach = todo;
    }
    Bits<W> next = {};
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const uint32_t t = todo.w[i];
      const Bits<W> a = row<W>(adj, t ? 32 * i + __ffs(t) - 1 : kHMaxN);
      uint32_t left = t & (t - 1u);
#pragma unroll
      for (int k = 0; k < W; ++k)
        next.w[k] |= a.w[k];
      if constexpr (W <= 2) {
        const int top = 31 - __clz(left);
        const Bits<W> b = row<W>(adj, left ? 32 * i + top : kHMaxN);
        left &= ~(left ? 1u << top : 0u);
#pragma unroll
        for (int k = 0; k < W; ++k)
          next.w[k] |= b.w[k];
      }
      todo.w[i] = left;
    }
    uint32_t missing = 0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const uint32_t fresh = next.w[k] & S.w[k] & ~reach.w[k];
      reach.w[k] |= fresh;
      todo.w[k] |= fresh;
      missing |= reach.w[k] ^ S.w[k];
    }
    if (missing == 0 || !any(todo)) {
      f(reach);
#pragma unroll
      for (int k = 0; k < W; ++k) {
        S.w[k] &= ~reach.w[k];
        todo.w[k] = 0u;
      }
    }
  }
}

// The order of the variance scores of the vertices that leave nc > 1 parts of
// a component, `total` vertices together (variance_heuristic.hpp:40-56 as
// restated on the host: gamma is the sum of the squared distances from the mean
// size, the score D / sqrt(gamma + A) + E nc). Every score of the component has
// the same nc, so a smaller gamma wins. For nc a power of two the host's gamma
// is exact: gamma = (nc sum s^2 - total^2) / nc, whose steps of 1 / nc (gamma
// below 2^14) move the score by more than 1e-9, and the integer orders as the
// doubles do. Otherwise the host's double operations in their order, each
// rounded to nearest (no contraction into FMAs).
__device__ __forceinline__ unsigned long long variance_key(const uint8_t* sizes, int nc, int total) {
  if ((nc & (nc - 1)) == 0) {
    int squares = 0;
    for (int i = 0; i < nc; ++i)
      squares += static_cast<int>(sizes[i]) * sizes[i];
    return (1ull << 32) - static_cast<unsigned long long>(nc * squares - total * total);
  }
  const float A = 1.0f, D = 0.2f, E = 0.8f;
  double acc = 0.0, gamma = 0.0;
  for (int i = 0; i < nc; ++i)
    acc = __dadd_rn(acc, static_cast<double>(sizes[i]));
  const double avg = __ddiv_rn(acc, static_cast<double>(nc));
  for (int i = 0; i < nc; ++i) {
    const double d = __dsub_rn(static_cast<double>(sizes[i]), avg);
    gamma = __dadd_rn(gamma, __dmul_rn(d, d));
  }
  const float enc = __fmul_rn(E, static_cast<float>(nc));
  // positive doubles: their bits are in order
  return static_cast<unsigned long long>(__double_as_longlong(
      __dadd_rn(__ddiv_rn(static_cast<double>(D), __dsqrt_rn(__dadd_rn(gamma, static_cast<double>(A)))),
                static_cast<double>(enc))));
}

// One greedy elimination by a group of `threads` threads (its own barrier).
// Components are named by their lowest vertices.
struct RoundMem {
  alignas(16) uint32_t sets[4 * kHMaxN];   // the components
  alignas(16) uint32_t parts[4 * kHMaxN];  // per component eliminated from: the names of what is left of it
  unsigned long long best[kHMaxN];  // per component: the best score among those that leave the most parts
  unsigned long long own[kHMaxN];   // per vertex: its score
  uint32_t most[kHMaxN];            // per component: the most parts that a removal leaves
  uint32_t pick[kHMaxN];            // ... the best (degree, smallest id) among the best
  int32_t parent[kHMaxN];
  uint8_t leaves[kHMaxN];           // per vertex: parts that its removal leaves
  uint8_t name[kHMaxN];             // the vertex's component
  uint8_t inner[kHMaxN];            // the vertices to search from
  int32_t left, height, inners;
};

__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Rounds: every vertex scores itself within its component, each component
// eliminates its best. The number of rounds is the tree's height, not its
// size. The variance score needs a search of C - v per vertex, but not for a
// vertex with one neighbour left, and the searches are taken by the first
// threads, so that whole warps have none. A score lies in (E nc, E nc + D] and
// D < E: only the vertices that leave the most parts can win. What is left of a
// component is published by the thread that searched its vertex (which still
// has it up to kKeep parts; kind 1 searches only here), the others look
// themselves up in it. Bound by the latency of a search, |C| / 4 steps of some
// 100 cycles, once a round.
template <int W>
__device__ void greedy_rounds(const uint32_t* adj, int n, bool variance, RoundMem& m, int barrier, int threads) {
  constexpr int kKeep = 4;
  const int v = threadIdx.x % threads;
  const bool own = v < n;
  bool alive = own;
  int owner = -1, depth = 0, name = 0;
  auto store = [&](uint32_t* to, int at, const Bits<W>& s) {
#pragma unroll
    for (int i = 0; i < W; ++i)
      to[at * W + i] = s.w[i];
  };
  auto look_up = [&](int from) {
    Bits<W> names = row<W>(m.parts, from);
    while (any(names)) {
      name = first(names);
      if (has(row<W>(m.sets, name), v))
        break;
      set_bit(names, name, false);
    }
    m.name[v] = static_cast<uint8_t>(name);
  };
  auto publish = [&](const Bits<W>& S, int from) {
    Bits<W> names = {};
    for_components<W>(adj, S, [&](const Bits<W>& c) {
      store(m.sets, first(c), c);
      set_bit(names, first(c), true);
    });
    store(m.parts, from, names);
  };
  if (v == 0) {
    m.left = n;
    m.height = 0;
    Bits<W> all;
#pragma unroll
    for (int i = 0; i < W; ++i)
      all.w[i] = n >= 32 * (i + 1) ? ~0u : n > 32 * i ? (1u << (n - 32 * i)) - 1u : 0u;
    publish(all, 0);
  }
  group_sync(barrier, threads);
  if (own)
    look_up(0);
  for (;;) {
    if (own) {
      m.most[v] = 0u;
      m.best[v] = 0ull;
      m.pick[v] = 0u;
    }
    if (v == 0)
      m.inners = 0;
    group_sync(barrier, threads);
    if (m.left == 0)
      return;
    uint32_t key = 0, deg = 0;
    Bits<W> C = {};
    if (alive) {
      C = row<W>(m.sets, name);
      const Bits<W> mine = row<W>(adj, v);
#pragma unroll
      for (int i = 0; i < W; ++i)
        deg += __popc(mine.w[i] & C.w[i]);
      key = (deg + 1) << 8 | static_cast<uint32_t>(kHMaxN - 1 - v);  // > 0
      if (variance) {
        if (deg >= 2) {
          m.inner[atomicAdd(&m.inners, 1)] = static_cast<uint8_t>(v);
        } else {
          m.leaves[v] = static_cast<uint8_t>(deg);  // of a single vertex nothing is left
          atomicMax(&m.most[name], deg);
        }
      }
    }
    Bits<W> kept[kKeep];
    int u = -1, at = 0, nc = 0;
    if (variance) {
      group_sync(barrier, threads);
      uint8_t sizes[kHMaxN];
      int total = 0;
      if (v < m.inners) {
        u = m.inner[v];
        at = m.name[u];
        Bits<W> rest = row<W>(m.sets, at);
        set_bit(rest, u, false);
        total = size(rest);
        for_components<W>(adj, rest, [&](const Bits<W>& c) {
#pragma unroll
          for (int i = 0; i < kKeep; ++i)
            if (nc == i)
              kept[i] = c;
          sizes[nc++] = static_cast<uint8_t>(size(c));
        });
        m.leaves[u] = static_cast<uint8_t>(nc);
        atomicMax(&m.most[at], static_cast<uint32_t>(nc));
      }
      group_sync(barrier, threads);
      if (u >= 0 && nc > 1 && m.most[at] == static_cast<uint32_t>(nc)) {
        m.own[u] = variance_key(sizes, nc, total);
        atomicMax(&m.best[at], m.own[u]);
      }
      group_sync(barrier, threads);
    }
    bool candidate = alive;
    if (alive && variance) {
      const uint32_t most = m.most[name];  // of one part or none the scores are equal
      candidate = m.leaves[v] == most && (most <= 1 || m.best[name] == m.own[v]);
    }
    if (candidate)
      atomicMax(&m.pick[name], key);
    group_sync(barrier, threads);
    const int from = name;
    bool moved = false;
    if (u >= 0 && kHMaxN - 1 - static_cast<int>(m.pick[at] & 0xFFu) == u) {  // what this thread searched is eliminated
      if (nc <= kKeep) {
        Bits<W> names = {};
#pragma unroll
        for (int i = 0; i < kKeep; ++i)
          if (i < nc) {
            store(m.sets, first(kept[i]), kept[i]);
            set_bit(names, first(kept[i]), true);
          }
        store(m.parts, at, names);
      } else {
        Bits<W> rest = row<W>(m.sets, at);
        set_bit(rest, u, false);
        publish(rest, at);
      }
    }
    if (alive) {
      const int chosen = kHMaxN - 1 - static_cast<int>(m.pick[name] & 0xFFu);
      if (chosen == v) {
        m.parent[v] = owner;
        atomicMax(&m.height, depth + 1);
        atomicSub(&m.left, 1);
        alive = false;
        set_bit(C, v, false);
        if (!variance) {
          publish(C, name);
        } else if (deg == 1) {  // one part
          Bits<W> names = {};
          set_bit(names, first(C), true);
          store(m.sets, first(C), C);
          store(m.parts, name, names);
        }
      } else {
        owner = chosen;
        ++depth;
        moved = true;
      }
    }
    group_sync(barrier, threads);
    if (moved)
      look_up(from);
  }
}

// One CTA per graph; kind 0 runs kinds 1 and 2 side by side, `threads` threads
// each. Components that do not depend on where a search starts need symmetric
// masks: a graph without them gets the height -1 and is left to the host (the
// check adds nothing that shows). 1024 graphs of 20..80 vertices, kind 0:
// 1.48 ms with one warp per graph and one vertex per step, 627 us when every
// vertex searched its new component and scored itself in double, 324 us now
// (48 graphs of 24..36: 45 us).
__global__ void heuristic_rounds_kernel(const HeurGraph* graphs, const uint64_t* adj2, int kind, int threads,
                                        int32_t* td_out, int32_t* parent_out) {
  __shared__ __align__(16) uint32_t adj[4 * (kHMaxN + 1)];
  __shared__ RoundMem mem[2];
  const HeurGraph G = graphs[blockIdx.x];
  const int words = G.n <= 32 ? 1 : G.n <= 64 ? 2 : 4;
  const uint32_t* const rows = reinterpret_cast<const uint32_t*>(adj2 + 2 * size_t(G.off));
  for (int t = threadIdx.x; t < G.n * words; t += blockDim.x)
    adj[t] = rows[4 * (t / words) + t % words];
  if (threadIdx.x < words)
    adj[kHMaxN * words + threadIdx.x] = 0u;
  __syncthreads();
  bool one_way = false;
  if (threadIdx.x < G.n) {
    const int v = threadIdx.x;
    for (int i = 0; i < words; ++i)
      for (uint32_t left = adj[v * words + i]; left; left &= left - 1u) {
        const int u = 32 * i + __ffs(static_cast<int>(left)) - 1;
        one_way |= !((adj[u * words + (v >> 5)] >> (v & 31)) & 1u);
      }
  }
  if (__syncthreads_or(one_way)) {
    if (threadIdx.x == 0)
      td_out[blockIdx.x] = -1;
    return;
  }
  const int half = threadIdx.x / threads;
  const bool variance = kind == 2 || half == 1;
  if (words == 1)
    greedy_rounds<1>(adj, G.n, variance, mem[half], 1 + half, threads);
  else if (words == 2)
    greedy_rounds<2>(adj, G.n, variance, mem[half], 1 + half, threads);
  else
    greedy_rounds<4>(adj, G.n, variance, mem[half], 1 + half, threads);
  __syncthreads();
  // the variance tree only when strictly lower, as on the host
  const int from = kind == 0 && mem[1].height < mem[0].height ? 1 : 0;
  for (int u = threadIdx.x; u < G.n; u += blockDim.x)
    parent_out[G.off + u] = mem[from].parent[u];
  if (threadIdx.x == 0)
    td_out[blockIdx.x] = mem[from].height;
}

}  // namespace
}  // namespace gtd

using gtd::DeviceGuard;
using gtd::ensure_device;
using gtd::fail;

extern "C" gtd_status gtd_heuristic_batch(gtd_handle h, const gtd_graph_desc* descs, int count,
                                          const uint64_t* adj2_pool, int64_t pool_len, int kind,
                                          const float* scores_pool, int32_t* td_out, int32_t* parent_out) {
  if (!h)
    return GTD_INVALID_ARG;
  if (!descs || count < 1 || !adj2_pool || pool_len < 1 || !td_out || !parent_out || kind < 0 || kind > 3 ||
      (kind == 3 && !scores_pool))
    return fail(h, GTD_INVALID_ARG, "null pointer argument, empty batch, or kind outside 0..3 (3 needs scores)");
  std::vector<gtd::HeurGraph> graphs(count);
  int max_n = 1;
  for (int i = 0; i < count; ++i) {
    const gtd_graph_desc& d = descs[i];
    if (d.n < 1 || d.n > gtd::kHMaxN || d.offset < 0 || int64_t(d.offset) + d.n > pool_len)
      return fail(h, GTD_INVALID_ARG, "graph " + std::to_string(i) + ": n outside [1, 128] or outside the pool");
    const uint64_t* a = adj2_pool + 2 * size_t(d.offset);
    const uint64_t lo_ok = d.n >= 64 ? ~0ull : ((1ull << d.n) - 1);
    const uint64_t hi_ok = d.n <= 64 ? 0ull : (d.n >= 128 ? ~0ull : ((1ull << (d.n - 64)) - 1));
    for (int v = 0; v < d.n; ++v) {
      const bool self = v < 64 ? ((a[2 * v] >> v) & 1ull) : ((a[2 * v + 1] >> (v - 64)) & 1ull);
      const bool beyond = (a[2 * v] & ~lo_ok) != 0 || (a[2 * v + 1] & ~hi_ok) != 0;
      if (self || beyond)
        return fail(h, GTD_INVALID_ARG, "graph " + std::to_string(i) + ": self loop or adjacency bit >= n");
    }
    graphs[i] = gtd::HeurGraph{d.n, d.offset};
    max_n = std::max(max_n, d.n);
  }
  DeviceGuard guard(h->device);
  const size_t n_pool = static_cast<size_t>(pool_len);
  const size_t bytes = 256 + count * sizeof(gtd::HeurGraph) + 2 * n_pool * sizeof(uint64_t) +
                       (scores_pool ? n_pool * sizeof(float) : 0) + size_t(count) * 4 + n_pool * 4 + 1024;
  GTD_CUDA(h, ensure_device(&h->d_scratch, &h->scratch_cap, bytes));
  char* base = static_cast<char*>(h->d_scratch);
  auto carve = [&](size_t b) {
    char* p = base;
    base += (b + 255) & ~size_t(255);
    return p;
  };
  auto* d_graphs = reinterpret_cast<gtd::HeurGraph*>(carve(count * sizeof(gtd::HeurGraph)));
  auto* d_adj = reinterpret_cast<uint64_t*>(carve(2 * n_pool * sizeof(uint64_t)));
  auto* d_scores = scores_pool ? reinterpret_cast<float*>(carve(n_pool * sizeof(float))) : nullptr;
  auto* d_td = reinterpret_cast<int32_t*>(carve(size_t(count) * 4));
  auto* d_par = reinterpret_cast<int32_t*>(carve(n_pool * 4));
  cudaStream_t s = h->stream;
  GTD_CUDA(h, cudaMemcpyAsync(d_graphs, graphs.data(), count * sizeof(gtd::HeurGraph), cudaMemcpyHostToDevice, s));
  GTD_CUDA(h, cudaMemcpyAsync(d_adj, adj2_pool, 2 * n_pool * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  if (d_scores)
    GTD_CUDA(h, cudaMemcpyAsync(d_scores, scores_pool, n_pool * sizeof(float), cudaMemcpyHostToDevice, s));
  if (kind == 3) {
    const int blocks = std::min(4096, (count + gtd::kHWarps - 1) / gtd::kHWarps);
    gtd::heuristic_kernel<<<blocks, 32 * gtd::kHWarps, 0, s>>>(d_graphs, count, d_adj, d_scores, d_td, d_par);
  } else {
    const int threads = (max_n + 31) / 32 * 32;
    gtd::heuristic_rounds_kernel<<<count, kind == 0 ? 2 * threads : threads, 0, s>>>(d_graphs, d_adj, kind, threads,
                                                                                    d_td, d_par);
  }
  GTD_CUDA(h, cudaGetLastError());
  GTD_CUDA(h, cudaMemcpyAsync(td_out, d_td, size_t(count) * 4, cudaMemcpyDeviceToHost, s));
  GTD_CUDA(h, cudaMemcpyAsync(parent_out, d_par, n_pool * 4, cudaMemcpyDeviceToHost, s));
  GTD_CUDA(h, cudaStreamSynchronize(s));
  for (int i = 0; i < count; ++i)
    if (td_out[i] < 0) {  // masks that are not symmetric
      const size_t off = size_t(descs[i].offset);
      const gtd_status st = gtd_heuristic(adj2_pool + 2 * off, descs[i].n, kind, nullptr, td_out + i, parent_out + off);
      if (st != GTD_OK)
        return fail(h, st, "graph " + std::to_string(i));
    }
  return GTD_OK;
}
