// The bottom-up union-find heuristic DP on sm_103a.
//
// Reference: BottomUpHeuristicGPU (Treedepth/src/branch_and_bound/heuristics/
// bottom_up_heuristic.hpp:18-33) over BottomUpHeuristicGPUAlgorithm
// (bottom_up_heuristic_gpu_algorithm.cu:57-258). Level by level over subset
// sizes, every subset S keeps ONE elimination forest: the forest of a child
// S - v with v added as the root over the trees of its neighbours in S,
// for the first v (ascending) giving the least forest height. The last
// vertex added to each subset is kept for every level; GetElimination reads
// the last vertex of V, of V minus it, and so on, and the heuristic's tree is
// the elimination-tree replay of that order. It is the innermost heuristic of
// the reference's bnbGPU / bnbCPU incumbent chains (main.cpp:170-186).
//
// The reference runs one thread per subset with a union-find array per
// thread in shared memory (int8, n + 2 entries) and path-compressed Find.
// Here:
//  * A tree of the forest of S is a connected component of G[S] (adding v joins
//    exactly the trees that hold a neighbour of v), and only its height enters
//    the recurrence. With hc the height of the forest of S - v, adding v gives
//    hc + 1 if v has a neighbour in a tree of height hc, else hc. So a
//    candidate needs 8 bytes of its child: hc and the set of vertices in trees
//    of height hc (BuKey).
//  * The chosen candidate's forest is then carried over: the tree height of
//    every vertex as six bit planes of 32 vertices (BuRow, 24 bytes), v's new
//    tree found by a search in G[S], its height from the planes of v's
//    neighbours.
//  * One thread per subset; subsets of a level are ranked in colex order (the
//    reference's set_encoder), children are ranked while the subset is
//    unranked. One launch: chunks of a level by ticket, a chunk waits for the
//    count of finished chunks of the level below.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "gtd_handle.h"

namespace gtd {
namespace {

constexpr int kBuMaxN = GTD_BOTTOM_UP_MAX_N;  // 32: a set of vertices is one word
constexpr int kBuThreads = 256;
constexpr int kBuLow = 12;  // low vertices whose subsets are looked up instead of (un)ranked
constexpr int kBuPlanes = 6;  // heights 0..32

struct BuKey {
  uint32_t top;     // vertices in trees of the forest's height
  uint32_t height;  // of the forest (the empty set's: 1)
};
struct BuRow {
  uint2 pair[kBuPlanes / 2];  // bit b of every vertex's tree height: half b & 1 of pair[b / 2]
};

struct BuParams {
  uint32_t adj[kBuMaxN];        // adjacency masks
  int n = 0;
  int per_thread = 1;           // subsets per thread of a chunk
  uint32_t chunks = 0;          // tickets: chunks of all levels
  BuKey* keys[2] = {};          // by parity of the level
  BuRow* rows[2] = {};
  uint8_t* last = nullptr;      // history: last vertex of every subset, level-major
  uint32_t* ticket = nullptr;
  uint32_t* level_done = nullptr;
  int32_t* error = nullptr;
  uint64_t timeout_ns = 0;
  int32_t* order = nullptr;
};

using BuBinom = uint32_t[kBuMaxN + 1][kBuMaxN + 1];

// C(a, b), row by row by the first warp (column 32 holds only C(32, 32)).
__device__ __forceinline__ void bu_fill_binom(BuBinom& binom) {
  if (threadIdx.x < 32) {
    uint32_t c = threadIdx.x == 0 ? 1u : 0u;
    for (int a = 0; a <= kBuMaxN; ++a) {
      binom[a][threadIdx.x] = c;
      if (threadIdx.x == 0)
        binom[a][kBuMaxN] = a == kBuMaxN ? 1u : 0u;
      const uint32_t left = __shfl_up_sync(0xffffffffu, c, 1);
      if (threadIdx.x > 0)
        c += left;
    }
  }
}

// Bound by instruction issue (63 % of the slots, 28 warp instructions per
// subset at n = 26) and the latency of the key and row loads. A subset's low
// part is looked up in the list of the subsets of the low vertices by size, the
// ranks of its children in the inverse; a component search takes four lookups
// a round, of the joint neighbours of eight vertices each. n = 26: 53.8 ms with
// a warp per subset and 32-byte rows of roots, 2.73 with a thread per subset,
// 2.45 with the tables.
__global__ void __launch_bounds__(kBuThreads) bu_kernel(const __grid_constant__ BuParams p) {
  extern __shared__ uint32_t kid_rows[];  // child i of this thread's subset: kids[i * kBuThreads]
  __shared__ BuBinom binom;
  __shared__ uint32_t adj[kBuMaxN];
  __shared__ uint32_t joint[4][256];            // neighbours of any vertex of a set inside byte q
  __shared__ uint16_t low_set[1 << kBuLow];     // subsets of the low vertices by size, colex inside
  __shared__ uint16_t low_rank[1 << kBuLow];    // colex rank among those of its size
  __shared__ uint32_t low_off[kBuLow + 1];
  __shared__ uint32_t sTicket;
  __shared__ int sStop;
  const uint32_t tid = threadIdx.x;
  const int n = p.n;
  uint32_t* const kids = kid_rows + tid;
  bu_fill_binom(binom);
  if (tid < kBuMaxN)
    adj[tid] = p.adj[tid];
  __syncthreads();
  const int low_n = min(n, kBuLow);
  if (tid <= kBuLow) {
    uint32_t off = 0;
    for (int k = 0; k < static_cast<int>(tid); ++k)
      off += binom[low_n][k];
    low_off[tid] = off;
  }
  for (uint32_t i = tid; i < 4 * 256; i += kBuThreads) {
    uint32_t all = 0;
    for (uint32_t f = i & 255u; f; f &= f - 1)
      all |= adj[(i >> 8) * 8 + __ffs(static_cast<int>(f)) - 1];
    joint[i >> 8][i & 255u] = all;
  }
  __syncthreads();
  for (uint32_t w = tid; w < (1u << low_n); w += kBuThreads) {
    uint32_t rank = 0;
    int k = 0;
    for (uint32_t f = w; f; f &= f - 1)
      rank += binom[__ffs(static_cast<int>(f)) - 1][++k];
    low_rank[w] = static_cast<uint16_t>(rank);
    low_set[low_off[k] + rank] = static_cast<uint16_t>(w);
  }
  uint32_t ticket = 0;
  if (tid == 0)
    ticket = atomicAdd(p.ticket, 1u);
  const uint32_t chunk_size = kBuThreads * static_cast<uint32_t>(p.per_thread);
  int level = 0;                     // tickets only grow: the level of the last one and what lies below it
  uint32_t first_chunk = 0, chunks_prev = 0;
  uint32_t level_off = 0;            // subsets of the lower levels
  for (;;) {
    if (tid == 0)
      sTicket = ticket;
    __syncthreads();
    const uint32_t chunk = sTicket;
    if (chunk >= p.chunks)
      return;
    if (tid == 0)
      ticket = atomicAdd(p.ticket, 1u);
    for (;;) {
      const uint32_t count = binom[n][level], chunks = (count + chunk_size - 1u) / chunk_size;
      if (chunk - first_chunk < chunks)
        break;
      first_chunk += chunks;
      chunks_prev = chunks;
      level_off += count;
      ++level;
    }
    if (level > 0) {
      if (tid == 0)
        sStop = wait_count(p.level_done + (level - 1), chunks_prev, p.timeout_ns, p.error) ? 0 : 1;
      __syncthreads();
      if (sStop)
        return;
    }
    const uint32_t count = binom[n][level], begin = (chunk - first_chunk) * chunk_size;
    const BuKey* const keys = p.keys[(level & 1) ^ 1];
    const BuRow* const rows = p.rows[(level & 1) ^ 1];
    BuKey* const keys_out = p.keys[level & 1];
    BuRow* const rows_out = p.rows[level & 1];
    for (uint32_t rank = begin + tid; rank < count && rank - begin < chunk_size; rank += kBuThreads) {
      // unrank the high part (colex, descending), ranking the children S - a
      // on the way: the terms below a stay, those above shift down one place
      uint32_t S = 0, rest = rank, shifted = 0;
      int k = level;
      {
        uint32_t* at = kids;
        for (int a = n - 1; a >= low_n; --a) {  // k = 0: C(a, 0) = 1 > rest = 0
          const uint32_t c = binom[a][k], d = binom[a][max(k - 1, 0)];
          if (rest >= c) {
            rest -= c;
            S |= 1u << a;
            *at = rest + shifted;
            at += kBuThreads;
            shifted += d;
            --k;
          }
        }
      }
      uint32_t low = low_set[low_off[k] + rest];
      const int high_count = level - k;
      uint32_t todo = S;
      S |= low;
      if (level == 0) {
        keys_out[0] = BuKey{0u, 1u};
        rows_out[0] = BuRow{};
        p.last[0] = 0xFF;
        continue;
      }
      // the first v with the least height; the children run from the largest v
      // down, so the last one at the least wins. Four loads in flight.
      uint32_t best = 0xFFFFFFFFu, v = 0, kid = 0, top = 0;
      auto consider = [&](const uint2& key, uint32_t child, int a) {
        const uint32_t h = key.y + ((key.x & adj[a]) ? 1u : 0u);
        if (h <= best) {
          best = h;
          v = static_cast<uint32_t>(a);
          kid = child;
          top = key.x;
        }
      };
      auto key_of = [&](uint32_t child) { return __ldcg(reinterpret_cast<const uint2*>(keys) + child); };
      for (int i = 0; i < high_count; i += 4) {
        uint32_t c[4];
        uint2 key[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + u < high_count) {
            c[u] = kids[(i + u) * kBuThreads];
            key[u] = key_of(c[u]);
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i + u < high_count) {
            const int a = 31 - __clz(static_cast<int>(todo));
            todo ^= 1u << a;
            consider(key[u], c[u], a);
          }
      }
      todo = low;
      while (todo) {
        uint32_t c[4], bit[4];
        uint2 key[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          bit[u] = todo ? 0x80000000u >> __clz(static_cast<int>(todo)) : 0u;
          todo ^= bit[u];
          if (bit[u]) {
            c[u] = shifted + low_rank[low ^ bit[u]];
            key[u] = key_of(c[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (bit[u])
            consider(key[u], c[u], 31 - __clz(static_cast<int>(bit[u])));
      }
      uint32_t plane[kBuPlanes];
#pragma unroll
      for (int b = 0; b < kBuPlanes / 2; ++b) {
        const uint2 x = __ldcg(&rows[kid].pair[b]);
        plane[2 * b] = x.x;
        plane[2 * b + 1] = x.y;
      }
      // v's tree: its component in G[S]
      const uint32_t nbrs = adj[v] & S;
      uint32_t tree = 1u << v, front = nbrs;
      while (front) {
        tree |= front;
        if (tree == S)
          break;
        front = (joint[0][front & 255u] | joint[1][front >> 8 & 255u] | joint[2][front >> 16 & 255u] |
                 joint[3][front >> 24]) & S & ~tree;
      }
      // its height: one more than the greatest among v's neighbours
      uint32_t m = 0, at_most = nbrs;
#pragma unroll
      for (int b = kBuPlanes - 1; b >= 0; --b)
        if (at_most & plane[b]) {
          at_most &= plane[b];
          m |= 1u << b;
        }
      ++m;
      // top: those that were there stay unless the height grew; v's tree joins
      // when it has the forest's height
      const uint32_t new_top = m == best ? ((best == m && (top & nbrs)) ? tree : top | tree) : top;
      BuRow out;
#pragma unroll
      for (int b = 0; b < kBuPlanes; ++b)
        plane[b] = (plane[b] & ~tree) | ((m >> b & 1u) ? tree : 0u);
#pragma unroll
      for (int b = 0; b < kBuPlanes / 2; ++b)
        out.pair[b] = make_uint2(plane[2 * b], plane[2 * b + 1]);
      keys_out[rank] = BuKey{new_top, best};
      rows_out[rank] = out;
      p.last[level_off + rank] = static_cast<uint8_t>(v);
    }
    // as in dp_level_kernel: stores, barrier, release count
    __syncthreads();
    if (tid == 0 && level < n)
      red_release_add_u32(p.level_done + level, 1u);
  }
}

// GetElimination(n, n, 0) (bottom_up_heuristic_gpu_algorithm.hpp:104-120):
// the last vertex of the remaining set, level by level down from V. One warp:
// lane b ranks bit b.
__global__ void __launch_bounds__(32) bu_order_kernel(const __grid_constant__ BuParams p) {
  __shared__ BuBinom binom;
  const uint32_t lane = threadIdx.x;
  bu_fill_binom(binom);
  __syncwarp();
  const int n = p.n;
  uint32_t S = n == 32 ? 0xffffffffu : ((1u << n) - 1u), off = 0;
  for (int i = static_cast<int>(lane); i < n; i += 32)
    off += binom[n][i];
  off = __reduce_add_sync(0xffffffffu, off);  // first history entry of level n
  for (int step = 0; step < n; ++step) {
    const uint32_t below = __popc(S & ((1u << lane) - 1u));
    const uint32_t rank = __reduce_add_sync(0xffffffffu, (S >> lane & 1u) ? binom[lane][below + 1] : 0u);
    const uint32_t v = __ldcg(p.last + off + rank) & 31u;
    if (lane == 0)
      p.order[step] = static_cast<int32_t>(v);
    S &= ~(1u << v);
    off -= binom[n][n - step - 1];
  }
}

uint64_t binom64(int a, int b) {
  if (b < 0 || b > a)
    return 0;
  uint64_t r = 1;
  for (int i = 1; i <= b; ++i)
    r = r * uint64_t(a - b + i) / uint64_t(i);
  return r;
}

// The elimination-tree replay of an order (elimination_tree.cpp:24-70, as
// BottomUpHeuristicGPU::Get eliminates its order): each vertex's parent is
// the last eliminated vertex whose component contained it.
int replay_order(const uint64_t* adj, int n, const int32_t* order, int32_t* parent) {
  uint64_t remaining = n == 64 ? ~0ull : ((1ull << n) - 1);
  std::vector<int> owner(n, -1), depth(n, 0);
  int height = 0;
  for (int i = 0; i < n; ++i) {
    const int v = order[i];
    if (v < 0 || v >= n || !((remaining >> v) & 1ull))
      return -1;
    parent[v] = owner[v];
    height = std::max(height, depth[v] + 1);
    uint64_t reach = 1ull << v, frontier = reach;
    while (frontier) {
      uint64_t nb = 0;
      for (uint64_t f = frontier; f; f &= f - 1)
        nb |= adj[__builtin_ctzll(f)];
      nb &= remaining & ~reach;
      reach |= nb;
      frontier = nb;
    }
    remaining &= ~(1ull << v);
    for (uint64_t s = reach & ~(1ull << v); s; s &= s - 1) {
      const int u = __builtin_ctzll(s);
      owner[u] = v;
      depth[u] = depth[v] + 1;
    }
  }
  return height;
}

}  // namespace
}  // namespace gtd

using namespace gtd;

extern "C" gtd_status gtd_bottom_up(gtd_handle h, const uint64_t* adj, int n, int32_t* td_out, int32_t* parent_out,
                                    int32_t* order_out) {
  if (!h)
    return GTD_INVALID_ARG;
  if (!adj || !td_out || !parent_out)
    return fail(h, GTD_INVALID_ARG, "null pointer argument");
  if (n < 1)
    return fail(h, GTD_INVALID_ARG, "n must be at least 1");
  if (n > kBuMaxN)
    return fail(h, GTD_NO_RESULT, "the bottom-up heuristic keeps sets of vertices in 32-bit words: n <= " +
                                      std::to_string(kBuMaxN));
  gtd_status s = check_adjacency(h, adj, n);
  if (s != GTD_OK)
    return s;
  DeviceGuard guard(h->device);
  uint64_t max_c = 0;
  for (int k = 0; k <= n; ++k)
    max_c = std::max(max_c, binom64(n, k));
  // [rows, two levels][keys, two levels][history][order]
  const size_t rows = max_c * sizeof(BuRow), keys = max_c * sizeof(BuKey), hist = size_t(1) << n;
  const size_t off_keys = 2 * rows, off_hist = off_keys + 2 * keys;
  const size_t off_order = (off_hist + hist + 15) & ~size_t(15);
  GTD_CUDA(h, ensure_field(&h->d_bu, &h->bu_cap, off_order + 64 * sizeof(int32_t)));
  uint8_t* base = h->d_bu;

  BuParams p;
  for (int v = 0; v < kBuMaxN; ++v)
    p.adj[v] = v < n ? static_cast<uint32_t>(adj[v]) : 0u;
  p.n = n;
  p.per_thread = n >= 24 ? 4 : 1;  // wide levels: fewer tickets and counts
  const uint64_t chunk = uint64_t(kBuThreads) * p.per_thread;
  for (int k = 0; k <= n; ++k)
    p.chunks += static_cast<uint32_t>((binom64(n, k) + chunk - 1) / chunk);
  for (int i = 0; i < 2; ++i) {
    p.rows[i] = reinterpret_cast<BuRow*>(base + i * rows);
    p.keys[i] = reinterpret_cast<BuKey*>(base + off_keys + i * keys);
  }
  p.last = base + off_hist;
  p.order = reinterpret_cast<int32_t*>(base + off_order);
  p.ticket = reinterpret_cast<uint32_t*>(h->d_io + kIoTicket);
  p.level_done = reinterpret_cast<uint32_t*>(h->d_io + kIoLevels);
  p.error = h->d_io + kIoError;
  p.timeout_ns = 10ull * 1000 * 1000 * 1000;
  const size_t smem = sizeof(uint32_t) * kBuThreads * size_t(n > kBuLow ? n - kBuLow : 0);
  int occ = 0;
  GTD_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, bu_kernel, kBuThreads, smem));
  const unsigned ctas = static_cast<unsigned>(
      std::min<uint64_t>(uint64_t(h->num_sms) * static_cast<unsigned>(std::max(1, occ)), p.chunks));
  // a solve enqueued before may not have been asked for its errors yet: its
  // words outlive this call, which has its own in their place meanwhile
  int32_t* const kept = reinterpret_cast<int32_t*>(static_cast<char*>(h->h_pinned) + kPinnedError);
  if (h->uncollected)
    GTD_CUDA(h, cudaMemcpyAsync(kept, h->d_io + kIoError, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
  GTD_CUDA(h, cudaMemsetAsync(h->d_io, 0, kIoWords * sizeof(int32_t), h->stream));
  GTD_CUDA(h, cudaEventRecord(h->ev[0], h->stream));
  bu_kernel<<<ctas, kBuThreads, smem, h->stream>>>(p);
  GTD_CUDA(h, cudaGetLastError());
  bu_order_kernel<<<1, 32, 0, h->stream>>>(p);
  GTD_CUDA(h, cudaGetLastError());
  GTD_CUDA(h, cudaEventRecord(h->ev[1], h->stream));
  std::vector<int32_t> order(n);
  int32_t io[4] = {0, 0, 0, 0};
  GTD_CUDA(h, cudaMemcpyAsync(order.data(), p.order, n * sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
  GTD_CUDA(h, cudaMemcpyAsync(io, h->d_io, sizeof(io), cudaMemcpyDeviceToHost, h->stream));
  if (h->uncollected)  // the words kept have arrived by the time these are put back
    GTD_CUDA(h, cudaMemcpyAsync(h->d_io + kIoError, kept, 2 * sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
  GTD_CUDA(h, cudaStreamSynchronize(h->stream));
  s = map_device_error(h, io[kIoError], io[kIoError + 1]);
  if (s != GTD_OK)
    return s;
  const int height = replay_order(adj, n, order.data(), parent_out);
  if (height < 0)
    return fail(h, GTD_ABORTED, "the bottom-up order is not a permutation");
  *td_out = height;
  if (order_out)
    std::memcpy(order_out, order.data(), n * sizeof(int32_t));
  return GTD_OK;
}
