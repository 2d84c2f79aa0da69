// K1: the level-by-level subset DP for exact treedepth on sm_103a.
//
// Reference: DynamicGPU (Treedepth/src/dynamic_gpu/dynamic_gpu.cu:40-201),
// which runs one thread per k-subset per level, labels components by repeated
// CSR sweeps, re-encodes S - v with 64-bit divides and gathers 8-byte
// {td, root} entries at random. This kernel computes the same values with a
// different schedule and layout:
//
//  * Recurrence. For |S| >= 3, S is connected iff at least two v in S leave
//    S - v connected (a connected graph has >= 2 non-cut vertices, and if
//    S - u and S - v are connected, u has a neighbour in S - v). For a
//    disconnected S, td(S) = max_v td(S - v) (treedepth is monotone under
//    vertex deletion, and deleting a vertex outside a deepest component keeps
//    it). So every subset is resolved from its |S| children S - v alone:
//      T[S] = 1 + min_v T[S - v]   (connected; dynamic_gpu.cu:68-89)
//      T[S] = max_v T[S - v]       (disconnected; = max over components,
//                                   dynamic_gpu.cu:90-111)
//    No per-subset BFS, no ranking per child.
//  * Bit slicing. Deleting a vertex lowers treedepth by at most one, so the
//    children's treedepths are a or a + 1 with a = td(S) - 1 or td(S), and
//    residues modulo 3 tell which: the table keeps three bits per subset
//    (planes "td = 0 mod 3", "td = 1 mod 3", "connected"), 32 subsets per
//    word. Children are reduced by OR per residue and a two-bit saturating
//    count of connected ones: 3.5 logic operations per child and 32 subsets,
//    where one byte per subset took 2 per child and 4 subsets (2.67 times
//    the bytes from L2 and DRAM too). Full treedepths are read back along a
//    chain of deletions (chain_td).
//  * Layout (gtd_dp_layout.h). Tiles of 2^lb subsets share a high part H; a
//    tile is its three planes, 2^(lb-5) words each. The cross-tile children
//    are whole tiles H - h one level down, read as 16-byte vectors; the
//    in-tile children are other words of the tile, resolved in popcount order
//    of the word index; the five lowest vertices live inside the word. There
//    the children of a subset are shifts of the word itself, one round per
//    subset size; four tiles are resolved together (resolve_quad), their
//    words transposed by bytes so that only three vertices are left inside.
//  * Schedule. One persistent launch; a CTA takes a group of consecutive
//    tiles of one level by ticket (atomicAdd, level-major), unranks them one
//    per thread, checks the ready flags of their children's groups, reduces
//    the cross-tile children, resolves the tiles in shared memory, stores
//    them and publishes the group's flag with a release store. A group only
//    waits on groups with smaller tickets, and tickets are only taken by
//    running CTAs, so the smallest unfinished ticket can always proceed; each
//    wait is bounded by a deadline.
//
// Reconstruction (dp_tree_kernel): one warp, one lane per vertex, rebuilds
// the reference's tree (first-argmin root per component, dynamic_gpu.cu:84-87,
// dynamic_cpu.hpp:59-81) and GetElimination order (dynamic_gpu.hpp:48-64).
#include <cuda_runtime.h>

#include <cstdint>

#include "gtd_device.cuh"
#include "gtd_dp_kernels.h"

namespace gtd {

// A group of tiles of LB bits in shared memory: five planes of kWords x
// kGroup words (the cross-tile children's summary: residues 0, 1, 2 present,
// at least one and at least two connected; the first three then receive the
// tiles).
template <int LB>
struct TileShape {
  static constexpr uint32_t kWords = 1u << (LB - 5);         // words of a plane of a tile
  static constexpr uint32_t kGroup = dp_group_tiles(LB);     // tiles of a group
  static constexpr uint32_t kQuads = kGroup / 4;             // sets of four tiles resolved together
  static constexpr uint32_t kPlane = kWords * kGroup;
  static constexpr uint32_t kChunks = kWords / 4;            // 16-byte parts of a plane of a tile
  static constexpr uint32_t kTileBytes = dp_tile_bytes(LB);
};

using Binom = uint32_t[kDpMaxHigh + 1][kDpMaxHigh + 1];

// Offset of word w of tile q in a shared-memory plane. The four tiles of a
// quad are adjacent (one 16-byte access in the in-tile phase, a warp on one w
// covers a row); the quads of a row are permuted by the word's chunk so that
// the chunk-wise accesses of the other phases spread over the banks.
template <int LB>
__device__ __forceinline__ uint32_t plane_at(uint32_t q, uint32_t w) {
  using Shape = TileShape<LB>;
  constexpr uint32_t kStep = Shape::kChunks >= 8 ? 4u : 32u / Shape::kChunks;
  return (w * Shape::kGroup + q) ^ (((w >> 2) * kStep) & 28u);
}

// What the children of 32 subsets have: residue k of their treedepths
// present (o0, o1, o2), at least one (c1) and two (c2) connected.
struct Acc {
  uint32_t o0 = 0u, o1 = 0u, o2 = 0u, c1 = 0u, c2 = 0u;
};

__device__ __forceinline__ void acc_add1(Acc& a, uint32_t p0, uint32_t p1, uint32_t c) {
  a.o0 |= p0;
  a.o1 |= p1;
  a.o2 |= ~(p0 | p1);
  a.c2 |= a.c1 & c;
  a.c1 |= c;
}

__device__ __forceinline__ void acc_add2(Acc& a, uint32_t p0, uint32_t p1, uint32_t c, uint32_t q0, uint32_t q1,
                                         uint32_t d) {
  a.o0 |= p0 | q0;
  a.o1 |= p1 | q1;
  a.o2 |= ~(p0 | p1);
  a.o2 |= ~(q0 | q1);
  a.c2 |= (a.c1 & (c | d)) | (c & d);
  a.c1 |= c | d;
}

struct Planes {
  uint32_t p0, p1, c;
};

// The binomial table (C(a, b) = 0 for b > a), row by row by the first warp; a
// CTA barrier must follow.
__device__ __forceinline__ void fill_binom(Binom& binom) {
  if (threadIdx.x < 32) {
    uint32_t c = threadIdx.x == 0 ? 1u : 0u;
    for (int a = 0; a <= kDpMaxHigh; ++a) {
      if (threadIdx.x <= kDpMaxHigh)
        binom[a][threadIdx.x] = c;
      const uint32_t left = __shfl_up_sync(0xffffffffu, c, 1);
      if (threadIdx.x > 0)
        c += left;
    }
  }
}

// Connectivity of the subsets of size <= 2 of a word (the count of connected
// children only decides it from size 3 on): conn = (count & keep) | set.
struct SmallSets {
  uint32_t keep = 0xFFFFFFFFu, set = 0u, zero = 0u;  // zero: the empty set's position (td 0)
};

// Residues of the subsets: 1 + min over the children when connected, else
// the max; the children hold a and possibly a + 1, so residue k is the result
// iff k + 1 is absent and (connected) k - 1 or (disconnected) k is present.
__device__ __forceinline__ Planes finish(const Acc& a, const SmallSets& s) {
  Planes r;
  r.c = (a.c2 & s.keep) | s.set;
  r.p0 = (~a.o1 & ((r.c & a.o2) | (~r.c & a.o0))) | s.zero;
  r.p1 = ~a.o2 & ((r.c & a.o0) | (~r.c & a.o1));
  return r;
}

// Four sets of 8 subsets, one per byte, each over the three lowest vertices
// (position x in the byte = the subset x), from the summary of their other
// children, by size of x: position 0; its broadcast to positions 1, 2, 4;
// 3, 5, 6 from those by one shift per vertex; 7 from 3, 5, 6.
__device__ __forceinline__ Planes resolve_octets(const Acc& ext, const SmallSets& s) {
  Planes r = finish(ext, s);
  Acc a = ext;
  a.o0 |= (r.p0 & 0x01010101u) * 0x16u;
  a.o1 |= (r.p1 & 0x01010101u) * 0x16u;
  a.o2 |= (~(r.p0 | r.p1) & 0x01010101u) * 0x16u;
  a.c2 |= a.c1 & ((r.c & 0x01010101u) * 0x16u);
  r = finish(a, s);

  constexpr uint32_t kHas0 = 0xAAAAAAAAu, kHas1 = 0xCCCCCCCCu, kHas2 = 0xF0F0F0F0u;
  uint32_t p2 = ~(r.p0 | r.p1);
  a = ext;
  a.o0 |= (r.p0 << 1) & kHas0;
  a.o1 |= (r.p1 << 1) & kHas0;
  a.o2 |= (p2 << 1) & kHas0;
  a.o0 |= (r.p0 << 2) & kHas1;
  a.o1 |= (r.p1 << 2) & kHas1;
  a.o2 |= (p2 << 2) & kHas1;
  a.o0 |= (r.p0 << 4) & kHas2;
  a.o1 |= (r.p1 << 4) & kHas2;
  a.o2 |= (p2 << 4) & kHas2;
  {
    const uint32_t x = (r.c << 1) & kHas0, y = (r.c << 2) & kHas1, z = (r.c << 4) & kHas2;
    a.c2 |= ((x & y) | (x & z) | (y & z)) | (a.c1 & (x | y | z));
  }
  r = finish(a, s);

  // bits 3, 5, 6 of a byte plus 0x78 carry into its bit 7 iff one is set
  constexpr uint32_t kPairs = 0x68686868u, kCarry = 0x78787878u, kTop = 0x80808080u;
  p2 = ~(r.p0 | r.p1);
  a = ext;
  a.o0 |= ((r.p0 & kPairs) + kCarry) & kTop;
  a.o1 |= ((r.p1 & kPairs) + kCarry) & kTop;
  a.o2 |= ((p2 & kPairs) + kCarry) & kTop;
  {
    const uint32_t x = r.c << 4, y = r.c << 2, z = r.c << 1;
    a.c2 |= (((x & y) | (x & z) | (y & z)) | (a.c1 & (x | y | z))) & kTop;
  }
  const Planes t = finish(a, s);
  r.p0 = (r.p0 & ~kTop) | (t.p0 & kTop);
  r.p1 = (r.p1 & ~kTop) | (t.p1 & kTop);
  r.c = (r.c & ~kTop) | (t.c & kTop);
  return r;
}

// Byte t of x[b] to byte b of x[t].
__device__ __forceinline__ void transpose_bytes(uint32_t& x0, uint32_t& x1, uint32_t& x2, uint32_t& x3) {
  const uint32_t a = __byte_perm(x0, x1, 0x5140u), b = __byte_perm(x2, x3, 0x5140u);
  const uint32_t c = __byte_perm(x0, x1, 0x7362u), d = __byte_perm(x2, x3, 0x7362u);
  x0 = __byte_perm(a, b, 0x5410u);
  x1 = __byte_perm(a, b, 0x7632u);
  x2 = __byte_perm(c, d, 0x5410u);
  x3 = __byte_perm(c, d, 0x7632u);
}

// The word of four tiles (32 subsets each, the five lowest vertices inside
// the word) from the summary a[b] of tile b's children outside the word.
// Byte t of a word holds the subsets whose vertices 3 and 4 are the bits of
// t: after a byte transpose a[t] holds them for all four tiles, t = 0 is a
// child of t = 1 and 2, and those are of 3. Resolving the words one by one
// with all five vertices inside takes three rounds of five shifts instead of
// this one round of three per octet: 210 operations a word against 120.
__device__ __forceinline__ void resolve_quad(Acc (&a)[4], SmallSets (&s)[4], Planes (&r)[4]) {
  transpose_bytes(a[0].o0, a[1].o0, a[2].o0, a[3].o0);
  transpose_bytes(a[0].o1, a[1].o1, a[2].o1, a[3].o1);
  transpose_bytes(a[0].o2, a[1].o2, a[2].o2, a[3].o2);
  transpose_bytes(a[0].c1, a[1].c1, a[2].c1, a[3].c1);
  transpose_bytes(a[0].c2, a[1].c2, a[2].c2, a[3].c2);
  transpose_bytes(s[0].keep, s[1].keep, s[2].keep, s[3].keep);
  transpose_bytes(s[0].set, s[1].set, s[2].set, s[3].set);
  transpose_bytes(s[0].zero, s[1].zero, s[2].zero, s[3].zero);
  r[0] = resolve_octets(a[0], s[0]);
  acc_add1(a[1], r[0].p0, r[0].p1, r[0].c);
  r[1] = resolve_octets(a[1], s[1]);
  acc_add1(a[2], r[0].p0, r[0].p1, r[0].c);
  r[2] = resolve_octets(a[2], s[2]);
  acc_add2(a[3], r[1].p0, r[1].p1, r[1].c, r[2].p0, r[2].p1, r[2].c);
  r[3] = resolve_octets(a[3], s[3]);
  transpose_bytes(r[0].p0, r[1].p0, r[2].p0, r[3].p0);
  transpose_bytes(r[0].p1, r[1].p1, r[2].p1, r[3].p1);
  transpose_bytes(r[0].c, r[1].c, r[2].c, r[3].c);
}

// Bits 0..4 to the positions of the singles.
__device__ __forceinline__ uint32_t spread5(uint32_t a) {
  return (a & 1u) << 1 | (a & 2u) << 1 | (a & 4u) << 2 | (a & 8u) << 5 | (a & 16u) << 12;
}

// SmallSets of the word whose position 0 is the set S0 of k <= 2 vertices
// >= 5 (vertices >= n are padding, isolated).
__device__ __noinline__ SmallSets small_sets(uint64_t S0, int k, const uint64_t* adj, int n) {
  auto at = [&](int v) -> uint64_t { return v < n ? adj[v] : 0ull; };
  constexpr uint32_t kSingles = 0x00010116u, kPairs = 0x01161668u;  // |x| = 1, 2
  SmallSets s;
  if (k == 2) {
    const int u = __ffsll(static_cast<long long>(S0)) - 1, v = 63 - __clzll(static_cast<long long>(S0));
    s.keep = ~1u;
    s.set = static_cast<uint32_t>(at(u) >> v) & 1u;
  } else if (k == 1) {
    s.keep = ~(1u | kSingles);
    s.set = 1u | spread5(static_cast<uint32_t>(at(__ffsll(static_cast<long long>(S0)) - 1)));
  } else {
    s.keep = ~(1u | kSingles | kPairs);
    s.set = kSingles;
    for (int i = 1; i < 5; ++i)
      s.set |= spread5(static_cast<uint32_t>(at(i)) & ((1u << i) - 1u)) << (1u << i);
    s.zero = 1u;
  }
  return s;
}

__device__ __forceinline__ uint32_t rank_colex(const Binom& binom, uint32_t H) {
  uint32_t r = 0;
  int q = 0;
  for (; H; H &= H - 1)
    r += binom[__ffs(H) - 1][++q];
  return r;
}

// Are a graph's adjacency masks well formed — no self loop, no bit >= n,
// symmetric? Whole warp, lane v checking vertex v (and v + 32).
__device__ __forceinline__ bool adjacency_ok(const uint64_t* adj, int n) {
  const uint64_t allowed = n >= 64 ? ~0ull : ((1ull << n) - 1);
  bool ok = true;
  for (int v = threadIdx.x & 31; v < n && ok; v += 32) {
    const uint64_t a = adj[v];
    if (((a >> v) & 1ull) || (a & ~allowed))
      ok = false;
    for (uint64_t s = a; s && ok; s &= s - 1)
      if (!((adj[__ffsll(static_cast<long long>(s)) - 1] >> v) & 1ull))
        ok = false;
  }
  return __all_sync(0xffffffffu, ok);
}

// What the first kernel of a single solve does with its input (one CTA; a
// barrier before the adjacency or the control words are used). Together with
// results written to pinned memory by the last kernel, a copy in, a memset, a
// copy out and an event fewer per call (n = 12: 50 -> 37 us, n = 20: 104 -> 95).
__device__ __forceinline__ void take_input(const DpBatchParams& p, const DpInput& in) {
  for (int i = threadIdx.x; i < in.clear_words; i += blockDim.x)
    in.clear[i] = 0;
  if (in.by_value && threadIdx.x < p.single.n)
    const_cast<uint64_t*>(p.adj)[threadIdx.x] = in.adj[threadIdx.x];
}

// Checks every graph, one warp per graph.
__global__ void dp_validate_kernel(const __grid_constant__ DpBatchParams p, const __grid_constant__ DpInput in) {
  if (!p.graphs) {
    take_input(p, in);
    __syncthreads();
  }
  const int g = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (g >= p.num_graphs)
    return;  // the whole warp
  const DpGraph G = p.graphs ? p.graphs[g] : p.single;
  if (!adjacency_ok(p.adj + G.adj_off, G.n) && (threadIdx.x & 31) == 0)
    raise_error(p.error, kDevInvalidInput, g);
}

// Batches issue tickets level-major across graphs (every graph's level-0
// groups, then every level-1 group, ...), so that a tile's children lie far
// back in the ticket stream; tables and flags stay graph-major.
__global__ void dp_fill_tile_map_kernel(const __grid_constant__ DpBatchParams p) {
  __shared__ Binom binom;
  fill_binom(binom);
  __syncthreads();
  for (int g = blockIdx.x; g < p.num_graphs; g += gridDim.x) {
    const DpGraph G = p.graphs[g];
    const uint32_t per = dp_chunk_tiles(G.lb);
    uint32_t local = 0;
    for (int j = 0; j <= G.nh; ++j) {
      const uint32_t count = (binom[G.nh][j] + per - 1u) / per;
      const uint32_t base = p.level_base[size_t(g) * (kDpMaxHigh + 2) + j];
      for (uint32_t i = threadIdx.x; i < count; i += blockDim.x)
        p.tile_map[base + i] = make_uint2(static_cast<uint32_t>(g), local + i);
      local += count;
    }
  }
}

// Word indices of `bits` bits ordered by popcount, colex rank inside each
// popcount class. For a tile of fewer word bits the words of class s are the
// first C(wb, s) entries of the class (colex order lists the subsets of the
// lower positions first), so one table serves every smaller tile size.
__device__ void build_word_order(uint8_t* sOrder, const Binom& binom, int bits) {
  for (int w = threadIdx.x; w < (1 << bits); w += blockDim.x) {
    const int i = __popc(w);
    uint32_t pos = 0;
    for (int q = 0; q < i; ++q)
      pos += binom[bits][q];
    pos += rank_colex(binom, static_cast<uint32_t>(w));
    sOrder[pos] = static_cast<uint8_t>(w);
  }
}

__device__ __forceinline__ uint4 ldcg128(const uint8_t* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }

// Dynamic shared memory of a launch: the planes of a group, the child lists
// (kid_rows children of every tile of a group, the launch's largest number of
// high vertices), the tiles' high parts, the binomial table, the word order.
struct SmemLayout {
  uint32_t kids_off, high_off, binom_off, order_off, bytes;
};

__host__ __device__ constexpr SmemLayout smem_layout(uint32_t plane_words, uint32_t tiles, int kid_rows,
                                                     int order_bits) {
  SmemLayout s{};
  s.kids_off = 5u * 4u * plane_words;
  s.high_off = s.kids_off + 4u * tiles * static_cast<uint32_t>(kid_rows);
  s.binom_off = s.high_off + 4u * tiles;
  s.order_off = s.binom_off + static_cast<uint32_t>(sizeof(Binom));
  s.bytes = s.order_off + (1u << order_bits);
  return s;
}

// Tiles of up to lb bits (min_lb = lb: the launch's only size).
__host__ __device__ constexpr SmemLayout smem_layout_for(int min_lb, int lb, int kid_rows) {
  uint32_t planes = 0, tiles = 0;
  for (int b = min_lb; b <= lb; ++b) {
    const uint32_t t = dp_group_tiles(b);
    tiles = t > tiles ? t : tiles;
    planes = (t << (b - 5)) > planes ? (t << (b - 5)) : planes;
  }
  return smem_layout(planes, tiles, kid_rows, lb - 5);
}

struct Workspace {
  uint32_t* planes;
  uint32_t* kids;
  uint32_t* high;
  const Binom& binom;
  const uint8_t* order;  // word order table of order_bits bits
  int order_bits;
};

__device__ __forceinline__ Workspace make_workspace(const DpBatchParams& p, const SmemLayout& L, int order_bits) {
  extern __shared__ __align__(16) uint8_t smem[];
  Binom& sBinom = *reinterpret_cast<Binom*>(smem + L.binom_off);
  fill_binom(sBinom);
  __syncthreads();
  build_word_order(smem + L.order_off, sBinom, order_bits);
  return Workspace{reinterpret_cast<uint32_t*>(smem), reinterpret_cast<uint32_t*>(smem + L.kids_off),
                   reinterpret_cast<uint32_t*>(smem + L.high_off), sBinom, smem + L.order_off, order_bits};
}

// The CTA resolves group `group` of graph G (tiles of LB bits, level-major
// group numbers): waits for its child tiles' groups, reduces them, resolves
// the tiles in shared memory and stores them; the caller publishes the group
// after a CTA barrier. False (for every thread) if a wait gave up.
//
// Bound by latency: 37 % of issue slots at n = 30 (16 warps per SM, as many as
// shared memory and registers take), a group's time going to unranking and
// flags (15 %), the gathers (27 %), the classes of the in-tile phase (33 %)
// and waits at the narrow levels (16 %). 8.5 warp instructions per word of 32
// subsets; the kernel alone takes 0.68 ms at n = 30 and 4.7 ms at n = 33 (whole
// calls one after another 0.73 and 4.82; at one byte per subset and one warp per
// tile, 1.52 warp instructions per subset: 1.92 and 14.9 ms). Tried
// and not kept: a warp per group (0.91 ms), 64 threads per CTA (0.79), the next
// group unranked by an idle warp beside the in-tile phase (0.72 and 5.2).
template <int LB>
__device__ __forceinline__ bool group_work(const DpBatchParams& p, const DpGraph& G, uint32_t group,
                                           const Workspace& ws) {
  using Shape = TileShape<LB>;
  constexpr uint32_t kQ = Shape::kGroup, kW = Shape::kWords, kPlane = Shape::kPlane, kChunks = Shape::kChunks;
  constexpr int kWordBits = LB - 5;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  uint8_t* const table = p.table + G.table_off;
  const uint32_t* const flags = p.flags + G.flag_base;
  const Binom& binom = ws.binom;
  const int nh = G.nh;

  // Level j of the group: running totals over the levels, lane i holding the
  // tiles (cumT) and groups (cumG) of levels 0..i (every warp alike).
  const uint32_t level_tiles = static_cast<int>(lane) <= nh ? binom[nh][lane] : 0u;
  uint32_t cumT = level_tiles, cumG = (level_tiles + kQ - 1u) / kQ;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, cumT, d);
    const uint32_t y = __shfl_up_sync(0xffffffffu, cumG, d);
    if (static_cast<int>(lane) >= d) {
      cumT += x;
      cumG += y;
    }
  }
  const int j = __popc(__ballot_sync(0xffffffffu, static_cast<int>(lane) <= nh && cumG <= group));
  const uint32_t tiles_j = __shfl_sync(0xffffffffu, level_tiles, j);
  uint32_t off_j = __shfl_sync(0xffffffffu, cumT, (j + 31) & 31);        // first tile of level j
  uint32_t groups_j = __shfl_sync(0xffffffffu, cumG, (j + 31) & 31);     // first group of level j
  uint32_t off_prev = __shfl_sync(0xffffffffu, cumT, (j + 30) & 31);     // ... of level j - 1
  uint32_t groups_prev = __shfl_sync(0xffffffffu, cumG, (j + 30) & 31);
  if (j < 1)
    off_j = groups_j = 0u;
  if (j < 2)
    off_prev = groups_prev = 0u;
  const uint32_t r0 = (group - groups_j) * kQ;          // rank of the first tile in its level
  const uint32_t count = min(kQ, tiles_j - r0);

  // Thread q unranks tile r0 + q (colex, descending) and ranks its children
  // on the way: deleting element a keeps the terms below it (`rest`) and
  // shifts those above down one place (`shifted`). Child i of tile q:
  // kids[i * kQ + q].
  if (tid < count) {
    uint32_t rest = r0 + tid, kid = off_prev, at = tid, H = 0;  // kid: off_prev + `shifted`
    int k = j;
    for (int a = nh - 1; a >= 0; --a) {  // k = 0: C(a, 0) = 1 > rest = 0
      const uint32_t c = binom[a][k], d = binom[a][max(k - 1, 0)];
      if (rest >= c) {
        rest -= c;
        H |= 1u << a;
        ws.kids[at] = kid + rest;
        at += kQ;
        kid += d;
        --k;
      }
    }
    ws.high[tid] = H;
  }
  __syncthreads();

  // The children's groups: every thread looks at some (tile, child) pairs,
  // four loads in flight. Relaxed flag loads followed by a gpu-scope fence
  // acquire the groups whose flags they read; the barrier hands that to every
  // thread.
  const uint32_t pairs = static_cast<uint32_t>(j) * kQ;
  auto flag_of = [&](uint32_t i) { return flags + groups_prev + (ws.kids[i] - off_prev) / kQ; };
  bool ok = true;
  for (uint32_t i0 = tid; i0 < pairs; i0 += 4 * kDpThreads) {
    uint32_t seen[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) {
      const uint32_t i = i0 + u * kDpThreads;
      seen[u] = i < pairs && i % kQ < count ? ld_relaxed_u32(flag_of(i)) : p.epoch;
    }
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u)
      ok &= seen[u] == p.epoch;
  }
  fence_acq_rel_gpu();
  if (!__syncthreads_and(ok)) {  // some child is still being resolved
    ok = true;
    for (uint32_t i = tid; i < pairs && ok; i += kDpThreads)
      if (i % kQ < count)
        ok = wait_flag(flag_of(i), p.epoch, p.timeout_ns, p.error);
    if (!__syncthreads_and(ok))
      return false;
  }

  // Cross-tile children, 16 bytes (4 words) of a plane per thread and load.
#pragma unroll 1
  for (uint32_t ci = tid; ci < count * kChunks; ci += kDpThreads) {
    const uint32_t q = ci / kChunks, k = ci % kChunks;
    Acc a[4];
    const uint8_t* const base = table + k * 16u;
    const uint32_t* kid = ws.kids + q;
    int m = 0;
#pragma unroll 2
    for (; m + 2 <= j; m += 2) {
      const uint8_t* s = base + size_t(kid[0]) * Shape::kTileBytes;
      const uint8_t* t = base + size_t(kid[kQ]) * Shape::kTileBytes;
      kid += 2 * kQ;
      const uint4 s0 = ldcg128(s), s1 = ldcg128(s + 4 * kW), sc = ldcg128(s + 8 * kW);
      const uint4 t0 = ldcg128(t), t1 = ldcg128(t + 4 * kW), tc = ldcg128(t + 8 * kW);
      acc_add2(a[0], s0.x, s1.x, sc.x, t0.x, t1.x, tc.x);
      acc_add2(a[1], s0.y, s1.y, sc.y, t0.y, t1.y, tc.y);
      acc_add2(a[2], s0.z, s1.z, sc.z, t0.z, t1.z, tc.z);
      acc_add2(a[3], s0.w, s1.w, sc.w, t0.w, t1.w, tc.w);
    }
    if (m < j) {
      const uint8_t* s = base + size_t(kid[0]) * Shape::kTileBytes;
      const uint4 s0 = ldcg128(s), s1 = ldcg128(s + 4 * kW), sc = ldcg128(s + 8 * kW);
      acc_add1(a[0], s0.x, s1.x, sc.x);
      acc_add1(a[1], s0.y, s1.y, sc.y);
      acc_add1(a[2], s0.z, s1.z, sc.z);
      acc_add1(a[3], s0.w, s1.w, sc.w);
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
      uint32_t* const at = ws.planes + plane_at<LB>(q, 4 * k + i);
      at[0] = a[i].o0;
      at[kPlane] = a[i].o1;
      at[2 * kPlane] = a[i].o2;
      at[3 * kPlane] = a[i].c1;
      at[4 * kPlane] = a[i].c2;
    }
  }
  __syncthreads();

  // In-tile children: words in popcount order of the word index, a thread per
  // word and quad of tiles (from 32 quads on a warp is on one word). Tiles
  // past `count` in the last quad come along and are not stored.
  const uint32_t quads = (count + 3u) / 4u;
  const uint8_t* order = ws.order;
#pragma unroll 1
  for (int s = 0; s <= kWordBits; ++s) {
    const uint32_t items = binom[kWordBits][s] * Shape::kQuads;
#pragma unroll 1
    for (uint32_t e = tid; e < items; e += kDpThreads) {
      const uint32_t q = (e % Shape::kQuads) * 4u, w = order[e / Shape::kQuads];
      if (q >= quads * 4u)
        continue;
      uint32_t* const at = ws.planes + plane_at<LB>(q, w);
      auto load = [](const uint32_t* from) { return *reinterpret_cast<const uint4*>(from); };
      const uint4 o0 = load(at), o1 = load(at + kPlane), o2 = load(at + 2 * kPlane), c1 = load(at + 3 * kPlane),
                  c2 = load(at + 4 * kPlane);
      Acc a[4] = {{o0.x, o1.x, o2.x, c1.x, c2.x},
                  {o0.y, o1.y, o2.y, c1.y, c2.y},
                  {o0.z, o1.z, o2.z, c1.z, c2.z},
                  {o0.w, o1.w, o2.w, c1.w, c2.w}};
#pragma unroll 1
      for (uint32_t bits = w; bits; bits &= bits - 1u) {
        const uint32_t* const child = ws.planes + plane_at<LB>(q, w ^ (bits & (0u - bits)));
        const uint4 p0 = load(child), p1 = load(child + kPlane), c = load(child + 2 * kPlane);
        acc_add1(a[0], p0.x, p1.x, c.x);
        acc_add1(a[1], p0.y, p1.y, c.y);
        acc_add1(a[2], p0.z, p1.z, c.z);
        acc_add1(a[3], p0.w, p1.w, c.w);
      }
      SmallSets small[4];
      Planes r[4];
      if (j + s > 2) {
        resolve_quad(a, small, r);
      } else {
        for (uint32_t b = 0; b < 4; ++b)
          if (q + b < count)
            small[b] = small_sets((uint64_t(ws.high[q + b]) << LB) | (uint64_t(w) << 5), j + s, p.adj + G.adj_off, G.n);
        resolve_quad(a, small, r);
      }
      *reinterpret_cast<uint4*>(at) = make_uint4(r[0].p0, r[1].p0, r[2].p0, r[3].p0);
      *reinterpret_cast<uint4*>(at + kPlane) = make_uint4(r[0].p1, r[1].p1, r[2].p1, r[3].p1);
      *reinterpret_cast<uint4*>(at + 2 * kPlane) = make_uint4(r[0].c, r[1].c, r[2].c, r[3].c);
    }
    order += binom[ws.order_bits][s];
    __syncthreads();
  }

  // Store the tiles.
  uint8_t* const dst = table + size_t(off_j + r0) * Shape::kTileBytes;
#pragma unroll 1
  for (uint32_t ci = tid; ci < count * kChunks; ci += kDpThreads) {
    const uint32_t q = ci / kChunks, k = ci % kChunks;
    uint8_t* const out = dst + q * Shape::kTileBytes + k * 16u;
#pragma unroll
    for (uint32_t plane = 0; plane < 3; ++plane) {
      const uint32_t* const from = ws.planes + plane * kPlane;
      *reinterpret_cast<uint4*>(out + plane * 4 * kW) =
          make_uint4(from[plane_at<LB>(q, 4 * k)], from[plane_at<LB>(q, 4 * k + 1)], from[plane_at<LB>(q, 4 * k + 2)],
                     from[plane_at<LB>(q, 4 * k + 3)]);
    }
  }
  return true;
}

constexpr uint32_t kNone = 0xFFFFFFFFu;

// The launch's loop: the ticket of the next group (and the error word) is on
// its way while `work` resolves a group; a CTA works its tickets in order, so
// taking one early holds nothing up that the ticket before it does not.
//
// Publication: the group's stores are ordered before thread 0's flag store by
// the CTA barrier, and that store is a gpu-scope release, which is cumulative:
// a reader that acquires the flag sees every byte of the group's tiles.
template <typename Work>
__device__ __forceinline__ void group_loop(const DpBatchParams& p, Work work) {
  __shared__ uint2 sNext;  // (graph, group); graph kNone: no more
  uint32_t pending = kNone, ticket = 0;
  int32_t error = 0;
  if (threadIdx.x == 0) {
    error = ld_relaxed_s32(p.error);
    ticket = atomicAdd(p.ticket, 1u);
  }
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0)
      sNext = error != 0 || ticket >= p.total_groups ? make_uint2(kNone, 0u)
              : p.graphs                             ? __ldg(p.tile_map + ticket)
                                                     : make_uint2(0u, ticket);
    if (threadIdx.x == 32 && pending != kNone)
      st_release_u32(p.flags + pending, p.epoch);
    __syncthreads();
    const uint2 next = sNext;
    if (next.x == kNone)
      return;
    if (threadIdx.x == 0) {
      error = ld_relaxed_s32(p.error);
      ticket = atomicAdd(p.ticket, 1u);
    }
    const DpGraph G = p.graphs ? p.graphs[next.x] : p.single;
    if (!work(G, next.x, next.y))
      return;
    pending = G.flag_base + next.y;
  }
}

// Tiles of one size (single-graph solves, and batches that use one).
template <int LB>
__global__ void __launch_bounds__(kDpThreads, 4) dp_tile_kernel(const __grid_constant__ DpBatchParams p) {
  const Workspace ws = make_workspace(p, smem_layout_for(LB, LB, p.kid_rows), LB - 5);
  group_loop(p, [&](const DpGraph& G, uint32_t, uint32_t group) { return group_work<LB>(p, G, group, ws); });
}

// Batches whose graphs use different tile sizes (DpGraph::lb, 8 .. p.lb):
// shared memory is laid out for the largest (p.lb, a runtime value) and each
// group dispatches on its graph's lb. The autotuner measures what the
// dispatch costs against one size and the planner only mixes sizes when the
// per-size gains outweigh it.
__global__ void __launch_bounds__(kDpThreads, 4) dp_tile_kernel_mixed(const __grid_constant__ DpBatchParams p) {
  const Workspace ws = make_workspace(p, smem_layout_for(kDpMinTileBits, p.lb, p.kid_rows), p.lb - 5);
  group_loop(p, [&](const DpGraph& G, uint32_t graph, uint32_t group) {
    switch (G.lb <= p.lb ? G.lb : 0) {
      case 8: return group_work<8>(p, G, group, ws);
      case 9: return group_work<9>(p, G, group, ws);
      case 10: return group_work<10>(p, G, group, ws);
      case 11: return group_work<11>(p, G, group, ws);
      case 12: return group_work<12>(p, G, group, ws);
      default:  // the planner never does this: the tile would not fit
        if (threadIdx.x == 0)
          raise_error(p.error, kDevInvalidInput, static_cast<int32_t>(graph));
        return false;
    }
  });
}

// ---------------------------------------------------------------------------
// Narrow levels: a thread per tile of 7 bits, level by level.
// ---------------------------------------------------------------------------

// A word's 32 subsets (bit x = the subset x of the five lowest vertices) from
// the summary of their children outside the word, by size of x: position 0,
// its broadcast to the singles, three rounds over the five vertices (round r
// settles size r; smaller sizes come out as before, larger ones are not
// final), then position 31 from its five children.
__device__ __forceinline__ Planes resolve_word(const Acc& ext, const SmallSets& s) {
  constexpr uint32_t kSingles = 0x00010116u, kFours = 0x68808000u, kTop = 0x80000000u;  // |x| = 1, 4, 5
  Planes r = finish(ext, s);
  Acc a = ext;
  a.o0 |= (r.p0 & 1u) * kSingles;
  a.o1 |= (r.p1 & 1u) * kSingles;
  a.o2 |= (~(r.p0 | r.p1) & 1u) * kSingles;
  a.c2 |= a.c1 & ((r.c & 1u) * kSingles);
  r = finish(a, s);
#pragma unroll
  for (int round = 2; round <= 4; ++round) {
    constexpr uint32_t kHas[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
    const uint32_t p2 = ~(r.p0 | r.p1);
    a = ext;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int sh = 1 << i;
      a.o0 |= (r.p0 << sh) & kHas[i];
      a.o1 |= (r.p1 << sh) & kHas[i];
      a.o2 |= (p2 << sh) & kHas[i];
      const uint32_t x = (r.c << sh) & kHas[i];
      a.c2 |= a.c1 & x;
      a.c1 |= x;
    }
    r = finish(a, s);
  }
  const uint32_t p2 = ~(r.p0 | r.p1), k = r.c & kFours;
  a = ext;
  a.o0 |= (r.p0 & kFours) ? kTop : 0u;
  a.o1 |= (r.p1 & kFours) ? kTop : 0u;
  a.o2 |= (p2 & kFours) ? kTop : 0u;
  a.c2 |= (k ? a.c1 & kTop : 0u) | ((k & (k - 1u)) ? kTop : 0u);
  const Planes t = finish(a, s);
  r.p0 = (r.p0 & ~kTop) | (t.p0 & kTop);
  r.p1 = (r.p1 & ~kTop) | (t.p1 & kTop);
  r.c = (r.c & ~kTop) | (t.c & kTop);
  return r;
}

constexpr int kLevelThreads = kDpLevelChunk;

// Thread r of a chunk resolves the tile of rank r: unranks it, gathers its
// child tiles (48 bytes each), resolves its four words in order 00, 01 and
// 10, 11 of vertices 5 and 6. A chunk of level j waits until every chunk of
// level j - 1 is done (one counter per level, acquired by one thread), after
// unranking: no flags to look up per child. Tickets as in the tile kernel.
//
// For levels too narrow to fill the GPU, where the latency of the tile
// kernel's groups (15 us a level at 11 bits) leaves most SMs idle: a level costs
// 2.5 to 3 us here (n = 20: 45 us), most of it the count, the gathers and the
// chain through three words. A tile of 48 bytes is also the widest load that
// the gathers can use, so tables beyond the L2 (n >= 29) go to the tile kernel.
//
// BATCH: chunks of many graphs, level-major as in the tile kernel, counters
// per graph.
template <bool BATCH>
__global__ void __launch_bounds__(kLevelThreads, 4) dp_level_kernel(const __grid_constant__ DpBatchParams p) {
  constexpr int LB = kDpLevelTileBits;
  constexpr uint32_t kTileBytes = dp_tile_bytes(LB);
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t* const kids = reinterpret_cast<uint32_t*>(smem) + threadIdx.x;  // kids[i * kLevelThreads]
  __shared__ Binom binom;
  __shared__ uint32_t sTicket;
  __shared__ int sStop;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  fill_binom(binom);
  uint32_t ticket = 0;
  if (tid == 0)
    ticket = atomicAdd(p.ticket, 1u);
  for (;;) {
    if (tid == 0)
      sTicket = ticket;
    __syncthreads();
    uint32_t chunk = sTicket;
    if (chunk >= p.total_groups)
      return;
    uint32_t g = 0;
    if (BATCH) {
      const uint2 at = __ldg(p.tile_map + chunk);
      g = at.x;
      chunk = at.y;
    }
    const DpGraph G = BATCH ? p.graphs[g] : p.single;
    uint8_t* const table = p.table + G.table_off;
    uint32_t* const level_done = p.level_done + 32u * g;
    const int nh = G.nh;
    if (tid == 0)
      ticket = atomicAdd(p.ticket, 1u);
    // Level j of the chunk: lane i holds the tiles and chunks of levels 0..i.
    const uint32_t level_tiles = static_cast<int>(lane) <= nh ? binom[nh][lane] : 0u;
    const uint32_t level_chunks = (level_tiles + kLevelThreads - 1u) / kLevelThreads;
    uint32_t cumT = level_tiles, cumG = level_chunks;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, cumT, d);
      const uint32_t y = __shfl_up_sync(0xffffffffu, cumG, d);
      if (static_cast<int>(lane) >= d) {
        cumT += x;
        cumG += y;
      }
    }
    const int j = __popc(__ballot_sync(0xffffffffu, static_cast<int>(lane) <= nh && cumG <= chunk));
    const uint32_t tiles_j = __shfl_sync(0xffffffffu, level_tiles, j);
    const uint32_t off_j = __shfl_sync(0xffffffffu, cumT, j) - tiles_j;
    const uint32_t first = __shfl_sync(0xffffffffu, cumG - level_chunks, j);
    const uint32_t off_prev = off_j - __shfl_sync(0xffffffffu, level_tiles, (j + 31) & 31);
    const uint32_t chunks_prev = __shfl_sync(0xffffffffu, level_chunks, (j + 31) & 31);
    const uint32_t rank = (chunk - first) * kLevelThreads + tid;
    const bool mine = rank < tiles_j;
    uint32_t H = 0;
    if (mine) {
      uint32_t rest = rank, kid = off_prev;
      uint32_t* at = kids;
      int k = j;
      for (int a = nh - 1; a >= 0; --a) {  // as in the tile kernel
        const uint32_t c = binom[a][k], d = binom[a][max(k - 1, 0)];
        if (rest >= c) {
          rest -= c;
          H |= 1u << a;
          *at = kid + rest;
          at += kLevelThreads;
          kid += d;
          --k;
        }
      }
    }
    if (j > 0) {
      if (tid == 0)
        sStop = wait_count(level_done + (j - 1), chunks_prev, p.timeout_ns, p.error) ? 0 : 1;
      __syncthreads();
      if (sStop)
        return;
    }
    if (mine) {
      Acc a[4];
      const uint32_t* kid = kids;
      auto child = [&](uint32_t t, uint4& p0, uint4& p1, uint4& c) {
        const uint8_t* from = table + size_t(t) * kTileBytes;
        p0 = ldcg128(from);
        p1 = ldcg128(from + 16);
        c = ldcg128(from + 32);
      };
      int m = 0;
#pragma unroll 2
      for (; m + 2 <= j; m += 2) {
        uint4 s0, s1, sc, t0, t1, tc;
        child(kid[0], s0, s1, sc);
        child(kid[kLevelThreads], t0, t1, tc);
        kid += 2 * kLevelThreads;
        acc_add2(a[0], s0.x, s1.x, sc.x, t0.x, t1.x, tc.x);
        acc_add2(a[1], s0.y, s1.y, sc.y, t0.y, t1.y, tc.y);
        acc_add2(a[2], s0.z, s1.z, sc.z, t0.z, t1.z, tc.z);
        acc_add2(a[3], s0.w, s1.w, sc.w, t0.w, t1.w, tc.w);
      }
      if (m < j) {
        uint4 s0, s1, sc;
        child(kid[0], s0, s1, sc);
        acc_add1(a[0], s0.x, s1.x, sc.x);
        acc_add1(a[1], s0.y, s1.y, sc.y);
        acc_add1(a[2], s0.z, s1.z, sc.z);
        acc_add1(a[3], s0.w, s1.w, sc.w);
      }
      Planes r[4];
      if (j > 2) {
        const SmallSets any;
        r[0] = resolve_word(a[0], any);
        acc_add1(a[1], r[0].p0, r[0].p1, r[0].c);
        acc_add1(a[2], r[0].p0, r[0].p1, r[0].c);
        r[1] = resolve_word(a[1], any);
        r[2] = resolve_word(a[2], any);
        acc_add2(a[3], r[1].p0, r[1].p1, r[1].c, r[2].p0, r[2].p1, r[2].c);
        r[3] = resolve_word(a[3], any);
      } else {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          if (w == 3) {
            acc_add2(a[3], r[1].p0, r[1].p1, r[1].c, r[2].p0, r[2].p1, r[2].c);
          } else if (w > 0) {
            acc_add1(a[w], r[0].p0, r[0].p1, r[0].c);
          }
          const int size = j + __popc(w);
          r[w] = resolve_word(a[w], size <= 2 ? small_sets((uint64_t(H) << LB) | (uint64_t(w) << 5), size,
                                                           p.adj + G.adj_off, G.n)
                                              : SmallSets{});
        }
      }
      uint4* const out = reinterpret_cast<uint4*>(table + size_t(off_j + rank) * kTileBytes);
      out[0] = make_uint4(r[0].p0, r[1].p0, r[2].p0, r[3].p0);
      out[1] = make_uint4(r[0].p1, r[1].p1, r[2].p1, r[3].p1);
      out[2] = make_uint4(r[0].c, r[1].c, r[2].c, r[3].c);
    }
    // The chunk's stores are ordered before the count by the barrier; the
    // count is a gpu-scope release, and a chain of such additions hands every
    // chunk's stores to the thread that acquires the final value.
    __syncthreads();
    if (tid == 0)
      red_release_add_u32(level_done + j, 1u);
  }
}

// ---------------------------------------------------------------------------
// Reconstruction: one warp per graph.
// ---------------------------------------------------------------------------

constexpr int kTreeWarps = 4;

__device__ __forceinline__ uint64_t ballot64(bool lo, bool hi) {
  const uint32_t a = __ballot_sync(0xffffffffu, lo);
  const uint32_t b = __ballot_sync(0xffffffffu, hi);
  return (static_cast<uint64_t>(b) << 32) | a;
}

__device__ __forceinline__ uint64_t warp_or64(uint64_t x) {
  const uint32_t lo = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(x));
  const uint32_t hi = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(x >> 32));
  return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Subsets of a table in global memory.
struct TreeCtx {
  const Binom& binom;
  const uint32_t* off;  // first tile of every level
  const uint8_t* table;
  int lb, n;
  // The first plane's word that holds S (the other planes: 2^(lb-5) words on).
  __device__ const uint32_t* word(uint64_t S) const {
    uint32_t H = static_cast<uint32_t>(S >> lb), rank = off[__popc(H)];
    const uint32_t* col = &binom[0][1];
#pragma unroll 4
    for (; H; H &= H - 1, ++col)
      rank += col[(__ffs(H) - 1) * (kDpMaxHigh + 1)];
    return reinterpret_cast<const uint32_t*>(table + size_t(rank) * dp_tile_bytes(lb)) +
           ((static_cast<uint32_t>(S) >> 5) & ((1u << (lb - 5)) - 1u));
  }
  // td(S) mod 3 (one lane).
  __device__ uint32_t residue(uint64_t S) const {
    const uint32_t* t = word(S);
    const uint32_t bit = static_cast<uint32_t>(S) & 31u;
    const uint32_t p0 = (t[0] >> bit) & 1u, p1 = (t[1u << (lb - 5)] >> bit) & 1u;
    return p0 ? 0u : 2u - p1;
  }
};

// First tiles of the levels of a graph with nh high vertices (whole warp).
__device__ __forceinline__ void level_offsets(const Binom& binom, int nh, uint32_t* off) {
  const int lane = threadIdx.x & 31;
  const uint32_t own = lane <= nh ? binom[nh][lane] : 0u;
  uint32_t cum = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, cum, d);
    if (lane >= d)
      cum += x;
  }
  off[lane] = cum - own;
  __syncwarp();
}

// Residues of the chain S & {v, v + 1, ...}, v = lane and lane + 32 (0 .. n),
// and from them td(S): each deletion lowers the treedepth by 0 or 1, which the
// residues tell. (Two parts, so that the loads can be on their way meanwhile.)
struct Chain {
  uint32_t lo, hi;
};
template <class Ctx>
__device__ __forceinline__ Chain load_chain(const Ctx& ctx, uint64_t S) {
  const int lane = threadIdx.x & 31;
  return Chain{lane <= ctx.n ? ctx.residue(S & (~0ull << lane)) : 0u,
               lane + 32 <= ctx.n ? ctx.residue(S & (~0ull << (lane + 32))) : 0u};
}
__device__ __forceinline__ uint32_t chain_td(const Chain& c, int n) {
  const int lane = threadIdx.x & 31;
  uint32_t next_lo = __shfl_down_sync(0xffffffffu, c.lo, 1);
  const uint32_t first_hi = __shfl_sync(0xffffffffu, c.hi, 0), next_hi = __shfl_down_sync(0xffffffffu, c.hi, 1);
  if (lane == 31)
    next_lo = first_hi;
  return __reduce_add_sync(0xffffffffu, (lane < n && c.lo != next_lo ? 1u : 0u) +
                                            (lane + 32 < n && c.hi != next_hi ? 1u : 0u));
}

// Shared memory of one warp's reconstruction.
struct TreeMem {
  uint64_t set[2][kDpMaxN];       // components of the depth in work and of the next
  unsigned long long kids[kDpMaxN];  // children of each vertex
  int32_t owner[2][kDpMaxN];
  int32_t par[kDpMaxN];           // the canonical tree
  int32_t dep[kDpMaxN];           // depth of each vertex in it
  uint32_t hgt[kDpMaxN];          // subtree height (in vertices)
  uint32_t low[kDpMaxN];          // 255 - the subtree's lowest vertex
  uint8_t comp[64];               // component of each vertex, of the depth in work
  uint32_t off[32];
};

// The canonical tree of `query` and what p asks of it (whole warp): every
// component is rooted at the first vertex v with td(C - v) = td(C) - 1 and its
// sub-components hang below that root (dynamic_cpu.hpp:59-81). All components
// of a depth are taken together. They are the components of the graph on the
// vertices not yet placed (an edge between two of them would have kept them in
// one), so lane v holds the set C(v) of its vertex in a register: one round of
// loads reads C(v) - v, three ballots of the residues give every component its
// root, and a root's C is its subtree. The latency of one warp bounds
// it: with lists of components in shared memory, taken one after another, and
// the order from shared-memory atomics it took 15 us at n = 16 (9 depths, 11
// components; the small kernel as a whole 29 us, now 22; n = 12 19, now 15).
template <class Ctx>
__device__ __forceinline__ bool build_tree(const DpBatchParams& p, const DpGraph& G, const uint64_t* adj_masks,
                                           const Ctx& ctx, uint32_t query) {
  const int lane = threadIdx.x & 31, n = G.n;
  const uint32_t adj = lane < n ? static_cast<uint32_t>(adj_masks[lane]) : 0u;
  const Chain chain = load_chain(ctx, query);
  uint32_t comp = 0u, sub = 0u;  // the vertex's component; its subtree once placed
  int parent = -1, owner = -1;   // owner: root of the component around it
  int dep = 0, deepest = 0, height = 0;
  for (uint32_t rest = query; rest;) {
    ++height;
    const bool in = (rest >> lane) & 1u, alone = in && (adj & rest) == 0u;
    if (alone)
      comp = 1u << lane;
    uint32_t todo = rest & ~__ballot_sync(0xffffffffu, alone);
    while (todo) {
      uint32_t reach = todo & (0u - todo), front = reach;
      while (front) {
        front = __reduce_or_sync(0xffffffffu, ((front >> lane) & 1u) ? adj : 0u) & todo & ~reach;
        reach |= front;
      }
      if ((reach >> lane) & 1u)
        comp = reach;
      todo &= ~reach;
    }
    const bool look = in && !alone;
    const uint32_t t = look ? ctx.residue(comp & ~(1u << lane)) : 3u;
    const uint32_t h0 = __ballot_sync(0xffffffffu, t == 0u) & comp, h1 = __ballot_sync(0xffffffffu, t == 1u) & comp,
                   h2 = __ballot_sync(0xffffffffu, t == 2u) & comp;
    // td(C - v) over v in C is a and possibly a + 1: residue a is the one
    // present whose predecessor is absent (three: a corrupt table)
    const uint32_t hits = h0 && h2 ? h2 : h0 ? h0 : h1 ? h1 : h2;
    if (__any_sync(0xffffffffu, look && ((h0 && h1 && h2) || hits == 0u)))
      return false;
    const int root = look ? __ffs(hits) - 1 : lane;
    const bool placed = in && root == lane;
    if (placed) {
      parent = owner;
      dep = height;
      sub = comp;
    }
    owner = root;
    const uint32_t now = __ballot_sync(0xffffffffu, placed);
    if (now & sub)
      deepest = height;
    rest &= ~now;
  }
  const uint32_t td = chain_td(chain, n);
  if (lane == 0 && p.td_out)
    p.td_out[G.out_idx] = static_cast<int32_t>(td);
  if (static_cast<uint32_t>(height) != td)
    return false;
  const bool in = (query >> lane) & 1u;
  if (p.parent_out && in)
    p.parent_out[G.adj_off + lane] = parent;
  if (p.order_out) {
    // GetElimination (dynamic_gpu.hpp:58-63): repeatedly remove the stored
    // root of the remaining set; for a disconnected set that is the root of
    // its first deepest component, components taken in order of their
    // lowest vertex (dynamic_gpu.cu:92-103). The components of the
    // remaining set are subtrees of the canonical tree and a component's
    // treedepth is its subtree's height, so the order is read off the tree:
    // the active subtree of greatest height, ties to the lowest vertex,
    // gives its root and is replaced by its children's subtrees.
    const uint32_t key = static_cast<uint32_t>(deepest - dep + 1) << 10 |
                         static_cast<uint32_t>(32 - __ffs(sub)) << 5 | static_cast<uint32_t>(lane);
    bool active = in && parent < 0;
    const int count = __popc(query);
    int own = 0;
    for (int step = 0; step < count; ++step) {
      const int v = static_cast<int>(__reduce_max_sync(0xffffffffu, active ? key : 0u) & 31u);
      if (lane == step)
        own = v;
      active = (active && lane != v) || (in && parent == v);
    }
    if (lane < count)
      p.order_out[G.adj_off + lane] = own;
  }
  return true;
}

// The same for more than 32 vertices, two to a lane, the components of a depth
// in lists in shared memory. A table of this size takes milliseconds, its tree
// a few dozen microseconds.
template <class Ctx>
__device__ __noinline__ bool build_wide_tree(const DpBatchParams& p, const DpGraph& G, const uint64_t* adj, const Ctx& ctx, TreeMem& m,
                           uint64_t query) {
  const int lane = threadIdx.x & 31, n = G.n;
  const uint64_t adj_lo = lane < n ? adj[lane] : 0ull;
  const uint64_t adj_hi = lane + 32 < n ? adj[lane + 32] : 0ull;
  const Chain chain = load_chain(ctx, query);
  int height = 0, count = 0;      // count: components of the next depth
  uint64_t in_next = 0;           // their union
  // The components of `rest`, below `owner` at depth d: single vertices are
  // done, the others join list `to`.
  auto split = [&](uint64_t rest, int owner, int d, int to) {
    if (rest)
      height = max(height, d);
    // the vertices without a neighbour left, all at once
    const bool one_lo = ((rest >> lane) & 1ull) && (adj_lo & rest) == 0ull;
    const bool one_hi = ((rest >> (lane + 32)) & 1ull) && (adj_hi & rest) == 0ull;
    if (one_lo) {
      m.par[lane] = owner;
      m.dep[lane] = d;
    }
    if (one_hi) {
      m.par[lane + 32] = owner;
      m.dep[lane + 32] = d;
    }
    rest &= ~ballot64(one_lo, one_hi);
    while (rest) {
      uint64_t reach = rest & (0ull - rest), frontier = reach;
      while (frontier) {
        const uint64_t nb = (((frontier >> lane) & 1ull) ? adj_lo : 0ull) |
                            (((frontier >> (lane + 32)) & 1ull) ? adj_hi : 0ull);
        frontier = warp_or64(nb) & rest & ~reach;
        reach |= frontier;
      }
      rest &= ~reach;
      if (lane == 0) {
        m.set[to][count] = reach;
        m.owner[to][count] = owner;
      }
      if ((reach >> lane) & 1ull)
        m.comp[lane] = static_cast<uint8_t>(count);
      if ((reach >> (lane + 32)) & 1ull)
        m.comp[lane + 32] = static_cast<uint8_t>(count);
      in_next |= reach;
      ++count;
    }
  };
  split(query, -1, 1, 0);
  for (int depth = 1, cur = 0; count > 0; ++depth, cur ^= 1) {
    __syncwarp();
    const bool in_lo = (in_next >> lane) & 1ull, in_hi = (in_next >> (lane + 32)) & 1ull;
    const uint32_t t_lo = in_lo ? ctx.residue(m.set[cur][m.comp[lane]] & ~(1ull << lane)) : 0u;
    const uint32_t t_hi = in_hi ? ctx.residue(m.set[cur][m.comp[lane + 32]] & ~(1ull << (lane + 32))) : 0u;
    const int here = count;
    count = 0;
    in_next = 0;
    __syncwarp();  // comp[] read above, rewritten by split
    for (int i = 0; i < here; ++i) {
      const uint64_t C = m.set[cur][i];
      const bool c_lo = (C >> lane) & 1ull, c_hi = (C >> (lane + 32)) & 1ull;
      // td(C - v) over v in C is a and possibly a + 1: residue a is the one
      // present whose predecessor is absent (three: a corrupt table)
      const uint32_t have = __reduce_or_sync(0xffffffffu, (c_lo ? 1u << t_lo : 0u) | (c_hi ? 1u << t_hi : 0u));
      const uint32_t a = (have & 5u) == 5u ? 2u : (have & 1u) ? 0u : (have & 2u) ? 1u : 2u;
      const uint64_t hits = ballot64(c_lo && t_lo == a, c_hi && t_hi == a);
      if (have == 7u || hits == 0ull)
        return false;
      const int root = __ffsll(static_cast<long long>(hits)) - 1, owner = m.owner[cur][i];
      if (lane == 0) {
        m.par[root] = owner;
        m.dep[root] = depth;
      }
      split(C & ~(1ull << root), root, depth + 1, cur ^ 1);
    }
  }
  __syncwarp();
  const uint32_t td = chain_td(chain, n);
  if (lane == 0 && p.td_out)
    p.td_out[G.out_idx] = static_cast<int32_t>(td);
  if (static_cast<uint32_t>(height) != td)
    return false;
  if (p.parent_out) {
    int32_t* parent = p.parent_out + G.adj_off;
    for (int v = lane; v < n; v += 32)
      if ((query >> v) & 1ull)
        parent[v] = m.par[v];
  }

  if (p.order_out) {
    for (int v = lane; v < n; v += 32) {
      m.hgt[v] = 0u;  // the tallest child so far
      m.low[v] = 255u - static_cast<uint32_t>(v);
      m.kids[v] = 0ull;
    }
    __syncwarp();
    for (int d = height; d >= 1; --d) {  // deepest first: children before parents
      for (int v = lane; v < n; v += 32) {
        if (((query >> v) & 1ull) && m.dep[v] == d) {
          const uint32_t h = m.hgt[v] + 1u;  // own height = tallest child + 1
          m.hgt[v] = h;
          const int pv = m.par[v];
          if (pv >= 0) {
            atomicMax(&m.hgt[pv], h);
            atomicMax(&m.low[pv], m.low[v]);
            atomicOr(&m.kids[pv], 1ull << v);
          }
        }
      }
      __syncwarp();
    }
    int32_t* order = p.order_out + G.adj_off;
    uint64_t active = 0;
    for (int v = lane; v < n; v += 32)
      if (((query >> v) & 1ull) && m.par[v] < 0)
        active |= 1ull << v;
    active = warp_or64(active);
    // key: height << 8 | 255 - lowest vertex (unique: the subtrees are disjoint)
    const uint32_t key_lo = lane < n ? m.hgt[lane] << 8 | m.low[lane] : 0u;
    const uint32_t key_hi = lane + 32 < n ? m.hgt[lane + 32] << 8 | m.low[lane + 32] : 0u;
    for (int step = 0; active; ++step) {
      const uint32_t k_lo = ((active >> lane) & 1ull) ? key_lo : 0u;
      const uint32_t k_hi = ((active >> (lane + 32)) & 1ull) ? key_hi : 0u;
      const uint32_t best = __reduce_max_sync(0xffffffffu, max(k_lo, k_hi));
      const uint64_t hit = ballot64(k_lo == best && k_lo != 0u, k_hi == best && k_hi != 0u);
      const int v = __ffsll(static_cast<long long>(hit)) - 1;
      if (lane == 0)
        order[step] = v;
      active = (active & ~(1ull << v)) | m.kids[v];
    }
  }
  return true;
}

// The error words of a single solve for the host (its graph is warp 0's).
__device__ __forceinline__ void report_error(const DpBatchParams& p) {
  if (p.report && blockIdx.x == 0 && threadIdx.x == 0) {
    p.report[0] = ld_relaxed_s32(p.error);
    p.report[1] = ld_relaxed_s32(p.error + 1);
  }
}

__global__ void __launch_bounds__(32 * kTreeWarps)
    dp_tree_kernel(const __grid_constant__ DpBatchParams p) {
  __shared__ Binom sBinom;
  __shared__ TreeMem mem[kTreeWarps];
  fill_binom(sBinom);
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  const bool failed = ld_relaxed_s32(p.error) != 0;
  for (int g = blockIdx.x * kTreeWarps + warp; g < p.num_graphs && !failed; g += gridDim.x * kTreeWarps) {
    const DpGraph G = p.graphs ? p.graphs[g] : p.single;
    level_offsets(sBinom, G.nh, mem[warp].off);
    const TreeCtx ctx{sBinom, mem[warp].off, p.table + G.table_off, G.lb, G.n};
    const uint64_t query = p.query ? p.query : (1ull << G.n) - 1ull;
    const uint64_t* const adj = p.adj + G.adj_off;
    if (!(G.n <= 32 ? build_tree(p, G, adj, ctx, static_cast<uint32_t>(query))
                    : build_wide_tree(p, G, adj, ctx, mem[warp], query))) {
      if ((threadIdx.x & 31) == 0)
        raise_error(p.error, kDevNoRoot, g);
      break;
    }
    __syncwarp();
  }
  report_error(p);
}

// ---------------------------------------------------------------------------
// Small graphs: check, table and tree in one CTA.
// ---------------------------------------------------------------------------

// Subsets of a table in shared memory, words in natural order.
struct SmallCtx {
  const uint32_t* p0;
  const uint32_t* p1;
  int n;
  __device__ uint32_t residue(uint64_t S) const {
    const uint32_t w = static_cast<uint32_t>(S) >> 5, bit = static_cast<uint32_t>(S) & 31u;
    return ((p0[w] >> bit) & 1u) ? 0u : 2u - ((p1[w] >> bit) & 1u);
  }
};

// Place of every word among all words by size and colex rank: f(word, place)
// for the words base << mh + ..., by the given warps, the m < 5 case in one of
// them. 32 words of one h = word / 32 at a time: the rank is that of the five
// low bits plus, by their number, one of six sums over the bits of h (a lane
// each); a loop over the bits of every word took 7 of the 62 us at n = 20.
template <class F>
__device__ __forceinline__ void for_places(const Binom& binom, const uint32_t* off, uint32_t base, int m, int warp,
                                           int warps, F&& f) {
  const int lane = threadIdx.x & 31, q = __popc(lane), mh = m > 5 ? m - 5 : 0;
  const uint32_t low = rank_colex(binom, static_cast<uint32_t>(lane));
  for (uint32_t h = warp; h < (1u << mh); h += warps) {
    const uint32_t H = base << mh | h;
    const bool in_H = (H >> lane) & 1u;
    const int k = __popc(H & ((2u << lane) - 1u));
    uint32_t high = 0;
#pragma unroll
    for (int i = 0; i <= 5; ++i) {
      const uint32_t sum = __reduce_add_sync(0xffffffffu, in_H ? binom[5 + lane][k + i] : 0u);
      high = i == q ? sum : high;
    }
    if (lane < (1 << m))
      f(h << 5 | lane, off[__popc(H) + q] + low + high);
  }
}

// Dynamic shared memory for graphs of up to n vertices: three planes of
// 2^(n-5) words and the words' order.
__host__ __device__ constexpr uint32_t small_words(int n) { return n > 5 ? 1u << (n - 5) : 1u; }
constexpr size_t small_smem(int n) { return size_t(small_words(n)) * (3 * 4 + 2); }

// One CTA per graph of n <= kDpSmallMaxN vertices: a thread per word of 32
// subsets, the words of a level between two CTA barriers, children at W ^ bit
// in shared memory; then the first warp builds the tree from there while the
// others copy the planes out (single-graph solves: tiles of 5 bits, for later
// queries). One launch and no flag, count or gather from L2, each of which
// costs a microsecond a level in the other kernels: bound by the latency of a
// level's word chain, about 0.8 us, and half as much again for the tree (n = 12,
// all of check, table and tree: 15 us against 4 + 21 + 9 in the level kernel's
// three; n = 16: 22 against 4 + 30 + 11).
__global__ void __launch_bounds__(512)
    dp_small_kernel(const __grid_constant__ DpBatchParams p, int max_n, const __grid_constant__ DpInput in) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ Binom binom;
  __shared__ uint32_t off[32];  // first place of a level
  __shared__ int sBad;
  const uint32_t tid = threadIdx.x, threads = blockDim.x;
  const int g = p.first_graph + static_cast<int>(blockIdx.x);
  const DpGraph G = p.graphs ? p.graphs[g] : p.single;
  __shared__ uint64_t adj[kDpSmallMaxN];
  const int n = G.n, m = n > 5 ? n - 5 : 0;
  const uint32_t words = 1u << m, stride = small_words(max_n);
  uint32_t* const p0 = reinterpret_cast<uint32_t*>(smem);
  uint32_t* const p1 = p0 + stride;
  uint32_t* const pc = p1 + stride;
  uint16_t* const order = reinterpret_cast<uint16_t*>(pc + stride);
  if (!p.graphs)
    take_input(p, in);
  if (tid < n)
    adj[tid] = in.by_value ? in.adj[tid] : p.adj[G.adj_off + tid];
  fill_binom(binom);
  __syncthreads();
  if (tid < 32) {
    level_offsets(binom, m, off);
    const bool bad = !adjacency_ok(adj, n);
    if (tid == 0) {
      sBad = bad ? 1 : 0;
      if (bad)
        raise_error(p.error, kDevInvalidInput, g);
    }
  }
  __syncthreads();
  if (sBad) {
    report_error(p);
    return;
  }
  for_places(binom, off, 0u, m, tid >> 5, threads >> 5,
             [&](uint32_t w, uint32_t at) { order[at] = static_cast<uint16_t>(w); });
  for (int j = 0; j <= m; ++j) {
    __syncthreads();
    const uint32_t begin = off[j], count = binom[m][j];
    for (uint32_t e = tid; e < count; e += threads) {
      const uint32_t w = order[begin + e];
      Acc a;
      for (uint32_t bits = w; bits; bits &= bits - 1u) {
        const uint32_t child = w ^ (bits & (0u - bits));
        acc_add1(a, p0[child], p1[child], pc[child]);
      }
      const Planes r = j > 2 ? resolve_word(a, SmallSets{})
                             : resolve_word(a, small_sets(static_cast<uint64_t>(w) << 5, j, adj, n));
      p0[w] = r.p0;
      p1[w] = r.p1;
      pc[w] = r.c;
    }
  }
  __syncthreads();
  if (tid < 32) {
    const SmallCtx ctx{p0, p1, n};
    if (!build_tree(p, G, adj, ctx, (1u << n) - 1u) && tid == 0)
      raise_error(p.error, kDevNoRoot, g);
    report_error(p);
  } else if (p.table) {
    uint32_t* const out = reinterpret_cast<uint32_t*>(p.table + G.table_off);
    for (uint32_t t = tid - 32; t < words; t += threads - 32) {
      const uint32_t w = order[t];
      out[3 * t] = p0[w];
      out[3 * t + 1] = p1[w];
      out[3 * t + 2] = pc[w];
    }
  }
}

// ---------------------------------------------------------------------------
// Middle-sized graphs: the table in the shared memory of one cluster.
// ---------------------------------------------------------------------------

constexpr int kClusterBits = 4, kClusterThreads = 512;
static_assert(1 << kClusterBits == kDpClusterCtas);

// Three planes and the words' order, of a CTA's share.
constexpr size_t cluster_smem(int n) { return size_t(14) << (n - 5 - kClusterBits); }

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// Shared-memory address `a` of this CTA as that of CTA `rank`.
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

__device__ __forceinline__ uint32_t ld_cluster(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}

// All threads of the cluster; stores to shared memory before it are seen after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// Words of a table over the cluster's CTAs, by the top bits of the word.
struct ClusterCtx {
  uint32_t p0, p1;  // shared-memory addresses of the planes
  int m, n;         // bits of a word within a CTA
  __device__ uint32_t residue(uint64_t S) const {
    const uint32_t w = static_cast<uint32_t>(S) >> 5, bit = static_cast<uint32_t>(S) & 31u;
    const uint32_t rank = w >> m, at = 4u * (w & ((1u << m) - 1u));
    const uint32_t a = ld_cluster(map_rank(p0 + at, rank)), b = ld_cluster(map_rank(p1 + at, rank));
    return ((a >> bit) & 1u) ? 0u : 2u - ((b >> bit) & 1u);
  }
};

// The small kernel over a cluster, a CTA per value of the word's top bits (a
// single graph of kDpSmallBestN < n <= kDpClusterMaxN vertices): every CTA has
// the same words of 2^(n-9) to go through, a level later for every top bit it
// has; children without one of those are read from the neighbour CTAs' shared
// memory, and a cluster barrier parts the levels. Bound by the word chain and
// the barrier of its levels (0.8 us), the widest ones by what 16 SMs issue.
// Kernel time, us, against the small / the level and tree kernels: n = 16 25 /
// 22, 17 26 / 28, 18 29 / 39, 19 35 / 59, 20 45 / 61, 21 61 / 67, 22 - / 80.
// 8 CTAs: n = 18 30, 20 50, 21 74.
__global__ void __launch_bounds__(kClusterThreads)
    dp_cluster_kernel(const __grid_constant__ DpBatchParams p, const __grid_constant__ DpInput in) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ Binom binom;
  __shared__ uint32_t off[32];        // first place of a level within the CTA
  __shared__ uint32_t table_off[32];
  __shared__ uint64_t adj[kDpClusterMaxN];
  const uint32_t tid = threadIdx.x, threads = blockDim.x, cta = cluster_rank();
  const DpGraph G = p.single;
  const int n = G.n, M = n - 5, m = M - kClusterBits, top = __popc(cta);
  const uint32_t words = 1u << m;
  uint32_t* const p0 = reinterpret_cast<uint32_t*>(smem);
  uint32_t* const p1 = p0 + words;
  uint32_t* const pc = p1 + words;
  uint16_t* const order = reinterpret_cast<uint16_t*>(pc + words);
  if (cta == 0)
    take_input(p, in);
  if (tid < n)
    adj[tid] = in.by_value ? in.adj[tid] : p.adj[tid];
  fill_binom(binom);
  __syncthreads();
  bool bad = false;
  if (tid < 32) {
    level_offsets(binom, m, off);
    level_offsets(binom, M, table_off);
    bad = cta == 0 && !adjacency_ok(adj, n);
  }
  __syncthreads();
  for_places(binom, off, 0u, m, tid >> 5, threads >> 5,
             [&](uint32_t w, uint32_t at) { order[at] = static_cast<uint16_t>(w); });
  const uint32_t a0 = static_cast<uint32_t>(__cvta_generic_to_shared(p0)), plane = 4u * words;
  uint32_t other[kClusterBits];
  bool has[kClusterBits];
#pragma unroll
  for (int i = 0; i < kClusterBits; ++i) {
    has[i] = (cta >> i) & 1u;
    other[i] = map_rank(a0, has[i] ? cta ^ (1u << i) : cta);
  }
  for (int j = 0; j <= M; ++j) {
    cluster_sync();
    const int own = j - top;
    if (own < 0 || own > m)
      continue;
    const uint32_t begin = off[own], count = binom[m][own];
    for (uint32_t e = tid; e < count; e += threads) {
      const uint32_t w = order[begin + e];
      Acc a;
      uint32_t r0[kClusterBits], r1[kClusterBits], rc[kClusterBits];
#pragma unroll
      for (int i = 0; i < kClusterBits; ++i) {
        r0[i] = r1[i] = rc[i] = 0u;
        if (has[i]) {
          r0[i] = ld_cluster(other[i] + 4u * w);
          r1[i] = ld_cluster(other[i] + 4u * w + plane);
          rc[i] = ld_cluster(other[i] + 4u * w + 2u * plane);
        }
      }
      for (uint32_t bits = w; bits; bits &= bits - 1u) {
        const uint32_t child = w ^ (bits & (0u - bits));
        acc_add1(a, p0[child], p1[child], pc[child]);
      }
#pragma unroll
      for (int i = 0; i < kClusterBits; ++i)
        if (has[i])
          acc_add1(a, r0[i], r1[i], rc[i]);
      const uint64_t S0 = (static_cast<uint64_t>(cta) << m | w) << 5;
      const Planes r = j > 2 ? resolve_word(a, SmallSets{}) : resolve_word(a, small_sets(S0, j, adj, n));
      p0[w] = r.p0;
      p1[w] = r.p1;
      pc[w] = r.c;
    }
  }
  cluster_sync();
  if (cta == 0 && tid < 32) {
    if (bad) {
      if (tid == 0)
        raise_error(p.error, kDevInvalidInput, 0);
    } else {
      const ClusterCtx ctx{a0, a0 + plane, m, n};
      if (!build_tree(p, G, adj, ctx, (1u << n) - 1u) && tid == 0)
        raise_error(p.error, kDevNoRoot, 0);
    }
    report_error(p);
  } else {
    uint32_t* const out = reinterpret_cast<uint32_t*>(p.table + G.table_off);
    const int first = cta == 0 ? 1 : 0;
    for_places(binom, table_off, cta, m, (tid >> 5) - first, (threads >> 5) - first, [&](uint32_t w, size_t t) {
      out[3 * t] = p0[w];
      out[3 * t + 1] = p1[w];
      out[3 * t + 2] = pc[w];
    });
  }
  cluster_sync();  // CTA 0's tree reads every CTA's planes
}

// ---------------------------------------------------------------------------
// Host-side launch helpers.
// ---------------------------------------------------------------------------

// A launch of the cluster kernel. 16 CTAs are above the portable cluster size:
// dp_cluster_fits says whether the device has room for them.
struct ClusterLaunch {
  cudaLaunchAttribute attr = {};
  cudaLaunchConfig_t cfg = {};
  cudaError_t status;
  ClusterLaunch(int n, cudaStream_t s) {
    status = cudaFuncSetAttribute(dp_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(cluster_smem(kDpClusterMaxN)));
    if (status == cudaSuccess)
      status = cudaFuncSetAttribute(dp_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kDpClusterCtas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(kDpClusterCtas);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = cluster_smem(n);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
  }
};

bool dp_cluster_fits() {
  ClusterLaunch l(kDpClusterMaxN, nullptr);
  int clusters = 0;
  if (l.status == cudaSuccess)
    l.status = cudaOccupancyMaxActiveClusters(&clusters, dp_cluster_kernel, &l.cfg);
  if (l.status != cudaSuccess)
    cudaGetLastError();  // not an error of the call that asked
  return l.status == cudaSuccess && clusters > 0;
}

cudaError_t dp_launch_cluster(const DpBatchParams& p, cudaStream_t s, const DpInput& in) {
  ClusterLaunch l(p.single.n, s);
  return l.status != cudaSuccess ? l.status : cudaLaunchKernelEx(&l.cfg, dp_cluster_kernel, p, in);
}

template <int LB>
static cudaError_t launch_tiles(const DpBatchParams& p, int ctas, cudaStream_t s) {
  dp_tile_kernel<LB><<<ctas, kDpThreads, smem_layout_for(LB, LB, p.kid_rows).bytes, s>>>(p);
  return cudaGetLastError();
}

template <typename Kernel>
static int occupancy_of(Kernel kernel, const SmemLayout& at, const SmemLayout& most) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most.bytes)) !=
      cudaSuccess)
    return 0;
  int blocks = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, kDpThreads, at.bytes);
  return blocks;
}

int dp_tile_occupancy(int lb, int kid_rows) {
  switch (lb) {
#define GTD_CASE(X) \
  case X:           \
    return occupancy_of(dp_tile_kernel<X>, smem_layout_for(X, X, kid_rows), smem_layout_for(X, X, kDpMaxHigh));
    GTD_CASE(8) GTD_CASE(9) GTD_CASE(10) GTD_CASE(11) GTD_CASE(12)
#undef GTD_CASE
    default:
      return 0;
  }
}

cudaError_t dp_launch_validate(const DpBatchParams& p, cudaStream_t s, const DpInput& in) {
  dp_validate_kernel<<<(p.num_graphs + 3) / 4, 128, 0, s>>>(p, in);  // one warp per graph
  return cudaGetLastError();
}

cudaError_t dp_launch_fill_tile_map(const DpBatchParams& p, cudaStream_t s) {
  const int blocks = p.num_graphs < 4096 ? p.num_graphs : 4096;
  dp_fill_tile_map_kernel<<<blocks, 256, 0, s>>>(p);
  return cudaGetLastError();
}

int dp_mixed_occupancy(int lb, int kid_rows) {
  return occupancy_of(dp_tile_kernel_mixed, smem_layout_for(kDpMinTileBits, lb, kid_rows),
                      smem_layout_for(kDpMinTileBits, kDpMaxTileBits, kDpMaxHigh));
}

cudaError_t dp_launch_small(const DpBatchParams& p, int max_n, cudaStream_t s, const DpInput& in) {
  const size_t smem = small_smem(max_n);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(dp_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(small_smem(kDpSmallMaxN)));
    if (e != cudaSuccess)
      return e;
  }
  // threads: the words of the widest level, 64 to 512 (128 for thousands of
  // graphs, which fill the GPU side by side; with 512, 48 graphs of up to 16
  // vertices take 24 us instead of 29, 300 of 16 31 instead of 34, 1000 the same)
  const bool many = p.num_graphs > 1024;
  const int threads = max_n <= 13 ? 64 : max_n == 14 || many ? 128 : max_n == 15 ? 256 : 512;
  dp_small_kernel<<<p.num_graphs, threads, smem, s>>>(p, max_n, in);
  return cudaGetLastError();
}

int dp_level_occupancy(int kid_rows) {
  const int smem = static_cast<int>(sizeof(uint32_t)) * kLevelThreads * kid_rows;
  int blocks = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, dp_level_kernel<true>, kLevelThreads, smem);
  return blocks;
}

cudaError_t dp_launch_levels(const DpBatchParams& p, int ctas, cudaStream_t s) {
  const size_t smem = sizeof(uint32_t) * kLevelThreads * p.kid_rows;
  if (p.graphs)
    dp_level_kernel<true><<<ctas, kLevelThreads, smem, s>>>(p);
  else
    dp_level_kernel<false><<<ctas, kLevelThreads, smem, s>>>(p);
  return cudaGetLastError();
}

cudaError_t dp_launch_tiles(const DpBatchParams& p, int ctas, cudaStream_t s) {
  if (p.mixed) {
    if (p.lb < kDpMinTileBits || p.lb > kDpMaxTileBits)
      return cudaErrorInvalidValue;
    dp_tile_kernel_mixed<<<ctas, kDpThreads, smem_layout_for(kDpMinTileBits, p.lb, p.kid_rows).bytes, s>>>(p);
    return cudaGetLastError();
  }
  switch (p.lb) {
#define GTD_CASE(X) \
  case X:           \
    return launch_tiles<X>(p, ctas, s);
    GTD_CASE(8) GTD_CASE(9) GTD_CASE(10) GTD_CASE(11) GTD_CASE(12)
#undef GTD_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t dp_launch_tree(const DpBatchParams& p, cudaStream_t s) {
  int blocks = (p.num_graphs + kTreeWarps - 1) / kTreeWarps;
  if (blocks > 4096)
    blocks = 4096;
  dp_tree_kernel<<<blocks, 32 * kTreeWarps, 0, s>>>(p);
  return cudaGetLastError();
}

// Training labels from a solved table (single graph): for each subset S,
// td(S) and, when S is connected, its optimal-root set
// R(S) = {v in S : td(S - v) = td(S) - 1} (one warp per subset).
__global__ void __launch_bounds__(32 * kTreeWarps)
    dp_labels_kernel(const __grid_constant__ DpBatchParams p, const uint64_t* subsets, int count, int32_t* td_out,
                     uint64_t* roots_out) {
  __shared__ Binom sBinom;
  fill_binom(sBinom);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const DpGraph G = p.single;
  __shared__ uint32_t sOff[32];
  if (warp == 0)
    level_offsets(sBinom, G.nh, sOff);
  __syncthreads();
  const TreeCtx ctx{sBinom, sOff, p.table + G.table_off, G.lb, G.n};
  for (int i = blockIdx.x * kTreeWarps + warp; i < count; i += gridDim.x * kTreeWarps) {
    const uint64_t S = subsets[i];
    if (S == 0) {
      if (lane == 0) {
        td_out[i] = 0;
        roots_out[i] = 0;
      }
      continue;
    }
    const Chain chain = load_chain(ctx, S);
    const bool in_lo = (S >> lane) & 1ull, in_hi = (S >> (lane + 32)) & 1ull;
    const uint32_t t_lo = in_lo ? ctx.residue(S & ~(1ull << lane)) : 3u;
    const uint32_t t_hi = in_hi ? ctx.residue(S & ~(1ull << (lane + 32))) : 3u;
    const uint32_t td = chain_td(chain, G.n), below = (td + 2u) % 3u;  // residue of td - 1
    const bool lo = t_lo == below, hi = t_hi == below;
    const uint64_t roots = ballot64(lo, hi);
    if (lane == 0) {
      td_out[i] = static_cast<int32_t>(td);
      roots_out[i] = roots;
    }
  }
}

cudaError_t dp_launch_labels(const DpBatchParams& p, const uint64_t* subsets, int count, int32_t* td_out,
                             uint64_t* roots_out, cudaStream_t s) {
  int blocks = (count + kTreeWarps - 1) / kTreeWarps;
  if (blocks > 8192)
    blocks = 8192;
  if (blocks < 1)
    blocks = 1;
  dp_labels_kernel<<<blocks, 32 * kTreeWarps, 0, s>>>(p, subsets, count, td_out, roots_out);
  return cudaGetLastError();
}

// Tiles [first, end) of the byte table of gtd_dp_table (td << 1 | connected per
// subset, tiles of 2^lb bytes in tile order; the planes may have tiles of
// another size), one warp per tile: td(H) from the warp's chain, each word's first subset along
// the chain of its bits, the word's subsets from one another.
__global__ void __launch_bounds__(32 * kTreeWarps)
    dp_expand_kernel(const __grid_constant__ DpBatchParams p, int lb, uint32_t first_tile, uint32_t end, uint8_t* out,
                     uint64_t bytes) {
  __shared__ Binom sBinom;
  fill_binom(sBinom);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const DpGraph G = p.single;
  __shared__ uint32_t sOff[32];
  if (warp == 0)
    level_offsets(sBinom, G.nh, sOff);
  __syncthreads();
  const TreeCtx ctx{sBinom, sOff, p.table + G.table_off, G.lb, G.n};
  const int nh = G.n > lb ? G.n - lb : 0;
  const uint32_t words = lb > 5 ? 1u << (lb - 5) : 1u;
  for (uint32_t t = first_tile + blockIdx.x * kTreeWarps + warp; t < end; t += gridDim.x * kTreeWarps) {
    uint32_t r = t, H = 0;
    int j = 0;
    while (r >= sBinom[nh][j])
      r -= sBinom[nh][j++];
    for (int a = nh - 1, k = j; k > 0; --a)
      if (r >= sBinom[a][k]) {
        r -= sBinom[a][k--];
        H |= 1u << a;
      }
    const uint64_t high = static_cast<uint64_t>(H) << lb;
    const uint32_t base = chain_td(load_chain(ctx, high), G.n);
    auto first = [&](uint32_t w) { return ctx.residue(high | (static_cast<uint64_t>(w) << 5)); };
    for (uint32_t w = lane; w < words; w += 32) {
      uint32_t td[32];
      td[0] = base;
      uint32_t here = first(w);
      for (uint32_t x = w; x; x &= x - 1) {
        const uint32_t next = first(x & (x - 1));
        td[0] += here != next;
        here = next;
      }
      const uint32_t* word = ctx.word(high | (static_cast<uint64_t>(w) << 5));
      const uint32_t stride = 1u << (G.lb - 5), p0 = word[0], p1 = word[stride], c = word[2 * stride];
      // residue changes between x and x without its lowest bit: treedepth + 1
#pragma unroll
      for (int x = 1; x < 32; ++x) {
        const int y = x & (x - 1);
        td[x] = td[y] + ((((p0 >> x) ^ (p0 >> y)) | ((p1 >> x) ^ (p1 >> y))) & 1u);
      }
      const uint64_t at = (static_cast<uint64_t>(t - first_tile) << lb) + w * 32u;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t v = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b)
          v |= (td[4 * i + b] << 1 | ((c >> (4 * i + b)) & 1u)) << (8 * b);
        if (at + 4 * i + 4 <= bytes)
          *reinterpret_cast<uint32_t*>(out + at + 4 * i) = v;
      }
    }
  }
}

cudaError_t dp_launch_expand(const DpBatchParams& p, int lb, uint32_t first, uint32_t end, uint8_t* out,
                             uint64_t bytes, cudaStream_t s) {
  const uint32_t ctas = (end - first + kTreeWarps - 1) / kTreeWarps;
  dp_expand_kernel<<<ctas < 16384u ? ctas : 16384u, 32 * kTreeWarps, 0, s>>>(p, lb, first, end, out, bytes);
  return cudaGetLastError();
}

}  // namespace gtd
