// Kernel parameters and launchers of the subset DP (K1). Host and device.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gtd_dp_layout.h"

namespace gtd {

// One graph of a DP launch (40 bytes). A graph with n < lb is padded with
// isolated vertices up to lb (one tile); padding changes no treedepth of a
// real subset and the reconstruction never touches padded vertices.
struct DpGraph {
  uint64_t table_off = 0;  // byte offset of the graph's table in the table pool
  uint32_t flag_base = 0;  // first flag of the graph (graph-major count of tile groups)
  uint32_t ntiles = 0;     // 2^nh
  uint32_t adj_off = 0;    // first adjacency mask; also the first output slot
  int32_t n = 0;           // real vertices
  int32_t nh = 0;          // high vertices (max(n - lb, 0))
  int32_t out_idx = 0;     // position of the graph in the caller's arrays (td_out)
  int32_t lb = 0;          // tile bits of this graph's table
};
static_assert(sizeof(DpGraph) == 40);

// Passed by value as a __grid_constant__ kernel parameter.
struct DpBatchParams {
  const DpGraph* graphs = nullptr;  // device descriptors; nullptr: only `single`
  DpGraph single;
  uint2* tile_map = nullptr;        // ticket -> (graph, its tile group) (batches)
  const uint32_t* level_base = nullptr;  // [graph][level] first ticket (batches)
  int num_graphs = 1;
  int first_graph = 0;              // number of graphs[0] (the small kernel starts there)
  int lb = 0;                       // tile bits of this launch (mixed batches: the largest)
  int kid_rows = 0;                 // largest nh of the launch's graphs
  int mixed = 0;                    // 1: graphs carry their own tile bits (DpGraph::lb)
  uint32_t total_groups = 0;        // tickets: groups of tiles of one level
  uint8_t* table = nullptr;         // table pool: tiles of three bit planes
  uint32_t* flags = nullptr;        // one ready stamp per tile group
  uint32_t* ticket = nullptr;       // work counter, zeroed before each launch
  uint32_t* level_done = nullptr;   // chunks done per level (level kernel), 32 words per graph, zeroed before each launch
  int32_t* error = nullptr;         // [0] code, [1] info
  const uint64_t* adj = nullptr;    // adjacency pool (device)
  uint32_t epoch = 0;               // flags equal to epoch are ready
  uint64_t timeout_ns = 0;          // bound of every dependency wait
  // reconstruction outputs (device): td_out[g], parent_out[adj_off + v],
  // order_out[adj_off + step]; query != 0 restricts a single graph to a subset
  uint64_t query = 0;
  int32_t* td_out = nullptr;
  int32_t* parent_out = nullptr;
  int32_t* order_out = nullptr;
  int32_t* report = nullptr;        // error code and info once the tree is built (host memory; may be null)
};

// What a single solve hands its first kernel instead of copying and clearing
// beforehand: the adjacency by value (put down at p.adj for the kernels after
// it) and the control words to zero.
struct DpInput {
  uint64_t adj[kDpMaxN] = {};
  int32_t by_value = 0;      // 1: adj holds the graph's masks
  int32_t clear_words = 0;
  int32_t* clear = nullptr;
};

// CTAs per SM with tiles of lb bits and up to kid_rows high vertices, and of
// the mixed-tile-size kernel with tiles of up to lb bits.
int dp_tile_occupancy(int lb, int kid_rows);
int dp_mixed_occupancy(int lb, int kid_rows);
cudaError_t dp_launch_validate(const DpBatchParams& p, cudaStream_t s, const DpInput& in = DpInput{});
cudaError_t dp_launch_fill_tile_map(const DpBatchParams& p, cudaStream_t s);
cudaError_t dp_launch_tiles(const DpBatchParams& p, int ctas, cudaStream_t s);
// The level kernel (tiles of kDpLevelTileBits, n >= that): total_groups counts
// chunks of kDpLevelChunk tiles of one level.
int dp_level_occupancy(int kid_rows);
cudaError_t dp_launch_levels(const DpBatchParams& p, int ctas, cudaStream_t s);
// The small kernel: p.num_graphs graphs, from p.first_graph on, of at most
// max_n <= kDpSmallMaxN vertices, checked, solved and reconstructed; p.table
// (tiles of kDpSmallTileBits) may be null.
cudaError_t dp_launch_small(const DpBatchParams& p, int max_n, cudaStream_t s, const DpInput& in = DpInput{});
// The cluster kernel: as the small kernel, for one graph of kDpSmallBestN <
// n <= kDpClusterMaxN vertices, on a device that has room for the cluster.
bool dp_cluster_fits();
cudaError_t dp_launch_cluster(const DpBatchParams& p, cudaStream_t s, const DpInput& in);
cudaError_t dp_launch_tree(const DpBatchParams& p, cudaStream_t s);
cudaError_t dp_launch_labels(const DpBatchParams& p, const uint64_t* subsets, int count, int32_t* td_out,
                             uint64_t* roots_out, cudaStream_t s);
// Tiles [first, end) (2^lb bytes each, `bytes` in all) of the byte table (td << 1
// | connected, 2^n bytes) of a solved single graph.
cudaError_t dp_launch_expand(const DpBatchParams& p, int lb, uint32_t first, uint32_t end, uint8_t* out,
                             uint64_t bytes, cudaStream_t s);

}  // namespace gtd
