// A small message-passing GNN that scores vertices as roots of an optimal
// elimination tree, with hand-written forward, backward and Adam kernels.
// It is used only to ORDER the branch and bound's candidates and to seed its
// incumbent (greedy elimination by score); it never prunes, so every
// treedepth stays proven by the exact search. No counterpart exists in the
// reference.
//
// Network (hidden H = 64 by default, L = 3 layers):
//   h0      = relu(x W_in + b_in)                       x: per-vertex features
//   a_l(v)  = mean_{u in N(v)} h_l(u)                   (0 for isolated v)
//   h_{l+1} = relu(h_l Ws_l + a_l Wn_l + b_l)
//   logit_v = h_L(v) . w_out + b_out                    root score
//   td_g    = mean_{v in g} h_L(v) . w_g + b_g          treedepth estimate
// Weights are stored in BF16 (a BF16 copy of an FP32 master kept by Adam);
// every product accumulates in FP32. Loss: masked mean binary cross entropy
// of the root logits + td_weight * mean squared td error.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <new>
#include <string>
#include <type_traits>
#include <vector>

#include "gtd_handle.h"

namespace gtd {
namespace {

constexpr int kNodesPerBlock = 16;
constexpr int kMaxK = 64;

__device__ __forceinline__ float bf(const __nv_bfloat16 x) { return __bfloat162float(x); }

// Z = X1 W1 (+ X2 W2) + bias; Hout = relu(Z). X rows of K floats, W K x H
// (row major, BF16), one thread per output channel, kNodesPerBlock nodes per
// block, weights staged in shared memory.
__global__ void node_linear(int N, int K, int H, const float* __restrict__ X1, const __nv_bfloat16* __restrict__ W1,
                            const float* __restrict__ X2, const __nv_bfloat16* __restrict__ W2,
                            const __nv_bfloat16* __restrict__ bias, float* __restrict__ Z, float* __restrict__ Hout) {
  __shared__ float w1[kMaxK * kMaxK], w2[kMaxK * kMaxK];
  __shared__ float x1[kNodesPerBlock][kMaxK], x2[kNodesPerBlock][kMaxK];
  const int j = threadIdx.x;
  for (int t = threadIdx.x; t < K * H; t += blockDim.x) {
    w1[t] = bf(W1[t]);
    if (X2)
      w2[t] = bf(W2[t]);
  }
  const int v0 = blockIdx.x * kNodesPerBlock;
  for (int t = threadIdx.x; t < kNodesPerBlock * K; t += blockDim.x) {
    const int r = t / K, i = t % K;
    const int v = v0 + r;
    x1[r][i] = v < N ? X1[size_t(v) * K + i] : 0.f;
    if (X2)
      x2[r][i] = v < N ? X2[size_t(v) * K + i] : 0.f;
  }
  __syncthreads();
  if (j >= H)
    return;
  float acc[kNodesPerBlock];
  const float b = bf(bias[j]);
#pragma unroll
  for (int r = 0; r < kNodesPerBlock; ++r)
    acc[r] = b;
  for (int i = 0; i < K; ++i) {
    const float wa = w1[i * H + j];
#pragma unroll
    for (int r = 0; r < kNodesPerBlock; ++r)
      acc[r] = fmaf(x1[r][i], wa, acc[r]);
  }
  if (X2)
    for (int i = 0; i < K; ++i) {
      const float wb = w2[i * H + j];
#pragma unroll
      for (int r = 0; r < kNodesPerBlock; ++r)
        acc[r] = fmaf(x2[r][i], wb, acc[r]);
    }
#pragma unroll
  for (int r = 0; r < kNodesPerBlock; ++r) {
    const int v = v0 + r;
    if (v < N) {
      Z[size_t(v) * H + j] = acc[r];
      Hout[size_t(v) * H + j] = fmaxf(acc[r], 0.f);
    }
  }
}

// dX = dZ W^T (W K x H): one thread per input channel i.
__global__ void node_linear_t(int N, int K, int H, const float* __restrict__ dZ, const __nv_bfloat16* __restrict__ W,
                              float* __restrict__ dX) {
  __shared__ float w[kMaxK * kMaxK];
  __shared__ float dz[kNodesPerBlock][kMaxK];
  for (int t = threadIdx.x; t < K * H; t += blockDim.x)
    w[t] = bf(W[t]);
  const int v0 = blockIdx.x * kNodesPerBlock;
  for (int t = threadIdx.x; t < kNodesPerBlock * H; t += blockDim.x) {
    const int r = t / H, j = t % H;
    const int v = v0 + r;
    dz[r][j] = v < N ? dZ[size_t(v) * H + j] : 0.f;
  }
  __syncthreads();
  const int i = threadIdx.x;
  if (i >= K)
    return;
  float acc[kNodesPerBlock] = {};
  for (int j = 0; j < H; ++j) {
    const float wij = w[i * H + j];
#pragma unroll
    for (int r = 0; r < kNodesPerBlock; ++r)
      acc[r] = fmaf(dz[r][j], wij, acc[r]);
  }
#pragma unroll
  for (int r = 0; r < kNodesPerBlock; ++r) {
    const int v = v0 + r;
    if (v < N)
      dX[size_t(v) * K + i] = acc[r];
  }
}

// Partial X^T dZ (and column sums of dZ) of a chunk of 64 nodes per block,
// written to part[block][K * H + H]; reduce_partials adds the chunks in a
// fixed order, so the gradient (and training) is deterministic.
__global__ void weight_grad(int N, int K, int H, const float* __restrict__ X, const float* __restrict__ dZ,
                            float* __restrict__ part) {
  constexpr int kChunk = 64;
  __shared__ float xs[kChunk][kMaxK], ds[kChunk][kMaxK];
  const int v0 = blockIdx.x * kChunk;
  const int nv = min(kChunk, N - v0);
  for (int t = threadIdx.x; t < kChunk * kMaxK; t += blockDim.x) {
    const int r = t / kMaxK, c = t % kMaxK;
    xs[r][c] = (r < nv && c < K) ? X[size_t(v0 + r) * K + c] : 0.f;
    ds[r][c] = (r < nv && c < H) ? dZ[size_t(v0 + r) * H + c] : 0.f;
  }
  __syncthreads();
  float* out = part + size_t(blockIdx.x) * (K * H + H);
  for (int t = threadIdx.x; t < K * H; t += blockDim.x) {
    const int i = t / H, j = t % H;
    float acc = 0.f;
    for (int r = 0; r < nv; ++r)
      acc = fmaf(xs[r][i], ds[r][j], acc);
    out[t] = acc;
  }
  for (int j = threadIdx.x; j < H; j += blockDim.x) {
    float acc = 0.f;
    for (int r = 0; r < nv; ++r)
      acc += ds[r][j];
    out[K * H + j] = acc;
  }
}

// dW += sum over chunks of the partials, db likewise (when non-null).
__global__ void reduce_partials(int chunks, int KH, int H, const float* __restrict__ part, float* __restrict__ dW,
                                float* __restrict__ db) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= KH + H || (t >= KH && !db))
    return;
  float acc = 0.f;
  for (int c = 0; c < chunks; ++c)
    acc += part[size_t(c) * (KH + H) + t];
  if (t < KH)
    dW[t] += acc;
  else
    db[t - KH] += acc;
}

// a(v) = mean over neighbours of h(u); one thread per (v, channel).
__global__ void aggregate(int N, int H, const int32_t* __restrict__ nbr_start, const int32_t* __restrict__ nbr,
                          const float* __restrict__ h, float* __restrict__ a) {
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(N) * H)
    return;
  const int v = static_cast<int>(t / H), j = static_cast<int>(t % H);
  const int s = nbr_start[v], e = nbr_start[v + 1];
  float acc = 0.f;
  for (int k = s; k < e; ++k)
    acc += h[size_t(nbr[k]) * H + j];
  a[t] = e > s ? acc / float(e - s) : 0.f;
}

// Backward of the mean: dh(u) += sum over neighbours v of da(v) / deg(v)
// (adjacency is symmetric, so this is a gather, no atomics).
__global__ void aggregate_t(int N, int H, const int32_t* __restrict__ nbr_start, const int32_t* __restrict__ nbr,
                            const float* __restrict__ da, float* __restrict__ dh) {
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(N) * H)
    return;
  const int u = static_cast<int>(t / H), j = static_cast<int>(t % H);
  float acc = 0.f;
  for (int k = nbr_start[u]; k < nbr_start[u + 1]; ++k) {
    const int v = nbr[k];
    const int dv = nbr_start[v + 1] - nbr_start[v];
    acc += da[size_t(v) * H + j] / float(dv);
  }
  dh[t] += acc;
}

__global__ void relu_mask(size_t count, const float* __restrict__ z, const float* __restrict__ dh,
                          float* __restrict__ dz) {
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < count)
    dz[t] = z[t] > 0.f ? dh[t] : 0.f;
}

// Heads: logits per node; pooled mean per graph; td estimate per graph.
__global__ void heads_forward(int N, int G, int H, const float* __restrict__ h, const int32_t* __restrict__ gstart,
                              const __nv_bfloat16* __restrict__ w_out, const __nv_bfloat16* __restrict__ b_out,
                              const __nv_bfloat16* __restrict__ w_g, const __nv_bfloat16* __restrict__ b_g,
                              float* __restrict__ logits, float* __restrict__ pooled, float* __restrict__ td_est) {
  // blocks [0, ceil(N/128)) do logits; the next G blocks do the graphs
  const int nb = (N + 127) / 128;
  if (static_cast<int>(blockIdx.x) < nb) {
    const int v = blockIdx.x * 128 + threadIdx.x;
    if (v < N) {
      float acc = bf(b_out[0]);
      for (int j = 0; j < H; ++j)
        acc = fmaf(h[size_t(v) * H + j], bf(w_out[j]), acc);
      logits[v] = acc;
    }
    return;
  }
  const int g = blockIdx.x - nb;
  if (g >= G)
    return;
  __shared__ float part[128];
  const int s = gstart[g], e = gstart[g + 1];
  const int j = threadIdx.x;
  float m = 0.f;
  if (j < H) {
    for (int v = s; v < e; ++v)
      m += h[size_t(v) * H + j];
    m = e > s ? m / float(e - s) : 0.f;
    pooled[size_t(g) * H + j] = m;
  }
  part[threadIdx.x] = j < H ? m * bf(w_g[j]) : 0.f;
  __syncthreads();
  for (int off = 64; off > 0; off >>= 1) {
    if (threadIdx.x < off)
      part[threadIdx.x] += part[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    td_est[g] = part[0] + bf(b_g[0]);
}

// Loss and the head gradients w.r.t. the logits and td estimates (a thread per
// node and per graph): writes dlogit (per node), dtd (per graph) and dh_L = dlogit w_out + dtd w_g / |g|.
__global__ void heads_backward(int N, int G, int H, const int32_t* __restrict__ gstart,
                               const int32_t* __restrict__ graph_of, const float* __restrict__ logits,
                               const float* __restrict__ td_est, const float* __restrict__ y,
                               const float* __restrict__ mask, const float* __restrict__ td_label, float inv_mask_sum,
                               float td_weight, const __nv_bfloat16* __restrict__ w_out,
                               const __nv_bfloat16* __restrict__ w_g, float* __restrict__ dlogit,
                               float* __restrict__ dtd, float* __restrict__ dh, float* __restrict__ loss) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < G) {  // graph v, which may have no node
    const float diff = td_est[v] - td_label[v];
    dtd[v] = 2.f * td_weight * diff / float(G);
    atomicAdd(loss, td_weight * diff * diff / float(G));
  }
  if (v >= N)
    return;
  const float z = logits[v];
  const float m = mask[v];
  const float sig = 1.f / (1.f + expf(-z));
  const float dl = m * (sig - y[v]) * inv_mask_sum;
  atomicAdd(loss, m * (fmaxf(z, 0.f) - z * y[v] + log1pf(expf(-fabsf(z)))) * inv_mask_sum);
  dlogit[v] = dl;
  const int g = graph_of[v];
  const float diff = td_est[g] - td_label[g];
  const float dt = 2.f * td_weight * diff / float(G);
  const float ng = float(gstart[g + 1] - gstart[g]);
  for (int j = 0; j < H; ++j)
    dh[size_t(v) * H + j] = dl * bf(w_out[j]) + dt * bf(w_g[j]) / ng;
}

__global__ void adam_step(int64_t n, float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                          const float* __restrict__ g, __nv_bfloat16* __restrict__ w, float lr, float b1, float b2,
                          float eps, float c1, float c2) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n)
    return;
  const float gt = g[t];
  const float mt = b1 * m[t] + (1.f - b1) * gt;
  const float vt = b2 * v[t] + (1.f - b2) * gt * gt;
  m[t] = mt;
  v[t] = vt;
  const float upd = lr * (mt / c1) / (sqrtf(vt / c2) + eps);
  const float nm = master[t] - upd;
  master[t] = nm;
  w[t] = __float2bfloat16_rn(nm);
}

__global__ void to_bf16(int64_t n, const float* __restrict__ src, __nv_bfloat16* __restrict__ dst) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < n)
    dst[t] = __float2bfloat16_rn(src[t]);
}

unsigned blocks_for(size_t n, unsigned t) { return static_cast<unsigned>((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// Whole network per tile. A node's neighbours lie in its own graph, so a CTA
// that holds a run of whole graphs (a tile, at most M nodes) computes every
// layer, and for training the backward pass, from shared memory in one launch.
// Training then takes the weight gradients of all layers in a second launch and
// their sums in a third. Every sum runs in the order of the layer-by-layer
// kernels above, so results are the same bit for bit (but for the loss, whose
// order those leave open). Width 64; other widths, graphs larger than a tile or
// without nodes and neighbours outside their graph take the layer-by-layer
// kernels.
// ---------------------------------------------------------------------------

constexpr int kWide = 64;            // hidden width
constexpr int kRow = kWide + 4;      // row stride in shared memory (16-byte rows, banks spread)
constexpr int kTileThreads = 256;
constexpr int kRowGroups = kTileThreads / 16;  // 16 threads take the 64 columns of a row
constexpr int kGradThreads = 256;

struct TileParams {
  int fin, layers;
  const float* x;
  const int32_t* gstart;
  const int32_t* nbr_start;
  const int32_t* nbr;
  const int32_t* tile_graph;   // [tiles + 1]: first graph of every tile
  const __nv_bfloat16* w;      // all parameters
  float* logits;
  float* td_est;
  int32_t* outside;            // set when a neighbour lies outside its tile
  // training
  const float* y;
  const float* mask;
  const float* td_label;
  float inv_mask_sum, td_weight;
  int num_nodes, num_graphs;
  float *hs, *as, *dzs;        // [layers + 1], [layers], [layers + 1] x nodes x 64: kept for the weight gradients
  float *pooled, *dlogit, *dtd;
  float* tile_loss;            // [tiles]
  int64_t nparams;
  float* part;                 // [kGradRun][nparams]: weight gradients of the chunks of 64 rows of a run
  int first_chunk;             // of the run
  float* grad_copy;            // the gradient once more next to the flag and the loss, for the one copy back (or null)
};

// Chunks whose weight gradients are held at a time (51 MB with three layers).
// More of them, from 32,769 nodes on, take further launches: all at once, with
// eight layers, a training step took 1.4 times the memory of the layer-by-layer
// kernels, which hold one matrix's.
constexpr int kGradRun = 512;

// BF16 weights (rows of 64, 16-byte aligned: every parameter block starts at a
// multiple of 64 values) to FP32 rows of kRow, in two halves: the loads can be
// on their way while the destination is still in use.
template <int ROWS>
struct WeightRegs {
  static constexpr int kVec = ROWS * kWide / 8 / kTileThreads;
  uint4 v[kVec];
  __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ w) {
#pragma unroll
    for (int q = 0; q < kVec; ++q)
      v[q] = __ldg(reinterpret_cast<const uint4*>(w) + threadIdx.x + q * kTileThreads);
  }
  __device__ __forceinline__ void store(float* out) const {
#pragma unroll
    for (int q = 0; q < kVec; ++q) {
      const int t = threadIdx.x + q * kTileThreads;
      float* const to = out + (t / 8) * kRow + 8 * (t % 8);
      const uint32_t w[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
      float f[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      }
      *reinterpret_cast<float4*>(to) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(to + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
  }
};

// x / d, correctly rounded as the division is, from inv = 1 / d correctly
// rounded: with the residue of q = x inv exact in a fused multiply-add,
// q + residue * inv rounds to the quotient (Markstein's theorem; compared in
// integers for every significand over every odd d below 300, and for random
// ones over every d up to 4096: a node may have more neighbours than a tile has
// nodes, where its list repeats them). The residue is exact above the denormal
// range; an infinite or NaN q is the quotient itself. One division per node in place of one per channel, which took 60 %
// of the aggregation.
__device__ __forceinline__ float quotient(float x, float d, float inv) {
  const float q = x * inv, residue = fmaf(-q, d, x);
  return residue == residue ? fmaf(residue, inv, q) : q;
}

// acc[i][c] += X[row i][k] W[k][4 col + c] for k < K (a multiple of 4), in
// ascending k: the same sums, bit for bit, as one thread per output. With few
// rows per thread the next four k are loaded while these are multiplied.
template <int R>
struct Step {
  float4 x[R], w[4];
};

template <int R>
__device__ __forceinline__ void step_mul(const Step<R>& s, float (&acc)[R][4]) {
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float xs[4] = {s.x[i].x, s.x[i].y, s.x[i].z, s.x[i].w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc[i][0] = fmaf(xs[q], s.w[q].x, acc[i][0]);
      acc[i][1] = fmaf(xs[q], s.w[q].y, acc[i][1]);
      acc[i][2] = fmaf(xs[q], s.w[q].z, acc[i][2]);
      acc[i][3] = fmaf(xs[q], s.w[q].w, acc[i][3]);
    }
  }
}

template <int R>
__device__ __forceinline__ void tile_product(const float* X, const float* W, int K, float (&acc)[R][4]) {
  const int col = 4 * (threadIdx.x % 16), row = threadIdx.x / 16;
  auto load = [&](int k, Step<R>& s) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      s.w[q] = *reinterpret_cast<const float4*>(W + (k + q) * kRow + col);
#pragma unroll
    for (int i = 0; i < R; ++i)
      s.x[i] = *reinterpret_cast<const float4*>(X + (i * kRowGroups + row) * kRow + k);
  };
  if constexpr (R > 4) {  // enough independent products per load; registers for two CTAs per SM
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
      Step<R> a;
      load(k, a);
      step_mul<R>(a, acc);
    }
    return;
  }
  Step<R> a, b;
  load(0, a);
#pragma unroll 1
  for (int k = 0; k < K; k += 8) {
    if (k + 4 < K)
      load(k + 4, b);
    step_mul<R>(a, acc);
    if (k + 8 < K)
      load(k + 8, a);
    if (k + 4 < K)
      step_mul<R>(b, acc);
  }
}

// out = relu(b + X1 W1 (+ X2 W2)), rows < kRowGroups R; out may be X1.
template <int R>
__device__ __forceinline__ void tile_layer(const float* X1, const float* W1, int K1, const float* X2, const float* W2,
                                           const __nv_bfloat16* __restrict__ bias, float* out) {
  const int col = 4 * (threadIdx.x % 16), row = threadIdx.x / 16;
  float acc[R][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float b = bf(bias[col + c]);
#pragma unroll
    for (int i = 0; i < R; ++i)
      acc[i][c] = b;
  }
  tile_product<R>(X1, W1, K1, acc);
  if (X2)
    tile_product<R>(X2, W2, kWide, acc);
  __syncthreads();  // every read of X1 before `out` is written
#pragma unroll
  for (int i = 0; i < R; ++i)
    *reinterpret_cast<float4*>(out + (i * kRowGroups + row) * kRow + col) =
        make_float4(fmaxf(acc[i][0], 0.f), fmaxf(acc[i][1], 0.f), fmaxf(acc[i][2], 0.f), fmaxf(acc[i][3], 0.f));
}

// out[v][i] = sum_j Z[v][j] W[i][j], rows < kRowGroups R; with `start` divided by the
// number of v's neighbours.
template <int R>
__device__ __forceinline__ void tile_product_t(const float* Z, const float* W, float* out,
                                               const int32_t* start = nullptr) {
  const int c = threadIdx.x % 16, row = threadIdx.x / 16;
  float acc[R][4] = {};
  auto load = [&](int j, Step<R>& s) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      s.w[q] = *reinterpret_cast<const float4*>(W + (c + 16 * q) * kRow + j);
#pragma unroll
    for (int i = 0; i < R; ++i)
      s.x[i] = *reinterpret_cast<const float4*>(Z + (i * kRowGroups + row) * kRow + j);
  };
  auto mul = [&](const Step<R>& s) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        acc[i][q] = fmaf(s.x[i].w, s.w[q].w,
                         fmaf(s.x[i].z, s.w[q].z, fmaf(s.x[i].y, s.w[q].y, fmaf(s.x[i].x, s.w[q].x, acc[i][q]))));
  };
  Step<R> s, t;
  load(0, s);
#pragma unroll 1
  for (int j = 0; j < kWide; j += 8) {
    load(j + 4, t);
    mul(s);
    if (j + 8 < kWide)
      load(j + 8, s);
    mul(t);
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int v = i * kRowGroups + row;
    if (start) {
      const float d = static_cast<float>(max(1, start[v + 1] - start[v]));  // without neighbours: not read
      const float inv = 1.f / d;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        out[v * kRow + c + 16 * q] = quotient(acc[i][q], d, inv);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        out[v * kRow + c + 16 * q] = acc[i][q];
    }
  }
}

// Rows per thread that hold nodes: only those are computed.
template <int M, typename F>
__device__ __forceinline__ void for_rows(int nodes, F f) {
  switch ((nodes + kRowGroups - 1) / kRowGroups) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: if constexpr (M >= 64) f(std::integral_constant<int, 3>{}); break;
    case 4: if constexpr (M >= 64) f(std::integral_constant<int, 4>{}); break;
    case 5: if constexpr (M >= 128) f(std::integral_constant<int, 5>{}); break;
    case 6: if constexpr (M >= 128) f(std::integral_constant<int, 6>{}); break;
    case 7: if constexpr (M >= 128) f(std::integral_constant<int, 7>{}); break;
    default: if constexpr (M >= 128) f(std::integral_constant<int, 8>{}); break;
  }
}

// Neighbour lists of a tile: first list entry of every node (relative to the
// tile's first) and, where they fit, the neighbours as node numbers inside the
// tile (else they are read from the batch's list each time).
struct TileGraph {
  const int32_t* start;   // [M + 1] shared; padding nodes have no neighbours
  const uint8_t* local;   // shared, or null
  const int32_t* nbr;     // the tile's part of the batch's list
  int v0;
  __device__ __forceinline__ int neighbour(int k) const { return local ? local[k] : __ldg(nbr + k) - v0; }
};

// Sum over v's neighbours, in list order, of h(u): 16 threads per node, 4
// channels each; each of the 16 fetches one neighbour's number, so that the
// rows follow one another without waiting for it. MEAN: out(v) = the sum over
// their number, 0 without any; else out(v) += the sum. Whole CTA.
template <bool MEAN>
__device__ __forceinline__ void tile_aggregate(const TileGraph& t, int nodes, const float* h, float* out) {
  const int sub = threadIdx.x % 16, col = 4 * sub, lane = threadIdx.x & 31;
  for (int v0 = 0; v0 < nodes; v0 += kRowGroups) {
    const int v = v0 + threadIdx.x / 16;
    const int s = v < nodes ? t.start[v] : 0, deg = v < nodes ? t.start[v + 1] - s : 0;
    const int most = max(deg, __shfl_xor_sync(0xffffffffu, deg, 16));  // of the warp's two nodes
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < most; k0 += 16) {
      const int mine = k0 + sub < deg ? t.neighbour(s + k0 + sub) : 0;
      const int trip = min(16, most - k0);
#pragma unroll 4
      for (int k = 0; k < trip; ++k) {
        const int u = __shfl_sync(0xffffffffu, mine, (lane & 16) + k);
        const float4 x = *reinterpret_cast<const float4*>(h + u * kRow + col);
        if (k0 + k < deg) {
          acc.x += x.x;
          acc.y += x.y;
          acc.z += x.z;
          acc.w += x.w;
        }
      }
    }
    if (v < nodes) {
      float4* const to = reinterpret_cast<float4*>(out + v * kRow + col);
      if constexpr (MEAN) {
        // without neighbours the sum is 0
        const float d = static_cast<float>(max(1, deg)), inv = 1.f / d;
        *to = make_float4(quotient(acc.x, d, inv), quotient(acc.y, d, inv), quotient(acc.z, d, inv),
                          quotient(acc.w, d, inv));
      } else {
        const float4 o = *to;
        *to = make_float4(o.x + acc.x, o.y + acc.y, o.z + acc.z, o.w + acc.w);
      }
    }
  }
}

// Neighbours held in shared memory per tile: a complete graph of 32 vertices,
// or sparse ones.
template <int M>
constexpr int kTileEdges = M == 32 ? 1024 : 4096;

// Shared memory (floats) of a tile: rows of activations (forward two buffers,
// training a third), two weight matrices, and for training the signs of every
// layer's activations and dlogit, dtd, loss terms.
template <int M>
size_t tile_smem(bool train, int layers) {
  return 4 * ((train ? 3 : 2) * size_t(M) * kRow + 2 * size_t(kWide) * kRow +
              (train ? (2 * (size_t(layers) + 1) + 3) * M : 0) + M + 32) + kTileEdges<M>;
}

// One tile: forward, and for TRAIN the backward pass up to the weight
// gradients. The products are bound by FP32 issue where two CTAs share an SM
// (forward, M = 128: 1024 graphs of 20..80 nodes 100 us, where the layer-by-layer
// kernels took 580), by the latency of shared loads at 8 warps per SM (training,
// M = 32: 256 graphs of 5..24 nodes 48 us, 18 with gnn_weight_grads and
// gnn_sum_chunks after it, against 530). 512 threads per CTA: 76 us in training.
template <int M, bool TRAIN>
__global__ void __launch_bounds__(kTileThreads, TRAIN ? 1 : 2) gnn_tile_kernel(const __grid_constant__ TileParams p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kBuf = M * kRow;
  const int tid = threadIdx.x, H = kWide, L = p.layers, fin = p.fin;
  const int g0 = p.tile_graph[blockIdx.x], g1 = p.tile_graph[blockIdx.x + 1];
  const int v0 = p.gstart[g0], nodes = p.gstart[g1] - v0, graphs = g1 - g0;
  float* const h = sm;            // the layer's activations; backward: dh
  float* const agg = sm + kBuf;   // neighbour means (first: input features); backward: dz
  float* const W1 = sm + (TRAIN ? 3 : 2) * kBuf;
  float* const W2 = W1 + H * kRow;
  int32_t* const start = reinterpret_cast<int32_t*>(W2 + H * kRow);  // [M + 32]
  uint8_t* const local = reinterpret_cast<uint8_t*>(start + M + 32);
  uint32_t* const sign = reinterpret_cast<uint32_t*>(local + kTileEdges<M>);  // training: [layer][node][2]
  const __nv_bfloat16* const w = p.w;
  const int64_t layer0 = int64_t(fin) * H + H, stride = 2 * int64_t(H) * H + H, head = layer0 + L * stride;
  const size_t NH = size_t(p.num_nodes) * H;

  // training keeps a layer for the weight gradients, and its signs here
  auto keep = [&](const float* from, float* to) {
    for (int t = tid; t < nodes * (H / 4); t += kTileThreads)
      reinterpret_cast<float4*>(to + size_t(v0) * H)[t] =
          *reinterpret_cast<const float4*>(from + (t / (H / 4)) * kRow + 4 * (t % (H / 4)));
  };
  auto keep_signs = [&](int l) {
    for (int t = tid; t < nodes * H; t += kTileThreads) {  // whole warps: H is 64
      const uint32_t bits = __ballot_sync(0xffffffffu, h[(t / H) * kRow + t % H] > 0.f);
      if ((tid & 31) == 0)
        sign[l * 2 * M + t / 32] = bits;
    }
  };

  // input features, padded with zeros to a multiple of 4 and to whole row groups
  const int fin4 = (fin + 3) & ~3, rows = (nodes + kRowGroups - 1) / kRowGroups * kRowGroups;
  for (int t = tid; t < rows * fin4; t += kTileThreads) {
    const int r = t / fin4, i = t % fin4;
    agg[r * kRow + i] = r < nodes && i < fin ? p.x[size_t(v0 + r) * fin + i] : 0.f;
  }
  for (int t = tid; t < fin4 * H; t += kTileThreads)
    W1[(t / H) * kRow + t % H] = t / H < fin ? bf(w[t]) : 0.f;
  // neighbour lists; a neighbour outside the tile is reported and the batch
  // taken up again layer by layer
  const int e0 = p.nbr_start[v0], edges = p.nbr_start[v0 + nodes] - e0;
  const TileGraph graph{start, edges <= kTileEdges<M> ? local : nullptr, p.nbr + e0, v0};
  for (int v = tid; v < rows + 1; v += kTileThreads)
    start[v] = v <= nodes ? p.nbr_start[v0 + v] - e0 : edges;
  int bad = 0;
  for (int k = tid; k < edges; k += kTileThreads) {
    const int u = p.nbr[e0 + k] - v0;
    bad |= static_cast<unsigned>(u) >= static_cast<unsigned>(nodes);
    if (graph.local)
      local[k] = static_cast<uint8_t>(u);
  }
  if (__syncthreads_or(bad)) {
    if (tid == 0)
      *p.outside = 1;
    return;
  }
  WeightRegs<kWide> r1, r2;
  for_rows<M>(nodes, [&](auto R) {
    tile_layer<decltype(R)::value>(agg, W1, fin4, nullptr, nullptr, w + int64_t(fin) * H, h);
  });
  for (int l = 0; l < L; ++l) {
    r1.load(w + layer0 + l * stride);
    r2.load(w + layer0 + l * stride + H * H);
    __syncthreads();
    tile_aggregate<true>(graph, nodes, h, agg);
    r1.store(W1);
    r2.store(W2);
    if constexpr (TRAIN) {
      keep(h, p.hs + l * NH);
      keep_signs(l);
    }
    __syncthreads();
    if constexpr (TRAIN)
      keep(agg, p.as + l * NH);
    for_rows<M>(nodes, [&](auto R) {
      tile_layer<decltype(R)::value>(h, W1, H, agg, W2, w + layer0 + l * stride + 2 * H * H, h);
    });
  }
  __syncthreads();

  // heads: a thread per node, then a warp per graph
  const __nv_bfloat16 *w_out = w + head, *w_g = w + head + H + 1;
  float* const dl = reinterpret_cast<float*>(sign + 2 * (L + 1) * M);  // training: dlogit per node
  float* const dt = dl + M;         // dtd per graph
  float* const loss = dt + M;       // loss terms per node
  if constexpr (TRAIN) {
    keep(h, p.hs + L * NH);
    keep_signs(L);
  }
  if (tid < H) {
    W1[tid] = bf(w_out[tid]);
    W1[kRow + tid] = bf(w_g[tid]);
  }
  __syncthreads();
  for (int v = tid; v < nodes; v += kTileThreads) {
    float acc = bf(w_out[H]);
    for (int j = 0; j < H; j += 4) {
      const float4 x = *reinterpret_cast<const float4*>(h + v * kRow + j);
      acc = fmaf(x.x, W1[j], acc);
      acc = fmaf(x.y, W1[j + 1], acc);
      acc = fmaf(x.z, W1[j + 2], acc);
      acc = fmaf(x.w, W1[j + 3], acc);
    }
    if constexpr (!TRAIN) {
      p.logits[v0 + v] = acc;
    } else {
      const float m = p.mask[v0 + v], y = p.y[v0 + v], sig = 1.f / (1.f + expf(-acc));
      const float d = m * (sig - y) * p.inv_mask_sum;
      dl[v] = d;
      p.dlogit[v0 + v] = d;
      loss[v] = m * (fmaxf(acc, 0.f) - acc * y + log1pf(expf(-fabsf(acc)))) * p.inv_mask_sum;
    }
  }
  for (int g = tid / 32; g < graphs; g += kTileThreads / 32) {
    const int lane = tid & 31, s = p.gstart[g0 + g] - v0, e = p.gstart[g0 + g + 1] - v0;
    float a = 0.f, b = 0.f;
    for (int v = s; v < e; ++v) {
      a += h[v * kRow + lane];
      b += h[v * kRow + lane + 32];
    }
    a = a / static_cast<float>(e - s);  // no empty graphs here
    b = b / static_cast<float>(e - s);
    float sum = __fadd_rn(__fmul_rn(a, W1[kRow + lane]), __fmul_rn(b, W1[kRow + lane + 32]));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      sum += __shfl_down_sync(0xffffffffu, sum, off);
    const float est = __shfl_sync(0xffffffffu, sum, 0) + bf(w_g[H]);
    if constexpr (!TRAIN) {
      if (lane == 0)
        p.td_est[g0 + g] = est;
    } else {
      const float diff = est - p.td_label[g0 + g], d = 2.f * p.td_weight * diff / static_cast<float>(p.num_graphs);
      if (lane == 0) {
        dt[g] = d;
        p.dtd[g0 + g] = d;
        W2[g] = p.td_weight * diff * diff / static_cast<float>(p.num_graphs);  // g < M <= 128: two rows
      }
      p.pooled[size_t(g0 + g) * H + lane] = a;
      p.pooled[size_t(g0 + g) * H + lane + 32] = b;
    }
  }
  if constexpr (TRAIN) {
    float* const dz = agg;
    float* const da = sm + 2 * kBuf;
    __syncthreads();
    if (tid == 0) {
      float a = 0.f;
      for (int v = 0; v < nodes; ++v)
        a += loss[v];
      for (int g = 0; g < graphs; ++g)
        a += W2[g];
      p.tile_loss[blockIdx.x] = a;
    }
    // dh of the last layer (over its activations: only their signs are needed)
    for (int g = tid / H; g < graphs; g += kTileThreads / H) {
      const int j = tid % H, s = p.gstart[g0 + g] - v0, e = p.gstart[g0 + g + 1] - v0;
      for (int v = s; v < e; ++v)
        h[v * kRow + j] = dl[v] * W1[j] + dt[g] * W1[kRow + j] / static_cast<float>(e - s);
    }
    for (int l = L; l >= 0; --l) {
      if (l > 0) {
        r1.load(w + layer0 + (l - 1) * stride);
        r2.load(w + layer0 + (l - 1) * stride + H * H);
      }
      __syncthreads();
      // dz = dh where the activation is positive; zero padding rows
      for (int t = tid; t < rows * H; t += kTileThreads) {
        const int v = t / H, j = t % H;
        const bool on = v < nodes && (sign[l * 2 * M + t / 32] >> (t & 31) & 1u);
        dz[v * kRow + j] = on ? h[v * kRow + j] : 0.f;
      }
      if (l > 0) {
        r1.store(W1);
        r2.store(W2);
      }
      __syncthreads();
      keep(dz, p.dzs + l * NH);
      if (l == 0)
        break;
      // dh of the layer below: dz Ws^T + aggregate^T(dz Wn^T)
      for_rows<M>(nodes, [&](auto R) {
        tile_product_t<decltype(R)::value>(dz, W2, da, start);
        tile_product_t<decltype(R)::value>(dz, W1, h);
      });
      __syncthreads();
      tile_aggregate<false>(graph, nodes, da, h);
    }
  }
}

// Weight gradients of a chunk of 64 rows: dW[i][j] = sum_v X[v][i] dZ[v][j] and
// the bias's column sums, in ascending v. blockIdx.y: 0 .. layers - 1 the two
// matrices of a layer, `layers` the input projection, then the node head and
// the graph head (rows: graphs).
__global__ void __launch_bounds__(kGradThreads) gnn_weight_grads(const __grid_constant__ TileParams p) {
  extern __shared__ __align__(16) float sm[];
  constexpr int kChunk = 64;
  const int tid = threadIdx.x, H = kWide, L = p.layers, fin = p.fin, what = static_cast<int>(blockIdx.y);
  const int total = what == L + 2 ? p.num_graphs : p.num_nodes;
  const int r0 = (p.first_chunk + static_cast<int>(blockIdx.x)) * kChunk, rows = min(kChunk, total - r0);
  if (rows <= 0)
    return;
  const int64_t layer0 = int64_t(fin) * H + H, stride = 2 * int64_t(H) * H + H, head = layer0 + L * stride;
  const size_t NH = size_t(p.num_nodes) * H;
  float* const out = p.part + size_t(blockIdx.x) * p.nparams;
  float *const X = sm, *const Y = sm + kChunk * kRow, *const Z = sm + 2 * kChunk * kRow;
  auto load = [&](const float* from, float* to) {
    for (int t = tid; t < rows * (H / 4); t += kGradThreads)
      *reinterpret_cast<float4*>(to + (t / (H / 4)) * kRow + 4 * (t % (H / 4))) =
          reinterpret_cast<const float4*>(from + size_t(r0) * H)[t];
  };
  if (what < L) {
    load(p.hs + what * NH, X);
    load(p.as + what * NH, Y);
    load(p.dzs + (what + 1) * NH, Z);
    __syncthreads();
    const int j0 = 4 * (tid % 16), i0 = 4 * (tid / 16);
    float a[4][4] = {}, b[4][4] = {};
#pragma unroll 2
    for (int v = 0; v < rows; ++v) {
      const float4 z = *reinterpret_cast<const float4*>(Z + v * kRow + j0);
      const float4 x = *reinterpret_cast<const float4*>(X + v * kRow + i0);
      const float4 y = *reinterpret_cast<const float4*>(Y + v * kRow + i0);
      const float zs[4] = {z.x, z.y, z.z, z.w}, xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          a[i][j] = fmaf(xs[i], zs[j], a[i][j]);
          b[i][j] = fmaf(ys[i], zs[j], b[i][j]);
        }
    }
    float* const g = out + layer0 + what * stride;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        g[(i0 + i) * H + j0 + j] = a[i][j];
        g[H * H + (i0 + i) * H + j0 + j] = b[i][j];
      }
    if (tid < H) {
      float sum = 0.f;
      for (int v = 0; v < rows; ++v)
        sum += Z[v * kRow + tid];
      g[2 * H * H + tid] = sum;
    }
  } else if (what == L) {
    load(p.dzs, Z);
    for (int t = tid; t < rows * fin; t += kGradThreads)
      X[(t / fin) * kRow + t % fin] = p.x[size_t(r0) * fin + t];
    __syncthreads();
    for (int t = tid; t < fin * H; t += kGradThreads) {
      float a = 0.f;
      for (int v = 0; v < rows; ++v)
        a = fmaf(X[v * kRow + t / H], Z[v * kRow + t % H], a);
      out[t] = a;
    }
    if (tid < H) {
      float sum = 0.f;
      for (int v = 0; v < rows; ++v)
        sum += Z[v * kRow + tid];
      out[int64_t(fin) * H + tid] = sum;
    }
  } else {
    const bool graph = what == L + 2;
    const float* const from = graph ? p.pooled : p.hs + L * NH;
    const float* const d = (graph ? p.dtd : p.dlogit) + r0;
    float* const g = out + head + (graph ? H + 1 : 0);
    if (tid < H) {
      float a = 0.f;
      for (int v = 0; v < rows; ++v)
        a = fmaf(from[size_t(r0 + v) * H + tid], d[v], a);
      g[tid] = a;
    } else if (tid == H) {
      float a = 0.f;
      for (int v = 0; v < rows; ++v)
        a += d[v];
      g[H] = a;
    }
  }
}

// The gradient: every parameter's chunks in ascending order, on top of those of
// earlier runs; the loss (with the first run): the tiles' likewise.
__global__ void __launch_bounds__(128) gnn_sum_chunks(const __grid_constant__ TileParams p, int tiles,
                                                      float* __restrict__ grad, float* __restrict__ loss) {
  const int64_t t = int64_t(blockIdx.x) * 128 + threadIdx.x;
  if (t > p.nparams)
    return;
  const int64_t graph_head = p.nparams - kWide - 1;
  const bool again = p.first_chunk > 0;
  if (again && t == p.nparams)
    return;
  const int chunks = ((t >= graph_head ? p.num_graphs : p.num_nodes) + 63) / 64 - p.first_chunk;
  const int count = t == p.nparams ? tiles : min(chunks, kGradRun);
  const float* from = t == p.nparams ? p.tile_loss : p.part + t;
  const int64_t step = t == p.nparams ? 1 : p.nparams;
  float acc = again ? grad[t] : 0.f;
#pragma unroll 8
  for (int c = 0; c < count; ++c)
    acc += from[c * step];
  if (t == p.nparams) {
    *loss = acc;
  } else {
    grad[t] = 0.f + acc;
    if (p.grad_copy)
      p.grad_copy[t] = 0.f + acc;
  }
}

}  // namespace
}  // namespace gtd

struct gtd_gnn_s {
  gtd_handle h = nullptr;
  int device = 0;  // the handle's, which may be gone when the network is destroyed
  int fin = 0, hid = 0, layers = 0;
  int64_t nparams = 0;
  float* master = nullptr;
  float* m = nullptr;
  float* v = nullptr;
  float* grad = nullptr;
  __nv_bfloat16* w = nullptr;
  int64_t step = 0;
  // batch and activation buffers (grown as needed)
  void* buf = nullptr;
  size_t buf_cap = 0;
  void* stage = nullptr;  // pinned: small arrays of a batch in, results out
  size_t stage_cap = 0;
  bool smem_set = false;  // the tile kernels' shared-memory limits are raised
};

namespace {

struct Layout {
  int64_t w_in, b_in, layer0, layer_stride, head;
  int64_t ws(int l, int H) const { return layer0 + l * layer_stride; }
  int64_t wn(int l, int H) const { return layer0 + l * layer_stride + int64_t(H) * H; }
  int64_t b(int l, int H) const { return layer0 + l * layer_stride + 2 * int64_t(H) * H; }
};

Layout layout_of(const gtd_gnn_s* g) {
  const int64_t H = g->hid;
  Layout L;
  L.w_in = 0;
  L.b_in = int64_t(g->fin) * H;
  L.layer0 = L.b_in + H;
  L.layer_stride = 2 * H * H + H;
  L.head = L.layer0 + g->layers * L.layer_stride;
  return L;
}

// Device views of one batch plus activations, carved from g->buf.
struct Views {
  float* x;
  int32_t *gstart, *nbr_start, *nbr, *graph_of;
  float *y, *mask, *td_label;
  float *Z, *Hs, *A;  // (L + 1) x N x H, (L + 1) x N x H, L x N x H
  float *logits, *pooled, *td_est, *loss;
  float *dh, *dz, *da, *tmp, *dlogit, *dtd;
  float* part;  // weight-gradient partials, one row per 64-node chunk
};

gtd_status prepare(gtd_gnn g, const gtd_gnn_batch* b, bool train, Views& V) {
  gtd_handle h = g->h;
  const size_t N = size_t(b->num_nodes), G = size_t(b->num_graphs), H = size_t(g->hid), L = size_t(g->layers);
  const size_t E = size_t(b->nbr_start[b->num_nodes]);
  auto al = [](size_t bytes) { return (bytes + 255) & ~size_t(255); };
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += al(bytes);
    return o;
  };
  const size_t ox = take(N * g->fin * 4), ogs = take((G + 1) * 4), ons = take((N + 1) * 4), onb = take(E * 4 + 4),
               ogo = take(N * 4), oy = take(N * 4), om = take(N * 4), otd = take(G * 4),
               oZ = take((L + 1) * N * H * 4), oH = take((L + 1) * N * H * 4), oA = take(L * N * H * 4),
               olog = take(N * 4), opool = take(G * H * 4), otde = take(G * 4), oloss = take(4), odh = take(N * H * 4),
               odz = take(N * H * 4), oda = take(N * H * 4), otmp = take(N * H * 4), odl = take(N * 4),
               odt = take(G * 4),
               opart = take(((std::max(N, G) + 63) / 64) * (size_t(std::max(g->fin, g->hid)) * H + H) * 4);
  GTD_CUDA(h, gtd::ensure_device(&g->buf, &g->buf_cap, off));
  char* base = static_cast<char*>(g->buf);
  V.x = reinterpret_cast<float*>(base + ox);
  V.gstart = reinterpret_cast<int32_t*>(base + ogs);
  V.nbr_start = reinterpret_cast<int32_t*>(base + ons);
  V.nbr = reinterpret_cast<int32_t*>(base + onb);
  V.graph_of = reinterpret_cast<int32_t*>(base + ogo);
  V.y = reinterpret_cast<float*>(base + oy);
  V.mask = reinterpret_cast<float*>(base + om);
  V.td_label = reinterpret_cast<float*>(base + otd);
  V.Z = reinterpret_cast<float*>(base + oZ);
  V.Hs = reinterpret_cast<float*>(base + oH);
  V.A = reinterpret_cast<float*>(base + oA);
  V.logits = reinterpret_cast<float*>(base + olog);
  V.pooled = reinterpret_cast<float*>(base + opool);
  V.td_est = reinterpret_cast<float*>(base + otde);
  V.loss = reinterpret_cast<float*>(base + oloss);
  V.dh = reinterpret_cast<float*>(base + odh);
  V.dz = reinterpret_cast<float*>(base + odz);
  V.da = reinterpret_cast<float*>(base + oda);
  V.tmp = reinterpret_cast<float*>(base + otmp);
  V.dlogit = reinterpret_cast<float*>(base + odl);
  V.dtd = reinterpret_cast<float*>(base + odt);
  V.part = reinterpret_cast<float*>(base + opart);
  cudaStream_t s = h->stream;
  GTD_CUDA(h, cudaMemcpyAsync(V.x, b->x, N * g->fin * 4, cudaMemcpyHostToDevice, s));
  GTD_CUDA(h, cudaMemcpyAsync(V.gstart, b->graph_start, (G + 1) * 4, cudaMemcpyHostToDevice, s));
  GTD_CUDA(h, cudaMemcpyAsync(V.nbr_start, b->nbr_start, (N + 1) * 4, cudaMemcpyHostToDevice, s));
  if (E)
    GTD_CUDA(h, cudaMemcpyAsync(V.nbr, b->nbr, E * 4, cudaMemcpyHostToDevice, s));
  // graph of every node, from the ranges
  std::vector<int32_t> go(N);
  for (size_t gi = 0; gi < G; ++gi)
    for (int32_t v = b->graph_start[gi]; v < b->graph_start[gi + 1]; ++v)
      go[v] = static_cast<int32_t>(gi);
  GTD_CUDA(h, cudaMemcpyAsync(V.graph_of, go.data(), N * 4, cudaMemcpyHostToDevice, s));
  if (train) {
    GTD_CUDA(h, cudaMemcpyAsync(V.y, b->root_label, N * 4, cudaMemcpyHostToDevice, s));
    GTD_CUDA(h, cudaMemcpyAsync(V.mask, b->node_mask, N * 4, cudaMemcpyHostToDevice, s));
    GTD_CUDA(h, cudaMemcpyAsync(V.td_label, b->td_label, G * 4, cudaMemcpyHostToDevice, s));
  }
  // the copies above read host arrays that the caller may reuse right after
  GTD_CUDA(h, cudaStreamSynchronize(s));
  return GTD_OK;
}

gtd_status forward(gtd_gnn g, const gtd_gnn_batch* b, const Views& V) {
  gtd_handle h = g->h;
  const int N = b->num_nodes, G = b->num_graphs, H = g->hid, L = g->layers;
  const Layout P = layout_of(g);
  cudaStream_t s = h->stream;
  const unsigned nb = gtd::blocks_for(size_t(N), gtd::kNodesPerBlock);
  const size_t NH = size_t(N) * H;
  gtd::node_linear<<<nb, 64, 0, s>>>(N, g->fin, H, V.x, g->w + P.w_in, nullptr, nullptr, g->w + P.b_in, V.Z, V.Hs);
  GTD_CUDA(h, cudaGetLastError());
  for (int l = 0; l < L; ++l) {
    gtd::aggregate<<<gtd::blocks_for(NH, 256), 256, 0, s>>>(N, H, V.nbr_start, V.nbr, V.Hs + l * NH, V.A + l * NH);
    gtd::node_linear<<<nb, 64, 0, s>>>(N, H, H, V.Hs + l * NH, g->w + P.ws(l, H), V.A + l * NH, g->w + P.wn(l, H),
                                       g->w + P.b(l, H), V.Z + (l + 1) * NH, V.Hs + (l + 1) * NH);
    GTD_CUDA(h, cudaGetLastError());
  }
  const unsigned hb = gtd::blocks_for(size_t(N), 128) + static_cast<unsigned>(G);
  gtd::heads_forward<<<hb, 128, 0, s>>>(N, G, H, V.Hs + L * NH, V.gstart, g->w + P.head, g->w + P.head + H,
                                        g->w + P.head + H + 1, g->w + P.head + 2 * H + 1, V.logits, V.pooled,
                                        V.td_est);
  GTD_CUDA(h, cudaGetLastError());
  return GTD_OK;
}

// Weight gradient of one linear map over N rows: per-chunk partials, then
// their ordered sum into dW (and db).
void wgrad(cudaStream_t s, int N, int K, int H, const float* X, const float* dZ, float* dW, float* db, float* part) {
  const unsigned chunks = gtd::blocks_for(size_t(N), 64);
  gtd::weight_grad<<<chunks, 256, 0, s>>>(N, K, H, X, dZ, part);
  gtd::reduce_partials<<<gtd::blocks_for(size_t(K) * H + H, 256), 256, 0, s>>>(static_cast<int>(chunks), K * H, H,
                                                                              part, dW, db);
}

gtd_status backward(gtd_gnn g, const gtd_gnn_batch* b, const Views& V, float td_weight) {
  gtd_handle h = g->h;
  const int N = b->num_nodes, G = b->num_graphs, H = g->hid, L = g->layers;
  const Layout P = layout_of(g);
  cudaStream_t s = h->stream;
  const size_t NH = size_t(N) * H;
  double msum = 0;
  for (int v = 0; v < N; ++v)
    msum += b->node_mask[v];
  const float inv = msum > 0 ? float(1.0 / msum) : 0.f;
  GTD_CUDA(h, cudaMemsetAsync(g->grad, 0, g->nparams * 4, s));
  GTD_CUDA(h, cudaMemsetAsync(V.loss, 0, 4, s));
  float* gr = g->grad;
  gtd::heads_backward<<<gtd::blocks_for(size_t(std::max(N, G)), 128), 128, 0, s>>>(
      N, G, H, V.gstart, V.graph_of, V.logits, V.td_est, V.y, V.mask, V.td_label, inv, td_weight, g->w + P.head,
      g->w + P.head + H + 1, V.dlogit, V.dtd, V.dh, V.loss);
  // w_out, b_out from h_L and dlogit; w_g, b_g from the pooled means and dtd
  wgrad(s, N, H, 1, V.Hs + L * NH, V.dlogit, gr + P.head, gr + P.head + H, V.part);
  wgrad(s, G, H, 1, V.pooled, V.dtd, gr + P.head + H + 1, gr + P.head + 2 * H + 1, V.part);
  GTD_CUDA(h, cudaGetLastError());
  const unsigned nb = gtd::blocks_for(size_t(N), gtd::kNodesPerBlock);
  const unsigned eb = gtd::blocks_for(NH, 256);
  for (int l = L - 1; l >= 0; --l) {
    // dz = dh * relu'(z_{l+1})
    gtd::relu_mask<<<eb, 256, 0, s>>>(NH, V.Z + (l + 1) * NH, V.dh, V.dz);
    wgrad(s, N, H, H, V.Hs + l * NH, V.dz, gr + P.ws(l, H), gr + P.b(l, H), V.part);
    wgrad(s, N, H, H, V.A + l * NH, V.dz, gr + P.wn(l, H), nullptr, V.part);
    // dh_l = dz Ws^T + aggregate^T(dz Wn^T)
    gtd::node_linear_t<<<nb, 64, 0, s>>>(N, H, H, V.dz, g->w + P.wn(l, H), V.da);
    gtd::node_linear_t<<<nb, 64, 0, s>>>(N, H, H, V.dz, g->w + P.ws(l, H), V.tmp);
    gtd::aggregate_t<<<eb, 256, 0, s>>>(N, H, V.nbr_start, V.nbr, V.da, V.tmp);
    GTD_CUDA(h, cudaMemcpyAsync(V.dh, V.tmp, NH * 4, cudaMemcpyDeviceToDevice, s));
    GTD_CUDA(h, cudaGetLastError());
  }
  gtd::relu_mask<<<eb, 256, 0, s>>>(NH, V.Z, V.dh, V.dz);
  wgrad(s, N, g->fin, H, V.x, V.dz, gr + P.w_in, gr + P.b_in, V.part);
  GTD_CUDA(h, cudaGetLastError());
  return GTD_OK;
}

// The most shared memory a CTA of these kernels may take (227 KB).
constexpr size_t kTileSmemMost = 227 * 1024;

template <int M, bool TRAIN>
cudaError_t launch_tile_kernel(const gtd::TileParams& p, int tiles, cudaStream_t s) {
  gtd::gnn_tile_kernel<M, TRAIN><<<tiles, gtd::kTileThreads, gtd::tile_smem<M>(TRAIN, p.layers), s>>>(p);
  return cudaGetLastError();
}

// Nodes per tile for this batch, 0 where the tile kernels do not apply: the
// largest graph decides, small tiles spread a small batch over more SMs.
int tile_nodes(const gtd_gnn_s* g, const gtd_gnn_batch* b) {
  if (g->hid != gtd::kWide)
    return 0;
  int most = 0;
  for (int i = 0; i < b->num_graphs; ++i) {
    const int n = b->graph_start[i + 1] - b->graph_start[i];
    if (n < 1)
      return 0;
    most = std::max(most, n);
  }
  if (most <= 32 && b->num_nodes <= 32 * 3 * g->h->num_sms)
    return 32;
  return most <= 64 ? 64 : most <= 128 ? 128 : 0;
}

// Forward (train = false: logits and td estimates) or loss and gradients
// (train = true: g->grad, grad_out and *loss_out) by tiles. *done is false, and
// no output written (g->grad is), where the batch needs the layer-by-layer
// kernels.
gtd_status run_tiles(gtd_gnn g, const gtd_gnn_batch* b, bool train, float td_weight, float* logits_out, float* td_out,
                     float* grad_out, float* loss_out, bool* done) {
  *done = false;
  const int M = tile_nodes(g, b);
  if (M == 0)
    return GTD_OK;
  gtd_handle h = g->h;
  cudaStream_t s = h->stream;
  const size_t N = size_t(b->num_nodes), G = size_t(b->num_graphs), E = size_t(b->nbr_start[b->num_nodes]);
  std::vector<int32_t> first;  // first graph of every tile
  int nodes = M + 1;
  for (size_t i = 0; i < G; ++i) {
    const int n = b->graph_start[i + 1] - b->graph_start[i];
    if (nodes + n > M) {
      first.push_back(static_cast<int32_t>(i));
      nodes = 0;
    }
    nodes += n;
  }
  const int tiles = static_cast<int>(first.size());
  first.push_back(static_cast<int32_t>(G));

  // one buffer: the batch's arrays, then results; the small ones (up to
  // kStaged bytes each) lie in front and go up in one copy from pinned memory,
  // the others straight from the caller's arrays (the host takes longer over a
  // pass of its own: 78 us against 18 for 1.6 MB)
  constexpr size_t kStaged = 64 * 1024;
  struct Array {
    const void* from;
    size_t bytes, at;
  };
  enum { kX, kGraphStart, kNbrStart, kNbr, kTiles, kY, kMask, kTd, kArrays };
  Array in[kArrays] = {{b->x, N * g->fin * 4, 0},
                       {b->graph_start, (G + 1) * 4, 0},
                       {b->nbr_start, (N + 1) * 4, 0},
                       {b->nbr, E * 4, 0},
                       {first.data(), first.size() * 4, 0},
                       {b->root_label, train ? N * 4 : 0, 0},
                       {b->node_mask, train ? N * 4 : 0, 0},
                       {b->td_label, train ? G * 4 : 0, 0}};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 255) & ~size_t(255);
    return o;
  };
  for (Array& a : in)
    if (a.bytes <= kStaged)
      a.at = take(a.bytes);
  const size_t staged = off;
  for (Array& a : in)
    if (a.bytes > kStaged)
      a.at = take(a.bytes);
  const size_t chunks = (std::max(N, G) + 63) / 64, NH = N * size_t(gtd::kWide), L = size_t(g->layers);
  // results, in one copy back: the flag, and the loss and the gradient or the td estimates and the logits
  const size_t grad_bytes = train && grad_out ? size_t(g->nparams) * 4 : 0;
  const size_t ores = take(256), ograd = take(grad_bytes), otde = take(G * 4), olog = take(N * 4);
  const size_t res_bytes = !train ? off - ores : grad_bytes ? ograd + grad_bytes - ores : 8;
  const size_t ohs = take(train ? (L + 1) * NH * 4 : 0), oas = take(train ? L * NH * 4 : 0),
               odz = take(train ? (L + 1) * NH * 4 : 0), opool = take(train ? G * gtd::kWide * 4 : 0),
               otl2 = take(train ? size_t(tiles) * 4 : 0), opart = take(train ? std::min(chunks, size_t(gtd::kGradRun)) * size_t(g->nparams) * 4 : 0);
  GTD_CUDA(h, gtd::ensure_device(&g->buf, &g->buf_cap, off));
  const size_t stage = std::max(staged, res_bytes);
  if (g->stage_cap < stage) {
    if (g->stage)
      cudaFreeHost(g->stage);
    g->stage = nullptr;
    g->stage_cap = 0;
    GTD_CUDA(h, cudaMallocHost(&g->stage, stage));
    g->stage_cap = stage;
  }
  if (!g->smem_set) {
    const int most = static_cast<int>(kTileSmemMost);
    for (auto kernel : {gtd::gnn_tile_kernel<32, false>, gtd::gnn_tile_kernel<64, false>,
                        gtd::gnn_tile_kernel<128, false>, gtd::gnn_tile_kernel<32, true>,
                        gtd::gnn_tile_kernel<64, true>, gtd::gnn_tile_kernel<128, true>, gtd::gnn_weight_grads})
      GTD_CUDA(h, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    g->smem_set = true;
  }
  char* const base = static_cast<char*>(g->buf);
  char* const pinned = static_cast<char*>(g->stage);
  for (const Array& a : in)
    if (a.bytes > kStaged)
      GTD_CUDA(h, cudaMemcpyAsync(base + a.at, a.from, a.bytes, cudaMemcpyHostToDevice, s));
    else if (a.bytes)
      std::memcpy(pinned + a.at, a.from, a.bytes);
  GTD_CUDA(h, cudaMemcpyAsync(base, pinned, staged, cudaMemcpyHostToDevice, s));
  GTD_CUDA(h, cudaMemsetAsync(base + ores, 0, 8, s));
  double msum = 0;
  for (size_t v = 0; train && v < N; ++v)
    msum += b->node_mask[v];
  auto f = [&](size_t o) { return reinterpret_cast<float*>(base + o); };
  auto i32 = [&](size_t o) { return reinterpret_cast<int32_t*>(base + o); };
  gtd::TileParams p = {};
  p.fin = g->fin;
  p.layers = g->layers;
  p.x = f(in[kX].at);
  p.gstart = i32(in[kGraphStart].at);
  p.nbr_start = i32(in[kNbrStart].at);
  p.nbr = i32(in[kNbr].at);
  p.tile_graph = i32(in[kTiles].at);
  p.w = g->w;
  p.logits = f(olog);
  p.td_est = f(otde);
  p.outside = i32(ores);
  p.y = f(in[kY].at);
  p.mask = f(in[kMask].at);
  p.td_label = f(in[kTd].at);
  p.inv_mask_sum = msum > 0 ? float(1.0 / msum) : 0.f;
  p.td_weight = td_weight;
  p.num_nodes = b->num_nodes;
  p.num_graphs = b->num_graphs;
  p.hs = f(ohs);
  p.as = f(oas);
  p.dzs = f(odz);
  p.pooled = f(opool);
  p.dlogit = f(olog);
  p.dtd = f(otde);
  p.tile_loss = f(otl2);
  p.nparams = g->nparams;
  p.part = f(opart);
  p.grad_copy = grad_bytes ? f(ograd) : nullptr;
  if (train) {
    GTD_CUDA(h, (M == 32   ? launch_tile_kernel<32, true>(p, tiles, s)
                 : M == 64 ? launch_tile_kernel<64, true>(p, tiles, s)
                           : launch_tile_kernel<128, true>(p, tiles, s)));
    for (size_t first = 0; first < chunks; first += gtd::kGradRun) {
      p.first_chunk = static_cast<int>(first);
      const dim3 grid(static_cast<unsigned>(std::min(chunks - first, size_t(gtd::kGradRun))),
                      static_cast<unsigned>(g->layers + 3));
      gtd::gnn_weight_grads<<<grid, gtd::kGradThreads, 3 * 64 * gtd::kRow * 4, s>>>(p);
      gtd::gnn_sum_chunks<<<gtd::blocks_for(size_t(g->nparams) + 1, 128), 128, 0, s>>>(p, tiles, g->grad,
                                                                                      f(ores) + 1);
    }
    GTD_CUDA(h, cudaGetLastError());
  } else {
    GTD_CUDA(h, (M == 32   ? launch_tile_kernel<32, false>(p, tiles, s)
                 : M == 64 ? launch_tile_kernel<64, false>(p, tiles, s)
                           : launch_tile_kernel<128, false>(p, tiles, s)));
  }
  GTD_CUDA(h, cudaMemcpyAsync(pinned, base + ores, res_bytes, cudaMemcpyDeviceToHost, s));
  GTD_CUDA(h, cudaStreamSynchronize(s));
  int32_t outside = 0;
  std::memcpy(&outside, pinned, 4);
  if (outside)
    return GTD_OK;  // a neighbour lies outside its graph: layer by layer
  *done = true;
  if (train) {
    if (loss_out)
      std::memcpy(loss_out, pinned + 4, 4);
    if (grad_bytes)
      std::memcpy(grad_out, pinned + (ograd - ores), grad_bytes);
  } else {
    if (td_out)
      std::memcpy(td_out, pinned + (otde - ores), G * 4);
    if (logits_out)
      std::memcpy(logits_out, pinned + (olog - ores), N * 4);
  }
  return GTD_OK;
}

uint64_t splitmix(uint64_t& s) {
  s += 0x9E3779B97F4A7C15ull;
  uint64_t z = s;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

using namespace gtd;

extern "C" {

gtd_status gtd_gnn_create(gtd_handle h, int in_features, int hidden, int layers, uint64_t seed, gtd_gnn* out) {
  if (!h || !out)
    return GTD_INVALID_ARG;
  if (in_features < 1 || in_features > kMaxK || hidden < 1 || hidden > kMaxK || layers < 1 || layers > 8)
    return fail(h, GTD_INVALID_ARG, "GNN shape out of range (features, hidden <= 64, layers <= 8)");
  DeviceGuard dg(h->device);
  gtd_gnn g = new (std::nothrow) gtd_gnn_s();
  if (!g)
    return GTD_OOM;
  g->h = h;
  g->device = h->device;
  g->fin = in_features;
  g->hid = hidden;
  g->layers = layers;
  const Layout P = layout_of(g);
  g->nparams = P.head + 2 * hidden + 2;
  const size_t bytes = size_t(g->nparams) * 4;
  cudaError_t e = cudaMalloc(&g->master, bytes);
  if (e == cudaSuccess)
    e = cudaMalloc(&g->m, bytes);
  if (e == cudaSuccess)
    e = cudaMalloc(&g->v, bytes);
  if (e == cudaSuccess)
    e = cudaMalloc(&g->grad, bytes);
  if (e == cudaSuccess)
    e = cudaMalloc(&g->w, size_t(g->nparams) * 2);
  if (e != cudaSuccess) {
    gtd_gnn_destroy(g);
    return cuda_fail(h, e, "gtd_gnn_create");
  }
  // Glorot-uniform weights, zero biases, from a seeded splitmix64 stream.
  std::vector<float> p(g->nparams, 0.f);
  uint64_t st = seed;
  auto fill = [&](int64_t off, int fan_in, int fan_out) {
    const double lim = std::sqrt(6.0 / (fan_in + fan_out));
    for (int64_t i = 0; i < int64_t(fan_in) * fan_out; ++i)
      p[off + i] = float((double(splitmix(st) >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0) * lim);
  };
  fill(P.w_in, in_features, hidden);
  for (int l = 0; l < layers; ++l) {
    fill(P.ws(l, hidden), hidden, hidden);
    fill(P.wn(l, hidden), hidden, hidden);
  }
  fill(P.head, hidden, 1);
  fill(P.head + hidden + 1, hidden, 1);
  gtd_status s = gtd_gnn_set_params(g, p.data());
  if (s != GTD_OK) {
    gtd_gnn_destroy(g);
    return s;
  }
  *out = g;
  return GTD_OK;
}

gtd_status gtd_gnn_destroy(gtd_gnn g) {
  if (!g)
    return GTD_INVALID_ARG;
  DeviceGuard dg(g->device);
  cudaFree(g->master);
  cudaFree(g->m);
  cudaFree(g->v);
  cudaFree(g->grad);
  cudaFree(g->w);
  cudaFree(g->buf);
  if (g->stage)
    cudaFreeHost(g->stage);
  delete g;
  return GTD_OK;
}

int64_t gtd_gnn_num_params(gtd_gnn g) { return g ? g->nparams : -1; }

gtd_status gtd_gnn_get_params(gtd_gnn g, float* out) {
  if (!g || !out)
    return GTD_INVALID_ARG;
  DeviceGuard dg(g->h->device);
  GTD_CUDA(g->h, cudaMemcpyAsync(out, g->master, g->nparams * 4, cudaMemcpyDeviceToHost, g->h->stream));
  GTD_CUDA(g->h, cudaStreamSynchronize(g->h->stream));
  return GTD_OK;
}

gtd_status gtd_gnn_set_params(gtd_gnn g, const float* in) {
  if (!g || !in)
    return GTD_INVALID_ARG;
  DeviceGuard dg(g->h->device);
  cudaStream_t s = g->h->stream;
  GTD_CUDA(g->h, cudaMemcpyAsync(g->master, in, g->nparams * 4, cudaMemcpyHostToDevice, s));
  GTD_CUDA(g->h, cudaMemsetAsync(g->m, 0, g->nparams * 4, s));
  GTD_CUDA(g->h, cudaMemsetAsync(g->v, 0, g->nparams * 4, s));
  to_bf16<<<blocks_for(size_t(g->nparams), 256), 256, 0, s>>>(g->nparams, g->master, g->w);
  GTD_CUDA(g->h, cudaGetLastError());
  GTD_CUDA(g->h, cudaStreamSynchronize(s));
  g->step = 0;
  return GTD_OK;
}

static gtd_status check_batch(gtd_gnn g, const gtd_gnn_batch* b, bool train) {
  if (!g || !b || b->num_nodes < 1 || b->num_graphs < 1 || !b->x || !b->graph_start || !b->nbr_start ||
      (b->nbr_start[b->num_nodes] > 0 && !b->nbr))
    return fail(g ? g->h : nullptr, GTD_INVALID_ARG, "malformed GNN batch");
  if (train && (!b->root_label || !b->node_mask || !b->td_label))
    return fail(g->h, GTD_INVALID_ARG, "training batch without labels");
  if (b->graph_start[0] != 0 || b->graph_start[b->num_graphs] != b->num_nodes)
    return fail(g->h, GTD_INVALID_ARG, "graph ranges do not cover the nodes");
  return GTD_OK;
}

gtd_status gtd_gnn_forward(gtd_gnn g, const gtd_gnn_batch* b, float* logits_out, float* td_out) {
  gtd_status s = check_batch(g, b, false);
  if (s != GTD_OK)
    return s;
  DeviceGuard dg(g->h->device);
  bool done = false;
  if ((s = run_tiles(g, b, false, 0.f, logits_out, td_out, nullptr, nullptr, &done)) != GTD_OK || done)
    return s;
  Views V;
  if ((s = prepare(g, b, false, V)) != GTD_OK)
    return s;
  if ((s = forward(g, b, V)) != GTD_OK)
    return s;
  cudaStream_t st = g->h->stream;
  if (logits_out)
    GTD_CUDA(g->h, cudaMemcpyAsync(logits_out, V.logits, size_t(b->num_nodes) * 4, cudaMemcpyDeviceToHost, st));
  if (td_out)
    GTD_CUDA(g->h, cudaMemcpyAsync(td_out, V.td_est, size_t(b->num_graphs) * 4, cudaMemcpyDeviceToHost, st));
  GTD_CUDA(g->h, cudaStreamSynchronize(st));
  return GTD_OK;
}

gtd_status gtd_gnn_gradients(gtd_gnn g, const gtd_gnn_batch* b, float td_weight, float* grad_out, float* loss_out) {
  gtd_status s = check_batch(g, b, true);
  if (s != GTD_OK)
    return s;
  DeviceGuard dg(g->h->device);
  bool done = false;
  if ((s = run_tiles(g, b, true, td_weight, nullptr, nullptr, grad_out, loss_out, &done)) != GTD_OK || done)
    return s;
  Views V;
  if ((s = prepare(g, b, true, V)) != GTD_OK)
    return s;
  if ((s = forward(g, b, V)) != GTD_OK)
    return s;
  if ((s = backward(g, b, V, td_weight)) != GTD_OK)
    return s;
  cudaStream_t st = g->h->stream;
  if (grad_out)
    GTD_CUDA(g->h, cudaMemcpyAsync(grad_out, g->grad, g->nparams * 4, cudaMemcpyDeviceToHost, st));
  if (loss_out)
    GTD_CUDA(g->h, cudaMemcpyAsync(loss_out, V.loss, 4, cudaMemcpyDeviceToHost, st));
  GTD_CUDA(g->h, cudaStreamSynchronize(st));
  return GTD_OK;
}

gtd_status gtd_gnn_train_step(gtd_gnn g, const gtd_gnn_batch* b, float lr, float td_weight, float* loss_out) {
  gtd_status s = check_batch(g, b, true);
  if (s != GTD_OK)
    return s;
  DeviceGuard dg(g->h->device);
  bool done = false;
  if ((s = run_tiles(g, b, true, td_weight, nullptr, nullptr, nullptr, loss_out, &done)) != GTD_OK)
    return s;
  Views V;
  if (!done) {
    if ((s = prepare(g, b, true, V)) != GTD_OK)
      return s;
    if ((s = forward(g, b, V)) != GTD_OK)
      return s;
    if ((s = backward(g, b, V, td_weight)) != GTD_OK)
      return s;
  }
  ++g->step;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, float(g->step)), c2 = 1.f - std::pow(b2, float(g->step));
  cudaStream_t st = g->h->stream;
  adam_step<<<blocks_for(size_t(g->nparams), 256), 256, 0, st>>>(g->nparams, g->master, g->m, g->v, g->grad, g->w,
                                                                  lr, b1, b2, 1e-8f, c1, c2);
  GTD_CUDA(g->h, cudaGetLastError());
  if (loss_out && !done)
    GTD_CUDA(g->h, cudaMemcpyAsync(loss_out, V.loss, 4, cudaMemcpyDeviceToHost, st));
  GTD_CUDA(g->h, cudaStreamSynchronize(st));
  return GTD_OK;
}

}  // extern "C"
