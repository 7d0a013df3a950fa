// A prompt's experts, rows sorted by expert, bfloat16: the passes around the two tensor-core products
// (gemm_bf16_wide.cu, or gemm_bf16_umma.cu where there are no pairs of SMs) in which every row multiplies its own expert only.
//
//   sort     the (token, choice) pairs in the order of their experts, each expert's on whole tiles of 128 rows
//   gather   x of every row's token
//   gate     y = weight(t, c) * act(gate, up) in the products' float32, rounded to bfloat16 as on the way over all
//            experts (moe.cu): in the first product's epilogue; the launch below makes the same bits (but for gates below -80,
//            silu.cuh) and is what tests compare with. 1,500 tokens, 2 of 8 experts of 2048 x 1024: product and gate 38 us (38 + 7 in two launches,
//            and 29 MB of float32 less to write and read)
//   combine  out[t] (+)= sum over a token's choices in their order
//
// The passes around the products wait for memory more than they read: what they need is asked for together, not number by number, and a
// warp of the sorting kernel goes over a run of pairs of its own, without meeting the others on the way. us over router, experts and sum, in
// brackets with a row a CTA and a meeting per 512 pairs: 2048 x 1024, 2 of 8 experts 1,500 tokens 78.8 (82.7), 2,048 96 (103), 4 of 16 1,000
// tokens 112 (120); 1024 x 512, 2 of 8 520 tokens 30.5 (31.8), 2,000 46.3 (54.2).
//
// Against the products over all experts (E / top times the arithmetic, E 2 ff float32 columns per token between them)
// this pays where experts are large or many: ops.moe_prefers_sorted and ops.moe_prefers_pairs have the lines and what both sides
// measured.
// What the launches before write is read through plain pointers: loads through `const __restrict__` ones may be moved ahead of
// the wait for those launches.
#include <climits>

#include "common.cuh"

namespace {

constexpr int kTileRows = 128;
constexpr int kSortThreads = 512;

__device__ __forceinline__ float activation(float g, float u, int act, float limit, float alpha) {
  if (act == 1) return g / (1.0f + expf(-g)) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
}

// A CTA per expert: every CTA counts all experts' pairs, so that it knows where its own begin, then lists its own in
// ascending order. rows[pos] = pair or -1 (padding up to whole tiles); places[pair] = pos, -1 for an identity expert;
// tile_experts[tile] = expert, -1 behind the last tile.
__global__ __launch_bounds__(kSortThreads) void moe_sort_kernel(const int* ids, int pairs, int experts,
                                                                int* __restrict__ rows, int* __restrict__ places,
                                                                int* __restrict__ tile_experts, int tiles) {
  extern __shared__ int counts[];  // [experts]
  __shared__ int warp_counts[kSortThreads / 32];
  __shared__ int before_all, total_all;
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mine = blockIdx.x;
  for (int e = tid; e < experts; e += kSortThreads) counts[e] = 0;
  if (tid == 0) before_all = total_all = 0;
  __syncthreads();
  for (int p0 = tid; p0 < pairs; p0 += 8 * kSortThreads) {
    int e[8];  // asked for together
#pragma unroll
    for (int u = 0; u < 8; ++u) e[u] = p0 + u * kSortThreads < pairs ? ids[p0 + u * kSortThreads] : INT_MAX;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (e[u] >= 0 && e[u] < experts) atomicAdd(counts + e[u], 1);
      else if (mine == 0 && p0 + u * kSortThreads < pairs) places[p0 + u * kSortThreads] = -1;
    }
  }
  __syncthreads();
  int before = 0, total = 0;
  for (int e = tid; e < experts; e += kSortThreads) {
    const int own = (counts[e] + kTileRows - 1) / kTileRows;
    total += own;
    if (e < mine) before += own;
  }
  atomicAdd(&before_all, before);
  atomicAdd(&total_all, total);
  __syncthreads();
  const int first = before_all, count = counts[mine], own_tiles = (count + kTileRows - 1) / kTileRows;
  for (int i = tid; i < own_tiles; i += kSortThreads) tile_experts[first + i] = mine;
  if (mine == experts - 1)
    for (int i = total_all + tid; i < tiles; i += kSortThreads) tile_experts[i] = -1;
  // a warp's run of pairs: how many are this expert's in the runs ahead, then its own in their order
  const int run = (pairs + kSortThreads - 1) / kSortThreads * 32, from = warp * run, upto = min(pairs, from + run);
  int own = 0;
  unsigned held[8];  // which of the first eight times 32
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int p = from + 32 * u + lane;
    held[u] = __ballot_sync(0xffffffffu, p < upto && ids[p] == mine);
    own += __popc(held[u]);
  }
#pragma unroll 4
  for (int p0 = from + 8 * 32; p0 < upto; p0 += 32) own += __popc(__ballot_sync(0xffffffffu, p0 + lane < upto && ids[p0 + lane] == mine));
  if (lane == 0) warp_counts[warp] = own;
  __syncthreads();
  const int ahead = lane < warp ? warp_counts[lane] : 0;
  int at = first * kTileRows + __reduce_add_sync(0xffffffffu, ahead);
  const auto place = [&](int p, unsigned which) {
    if (which >> lane & 1) {
      const int pos = at + __popc(which & ((1u << lane) - 1u));
      rows[pos] = p;
      places[p] = pos;
    }
    at += __popc(which);
  };
#pragma unroll
  for (int u = 0; u < 8; ++u) place(from + 32 * u + lane, held[u]);
#pragma unroll 4
  for (int p0 = from + 8 * 32; p0 < upto; p0 += 32)
    place(p0 + lane, __ballot_sync(0xffffffffu, p0 + lane < upto && ids[p0 + lane] == mine));
  for (int i = count + tid; i < own_tiles * kTileRows; i += kSortThreads) rows[first * kTileRows + i] = -1;
}

// A warp per row, eight of a lane's loads under way. Rows behind the last tile are nobody's: not read by the products.
__global__ __launch_bounds__(256) void moe_gather_kernel(const uint4* x, const int* rows,
                                                         const int* tile_experts, int top, int pieces,
                                                         uint4* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (tile_experts[row / kTileRows] < 0) return;
  const int p = rows[row];
  const uint4* from = x + static_cast<size_t>(max(p, 0) / top) * pieces;
  uint4* to = out + static_cast<size_t>(row) * pieces;
  for (int i0 = lane; i0 < pieces; i0 += 8 * 32) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = p >= 0 && i0 + 32 * u < pieces ? from[i0 + 32 * u] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + 32 * u < pieces) to[i0 + 32 * u] = v[u];
  }
}

__global__ __launch_bounds__(256) void moe_sorted_gate_kernel(const float* gu, const int* rows,
                                                              const int* tile_experts, const float* weights,
                                                              int ff, float limit, float alpha, int act,
                                                              __nv_bfloat16* __restrict__ y) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x;
  if (tile_experts[row / kTileRows] < 0) return;
  const int p = rows[row];
  const float w = p < 0 ? 0.f : weights[p];
  const float* g = gu + static_cast<size_t>(row) * 2 * ff;
  for (int f = threadIdx.x * 4; f < ff; f += blockDim.x * 4) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (w != 0.f) {
      const float4 a = *reinterpret_cast<const float4*>(g + f), b = *reinterpret_cast<const float4*>(g + ff + f);
      v[0] = activation(a.x, b.x, act, limit, alpha) * w, v[1] = activation(a.y, b.y, act, limit, alpha) * w;
      v[2] = activation(a.z, b.z, act, limit, alpha) * w, v[3] = activation(a.w, b.w, act, limit, alpha) * w;
    }
    __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(y + static_cast<size_t>(row) * ff + f) =
        make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
  }
}

__global__ __launch_bounds__(256) void moe_combine_kernel(const float* part, const int* places, int top,
                                                          int width, int add, float* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const size_t t = blockIdx.x;
  int first[4];  // the first choices' rows: asked for at once, as are their numbers
#pragma unroll
  for (int c = 0; c < 4; ++c) first[c] = c < top ? places[t * top + c] : -1;
#pragma unroll 2
  for (int i = threadIdx.x * 4; i < width; i += blockDim.x * 4) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f), v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (first[c] >= 0) v[c] = *reinterpret_cast<const float4*>(part + static_cast<size_t>(first[c]) * width + i);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (first[c] >= 0) sum.x += v[c].x, sum.y += v[c].y, sum.z += v[c].z, sum.w += v[c].w;
    for (int c = 4; c < top; ++c) {
      const int pos = places[t * top + c];
      if (pos < 0) continue;
      const float4 more = *reinterpret_cast<const float4*>(part + static_cast<size_t>(pos) * width + i);
      sum.x += more.x, sum.y += more.y, sum.z += more.z, sum.w += more.w;
    }
    float4* to = reinterpret_cast<float4*>(out + t * width + i);
    if (add) {
      const float4 old = *to;
      sum.x += old.x, sum.y += old.y, sum.z += old.z, sum.w += old.w;
    }
    *to = sum;
  }
}

}  // namespace

// Tiles of 128 rows that hold any choice of `pairs` pairs among `experts` experts.
LRM_API int lrm_moe_sorted_tiles_room(int pairs, int experts) { return pairs / kTileRows + experts; }

// ids int32 [pairs] -> rows int32 [tiles * 128], places int32 [pairs], tile_experts int32 [tiles].
LRM_API int lrm_moe_sort(const int* ids, int pairs, int experts, int* rows, int* places, int* tile_experts, int tiles,
                         cudaStream_t stream) {
  if (pairs <= 0) return 0;
  if (experts <= 0 || experts > 8192 || tiles < lrm_moe_sorted_tiles_room(pairs, experts)) return LRM_BAD_ARGUMENT;
  LRM_LAUNCH(moe_sort_kernel, experts, kSortThreads, sizeof(int) * experts, stream, ids, pairs, experts, rows, places, tile_experts,
             tiles);
  return 0;
}

// x bfloat16 [T, width] -> out [tiles * 128, width] (width a multiple of 8, rows 16-byte aligned).
LRM_API int lrm_moe_gather(const void* x, const int* rows, const int* tile_experts, int top, int width, int tiles, void* out,
                           cudaStream_t stream) {
  if (width <= 0 || width % 8 || top <= 0 || tiles <= 0) return LRM_BAD_ARGUMENT;
  LRM_LAUNCH(moe_gather_kernel, tiles * kTileRows / 8, 256, 0, stream, static_cast<const uint4*>(x), rows, tile_experts, top, width / 8,
             static_cast<uint4*>(out));
  return 0;
}

// gu float32 [tiles * 128, 2 ff] (gate columns, then up columns) -> y bfloat16 [tiles * 128, ff]; ff a multiple of 4.
LRM_API int lrm_moe_sorted_gate(const float* gu, const int* rows, const int* tile_experts, const float* weights, int ff, int tiles,
                                float limit, float alpha, int act, void* y, cudaStream_t stream) {
  if (ff <= 0 || ff % 4 || tiles <= 0 || (act != 0 && act != 1)) return LRM_BAD_ARGUMENT;
  LRM_LAUNCH(moe_sorted_gate_kernel, tiles * kTileRows, 256, 0, stream, gu, rows, tile_experts, weights, ff, limit, alpha, act,
             static_cast<__nv_bfloat16*>(y));
  return 0;
}

// part float32 [tiles * 128, width], places int32 [T * top]; out float32 [T, width], added to with `add`.
LRM_API int lrm_moe_combine(const float* part, const int* places, int tokens, int top, int width, int add, float* out,
                            cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (width <= 0 || width % 4 || top <= 0) return LRM_BAD_ARGUMENT;
  LRM_LAUNCH(moe_combine_kernel, tokens, 256, 0, stream, part, places, top, width, add, out);
  return 0;
}

LRM_API int lrm_gemm_bf16_wide_experts(const void* X, const void* W, void* out, int M, int N, int K, long long w_height, long long w_width,
                                       int w_rows, int w_cols, const int* tile_experts, int* status, cudaStream_t stream);
LRM_API int lrm_gemm_bf16_wide_experts_gated(const void* X, const void* W, void* out, int M, int ff, int K, long long w_height,
                                             const int* tile_experts, const int* rows, const float* weights, float limit, float alpha,
                                             int act, int* status, cudaStream_t stream);

namespace {

// How lrm_moe_sorted_step divides its scratch, in bytes from its start; M rows in `tiles` tiles.
struct SortedScratch {
  int tiles;
  long long M, y, part, rows, places, tile_experts, end;
  SortedScratch(int tokens, int width, int ff, int experts, int top) {
    const long long pairs = static_cast<long long>(tokens) * top;
    tiles = static_cast<int>(pairs / kTileRows) + experts, M = static_cast<long long>(tiles) * kTileRows;
    y = M * width * 2, part = y + M * ff * 2, rows = part + M * width * 4, places = rows + M * 4;
    tile_experts = places + (pairs + 3) / 4 * 16, end = tile_experts + (tiles + 3) / 4 * 16ll;
  }
};

}  // namespace

// Bytes of scratch that lrm_moe_sorted_step wants.
LRM_API long long lrm_moe_sorted_step_bytes(int tokens, int width, int ff, int experts, int top) {
  return SortedScratch(tokens, width, ff, experts, top).end;
}

// The five launches in one call, with the products on pairs of SMs: out float32 [T, width] (added to with `add`) from bfloat16 x
// [T, width], gate_up [experts, 2 ff, width], down [width, experts, ff] and the choices ids, weights [T, top]. width and ff multiples of
// 64; x, gate_up, down and scratch on 16 bytes.
LRM_API int lrm_moe_sorted_step(const void* x, const void* gate_up, const void* down, const int* ids, const float* weights, void* scratch,
                                float* out, int tokens, int width, int ff, int experts, int top, float limit, float alpha, int act, int add,
                                int* status, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (width <= 0 || width % 64 || ff <= 0 || ff % 64 || top <= 0 || experts <= 0 || experts > 8192 || (act != 0 && act != 1) ||
      scratch == nullptr || status == nullptr || static_cast<long long>(tokens) * top >= 1ll << 28)
    return LRM_BAD_ARGUMENT;
  const SortedScratch at(tokens, width, ff, experts, top);
  if (at.M >= 1ll << 31 || 2ll * experts * ff >= 1ll << 31) return LRM_UNSUPPORTED;
  char* const base = static_cast<char*>(scratch);
  int *rows = reinterpret_cast<int*>(base + at.rows), *places = reinterpret_cast<int*>(base + at.places);
  int* tile_experts = reinterpret_cast<int*>(base + at.tile_experts);
  float* part = reinterpret_cast<float*>(base + at.part);
  const int M = static_cast<int>(at.M);
  LRM_LAUNCH(moe_sort_kernel, experts, kSortThreads, sizeof(int) * experts, stream, ids, tokens * top, experts, rows, places, tile_experts,
             at.tiles);
  LRM_LAUNCH(moe_gather_kernel, M / 8, 256, 0, stream, static_cast<const uint4*>(x), rows, tile_experts, top, width / 8,
             reinterpret_cast<uint4*>(base));
  int code = lrm_gemm_bf16_wide_experts_gated(base, gate_up, base + at.y, M, ff, width, 2ll * experts * ff, tile_experts, rows, weights, limit,
                                              alpha, act, status, stream);
  if (code == 0)
    code = lrm_gemm_bf16_wide_experts(base + at.y, down, part, M, width, ff, width, static_cast<long long>(experts) * ff, 0, ff, tile_experts,
                                      status, stream);
  return code != 0 ? code : lrm_moe_combine(part, places, tokens, top, width, add, out, stream);
}
