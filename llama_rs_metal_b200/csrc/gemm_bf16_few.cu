// bfloat16 products of few rows (decoding) on the 5th-generation tensor cores, the weights as the wide operand:
// Y[M, N] = X[M, K] . W[N, K]^T, M <= 64.
//
// Bound by reading W. A tile of 128 weight rows is the A operand of tcgen05.mma (M 128), the activation rows are its 16, 32
// or 64 columns, so a stage of the TMA ring is 16 KB of weights and only 2 to 8 KB of activations, and some 200 KB per SM
// are on their way. The ring's first stages of weights are asked for before the kernel waits for its predecessor. The
// accumulator's lanes are weight rows: a thread has one output column for all activation rows, and neighbouring threads
// neighbouring columns.
//
// Persistent: CTA b works on items b, b + gridDim.x, ...; an item is a (K slice, tile) with the tiles fastest, two accumulators in
// turn, so an item's epilogue runs under the next one's reads. Narrow products, whose tiles leave SMs idle, are cut into K slices, each
// a float32 plane that the reader adds up in order (the next norm, or decode attention for q|k|v): 6144 x 4096, 32 rows, 10.3 us in three
// planes against 16.4 whole. No atomics: the result is the same every time. (A cluster of CTAs to a tile with the partial sums meeting
// in distributed shared memory was slower: 20.6 us.)
//
// Every weight is read once and leaves L2 first, so that the keys and values of short contexts are still there when attention comes: one
// sequence of 500 keys, 32 heads of 96 (two layers) 341 us a step, 16 of 256 (three) 3,482; with the copies' usual order 491 and 6,332
// (streamed 348 and 3,493), and steps that attend by the cluster kernel 2 to 4 % longer (8B shape, six layers, 561 -> 575).
//
// Epilogues as in gemm_bf16_stream.cu: 0 bf16, 1 f32, 3 SiLU gate (blocks of 8 gate / 8 up rows alternate), 4 f32 planes of K slices.
// Every mbarrier wait is bounded. Its times beside those of the kernels it replaces stand at gemm_dispatch.few_takes and few_plan.
#include "silu.cuh"
#include "umma.cuh"

namespace {

constexpr int kTileRows = 128, BK = 64, UMMA_K = 16, kThreads = 192;  // loader warp, issuer warp, four epilogue warps

enum : int { kStuckEmpty = 51, kStuckFull = 52, kStuckAccumulator = 53, kStuckDrain = 54, kStuckTmemFree = 55 };

template <int NC>
struct Few {
  static constexpr int STAGES = NC == 16 ? 11 : NC == 32 ? 9 : 7;
  static constexpr uint32_t W_BYTES = kTileRows * BK * 2, STAGE_BYTES = W_BYTES + NC * BK * 2;
  static constexpr uint32_t SET = NC < 32 ? 32 : NC;                 // tensor memory columns of an accumulator
  static constexpr size_t BYTES = 1024 + STAGES * STAGE_BYTES + 256;
};

// Column n, activation row m.
__device__ __forceinline__ void finish(float v, int m, int n, void* out, int N, int mode) {
  const size_t o = static_cast<size_t>(m) * N + n;
  if (mode == 0) static_cast<__nv_bfloat16*>(out)[o] = __float2bfloat16_rn(v);
  else static_cast<float*>(out)[o] = v;
}

// The gate over rows m0 .. m0 + ROWS - 1, a column per lane, 8 gate and 8 up columns in turn. The two lanes of a pair take half of
// the rows each, and their quotients go side by side. Every lane of the warp calls it; `stored`: this lane's column exists.
template <int ROWS>
__device__ __forceinline__ void finish_gated(const uint32_t (&r)[32], int m0, int M, int n, bool stored, __nv_bfloat16* out, int N) {
  constexpr int HALF = ROWS / 2;
  const bool is_up = n & 8;
  float g[HALF], u[HALF];
#pragma unroll
  for (int i = 0; i < HALF; ++i) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, is_up ? r[i] : r[i + HALF], 8);
    g[i] = __uint_as_float(is_up ? other : r[i]);
    u[i] = __uint_as_float(is_up ? r[i + HALF] : other);
  }
  silu_all(g);
  const int first = m0 + (is_up ? HALF : 0);
  out += static_cast<size_t>(first) * (N >> 1) + (n >> 4) * 8 + (n & 7);
#pragma unroll
  for (int i = 0; i < HALF; ++i)
    if (stored && first + i < M) out[static_cast<size_t>(i) * (N >> 1)] = __float2bfloat16_rn(g[i] * u[i]);
}

template <int NC>
__global__ __launch_bounds__(kThreads, 1) void gemm_bf16_few_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                    const __grid_constant__ CUtensorMap map_x, void* __restrict__ out,
                                                                    int M, int N, int K, int mode, int tile_rows, int kb_per_split,
                                                                    int splits, int* __restrict__ status) {
  using F = Few<NC>;
  constexpr int STAGES = F::STAGES;
  pdl_trigger();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + STAGES * F::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;  // [2]
  uint64_t* acc_free = acc_full + 2;    // [2] four warps arrive
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 2);
  volatile int* bail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t stage_bytes = tile_rows * BK * 2 + F::STAGE_BYTES - F::W_BYTES;  // of the copies
  const int tiles = (N + tile_rows - 1) / tile_rows, k_blocks = (K + BK - 1) / BK;
  const int items = tiles * splits, first_item = blockIdx.x, stride = gridDim.x;  // an item: (K slice, tile), the tiles fastest
  const int early = min(min(kb_per_split, k_blocks - first_item / tiles * kb_per_split), STAGES);  // stages of the first item's weights asked for ahead of the wait

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full + a, 1);
      mbar_init(acc_free + a, 4);
    }
    *bail = 0;
    mbar_fence_init();
    for (int kb = 0; kb < early; ++kb) {
      mbar_expect_tx(full + kb, stage_bytes);
      tma_load_2d_once(ring + kb * F::STAGE_BYTES, &map_w, full + kb, (first_item / tiles * kb_per_split + kb) * BK, first_item % tiles * tile_rows,
                       l2_evict_first());
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * F::SET);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();  // X is read from here on

  if (warp == 0) {
    if (lane == 0) {
      // The early stages' activations first, whatever happens: copies into those stages are under way.
      for (int kb = 0; kb < early; ++kb)
        tma_load_2d(ring + kb * F::STAGE_BYTES + F::W_BYTES, &map_x, full + kb, (first_item / tiles * kb_per_split + kb) * BK, 0);
      const uint64_t once = l2_evict_first();
      uint32_t it = early;  // blocks asked for so far
      int from = early;
      for (int item = first_item; item < items && !*bail; item += stride, from = 0) {
        const int slice = item / tiles, w_row = (item - slice * tiles) * tile_rows, kb0 = slice * kb_per_split;
        const int num_kb = min(kb_per_split, k_blocks - kb0);
        for (int kb = from; kb < num_kb; ++kb, ++it) {
          const uint32_t s = it % STAGES, round = it / STAGES;
          if (round > 0 && !mbar_wait(empty + s, (round - 1) & 1, status, kStuckEmpty)) {
            *bail = 1;
            break;
          }
          mbar_expect_tx(full + s, stage_bytes);
          tma_load_2d_once(ring + s * F::STAGE_BYTES, &map_w, full + s, (kb0 + kb) * BK, w_row, once);
          tma_load_2d(ring + s * F::STAGE_BYTES + F::W_BYTES, &map_x, full + s, (kb0 + kb) * BK, 0);
        }
      }
      if (*bail) {  // wait (bounded) for the copies already in flight before the CTA may exit
        const uint32_t oldest = it > STAGES ? it - STAGES : 0;
        for (uint32_t i = oldest; i < it; ++i) mbar_wait(full + i % STAGES, (i / STAGES) & 1, status, kStuckDrain);
      }
    }
  } else if (warp == 1) {
    // The warp stays together around its issuing lane and goes through all blocks that are there with one question, as in
    // gemm_bf16_umma.cu: a block's copies take some 600 cycles, a wait and four products by a lane of its own no fewer.
    constexpr uint32_t idesc = umma_idesc(kTileRows, NC);  // both operands K-major
    const uint32_t ring_at = __shfl_sync(0xffffffffu, smem_u32(ring), 0), tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    const bool chosen = elect_one();
    uint32_t it = 0, local = 0;
    bool going = true;
    for (int item = first_item; item < items && going; item += stride, ++local) {
      const int num_kb = min(kb_per_split, k_blocks - item / tiles * kb_per_split);
      const uint32_t acc = local & 1, use = local >> 1;
      if (__any_sync(0xffffffffu, *bail != 0) ||
          (use > 0 && !__all_sync(0xffffffffu, lane != 0 || mbar_wait(acc_free + acc, (use - 1) & 1, status, kStuckTmemFree)))) {
        *bail = 1;
        break;
      }
      tc_fence_after();
      for (int kb = 0; kb < num_kb;) {
        const int ready = min(ring_ready<STAGES>(full, it, lane, status, kStuckFull), num_kb - kb);
        if (ready == 0) {
          *bail = 1;
          going = false;
          break;
        }
        tc_fence_after();
        for (const int until = kb + ready; kb < until; ++kb, ++it) {
          const uint32_t s = it % STAGES;
          const uint32_t a = ring_at + s * F::STAGE_BYTES, b = a + F::W_BYTES;
          if (chosen) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16(tmem + acc * F::SET, smem_desc(a + k * UMMA_K * 2), smem_desc(b + k * UMMA_K * 2), idesc,
                        (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit(empty + s);
            if (kb + 1 == num_kb) umma_commit(acc_full + acc);  // (here and last: as in gemm_bf16_umma.cu)
          }
          __syncwarp();
        }
      }
    }
  } else {
    const int quarter = warp & 3, place = quarter * 32 + lane;  // a warp may touch only this quarter of the lanes
    uint32_t local = 0;
    for (int item = first_item; item < items; item += stride, ++local) {
      const int slice = item / tiles, tile = item - slice * tiles;
      void* plane = mode == 4 ? static_cast<void*>(static_cast<float*>(out) + static_cast<size_t>(slice) * M * N) : out;
      const uint32_t acc = local & 1;
      if (*bail || !mbar_wait(acc_full + acc, (local >> 1) & 1, status, kStuckAccumulator)) {
        *bail = 1;
        break;
      }
      tc_fence_after();
      const int n = tile * tile_rows + place;
      const bool stored = place < tile_rows && n < N;
#pragma unroll 1
      for (int c = 0; c < (NC + 31) / 32; ++c) {
        uint32_t r[32];
        tmem_load32(tmem_base + acc * F::SET + (static_cast<uint32_t>(quarter * 32) << 16) + c * 32, r);
        constexpr int ROWS = NC < 32 ? NC : 32;
        if (mode == 3) {
          finish_gated<ROWS>(r, c * 32, M, n, stored, static_cast<__nv_bfloat16*>(out), N);
          continue;
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
          const int m = c * 32 + i;
          if (m >= M || !stored) break;
          finish(__uint_as_float(r[i]), m, n, plane, N, mode);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free + acc);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 2 * F::SET);
}

template <int NC>
int launch(const void* X, const void* W, void* out, int M, int x_rows, int N, int K, int mode, int splits, int rows_wanted, int* status, cudaStream_t stream) {
  // Fewer weight rows to a tile where that leaves the CTA with the most tiles fewer rows to read (the others wait for it, and a part
  // of the SMs does not draw the whole bandwidth). The products work on 128 rows either way; those beyond are not stored. (8 rows:
  // what a tile costs beside its reads.) With the whole warp issuing and the gate's quotients side by side, us, 32 rows: 28672 x
  // 4096 43.1 -> 40.3 (gated 53.3 -> 41.0), 9472 x 22000 103 -> 84.
  int tile_rows = kTileRows, least = 0;
  for (int rows = kTileRows; rows >= 64; rows -= 16) {
    const int cost = ((N + rows - 1) / rows * splits + kSmCount - 1) / kSmCount * (rows + 8);
    if (least == 0 || cost < least) {
      least = cost;
      tile_rows = rows;
    }
  }
  if (rows_wanted > 0) tile_rows = rows_wanted;
  CUtensorMap map_w, map_x;
  if (!make_map_bf16(&map_w, W, N, K, tile_rows) || !make_map_bf16(&map_x, X, x_rows, K, NC)) return LRM_UNSUPPORTED;
  auto kernel = gemm_bf16_few_kernel<NC>;
  constexpr int smem = static_cast<int>(Few<NC>::BYTES);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int items = (N + tile_rows - 1) / tile_rows * splits, k_blocks = (K + BK - 1) / BK;
  LRM_LAUNCH(kernel, dim3(items < kSmCount ? items : kSmCount), kThreads, smem, stream, map_w, map_x, out, M, N, K, mode, tile_rows,
             (k_blocks + splits - 1) / splits, splits, status);
  return 0;
}

}  // namespace

// Shapes this kernel takes: up to 64 rows, K a multiple of 8 (TMA needs 16-byte row pitches).
LRM_API int lrm_gemm_bf16_few_supports(int M, int N, int K) {
  return M >= 1 && M <= 64 && N >= 1 && K >= 8 && K % 8 == 0 && encode_tiled() != nullptr ? 1 : 0;
}

// K slices a product in `wanted` slices really has: none is empty.
LRM_API int lrm_gemm_bf16_few_slices(int K, int wanted) {
  const int k_blocks = (K + BK - 1) / BK, per_split = (k_blocks + wanted - 1) / wanted;
  return (k_blocks + per_split - 1) / per_split;
}

// `x_rows` >= M: rows of X that may be read (TMA was measured slower on maps of fewer than 32 rows). `splits` (mode 4): as
// lrm_gemm_bf16_few_slices says; out is [splits, M, N]. `status`: one int in device memory, 0 before the launch.
LRM_API int lrm_gemm_bf16_few(const void* X, const void* W, void* out, int M, int x_rows, int N, int K, int mode, int splits, int tile_rows,
                              int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (!lrm_gemm_bf16_few_supports(M, N, K)) return LRM_UNSUPPORTED;
  if ((mode != 0 && mode != 1 && mode != 3 && mode != 4) || (mode == 3 && N % 16 != 0) || x_rows < M || status == nullptr || splits < 1 ||
      (splits > 1 && mode != 4) || splits != lrm_gemm_bf16_few_slices(K, splits) || tile_rows < 0 || tile_rows > kTileRows || tile_rows % 16)
    return LRM_BAD_ARGUMENT;
  if (reinterpret_cast<uintptr_t>(X) % 16 || reinterpret_cast<uintptr_t>(W) % 16) return LRM_UNSUPPORTED;
  if (M <= 16) return launch<16>(X, W, out, M, x_rows, N, K, mode, splits, tile_rows, status, stream);
  if (M <= 32) return launch<32>(X, W, out, M, x_rows, N, K, mode, splits, tile_rows, status, stream);
  return launch<64>(X, W, out, M, x_rows, N, K, mode, splits, tile_rows, status, stream);
}
