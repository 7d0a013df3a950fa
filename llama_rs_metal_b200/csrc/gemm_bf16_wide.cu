// bfloat16 products of more than 64 rows on pairs of SMs, the weights as the wide operand: Y[M, N] = X[M, K] . W[N, K]^T. Which products
// come here is estimated (gemm_dispatch.wide_plan): mostly those of up to some 1,300 rows, narrow ones of any number.
//
// A cluster of two CTAs makes a tile of 256 weight rows and BN activation rows with tcgen05.mma.cta_group::2 (M 256, N = BN): the
// weight rows are the A operand, so the activation rows are cut into tiles of any multiple of 32 up to 256 (529 rows: three of
// 192) where the kernels with activations as A fill whole tiles of 128 or 256 (640 or 768). CTA r of the pair loads weight rows
// [128 r, 128 r + 128) and activation rows [BN/2 r, BN/2 r + BN/2) of every stage.
//
// The accumulator's lanes are weight rows: a thread has one output column of its tokens, neighbouring lanes neighbouring columns, so
// a token's results leave a warp as a run of 128 bytes (float32), 64 (bfloat16, two columns a lane) or 32 (gated).
// Two sets of accumulators: a tile's epilogue runs under the next tile's products. The first stages' weights are asked for ahead of
// the kernel's wait for its predecessor.
//
// Sorted experts of a prompt (moe_sorted.cu): 128 rows of X are a tile of one expert, named by tile_experts; the first product's CTA
// takes 64 gate and 64 up rows of weights, and its epilogue writes weight * act(gate, up). 25 tiles (1,500 tokens, 2 of 8 experts of 2048 x
// 1024) on 74 pairs are three rounds of half a tile's time where 148 SMs of their own take two of a whole one: 35 and 21 us for the two
// products, 38 and 23 before. Tiles of 192 rows 34.5 and 18, but 125 against 120 us over all for 1,000 tokens, 4 of 16 experts, and 59
// against 54 for 2,000 tokens of 1024 x 512: more of them is filling.
//
// Epilogues: 0 bf16, 1 f32, 2 add into f32 in place (one add an element), 3 SiLU gate (blocks of 8 gate / 8 up rows alternate), 4 f32
// planes of K slices. No atomics where sums meet: the same result every time. Every mbarrier wait is bounded, and both CTAs of a pair
// always meet at the closing cluster barrier. The TMA loads carry no multicast.
#include "silu.cuh"
#include "umma_pair.cuh"

namespace {

constexpr int kWideRows = 128, BK = 64, UMMA_K = 16;  // weight rows per CTA, K per stage, K per instruction
constexpr int kSortedRows = 128;                      // of X in a tile of one expert
constexpr int kThreads = 352;                         // loader, tensor-memory/issuer warp, eight epilogue warps, second loader

enum : int { kStuckEmpty = 71, kStuckFull = 72, kStuckAccumulator = 73, kStuckDrain = 74, kStuckTmemFree = 75, kStuckGate = 76 };

template <int BN, bool GATED = false>
struct Wide {
  static constexpr uint32_t W_BYTES = kWideRows * BK * 2, STAGE_BYTES = W_BYTES + (BN / 2) * BK * 2;
  static constexpr int MEET = GATED ? 8 * 4096 : 0;  // where gates and ups meet: two pieces of 32 tokens per two epilogue warps, 4 KB each
  static constexpr int STAGES = (229376 - MEET) / STAGE_BYTES < 11 ? (229376 - MEET) / STAGE_BYTES : 11;
  static constexpr size_t BYTES = 1024 + STAGES * STAGE_BYTES + 256 + MEET;
  static constexpr int PIECE = BN % 64 == 0 ? 32 : 16;  // tokens that a thread takes out of tensor memory at a time
};

// A warp's 32 columns n0 .. of PIECE tokens from m0 on; r[i]: this lane's column of token m0 + i. Every lane calls it.
template <int PIECE>
__device__ __forceinline__ void store_columns(const uint32_t (&r)[PIECE], int m0, int M, int n, int N, void* __restrict__ out, int mode) {
  const bool odd = n & 1, stored = n < N;
  if (mode == 3) {  // the lanes of a gate and of its up row take half of the tokens each, then pairs of columns half of those
    constexpr int HALF = PIECE / 2;
    const bool is_up = n & 8;
    float g[HALF], u[HALF];
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, is_up ? r[i] : r[i + HALF], 8);
      g[i] = __uint_as_float(is_up ? other : r[i]);
      u[i] = __uint_as_float(is_up ? r[i + HALF] : other);
    }
    silu_all(g);
    const int first = m0 + (is_up ? HALF : 0) + odd;
    __nv_bfloat16* to = static_cast<__nv_bfloat16*>(out) + static_cast<size_t>(first) * (N >> 1) + (n >> 4) * 8 + (n & 6);
#pragma unroll
    for (int i = 0; i < HALF; i += 2) {
      const float even_token = g[i] * u[i], odd_token = g[i + 1] * u[i + 1];
      const float other = __shfl_xor_sync(0xffffffffu, odd ? even_token : odd_token, 1);
      if (stored && first + i < M)
        *reinterpret_cast<uint32_t*>(to + static_cast<size_t>(i) * (N >> 1)) = odd ? pack_bf16(other, odd_token) : pack_bf16(even_token, other);
    }
  } else if (mode == 0) {
    const int first = m0 + odd;
    __nv_bfloat16* to = static_cast<__nv_bfloat16*>(out) + static_cast<size_t>(first) * N + (n & ~1);
#pragma unroll
    for (int i = 0; i < PIECE; i += 2) {
      const float even_token = __uint_as_float(r[i]), odd_token = __uint_as_float(r[i + 1]);
      const float other = __shfl_xor_sync(0xffffffffu, odd ? even_token : odd_token, 1);
      if (stored && first + i < M)
        *reinterpret_cast<uint32_t*>(to + static_cast<size_t>(i) * N) = odd ? pack_bf16(other, odd_token) : pack_bf16(even_token, other);
    }
  } else if (stored) {
    float* to = static_cast<float*>(out) + static_cast<size_t>(m0) * N + n;
#pragma unroll
    for (int i = 0; i < PIECE; ++i) {
      if (m0 + i >= M) break;
      if (mode == 2) atomicAdd(to + static_cast<size_t>(i) * N, __uint_as_float(r[i]));  // no value comes back
      else to[static_cast<size_t>(i) * N] = __uint_as_float(r[i]);
    }
  }
}

// Row tile m multiplies the W of expert tile_experts[m] (-1: no tile, nor any after it), which begins w_rows rows and w_cols columns
// after the W of the expert before. From `rows` on for the gated product.
struct WideExperts {
  const int* tile_experts;
  int w_rows, w_cols;
  const int* rows;
  const float* weights;  // of a row's pair
  int ff, act;
  float limit, alpha;
};

// The gate over a piece of 32 tokens (m0 ..): the warps of 32 gate columns and of their up columns hold one of the two each, take 16 of
// the tokens each and hand the other's through `meet` (2 x 16 x 32 floats). f: this lane's column. Both warps call it; `both`: their
// barrier, two arrivals a phase. False: the other warp did not come.
__device__ __forceinline__ bool store_gated_columns(const uint32_t (&r)[32], bool is_up, float* meet, uint64_t* both, uint32_t parity, int m0,
                                                    int f, __nv_bfloat16* __restrict__ out, const WideExperts& a, int* status) {
  const int lane = threadIdx.x & 31, p = a.rows[m0 + lane];
  const float weight_of = p < 0 ? 0.f : a.weights[p];
  float* give = meet + (is_up ? 0 : 512);
  const float* take = meet + (is_up ? 512 : 0);
#pragma unroll
  for (int i = 0; i < 16; ++i) give[i * 32 + lane] = __uint_as_float(is_up ? r[i] : r[16 + i]);
  __syncwarp();
  if (lane == 0) mbar_arrive(both);
  if (!mbar_wait_warp(lane == 0, both, parity, status, kStuckGate)) return false;
  float g[16], u[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float other = take[i * 32 + lane];
    g[i] = is_up ? other : __uint_as_float(r[i]);
    u[i] = is_up ? __uint_as_float(r[16 + i]) : other;
    if (a.act != 1) g[i] = fminf(g[i], a.limit), u[i] = fminf(fmaxf(u[i], -a.limit), a.limit) + 1.f;
  }
  silu_all(g, a.act == 1 ? 1.f : a.alpha);
  const bool odd = lane & 1;
  const int first = is_up ? 16 : 0;
  __nv_bfloat16* to = out + static_cast<size_t>(m0 + first + odd) * a.ff + (f & ~1);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float weight = __shfl_sync(0xffffffffu, weight_of, first + i);
    g[i] = weight != 0.f ? g[i] * u[i] * weight : 0.f;
  }
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const float other = __shfl_xor_sync(0xffffffffu, odd ? g[i] : g[i + 1], 1);
    if (f < a.ff) *reinterpret_cast<uint32_t*>(to + static_cast<size_t>(i) * a.ff) = odd ? pack_bf16(other, g[i + 1]) : pack_bf16(g[i], other);
  }
  return true;
}

// Pair p (CTAs 2p and 2p + 1) works on items p, p + pairs, ...; an item is a (K slice, tile of weight rows, tile of activation rows)
// with the activation rows fastest, so that pairs that run together share weights in L2.
// Warps 0 and 10: TMA loaders. Warp 1: tensor memory, and in the leader the MMA issuer. Warps 2-9: epilogue.
template <int BN, bool EXPERTS = false, bool GATED = false>
__global__ __launch_bounds__(kThreads, 1) void gemm_bf16_wide_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                     const __grid_constant__ CUtensorMap map_x, void* __restrict__ out,
                                                                     int M, int N, int K, int mode, int kb_per_split, int splits,
                                                                     int* __restrict__ status, const __grid_constant__ WideExperts experts) {
  using S = Wide<BN, GATED>;
  static_assert(!GATED || (EXPERTS && S::PIECE == 32), "a tile of sorted rows");
  constexpr int STAGES = S::STAGES;
  constexpr uint32_t ALLOC = 512, SET = 256;  // two sets of accumulators, 256 columns apart
  static_assert(BN % 32 == 0 && BN >= 64 && BN <= 256 && S::STAGE_BYTES % 1024 == 0, "halves of 16 rows, stages aligned for the swizzle");
  pdl_trigger();
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + STAGES * S::STAGE_BYTES);  // the leader's are used
  uint64_t* empty = full + STAGES;       // each CTA's own: the leader's products have read the stage
  uint64_t* acc_full = empty + STAGES;   // [2] each CTA's own: accumulators written
  uint64_t* acc_free = acc_full + 2;     // [2] the leader's: read back by the epilogue warps of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 2);
  volatile int* bail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* gates_meet = reinterpret_cast<uint64_t*>(tmem_slot + 2);  // GATED: [two warps, piece], in `meet`
  float* const meet = reinterpret_cast<float*>(ring + STAGES * S::STAGE_BYTES + 256);
  static_assert((2 * STAGES + 4) * 8 + 8 + (GATED ? 64 : 0) <= 256, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  int m_tiles = (M + BN - 1) / BN;
  const int n_tiles = (N + 2 * kWideRows - 1) / (2 * kWideRows), k_blocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(acc_full + a, 1);
      mbar_init(acc_free + a, 16);  // eight epilogue warps in each of the two CTAs
    }
    if (GATED)
      for (int i = 0; i < 8; ++i) mbar_init(gates_meet + i, 2);
    *bail = 0;
    mbar_fence_init();
  }
  if (warp == 1) {  // the same warp of both CTAs, together
    tmem_alloc_pair(tmem_slot, ALLOC);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything of mine reaches them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (EXPERTS) {
    // The tiles there are, which come first: were the empty ones dealt out too, a pair in two had an item more than its share.
    pdl_wait();  // who names the experts is a kernel ahead
    int there = 0;
    for (int t = threadIdx.x; t - static_cast<int>(threadIdx.x) < m_tiles; t += kThreads)
      there += __syncthreads_count(t < m_tiles && experts.tile_experts[t] >= 0);
    m_tiles = there;
  }
  const int items = m_tiles * n_tiles * splits;

  if (warp == 0 || warp == 10) {
    // Two loaders, every other block each: one needs some 350 cycles a block (mbar_wait_warp), more than the products of narrow tiles.
    const uint32_t mine = warp == 0 ? 0 : 1;
    const uint32_t ring_at = __shfl_sync(0xffffffffu, smem_u32(ring), 0);
    const uint32_t bars = __shfl_sync(0xffffffffu, map_to_rank(smem_u32(full), 0), 0);  // the leader's
    const bool chosen = elect_one();
    int kb0, count, w_row, w_col = 0, x_row;  // an item's first block and how many, its first rows of W and X in this CTA
    const auto take = [&](int item) {
      const int slice = item / (m_tiles * n_tiles), tile = item - slice * (m_tiles * n_tiles), column = tile / m_tiles;
      kb0 = slice * kb_per_split;
      count = min(kb_per_split, k_blocks - kb0);
      w_row = GATED ? column * kWideRows + static_cast<int>(rank) * 64 : column * 2 * kWideRows + static_cast<int>(rank) * kWideRows;
      if (EXPERTS) {
        const int e = experts.tile_experts[tile - column * m_tiles];
        w_row += e * experts.w_rows, w_col = e * experts.w_cols;
      }
      x_row = (tile - column * m_tiles) * BN + static_cast<int>(rank) * (BN / 2);
    };
    const auto ask_weights = [&](uint32_t s, int kb) {
      if (leader) mbar_expect_tx(full + s, 2 * S::STAGE_BYTES);  // both CTAs' copies
      tma_load_2d_pair(ring_at + s * S::STAGE_BYTES, &map_w, bars + s * 8, kb * BK + w_col, w_row);
      if (GATED)  // (up rows; rows of columns beyond ff are others' or zeros, and not stored)
        tma_load_2d_pair(ring_at + s * S::STAGE_BYTES + S::W_BYTES / 2, &map_w, bars + s * 8, kb * BK, w_row + experts.ff);
    };
    const auto ask_rows = [&](uint32_t s, int kb) {
      tma_load_2d_pair(ring_at + s * S::STAGE_BYTES + S::W_BYTES, &map_x, bars + s * 8, kb * BK, x_row);
    };
    if (!EXPERTS) take(pair);
    const int early = EXPERTS ? 0 : min(count, STAGES);
    for (int i = mine; i < early; i += 2)
      if (chosen) ask_weights(i, kb0 + i);
    pdl_wait();  // X is read from here on
    for (int i = mine; i < early; i += 2)
      if (chosen) ask_rows(i, kb0 + i);
    uint32_t it = early;
    int from = early;
    bool going = true;
    for (int item = pair; item < items && going; item += pairs, from = 0) {
      if (__any_sync(0xffffffffu, *bail != 0)) break;
      take(item);
      for (int i = from; i < count; ++i, ++it) {
        if ((it & 1) != mine) continue;
        const uint32_t s = it % STAGES, round = it / STAGES;
        if (round > 0 && !mbar_wait_warp(chosen, empty + s, (round - 1) & 1, status, kStuckEmpty)) {
          *bail = 1;
          going = false;
          break;
        }
        if (chosen) {
          ask_weights(s, kb0 + i);
          ask_rows(s, kb0 + i);
        }
        __syncwarp();
      }
    }
    if (lane == 0 && *bail && leader) {  // wait (bounded) for the copies already in flight before the CTA may go on to exit
      const uint32_t first = it > STAGES ? it - STAGES : 0;
      for (uint32_t i = first; i < it; ++i)
        if ((i & 1) == mine) mbar_wait(full + i % STAGES, (i / STAGES) & 1, status, kStuckDrain);
    }
    // Nobody waits for the last stages to refill them, but the leader's commits signal them here all the same: not to leave before.
    if (lane == 0)
      for (uint32_t i = it > STAGES ? it - STAGES : 0; i < it && !*bail; ++i)
        if ((i & 1) == mine && !mbar_wait(empty + i % STAGES, (i / STAGES) & 1, status, kStuckEmpty)) *bail = 1;
  } else if (warp == 1) {
    if (leader) {
      // One lane of the leader drives the tensor cores of both SMs; the warp stays together around it, as in gemm_bf16_umma_pair.cu.
      constexpr uint32_t idesc = umma_idesc(2 * kWideRows, BN);
      const uint32_t ring_at = __shfl_sync(0xffffffffu, smem_u32(ring), 0), tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      const bool chosen = elect_one();
      uint32_t it = 0, local = 0;
      bool going = true;
      for (int item = pair; item < items && going; item += pairs, ++local) {
        const uint32_t acc = local & 1, use = local >> 1;
        if (__any_sync(0xffffffffu, *bail != 0) ||
            (use > 0 && !__all_sync(0xffffffffu, lane != 0 || mbar_wait(acc_free + acc, (use - 1) & 1, status, kStuckTmemFree)))) {
          *bail = 1;
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem + acc * SET;
        const int count = min(kb_per_split, k_blocks - item / (m_tiles * n_tiles) * kb_per_split);
        for (int kb = 0; kb < count;) {
          const int ready = min(ring_ready<STAGES>(full, it, lane, status, kStuckFull), count - kb);
          if (ready == 0) {
            *bail = 1;
            going = false;
            break;
          }
          tc_fence_after();
          for (const int until = kb + ready; kb < until; ++kb, ++it) {
            const uint32_t s = it % STAGES;
            const uint32_t a = ring_at + s * S::STAGE_BYTES, b = a + S::W_BYTES;
            if (chosen) {
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; ++k)
                umma_bf16_pair(tmem_d, smem_desc(a + k * UMMA_K * 2), smem_desc(b + k * UMMA_K * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
              umma_commit_pair(empty + s, 3);                            // both CTAs' loaders may refill the stage
              if (kb + 1 == count) umma_commit_pair(acc_full + acc, 3);  // both CTAs' epilogues may read (here and last: as in gemm_bf16_umma.cu)
            }
            __syncwarp();
          }
        }
      }
    }
  } else {
    // eight warps: a quarter of the CTA's 128 columns and half of the tokens each
    const int quarter = warp & 3, side = (warp - 2) >> 2;
    pdl_wait();  // `out` may be what kernels ahead read or add to
    uint32_t local = 0, met = 0;
    for (int item = pair; item < items; item += pairs, ++local) {
      const int tile = item % (m_tiles * n_tiles), slice = item / (m_tiles * n_tiles);
      const uint32_t acc = local & 1, use = local >> 1;
      if (*bail || !mbar_wait(acc_full + acc, use & 1, status, kStuckAccumulator)) {
        *bail = 1;
        break;
      }
      tc_fence_after();
      const int n = (tile / m_tiles) * 2 * kWideRows + static_cast<int>(rank) * kWideRows + quarter * 32 + lane, m0 = (tile % m_tiles) * BN;
      void* plane = mode == 4 ? static_cast<void*>(static_cast<float*>(out) + static_cast<size_t>(slice) * M * N) : out;
#pragma unroll 1
      for (int c = side * (BN / 2); c < (side + 1) * (BN / 2) && m0 + c < M; c += S::PIECE) {
        uint32_t r[S::PIECE];
        const uint32_t from = tmem_base + acc * SET + (static_cast<uint32_t>(quarter * 32) << 16) + c;
        if constexpr (S::PIECE == 32) tmem_load32(from, r);
        else tmem_load16(from, r);
        if constexpr (GATED) {
          // Lanes 0 to 63 are gates, the others their ups. The pieces take turns at two places: who meets the other at one of them has
          // taken what was left at the other.
          const int at = (side * 2 + (quarter & 1)) * 2 + static_cast<int>(met & 1);
          const uint32_t parity = met++ >> 1 & 1;
          if (!store_gated_columns(r, quarter >= 2, meet + at * 1024, gates_meet + at, parity, m0 + c,
                                   (tile / m_tiles) * kWideRows + static_cast<int>(rank) * 64 + (quarter & 1) * 32 + lane,
                                   static_cast<__nv_bfloat16*>(out), experts, status))
            *bail = 1;
          continue;
        }
        store_columns<S::PIECE>(r, m0 + c, M, n, N, plane, mode);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(acc_free + acc), 0));
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // nobody frees tensor memory or leaves while the other may still signal it
  if (warp == 1) tmem_dealloc_pair(tmem_base, ALLOC);
}

template <int BN, bool EXPERTS = false, bool GATED = false>
int wide_config(cudaLaunchConfig_t& config, cudaLaunchAttribute* attributes, int grid, cudaStream_t stream) {
  constexpr int smem = static_cast<int>(Wide<BN, GATED>::BYTES);
  static_assert(smem <= 232448, "a CTA's shared memory");
  cudaError_t e = cudaFuncSetAttribute((gemm_bf16_wide_kernel<BN, EXPERTS, GATED>), cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  config.gridDim = dim3(grid);
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = g_lrm_pdl ? 2 : 1;
  return 0;
}

// Pairs of CTAs the device runs at once (0: clusters of two cannot be launched).
template <int BN, bool EXPERTS = false, bool GATED = false> int wide_room() {
  static int pairs = -1;
  if (pairs < 0) {
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attributes[2];
    int n = 0;
    if (wide_config<BN, EXPERTS, GATED>(config, attributes, 2, nullptr) == 0) {
      config.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_bf16_wide_kernel<BN, EXPERTS, GATED>, &config) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
    }
    pairs = n;
  }
  return pairs;
}

template <int BN>
int launch_wide(const void* X, const void* W, void* out, int M, int N, int K, int mode, int splits, int* status, cudaStream_t stream) {
  const int room = wide_room<BN>();
  if (room <= 0) return LRM_UNSUPPORTED;
  CUtensorMap map_w, map_x;
  if (!make_map_bf16(&map_w, W, N, K, kWideRows) || !make_map_bf16(&map_x, X, M, K, BN / 2)) return LRM_UNSUPPORTED;
  const int k_blocks = (K + BK - 1) / BK, per_split = (k_blocks + splits - 1) / splits;
  const long long items = static_cast<long long>((N + 2 * kWideRows - 1) / (2 * kWideRows)) * ((M + BN - 1) / BN) * splits;
  const int pairs = static_cast<int>(items < room ? items : room);
  cudaLaunchConfig_t config = {};
  cudaLaunchAttribute attributes[2];
  const int code = wide_config<BN>(config, attributes, 2 * pairs, stream);
  if (code != 0) return code;
  const cudaError_t e = cudaLaunchKernelEx(&config, gemm_bf16_wide_kernel<BN>, map_w, map_x, out, M, N, K, mode, per_split, splits, status,
                                           WideExperts{});
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

// N: columns of the product, or with GATED twice the ff columns of the gated values, filled up to 256.
template <bool GATED>
int launch_wide_experts(const void* X, const void* W, void* out, int M, int N, int K, long long w_height, long long w_width, int* status,
                        const WideExperts& experts, cudaStream_t stream) {
  const int room = wide_room<kSortedRows, true, GATED>();
  if (room <= 0) return LRM_UNSUPPORTED;
  CUtensorMap map_w, map_x;
  if (!make_map_bf16(&map_w, W, w_height, w_width, GATED ? 64 : kWideRows) || !make_map_bf16(&map_x, X, M, K, kSortedRows / 2)) return LRM_UNSUPPORTED;
  const long long items = static_cast<long long>((N + 2 * kWideRows - 1) / (2 * kWideRows)) * (M / kSortedRows);
  const int pairs = static_cast<int>(items < room ? items : room);
  cudaLaunchConfig_t config = {};
  cudaLaunchAttribute attributes[2];
  const int code = wide_config<kSortedRows, true, GATED>(config, attributes, 2 * pairs, stream);
  if (code != 0) return code;
  const cudaError_t e = cudaLaunchKernelEx(&config, gemm_bf16_wide_kernel<kSortedRows, true, GATED>, map_w, map_x, out, M, N, K, 1, K / BK, 1, status,
                                           experts);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

}  // namespace

// K slices a product in `wanted` slices really has: none is empty.
LRM_API int lrm_gemm_bf16_wide_slices(int K, int wanted) {
  const int k_blocks = (K + BK - 1) / BK, per_split = (k_blocks + wanted - 1) / wanted;
  return (k_blocks + per_split - 1) / per_split;
}

// Y = X . W^T with epilogue `mode` (0-4) in tiles of 256 weight rows and `rows` activation rows (64 to 256, a multiple of 32).
// `splits` (mode 4): as lrm_gemm_bf16_wide_slices says; out is [splits, M, N]. `status`: one int in device memory, 0 before the launch.
LRM_API int lrm_gemm_bf16_wide(const void* X, const void* W, void* out, int M, int N, int K, int mode, int rows, int splits, int* status,
                               cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K < 8 || K % 8 != 0 || N % 2 != 0 || encode_tiled() == nullptr) return LRM_UNSUPPORTED;
  if (mode < 0 || mode > 4 || (mode == 3 && N % 16 != 0) || splits < 1 || (splits > 1 && mode != 4) || status == nullptr ||
      splits != lrm_gemm_bf16_wide_slices(K, splits))
    return LRM_BAD_ARGUMENT;
  if (reinterpret_cast<uintptr_t>(X) % 16 || reinterpret_cast<uintptr_t>(W) % 16 || reinterpret_cast<uintptr_t>(out) % 4) return LRM_UNSUPPORTED;
#define LRM_CASE(BN) \
  if (rows == BN) return launch_wide<BN>(X, W, out, M, N, K, mode, splits, status, stream);
  LRM_CASE(64)
  LRM_CASE(96)
  LRM_CASE(128)
  LRM_CASE(160)
  LRM_CASE(192)
  LRM_CASE(224)
  LRM_CASE(256)
#undef LRM_CASE
  return LRM_UNSUPPORTED;
}

// Sorted experts, as lrm_gemm_bf16_umma_experts and lrm_gemm_bf16_umma_experts_gated take them.
LRM_API int lrm_gemm_bf16_wide_experts(const void* X, const void* W, void* out, int M, int N, int K, long long w_height, long long w_width,
                                       int w_rows, int w_cols, const int* tile_experts, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % BK || M % kSortedRows || w_cols % 8 || w_width % 8 || w_height >= (1ll << 31) || w_width >= (1ll << 31) || encode_tiled() == nullptr)
    return LRM_UNSUPPORTED;
  if (tile_experts == nullptr || status == nullptr || w_rows < 0 || w_cols < 0) return LRM_BAD_ARGUMENT;
  if (reinterpret_cast<uintptr_t>(X) % 16 || reinterpret_cast<uintptr_t>(W) % 16 || reinterpret_cast<uintptr_t>(out) % 4) return LRM_UNSUPPORTED;
  return launch_wide_experts<false>(X, W, out, M, N, K, w_height, w_width, status,
                                    WideExperts{tile_experts, w_rows, w_cols, nullptr, nullptr, 0, 0, 0.f, 0.f}, stream);
}

LRM_API int lrm_gemm_bf16_wide_experts_gated(const void* X, const void* W, void* out, int M, int ff, int K, long long w_height,
                                             const int* tile_experts, const int* rows, const float* weights, float limit, float alpha,
                                             int act, int* status, cudaStream_t stream) {
  if (M <= 0 || ff <= 0) return 0;
  if (K <= 0 || K % BK || M % kSortedRows || ff % 64 || w_height >= (1ll << 31) || encode_tiled() == nullptr) return LRM_UNSUPPORTED;
  if (tile_experts == nullptr || rows == nullptr || weights == nullptr || status == nullptr || (act != 0 && act != 1)) return LRM_BAD_ARGUMENT;
  if (reinterpret_cast<uintptr_t>(X) % 16 || reinterpret_cast<uintptr_t>(W) % 16 || reinterpret_cast<uintptr_t>(out) % 4) return LRM_UNSUPPORTED;
  return launch_wide_experts<true>(X, W, out, M, (ff + 127) / 128 * 256, K, w_height, K, status,
                                   WideExperts{tile_experts, 2 * ff, 0, rows, weights, ff, act, limit, alpha}, stream);
}
