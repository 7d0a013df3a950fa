// float32 matrix product on the 5th-generation tensor cores: C[M,N] = X[M,K] . W[N,K]^T, for the larger matrices
// (gemm_dispatch.f32_takes_umma). Every float32 number is cut into three bfloat16 parts, each rounded, which hold all of it, and eight of
// the nine products of parts are added: the one left out is below 2^-34 of a product.
//
// The tensor core truncates where it adds (measured: to 2^-23 of the sum), with a bias towards zero that grows with the terms: 1.2e-7
// after 128, 2e-6 after 2,048. So the large products (of the first parts, 16 bits each) are added over 64 of K only, from zero, and the
// sums over K are float32 additions on the CUDA cores. The seven small ones have an accumulator of their own, over all of K, whose
// truncation is 2^-8 of that, and are added once, at the end. So a single product is rounded as a float32 FMA rounds it, and sums of
// any number of terms are no further off than with FMAs in ascending order. Distance from 64 bits, relative, normal numbers, rows with
// n of them (FMAs): 1 2.5e-8 (2.5e-8), 2 2.5e-8 (3.1e-8), 16 3.3e-8 (7.3e-8), 2,048 9.9e-8 (8.1e-7), 8,192 1.4e-7 (1.6e-6). (Six products,
// the first part cut off, all in one accumulator: 5.5e-8, 6.2e-8, 7.9e-8, 1.1e-7, 1.4e-7.)
//
// A tile of 128 weight rows is the A operand; the rows of X, in equal tiles of up to 128, are its columns. One thread brings the
// weights' blocks of 64 of K to shared memory by TMA, as float32. Eight or sixteen warps cut them, a row a lane, and put the parts into tensor
// memory (A from there leaves shared memory to the other operand). X's parts lie in shared memory in the
// swizzled layout of the instruction: up to 32 rows are cut there by four more warps; more rows, which many tiles share, have been cut by
// a launch ahead and come by TMA. One warp issues 32 products a block, the four large ones first, and four or twelve warps add those to
// their registers under the small ones, a thread per weight row and up to 48 rows of X. A matrix with few tiles is cut along K into
// slices of a cluster's CTAs, whose large and small sums meet in distributed shared memory, in order.
//
// An element's blocks and slices follow from N and K alone, so its value does not depend on M, on the tile it falls in, or on what
// else is in the batch.
//
// Both operands count 2^16 fold, so that parts of the smallest numbers are not lost, and the result is brought back. A row with a
// number of 2^32 or more or an infinity in a slice of K is marked for that slice, and its elements' sums over the slice are added once
// more with float32 FMAs.
//
// Bound, with many rows, by the tensor pipe: a block's 32 products take 72 cycles each with 112 rows of X a tile (56 by the
// instruction's size), and 6 us of start-up and drain a CTA beside that; with few rows by the chain of a block, 0.85 us (5.1 TB/s of weights).
// us, in brackets gemm_f32.cu's kernels: 1 row, 3072 x 2048 12.1 (24.8), 16384 x 2048 28 (36), 2048 x 8192 28 (94), 128256 x 2048 196
// (175; 4 rows 197 and 240); 32 rows 14 (66), 33 (147), 32 (221); 333 rows 60 (128), 139 (597), 99 (499); 512 rows 68, 202, 113. (With six
// products 333 rows 46, 115, 77.) Tried, 16384 x 2048, 333 rows: operands through registers (loads under way share scoreboards, so a
// use waits for the newest) 189 with six products; the large products behind the small ones, with a second wait of the issuer 169
// against 152; a look at the next barrier ahead of the last eight products 153, of the last sixteen 173; three stages of parts 154; sixteen
// warps cutting 185.
//
// Every wait is bounded (see umma.cuh).
#include "umma.cuh"

namespace {

constexpr int kRows = 128, BK = 64, kMaxSlices = 4;
constexpr int kLoader = 0, kIssuer = 1, kInputLoader = 2;  // (the fourth warp has no work)
constexpr uint32_t kHeld = BK / 2;  // columns of tensor memory of a part of the weights

// MAXC: rows of X in a tile at most. RAW: blocks of float32 in shared memory; two are held as parts. AHEAD: X has been cut before.
template <int MAXC, int RAW, bool AHEAD, int WW>
struct Cut {
  static constexpr int WEIGHT_WARPS = WW, INPUT_WARPS = AHEAD ? 0 : 4, ADDERS = MAXC > 32 ? 12 : 4, THREADS = (4 + WW + INPUT_WARPS + ADDERS) * 32;
  static constexpr uint32_t W_RAW = kRows * BK * 4, X_RAW = AHEAD ? 0 : MAXC * BK * 4, RAW_STAGE = W_RAW + X_RAW;
  static constexpr uint32_t PART = MAXC * BK * 2, STAGE = 3 * PART;
  static constexpr uint32_t AT_PARTS = RAW * RAW_STAGE, AT_BARRIERS = AT_PARTS + 2 * STAGE;
  static constexpr uint32_t WEIGHTS_AT = 2 * MAXC, COLUMNS = MAXC == 32 ? 256 : 512;  // of tensor memory: two accumulators, weights
  static constexpr size_t BYTES = 1024 + AT_BARRIERS + 256 + (kRows + MAXC) * sizeof(int);
  static constexpr int CHUNKS = (MAXC / 16 + ADDERS / 4 - 1) / (ADDERS / 4);  // pieces of 16 rows of X that an adding thread has
  static_assert(WEIGHTS_AT + 2 * 3 * kHeld <= COLUMNS && 2 * MAXC * kRows * 4 <= AT_PARTS && BYTES <= 227 * 1024, "room");
};

enum : int { kStuckEmpty = 61, kStuckFull = 62, kStuckAccumulator = 63, kStuckRaw = 64, kStuckDrain = 65, kStuckRawEmpty = 66, kStuckSmall = 67 };

// Two numbers, 2^16 fold, as three pairs of bfloat16; `most` collects the largest.
__device__ __forceinline__ void cut2(float x, float y, uint32_t& high, uint32_t& middle, uint32_t& low, float& most) {
  x *= 65536.f, y *= 65536.f;
  most = fmaxf(most, fmaxf(fabsf(x), fabsf(y)));  // (a NaN needs no mark: it is one in every product)
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(high) : "f"(y), "f"(x));
  const float ra = x - __uint_as_float(high << 16), rb = y - __uint_as_float(high & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(middle) : "f"(rb), "f"(ra));
  const float sa = ra - __uint_as_float(middle << 16), sb = rb - __uint_as_float(middle & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(low) : "f"(sb), "f"(sa));
}
constexpr float kTooLarge = 281474976710656.f;  // 2^32 2^16: products of smaller ones are below 2^96 and no sum over K leaves the range

// A bounded wait that also ends when another role of the CTA has given up.
__device__ __forceinline__ bool wait_or_bail(uint64_t* bar, uint32_t parity, int* status, int where, volatile int* bail) {
  for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 1023) == 1023 && *bail) return false;
  }
  atomicCAS(status, 0, where);
  *bail = 1;
  return false;
}

__device__ __forceinline__ uint32_t rank_in_cluster() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 load_from_rank(uint32_t local, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

// Numbers begin .. end - 1 of two rows, one after another.
__device__ __noinline__ float add_fma(const float* x, const float* w, int begin, int end) {
  float sum = 0.f;
#pragma unroll 4
  for (int k = begin; k < end; k += 4) {
    const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
    sum = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
  }
  return sum;
}

// X [rows, K] cut ahead: parts [3][rows][K], and for which slices of `of_slice` numbers a row is marked, a bit each. A CTA per row.
__global__ __launch_bounds__(256) void cut_rows_kernel(const float* X, uint2* __restrict__ parts, int* __restrict__ marks, int rows, int K,
                                                       int of_slice) {
  __shared__ int marked;
  pdl_trigger();
  if (threadIdx.x == 0) marked = 0;
  __syncthreads();
  pdl_wait();
  const int row = blockIdx.x;
  const float4* from = reinterpret_cast<const float4*>(X + static_cast<size_t>(row) * K);
  const size_t plane = static_cast<size_t>(rows) * (K / 4);
#pragma unroll 4
  for (int i = threadIdx.x; i < K / 4; i += 256) {
    const float4 x = from[i];
    float most = 0.f;
    uint2 part[3];
    cut2(x.x, x.y, part[0].x, part[1].x, part[2].x, most);
    cut2(x.z, x.w, part[0].y, part[1].y, part[2].y, most);
#pragma unroll
    for (int p = 0; p < 3; ++p) parts[p * plane + static_cast<size_t>(row) * (K / 4) + i] = part[p];
    if (most >= kTooLarge) atomicOr(&marked, 1 << (4 * i / of_slice));
  }
  __syncthreads();
  if (threadIdx.x == 0) marks[row] = marked;
}

// Item (n tile, m tile, slice), the slice fastest; a cluster is the slices of a tile. `columns`: rows of X in a tile, a multiple of 16.
// map_x: X as float32, or (AHEAD) its parts, one above the other, x_rows rows each, with `marks`.
template <int MAXC, int RAW, bool AHEAD, int WW>
__global__ __launch_bounds__(Cut<MAXC, RAW, AHEAD, WW>::THREADS, 1) void gemm_f32_umma_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* X, const float* W, const int* marks,
    float* __restrict__ C, int M, int N, int K, int mode, int group_cols, int group_rows, int x_rows, int columns, int m_tiles, int slices,
    int* __restrict__ status) {
  using T = Cut<MAXC, RAW, AHEAD, WW>;
  constexpr int kThreads = T::THREADS, kWeightWarps = WW, kInputWarps = T::INPUT_WARPS, kAdders = T::ADDERS;
  pdl_trigger();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(ring + T::AT_BARRIERS);
  uint64_t* raw_empty = raw_full + RAW;
  // A block's parts are there and the block before's large products have been added: one barrier, since each wait of the issuer
  // leaves the tensor pipe idle for some 500 cycles.
  uint64_t* full = raw_empty + RAW;      // [2]
  uint64_t* empty = full + 2;            // [2] a block's products are done with its parts
  uint64_t* acc_full = empty + 2;        // its large products are in their accumulator
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* bail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* any_marked = reinterpret_cast<int*>(tmem_slot + 2);
  int* marked = reinterpret_cast<int*>(ring + T::AT_BARRIERS + 256);  // [128 rows of W | rows of X]
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int slice = blockIdx.x % slices, tile = blockIdx.x / slices;
  const int m0 = tile % m_tiles * columns, n0 = tile / m_tiles * kRows;
  const int blocks_all = (K + BK - 1) / BK, per = (blocks_all + slices - 1) / slices;
  const int first = min(slice * per, blocks_all), blocks = min(per, blocks_all - first);
  const int x_row0 = (group_cols > 0 ? n0 / group_cols * group_rows : 0) + m0;

  if (tid == 0) {
    for (int s = 0; s < RAW; ++s) mbar_init(raw_full + s, 1), mbar_init(raw_empty + s, kWeightWarps + kInputWarps);
    for (int s = 0; s < 2; ++s) {
      mbar_init(full + s, kWeightWarps + (AHEAD ? 1 : kInputWarps) + kAdders), mbar_init(empty + s, 1);
    }
    mbar_init(acc_full, 1);
    *bail = 0;
    *any_marked = 0;
    mbar_fence_init();
  }
  for (int i = tid; i < kRows + MAXC; i += kThreads) marked[i] = 0;
  if (warp == kIssuer) {
    tmem_alloc(tmem_slot, T::COLUMNS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();
  if (AHEAD && warp == 3)
    for (int i = lane; i < columns; i += 32)
      if (m0 + i < M && (marks[x_row0 + i] >> slice & 1)) marked[kRows + i] = *any_marked = 1;
  auto all_meet = []() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); };

  if (warp == kLoader) {
    if (lane == 0) {
      const uint32_t bytes = T::W_RAW + (AHEAD ? 0 : columns * BK * 4);
      int block = 0;
      for (; block < blocks; ++block) {
        const int s = block % RAW;
        if (block >= RAW && !wait_or_bail(raw_empty + s, (block / RAW - 1) & 1, status, kStuckRawEmpty, bail)) break;
        unsigned char* stage = ring + s * T::RAW_STAGE;
        const int k = (first + block) * BK;
        mbar_expect_tx(raw_full + s, bytes);
#pragma unroll
        for (int half = 0; half < 2; ++half) {  // 32 of K each: rows of 128 bytes
          tma_load_2d(stage + half * (T::W_RAW / 2), &map_w, raw_full + s, k + 32 * half, n0);
          if (!AHEAD) tma_load_2d(stage + T::W_RAW + half * (T::X_RAW / 2), &map_x, raw_full + s, k + 32 * half, x_row0);
        }
      }
      if (*bail)  // wait (bounded) for the copies already in flight before the CTA may exit
        for (int i = max(0, block - RAW); i < block; ++i) mbar_wait(raw_full + i % RAW, (i / RAW) & 1, status, kStuckDrain);
    }
    __syncwarp();
    all_meet();
  } else if (AHEAD && warp == kInputLoader) {
    if (lane == 0) {
      int block = 0;
      for (; block < blocks; ++block) {
        const int s = block & 1;
        if (block >= 2 && !wait_or_bail(empty + s, ((block >> 1) - 1) & 1, status, kStuckEmpty, bail)) break;
        mbar_expect_tx(full + s, 3 * columns * BK * 2);
#pragma unroll
        for (int p = 0; p < 3; ++p)
          tma_load_2d(ring + T::AT_PARTS + s * T::STAGE + p * T::PART, &map_x, full + s, (first + block) * BK, p * x_rows + x_row0);
      }
      if (*bail)
        for (int i = max(0, block - 2); i < block; ++i) mbar_wait(full + (i & 1), (i >> 1) & 1, status, kStuckDrain);
    }
    __syncwarp();
    all_meet();
  } else if (warp == kIssuer) {
    // The warp stays together around its elected lane, on numbers the same in all lanes, so that descriptors are made in uniform registers.
    const uint32_t idesc = umma_idesc(kRows, __shfl_sync(0xffffffffu, columns, 0)), parts_at = __shfl_sync(0xffffffffu, smem_u32(ring), 0) + T::AT_PARTS;
    const bool leader = elect_one();
    bool ready = false;  // the next block, as seen while this one's products were under way
    for (int block = 0; block < blocks; ++block) {
      const int s = block & 1;
      if (!ready && !__all_sync(0xffffffffu, wait_or_bail(full + s, (block >> 1) & 1, status, kStuckFull, bail))) break;
      tc_fence_after();
      const uint32_t a = tmem + T::WEIGHTS_AT + s * 3 * kHeld, b = parts_at + s * T::STAGE;
      constexpr int kSmall = 7, of_w[kSmall] = {1, 2, 2, 0, 1, 1, 0}, of_x[kSmall] = {2, 1, 0, 2, 1, 0, 1};
      if (leader) {  // the large products first: they are added under the small ones
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16_a_tmem(tmem, a + k * 8, smem_desc(b + k * 32), idesc, k > 0 ? 1u : 0u);
        umma_commit(acc_full);
#pragma unroll
        for (int p = 0; p < kSmall; ++p)
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16_a_tmem(tmem + MAXC, a + of_w[p] * kHeld + k * 8, smem_desc(b + of_x[p] * T::PART + k * 32), idesc,
                             block > 0 || p > 0 || k > 0 ? 1u : 0u);
        umma_commit(empty + s);
      }
      __syncwarp();
      ready = block + 1 < blocks && __all_sync(0xffffffffu, mbar_try_wait(full + (s ^ 1), ((block + 1) >> 1) & 1));
    }
    all_meet();
    tmem_dealloc(tmem, T::COLUMNS);
  } else if (warp < 4) {
    all_meet();
  } else if (warp < 4 + kWeightWarps) {
    constexpr int SHARE = BK / (kWeightWarps / 4);  // numbers of a row and block that a thread has: 32 or 16
    const int quarter = warp & 3, share = (warp - 4) >> 2, place = quarter * 32 + lane;  // lanes of tensor memory, which of the shares
    const uint32_t to = tmem + T::WEIGHTS_AT + (static_cast<uint32_t>(quarter * 32) << 16) + share * (SHARE / 2);
    float most = 0.f;
    for (int block = 0; block < blocks; ++block) {
      const int r = block % RAW, s = block & 1;
      if (!wait_or_bail(raw_full + r, (block / RAW) & 1, status, kStuckRaw, bail) ||
          (block >= 2 && !wait_or_bail(empty + s, ((block >> 1) - 1) & 1, status, kStuckEmpty, bail)))
        break;
      tc_fence_after();
      const unsigned char* row = ring + r * T::RAW_STAGE + share * SHARE / 32 * (T::W_RAW / 2) + place * 128;
#pragma unroll
      for (int i = 0; i < SHARE / 16; ++i) {
        float4 x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = *reinterpret_cast<const float4*>(row + (((share * SHARE % 32 / 4 + 4 * i + e) ^ (place & 7)) << 4));
        uint32_t part[3][8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          cut2(x[e].x, x[e].y, part[0][2 * e], part[1][2 * e], part[2][2 * e], most);
          cut2(x[e].z, x[e].w, part[0][2 * e + 1], part[1][2 * e + 1], part[2][2 * e + 1], most);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_store8(to + (s * 3 + p) * kHeld + i * 8, part[p]);
      }
      tmem_store_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_empty + r), mbar_arrive(full + s);
    }
    if (most >= kTooLarge) marked[place] = *any_marked = 1;
    all_meet();
  } else if (!AHEAD && warp < 4 + kWeightWarps + kInputWarps) {
    constexpr int STEP = 8;  // rows that four warps have at a time
    const int row = (tid - (4 + kWeightWarps) * 32) >> 4, piece = tid & 15;  // rows row + STEP i, four numbers of K
    const uint32_t from = T::W_RAW + (piece >> 3) * (T::X_RAW / 2) + row * 128 + (((piece & 7) ^ (row & 7)) << 4);
    const uint32_t to = T::AT_PARTS + row * 128 + (((piece >> 1) ^ (row & 7)) << 4) + (piece & 1) * 8;  // (row + STEP i) & 7 is row & 7
    for (int block = 0; block < blocks; ++block) {
      const int r = block % RAW, s = block & 1;
      if (!wait_or_bail(raw_full + r, (block / RAW) & 1, status, kStuckRaw, bail) ||
          (block >= 2 && !wait_or_bail(empty + s, ((block >> 1) - 1) & 1, status, kStuckEmpty, bail)))
        break;
      const unsigned char* raw = ring + r * T::RAW_STAGE + from;
      unsigned char* stage = ring + s * T::STAGE + to;
#pragma unroll 1
      for (int i0 = 0; i0 * STEP < columns; i0 += 2) {  // two rows at a time: `columns` is a multiple of 16
        float4 x[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) x[i] = *reinterpret_cast<const float4*>(raw + (i0 + i) * STEP * 128);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint2 part[3];
          float most = 0.f;
          cut2(x[i].x, x[i].y, part[0].x, part[1].x, part[2].x, most);
          cut2(x[i].z, x[i].w, part[0].y, part[1].y, part[2].y, most);
          if (most >= kTooLarge) marked[kRows + row + STEP * (i0 + i)] = *any_marked = 1;
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(stage + p * T::PART + (i0 + i) * STEP * 128) = part[p];
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(raw_empty + r), mbar_arrive(full + s);
    }
    all_meet();
  } else {
    constexpr int CHUNKS = T::CHUNKS;
    float acc[CHUNKS][16];
#pragma unroll
    for (int i = 0; i < CHUNKS * 16; ++i) acc[i >> 4][i & 15] = 0.f;
    const int quarter = warp & 3, side = (warp - 4 - kWeightWarps - kInputWarps) >> 2;  // lanes of tensor memory, columns
    const int c0 = side * CHUNKS * 16, place = quarter * 32 + lane, n = n0 + place;
    constexpr float kBack = 2.3283064365386963e-10f;  // 2^-32
    float* sums = reinterpret_cast<float*>(ring);       // slices: [columns][128] of the large products, then of the small ones
    const uint32_t at = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c0;
    if (lane == 0) mbar_arrive(full);  // the accumulator is free
    for (int block = 0; block < blocks; ++block) {
      if (!wait_or_bail(acc_full, block & 1, status, kStuckAccumulator, bail)) break;
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        if (c0 + i * 16 >= columns) break;
        uint32_t r[16];
        tmem_load16(at + i * 16, r);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[i][j] += __uint_as_float(r[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(full + ((block + 1) & 1));
    }
    if (wait_or_bail(empty + ((blocks - 1) & 1), ((blocks - 1) >> 1) & 1, status, kStuckSmall, bail)) {  // (every block has been read)
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        if (c0 + i * 16 >= columns) break;
        uint32_t r[16];
        tmem_load16(at + MAXC + i * 16, r);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (slices == 1) acc[i][j] += __uint_as_float(r[j]);
          else sums[(MAXC + c0 + i * 16 + j) * kRows + place] = __uint_as_float(r[j]) * kBack;
        }
      }
      tc_fence_before();
    }
    all_meet();  // all marks are made
#pragma unroll
    for (int i = 0; i < CHUNKS * 16; ++i) acc[i >> 4][i & 15] *= kBack;
    if (*any_marked && n < N) {
      const int k_end = min(K, (first + blocks) * BK);
#pragma unroll
      for (int i = 0; i < CHUNKS * 16; ++i) {
        const int c = c0 + i;
        if (c < columns && m0 + c < M && (marked[place] || marked[kRows + c])) {
          acc[i >> 4][i & 15] = add_fma(X + static_cast<size_t>(x_row0 + c) * K, W + static_cast<size_t>(n) * K, first * BK, k_end);
          if (slices > 1) sums[(MAXC + c) * kRows + place] = 0.f;
        }
      }
    }
    if (slices == 1) {
      if (n < N) {
#pragma unroll
        for (int i = 0; i < CHUNKS * 16; ++i) {
          const int c = c0 + i, m = m0 + c;
          if (c < columns && m < M) {
            float* to = C + static_cast<size_t>(m) * N + n;
            *to = mode == 1 ? *to + acc[i >> 4][i & 15] : acc[i >> 4][i & 15];
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < CHUNKS * 16; ++i)
        if (c0 + i < columns) sums[(c0 + i) * kRows + place] = acc[i >> 4][i & 15];
    }
  }
  if (slices == 1) return;
  const float* sums = reinterpret_cast<const float*>(ring);
  cluster_meet();
  const uint32_t rank = rank_in_cluster();
  const int rows = min(columns, M - m0);
  const bool wide = N % 4 == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0;
  for (int i = tid; i < (rows - static_cast<int>(rank) + slices - 1) / slices * (kRows / 4); i += kThreads) {  // rows rank, rank + slices, ...
    const int c = static_cast<int>(rank) + i / (kRows / 4) * slices, col = i % (kRows / 4) * 4;
    float4 v = load_from_rank(smem_u32(sums + c * kRows + col), 0), small = load_from_rank(smem_u32(sums + (MAXC + c) * kRows + col), 0);
    for (int s = 1; s < slices; ++s) {
      const float4 more = load_from_rank(smem_u32(sums + c * kRows + col), s), less = load_from_rank(smem_u32(sums + (MAXC + c) * kRows + col), s);
      v.x += more.x, v.y += more.y, v.z += more.z, v.w += more.w;
      small.x += less.x, small.y += less.y, small.z += less.z, small.w += less.w;
    }
    v.x += small.x, v.y += small.y, v.z += small.z, v.w += small.w;
    float* to = C + static_cast<size_t>(m0 + c) * N + n0 + col;
    const float out[4] = {v.x, v.y, v.z, v.w};
    if (wide && n0 + col < N) {
      if (mode == 1) {
        const float4 old = *reinterpret_cast<const float4*>(to);
        v.x += old.x, v.y += old.y, v.z += old.z, v.w += old.w;
      }
      *reinterpret_cast<float4*>(to) = v;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + col + e < N) to[e] = mode == 1 ? to[e] + out[e] : out[e];
    }
  }
  cluster_meet();  // the others have read this CTA's sums
}

// Slices of K, from N and K alone: CTAs for two thirds of the SMs where one row tile would leave most of them idle, no slice shorter than 512.
int slices_of(int N, int K) {
  int s = 1;
  while (s < kMaxSlices && s * ((N + kRows - 1) / kRows) < 96 && K / (2 * s) >= 512) s *= 2;
  return s;
}

// Row-major [rows, width] float32 matrix, boxes of `box_rows` x 32 numbers, 128-byte swizzle, zeros out of range.
bool make_map_f32(CUtensorMap* map, const void* base, long long rows, long long width, int box_rows) {
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(width), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(width) * 4};
  const cuuint32_t box[2] = {32, static_cast<cuuint32_t>(box_rows)}, elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MAXC, int RAW, bool AHEAD, int WW>
int launch(const float* X, const float* W, float* C, int M, int N, int K, int mode, int group_cols, int group_rows, void* parts, int* status,
           cudaStream_t stream) {
  using T = Cut<MAXC, RAW, AHEAD, WW>;
  const int m_tiles = (M + MAXC - 1) / MAXC, columns = ((M + m_tiles - 1) / m_tiles + 15) / 16 * 16, slices = slices_of(N, K);
  const long long items = static_cast<long long>((N + kRows - 1) / kRows) * m_tiles * slices;
  const long long x_rows = static_cast<long long>(group_cols > 0 ? (N + group_cols - 1) / group_cols - 1 : 0) * group_rows + M;
  if (items > 0x7fffffffll || x_rows > 0x20000000ll) return LRM_UNSUPPORTED;
  int* marks = reinterpret_cast<int*>(static_cast<char*>(parts) + 6 * x_rows * K);
  CUtensorMap map_w, map_x;
  if (!make_map_f32(&map_w, W, N, K, kRows)) return LRM_UNSUPPORTED;
  if (!(AHEAD ? make_map_bf16(&map_x, parts, 3 * x_rows, K, columns) : make_map_f32(&map_x, X, x_rows, K, columns))) return LRM_UNSUPPORTED;
  auto kernel = gemm_f32_umma_kernel<MAXC, RAW, AHEAD, WW>;
  constexpr int bytes = static_cast<int>(T::BYTES);
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (AHEAD)
    LRM_LAUNCH(cut_rows_kernel, dim3(static_cast<unsigned>(x_rows)), 256, 0, stream, X, static_cast<uint2*>(parts), marks,
               static_cast<int>(x_rows), K, ((K + BK - 1) / BK + slices - 1) / slices * BK);
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(items));
  config.blockDim = dim3(T::THREADS);
  config.dynamicSmemBytes = bytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = slices, attributes[0].val.clusterDim.y = attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = g_lrm_pdl ? 2 : 1;
  const cudaError_t launched = cudaLaunchKernelEx(&config, kernel, map_w, map_x, X, W, static_cast<const int*>(marks), C, M, N, K, mode,
                                                  group_cols, group_rows, static_cast<int>(x_rows), columns, m_tiles, slices, status);
  return launched == cudaSuccess ? 0 : static_cast<int>(launched);
}

}  // namespace

// Bytes of `parts` for `rows` rows of X, all inputs together: scratch, 16-byte aligned.
LRM_API long long lrm_gemm_f32_umma_scratch(int rows_of_one, int rows, int K) {
  return rows_of_one <= 32 ? 0 : 6ll * rows * K + 4ll * rows;
}

// group_cols > 0 (a multiple of 128): several inputs `group_rows` rows apart in X. X and W start on 16 bytes, K a multiple of 8.
// mode 0: C = product, 1: C += product. `status`: one int in device memory, 0 before the launch.
LRM_API int lrm_gemm_f32_umma(const float* X, const float* W, float* C, int M, int N, int K, int mode, int group_cols, int group_rows,
                              void* parts, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (mode != 0 && mode != 1) || status == nullptr) return LRM_BAD_ARGUMENT;
  if (group_cols < 0 || group_cols % kRows || (group_cols > 0 && group_rows < M)) return LRM_BAD_ARGUMENT;
  if (K % 8 || reinterpret_cast<uintptr_t>(X) % 16 || reinterpret_cast<uintptr_t>(W) % 16) return LRM_UNSUPPORTED;
  if (M <= 32) return launch<32, 4, false, 16>(X, W, C, M, N, K, mode, group_cols, group_rows, nullptr, status, stream);
  if (parts == nullptr || reinterpret_cast<uintptr_t>(parts) % 16) return LRM_BAD_ARGUMENT;
  return launch<128, 4, true, 8>(X, W, C, M, N, K, mode, group_cols, group_rows, parts, status, stream);
}
