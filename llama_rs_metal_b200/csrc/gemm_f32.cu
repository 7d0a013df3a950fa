// True 32-bit matrix product on the CUDA cores: C[M,N] = X[M,K] . W[N,K]^T, for the smaller matrices and for operands off 16 bytes
// (gemm_f32_umma.cu has the others).
// W is a Linear weight as stored ([out][in]); every product and sum is an
// IEEE float32 fused multiply-add, with no tensor-core or reduced-precision
// mode anywhere. Each output element is accumulated over k = 0..K-1 in
// ascending order by one thread, so its value does not depend on M, on the
// tile it falls in, or on what else is in the batch.
// (Reference role: the F32 simdgroup GEMM/GEMV family,
// crates/metal-backend/src/shaders/matrix.metal:10-37,236-282.)
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16;
constexpr int kFewRows = 32;

// Up to kFewRows rows whose operands do not start on 16-byte boundaries.
// mode 0: C = acc;  mode 1: C += acc (the residual add folded into the epilogue)
__global__ __launch_bounds__(256) void gemm_f32_kernel(const float* __restrict__ X,
                                                       const float* __restrict__ W,
                                                       float* __restrict__ C, int M, int N, int K,
                                                       int mode, int group_cols, int group_rows) {
  __shared__ float Xs[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // grouped inputs: columns [i group_cols, (i + 1) group_cols) multiply the input that begins i group_rows
  // rows into X
  if (group_cols > 0) X += static_cast<size_t>(n0 / group_cols) * group_rows * K;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256, r = idx >> 4, c = idx & 15;
      const int gk = k0 + c;
      const int gm = m0 + r, gn = n0 + r;
      Xs[c][r] = (gm < M && gk < K) ? X[static_cast<size_t>(gm) * K + gk] : 0.f;
      Ws[c][r] = (gn < N && gk < K) ? W[static_cast<size_t>(gn) * K + gk] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = Xs[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      float* dst = C + static_cast<size_t>(gm) * N + gn;
      *dst = mode == 1 ? *dst + acc[i][j] : acc[i][j];
    }
  }
}

// The tiled kernel for prompts: BM x BN outputs per CTA, 8 x TN per thread (a warp covers 32 x 8 TN), K in
// blocks of 16 through two shared-memory buffers laid out [k][row]. Blocks are on their way to registers two
// ahead of the multiplications, the fragments of the next k one ahead. Two neighbouring columns are one
// fma.rn.f32x2, two IEEE float32 FMAs in one instruction; an element still adds its products over k in
// ascending order, so all tile sizes give the same bits. A tile of 128 x 64 keeps one warp on each of an SM's
// schedulers, which is what bounds it (an issue every 2.9 cycles, 2 of them the FMAs themselves). 384 rows, us, 64 x 64 tiles of 4 x 4 per thread and scalar loads before: 3072 x 2048 126
// (252), 16384 x 2048 607 (1248), 2048 x 8192 488 (1045); blocks one ahead only: 139, 637, 673.
constexpr int TK = 16, PAD = 4;

__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}

// VEC: rows of X, W and C start on 16-byte boundaries (K and N multiples of 4).
template <int BM_, int BN_, int TN, bool VEC>
__global__ __launch_bounds__(BM_ * BN_ / (8 * TN), BM_ == 128 ? 2 : 4) void gemm_f32_tiled_kernel(
    const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int mode,
    int group_cols, int group_rows) {
  constexpr int THREADS = BM_ * BN_ / (8 * TN), XL = BM_ * TK / 4 / THREADS, WL = BN_ * TK / 4 / THREADS;
  __shared__ __align__(16) float Xs[2][TK][BM_ + PAD];
  __shared__ __align__(16) float Ws[2][TK][BN_ + PAD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int WARPS_N = BN_ / (8 * TN), HALVES = TN / 4;  // warps side by side, pieces of 4 columns a thread has
  const int m_in = warp / WARPS_N * 32 + (lane >> 3) * 4, n_in = warp % WARPS_N * 8 * TN + (lane & 7) * 4;
  const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN_;
  if (group_cols > 0) X += static_cast<size_t>(n0 / group_cols) * group_rows * K;
  unsigned long long acc[8][2 * HALVES];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2 * HALVES; ++j) acc[i][j] = 0ull;

  float4 x0[XL], w0[WL], x1[XL], w1[WL];  // two blocks under way
  auto piece = [&](const float* __restrict__ base, int row, int rows, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= rows) return v;
    const float* p = base + static_cast<size_t>(row) * K + k;
    if (VEC) {
      if (k < K) v = *reinterpret_cast<const float4*>(p);
    } else {
      if (k < K) v.x = p[0];
      if (k + 1 < K) v.y = p[1];
      if (k + 2 < K) v.z = p[2];
      if (k + 3 < K) v.w = p[3];
    }
    return v;
  };
  auto load = [&](int k0, float4 (&xr)[XL], float4 (&wr)[WL]) {
#pragma unroll
    for (int i = 0; i < XL; ++i) {
      const int idx = tid + i * THREADS;
      xr[i] = piece(X, m0 + (idx >> 2), M, k0 + (idx & 3) * 4);
    }
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      const int idx = tid + i * THREADS;
      wr[i] = piece(W, n0 + (idx >> 2), N, k0 + (idx & 3) * 4);
    }
  };
  auto store = [&](int buffer, const float4 (&xr)[XL], const float4 (&wr)[WL]) {
#pragma unroll
    for (int i = 0; i < XL; ++i) {
      const int idx = tid + i * THREADS, r = idx >> 2, c = (idx & 3) * 4;
      Xs[buffer][c][r] = xr[i].x, Xs[buffer][c + 1][r] = xr[i].y, Xs[buffer][c + 2][r] = xr[i].z, Xs[buffer][c + 3][r] = xr[i].w;
    }
#pragma unroll
    for (int i = 0; i < WL; ++i) {
      const int idx = tid + i * THREADS, r = idx >> 2, c = (idx & 3) * 4;
      Ws[buffer][c][r] = wr[i].x, Ws[buffer][c + 1][r] = wr[i].y, Ws[buffer][c + 2][r] = wr[i].z, Ws[buffer][c + 3][r] = wr[i].w;
    }
  };
  float4 a[2][2];
  ulonglong2 b[2][HALVES];
  auto fragments = [&](int slot, int buffer, int kk) {
    a[slot][0] = *reinterpret_cast<const float4*>(&Xs[buffer][kk][m_in]);
    a[slot][1] = *reinterpret_cast<const float4*>(&Xs[buffer][kk][m_in + 16]);
#pragma unroll
    for (int j = 0; j < HALVES; ++j) b[slot][j] = *reinterpret_cast<const ulonglong2*>(&Ws[buffer][kk][n_in + 32 * j]);
  };
  // Block k0 lies in `buffer`; block k0 + TK is in `xn`, `wn` and goes to the other buffer (all threads are past the
  // barrier behind that buffer's last reads); block k0 + 2 TK is asked for into `xm`, `wm`.
  auto block = [&](int k0, int buffer, float4 (&xm)[XL], float4 (&wm)[WL], const float4 (&xn)[XL], const float4 (&wn)[WL]) {
    if (k0 + 2 * TK < K) load(k0 + 2 * TK, xm, wm);
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      if (kk + 1 < TK) {
        fragments((kk + 1) & 1, buffer, kk + 1);
      } else if (k0 + TK < K) {
        store(buffer ^ 1, xn, wn);
        __syncthreads();
        fragments((kk + 1) & 1, buffer ^ 1, 0);
      }
      const float4 lo = a[kk & 1][0], hi = a[kk & 1][1];
      const float rows[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long aa = twice(rows[i]);
#pragma unroll
        for (int j = 0; j < HALVES; ++j) fma2(acc[i][2 * j], aa, b[kk & 1][j].x), fma2(acc[i][2 * j + 1], aa, b[kk & 1][j].y);
      }
    }
  };
  load(0, x0, w0);
  if (TK < K) load(TK, x1, w1);
  store(0, x0, w0);
  __syncthreads();
  fragments(0, 0, 0);
  for (int k0 = 0; k0 < K; k0 += 2 * TK) {
    block(k0, 0, x0, w0, x1, w1);
    if (k0 + TK < K) block(k0 + TK, 1, x1, w1, x0, w0);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + m_in + (i & 3) + (i >> 2) * 16;
    if (m >= M) continue;
#pragma unroll
    for (int half = 0; half < HALVES; ++half) {
      const int n = n0 + n_in + half * 32;
      float* dst = C + static_cast<size_t>(m) * N + n;
      float v[4];
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][2 * half]));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][2 * half + 1]));
      if (VEC) {
        if (n >= N) continue;
        float4* to = reinterpret_cast<float4*>(dst);
        float4 o = make_float4(v[0], v[1], v[2], v[3]);
        if (mode == 1) {
          const float4 old = *to;
          o = make_float4(old.x + o.x, old.y + o.y, old.z + o.z, old.w + o.w);
        }
        *to = o;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < N) dst[e] = mode == 1 ? dst[e] + v[e] : v[e];
      }
    }
  }
}

template <int BM_, int BN_, int TN>
int launch_tiled(const float* X, const float* W, float* C, int M, int N, int K, int mode, int group_cols, int group_rows,
                 bool vec, cudaStream_t stream) {
  const dim3 grid((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_);
  // Launched behind the kernel before, not beside it: let in early, CTAs pile up on the SMs that kernel leaves first,
  // and a step whose tiles fill the SMs once then takes two rounds (384 x 3072 x 2048: 203 us against 126).
  if (vec)
    gemm_f32_tiled_kernel<BM_, BN_, TN, true><<<grid, BM_ * BN_ / (8 * TN), 0, stream>>>(X, W, C, M, N, K, mode, group_cols, group_rows);
  else
    gemm_f32_tiled_kernel<BM_, BN_, TN, false><<<grid, BM_ * BN_ / (8 * TN), 0, stream>>>(X, W, C, M, N, K, mode, group_cols, group_rows);
  LRM_LAUNCH_CHECK();
  return 0;
}

// 128 x 64 tiles (8 x 8 outputs per thread) where the busiest SM has no more work with them than with 64 x 64 tiles of 8 x 4,
// which read their operands more often. us, 128 x 64 against 64 x 64: 512 rows of 16384 x 2048 702 and 757, 384 rows of
// 3072 x 2048 127 and 125; 128 rows of 2048 x 8192 (32 and 64 tiles) 491 and 306, 64 rows of 3072 x 2048 121 and 78.
bool prefers_wide_tile(int M, int N) {
  const long long wide = static_cast<long long>((M + 127) / 128) * ((N + 63) / 64);
  const long long small = static_cast<long long>((M + 63) / 64) * ((N + 63) / 64);
  return 2 * ((wide + kSmCount - 1) / kSmCount) <= (small + kSmCount - 1) / kSmCount;
}

// Few rows (a head's logits, decoding): bound by reading W. A CTA owns 32 columns, a lane each, and its warps
// share the rows; W and X come in blocks of 64 k through kFewStages asynchronous stages. An element adds over k in
// ascending order here too, so the bits are the tiled kernel's. One row, us, in a tile of 64 rows before: 8192 x
// 2048 32 (186), 128256 x 2048 171 (1567); 8 rows: 2048 x 8192 112 (728).
constexpr int kFewK = 64, kFewStages = 4, kFewPitch = kFewK + 4, kFewWarps = 4;

template <int PER>  // rows per warp
__global__ __launch_bounds__(kFewWarps * 32) void gemm_f32_few_kernel(const float* __restrict__ X, const float* __restrict__ W,
                                                                       float* __restrict__ C, int M, int N, int K, int mode,
                                                                       int group_cols, int group_rows) {
  extern __shared__ __align__(16) float stages[];  // [kFewStages][32 + M rows][kFewPitch]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n0 = blockIdx.x * 32;
  const int rows = 32 + M, size = rows * kFewPitch, blocks = (K + kFewK - 1) / kFewK;
  pdl_trigger();
  pdl_wait();
  if (group_cols > 0) X += static_cast<size_t>(n0 / group_cols) * group_rows * K;
  auto issue = [&](int block) {
    if (block < blocks) {
      float* base = stages + block % kFewStages * size;
      for (int i = tid; i < rows * (kFewK / 4); i += kFewWarps * 32) {
        const int r = i / (kFewK / 4), c = i % (kFewK / 4) * 4, k = block * kFewK + c;
        const bool in = k < K && (r >= 32 || n0 + r < N);
        const float* src = r < 32 ? W + static_cast<size_t>(in ? n0 + r : 0) * K : X + static_cast<size_t>(r - 32) * K;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(base + r * kFewPitch + c));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src + (in ? k : 0)), "r"(in ? 16 : 0));
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  for (int s = 0; s < kFewStages - 1; ++s) issue(s);
  for (int block = 0; block < blocks; ++block) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kFewStages - 2));
    __syncthreads();
    issue(block + kFewStages - 1);
    const float* w = stages + block % kFewStages * size + lane * kFewPitch;
    const float* x = stages + block % kFewStages * size + 32 * kFewPitch;
    if (warp < M) {
#pragma unroll 4
      for (int k = 0; k < kFewK; k += 4) {  // beyond K both operands are zeros
        const float4 wv = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int m = min(warp + i * kFewWarps, M - 1);
          const float4 xv = *reinterpret_cast<const float4*>(x + m * kFewPitch + k);
          acc[i] = fmaf(xv.w, wv.w, fmaf(xv.z, wv.z, fmaf(xv.y, wv.y, fmaf(xv.x, wv.x, acc[i]))));
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (n0 + lane >= N) return;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int m = warp + i * kFewWarps;
    if (m >= M) continue;
    float* dst = C + static_cast<size_t>(m) * N + n0 + lane;
    *dst = mode == 1 ? *dst + acc[i] : acc[i];
  }
}

template <int PER>
int launch_few(const float* X, const float* W, float* C, int M, int N, int K, int mode, int group_cols, int group_rows,
               cudaStream_t stream) {
  const size_t bytes = sizeof(float) * kFewStages * (32 + M) * kFewPitch;
  constexpr int most = sizeof(float) * kFewStages * (32 + PER * kFewWarps) * kFewPitch;
  if (most > 48 * 1024) {  // the same for every M: a smaller one would take back what another thread's launch counts on
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<PER>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  LRM_LAUNCH((gemm_f32_few_kernel<PER>), (N + 31) / 32, kFewWarps * 32, bytes, stream, X, W, C, M, N, K, mode, group_cols,
             group_rows);
  return 0;
}
}  // namespace

// group_cols > 0 (a multiple of 64): several inputs `group_rows` rows apart in X.
LRM_API int lrm_gemm_f32_grouped(const float* X, const float* W, float* C, int M, int N, int K, int mode,
                                 int group_cols, int group_rows, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (group_cols < 0 || group_cols % BN || (group_cols > 0 && group_rows < M)) return LRM_BAD_ARGUMENT;
  if (K <= 0 || (mode != 0 && mode != 1)) return LRM_BAD_ARGUMENT;
  if ((M + BM - 1) / BM > 65535) return LRM_UNSUPPORTED;
  const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const bool rows_aligned = K % 4 == 0 && aligned(X) && aligned(W);
  if (M > kFewRows) {
    const bool vec = rows_aligned && N % 4 == 0 && aligned(C);
    if (prefers_wide_tile(M, N)) return launch_tiled<128, 64, 8>(X, W, C, M, N, K, mode, group_cols, group_rows, vec, stream);
    return launch_tiled<64, 64, 4>(X, W, C, M, N, K, mode, group_cols, group_rows, vec, stream);
  }
  if (rows_aligned) {
    if (M <= 4) return launch_few<1>(X, W, C, M, N, K, mode, group_cols, group_rows, stream);
    if (M <= 8) return launch_few<2>(X, W, C, M, N, K, mode, group_cols, group_rows, stream);
    if (M <= 16) return launch_few<4>(X, W, C, M, N, K, mode, group_cols, group_rows, stream);
    return launch_few<8>(X, W, C, M, N, K, mode, group_cols, group_rows, stream);
  }
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  gemm_f32_kernel<<<grid, 256, 0, stream>>>(X, W, C, M, N, K, mode, group_cols, group_rows);
  LRM_LAUNCH_CHECK();
  return 0;
}

LRM_API int lrm_gemm_f32(const float* X, const float* W, float* C, int M, int N, int K, int mode,
                         cudaStream_t stream) {
  return lrm_gemm_f32_grouped(X, W, C, M, N, K, mode, 0, 0, stream);
}
