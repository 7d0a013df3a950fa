// State scans of long sequences with float32 FMAs, a block of L tokens at a time (the formulas of recurrent_block.cuh): the way
// of steps whose sequences and heads make more CTAs than the SMs hold at once, where the tensor path of recurrent_block.cuh
// pays more for its preparation, once per head, than it gains in the walk (block_takes_fma says where the line lies).
//
// Quotients of decays are made as products of the decays between; every product and sum is float32. What does not depend on
// the column is made first, for all blocks at once: the vectors k G, q G, k (G_L / G_m) and G_L per head where decays differ by
// row, the bare k and q per key head where a token has one decay, and D, T and the other numbers per head. Then a CTA per
// (sequence, head, tile of columns) walks the blocks; a walking thread holds 4 NQ rows of C columns, two rows of a column in one
// 64-bit register for the packed FMAs. Bound by the shared-memory pipe (a vector goes to every warp: the wider a thread's
// tile, the less). 16 heads of 128 x 128, eight sequences of 1,024 tokens (1,024 CTAs at 16 columns): two quads of rows and two
// columns a thread 890 us, and 609 with four columns and 4 tokens a block (which leaves registers for them); a decay per
// token 524 and 428.
#pragma once
#include "recurrent_scan.cuh"

namespace {

constexpr int kWalkStage = 16;   // tokens of a stage
constexpr int kWalkTokens = 96;  // tokens of a sequence from which going in blocks pays

// Stages of sequence b are numbered from walk_base(b) on: a whole number of stages each, none shared. A launch takes a run of
// them: all, or as many as the workspace has room for.
struct WalkPiece {
  int first, count;
  bool whole;
};
__device__ __forceinline__ int walk_base(const int* cu_seqlens, int b) { return cu_seqlens[b] / kWalkStage + b; }

// The z-th sequence of at least `least` tokens, or -1. A warp per call, all with the same z. (A walk's grid has as many as the
// step's tokens can make, not all sequences: 128 of one token each would else be 16,384 CTAs of 16 heads that end at once, 35 us.)
__device__ __forceinline__ int walking_sequence(const int* cu_seqlens, int seqs, int least, int z) {
  const int lane = threadIdx.x & 31;
  for (int b0 = 0; b0 < seqs; b0 += 32) {
    const int b = b0 + lane;
    unsigned which = __ballot_sync(0xffffffffu, b < seqs && cu_seqlens[b + 1] - cu_seqlens[b] >= least);
    const int here = __popc(which);
    if (z >= here) {
      z -= here;
      continue;
    }
    for (; z > 0; --z) which &= which - 1;
    return b0 + __ffs(which) - 1;
  }
  return -1;
}

inline long long walk_stages(int tokens, int seqs) { return tokens / kWalkStage + seqs; }
inline int walk_padded(int d) { return d > 128 ? 256 : d > 64 ? 128 : 64; }

// Scratch of `floats` floats, 16-byte aligned.
struct Workspace {
  float* at;
  long long floats;
};

// Everything a walk is launched with.
struct WalkArgs {
  const float *q, *k, *v, *g, *head_decay, *beta, *look, *put;
  float *state, *out;
  const int *cu_seqlens, *slots;
  int seqs, H, KH, d, dv;
  Workspace workspace;
  cudaStream_t stream;
  Rows rows;
  int least;     // tokens of a sequence from which it walks (0: a step of one sequence, which has them)
  int walkers;   // sequences that may
};

template <int DP, int MODE, int L>
struct WalkShape {
  static constexpr bool DELTA = MODE == 1 || MODE == 5, ROW_DECAY = MODE == 1 || MODE == 4, BONUS = MODE == 4;
  static constexpr int BLOCKS = kWalkStage / L;                               // of a stage
  static constexpr int VECTORS = !ROW_DECAY ? 2 * L : DELTA ? 3 * L + 1 : 2 * L + 1;  // of DP floats, in a block
  static constexpr int AT_Q = DELTA || !ROW_DECAY ? L * DP : 0, AT_W = ROW_DECAY ? AT_Q + L * DP : 0, AT_G = AT_W + L * DP;
  static constexpr int STAGE = BLOCKS * VECTORS * DP;                        // floats of a stage's vectors
  // numbers of a block and head: D [L][L] | T [L][L] | G_j [L] | G_L / G_j [L] | G_L and what its rounding lost
  static constexpr int AT_T = L * L, AT_UPTO = 2 * L * L, AT_REST = AT_UPTO + L, AT_ALL = AT_REST + L, SCALARS = AT_ALL + 4;
};

// A CTA per stage and head (row decays) or key head.
template <int DP, int MODE, int L>
__global__ __launch_bounds__(128) void walk_prepare_kernel(
    const float* q, const float* k, const float* g, const float* __restrict__ head_decay, const float* beta,
    const float* __restrict__ look, const float* put, float* __restrict__ vectors_at, float* __restrict__ scalars_at,
    const int* __restrict__ cu_seqlens, int seqs, int H, int KH, int d, long long q_stride, int least, WalkPiece piece) {
  using W = WalkShape<DP, MODE, L>;
  constexpr bool DELTA = W::DELTA, ROW_DECAY = W::ROW_DECAY, BONUS = W::BONUS;
  constexpr int BLOCKS = W::BLOCKS, SUMS = L * L;
  __shared__ float partials[BLOCKS][4][SUMS];
  __shared__ float totals[BLOCKS][SUMS];
  pdl_trigger();
  pdl_wait();
  const int stage = blockIdx.x, vh = blockIdx.y, per_key = H / KH, kh = ROW_DECAY ? vh / per_key : vh;
  int b = 0;  // the last sequence whose stages begin no later
  for (int high = seqs; high - b > 1;) {
    const int middle = (b + high) >> 1;
    if (walk_base(cu_seqlens, middle) <= piece.first + stage) b = middle;
    else high = middle;
  }
  const int first = (piece.first + stage - walk_base(cu_seqlens, b)) * kWalkStage;  // token of the sequence
  const int start = cu_seqlens[b] + first, cn = min(kWalkStage, cu_seqlens[b + 1] - start);
  if (cn <= 0 || cu_seqlens[b + 1] - cu_seqlens[b] < least) return;
  const int tid = threadIdx.x, lane = tid & 31;
  constexpr int TPB = DP < 128 ? DP : 128, AT_ONCE = 128 / TPB, RPT = DP / TPB;  // threads per block, blocks at once, rows per thread
  float* to = vectors_at + (static_cast<size_t>(stage) * (ROW_DECAY ? H : KH) + vh) * W::STAGE;
#pragma unroll 1
  for (int it = 0; it < BLOCKS / AT_ONCE; ++it) {
    const int block = it * AT_ONCE + tid / TPB;
    float* vectors = to + block * W::VECTORS * DP;
    float sums[SUMS];
#pragma unroll
    for (int i = 0; i < SUMS; ++i) sums[i] = 0.f;
#pragma unroll
    for (int a = 0; a < RPT; ++a) {
      const int r = tid % TPB + a * TPB;
      const float factor = BONUS && r < d ? look[vh * d + r] : 0.f;
      float qr[L], kr[L], gr[L];
#pragma unroll
      for (int j = 0; j < L; ++j) {  // a token the sequence does not have: nothing read or written, no decay
        const bool is = block * L + j < cn && r < d;
        const size_t tok = static_cast<size_t>(start + block * L + j);
        qr[j] = is ? q[tok * q_stride + kh * d + r] : 0.f;
        kr[j] = is ? k[tok * q_stride + kh * d + r] : 0.f;
        gr[j] = ROW_DECAY && is ? g[(tok * H + vh) * d + r] : 1.f;
      }
      float upto = 1.f;
#pragma unroll
      for (int j = 0; j < L; ++j) {
        if (BONUS) vectors[W::AT_Q + j * DP + r] = qr[j] * upto;
        if (ROW_DECAY) upto *= gr[j];
        if (DELTA || !ROW_DECAY) vectors[j * DP + r] = kr[j] * upto;
        if (!BONUS) vectors[W::AT_Q + j * DP + r] = qr[j] * upto;
      }
      if (ROW_DECAY) vectors[W::AT_G + r] = upto;
#pragma unroll
      for (int m = 0; m < L; ++m) {  // token m's write on its way through the tokens behind it
        float w = kr[m];
        sums[(L + 1) * m] += qr[m] * (BONUS ? factor * w : w);
#pragma unroll
        for (int j = m + 1; j < L; ++j) {
          if (BONUS) sums[L * j + m] = fmaf(qr[j], w, sums[L * j + m]);
          if (ROW_DECAY) w *= gr[j];
          if (!BONUS) sums[L * j + m] = fmaf(qr[j], w, sums[L * j + m]);
          if (DELTA) sums[L * m + j] = fmaf(kr[j], w, sums[L * m + j]);
        }
        if (ROW_DECAY) vectors[W::AT_W + m * DP + r] = w;
      }
    }
    // sums over the rows: every exchange halves the sums a lane holds, down to SUMS / 32 or one
    constexpr int LEFT = SUMS > 32 ? SUMS / 32 : 1;
#pragma unroll
    for (int half = SUMS / 2, bit = 16; half >= LEFT; half >>= 1, bit >>= 1) {
      const bool high = (lane & bit) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float keep = high ? sums[i + half] : sums[i], give = high ? sums[i] : sums[i + half];
        sums[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
      }
    }
    if (SUMS == 16) sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], 1);
    if (SUMS > 16 || (lane & 1) == 0) {
#pragma unroll
      for (int i = 0; i < LEFT; ++i) partials[block][tid % TPB >> 5][(SUMS == 16 ? lane >> 1 : lane) * LEFT + i] = sums[i];
    }
  }
  __syncthreads();
  for (int i = tid; i < BLOCKS * SUMS; i += 128) {
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < TPB / 32; ++w) total += partials[i / SUMS][w][i % SUMS];
    totals[i / SUMS][i % SUMS] = total;  // [later j][earlier m] the D of j on m, [m][j] the C of j on m
  }
  __syncthreads();
  const int heads = ROW_DECAY ? 1 : per_key;
  for (int i = tid; i < heads * BLOCKS * L; i += 128) {  // a thread per head, block and earlier token m
    const int m = i % L, block = i / L % BLOCKS, h = ROW_DECAY ? vh : kh * per_key + i / (L * BLOCKS);
    float* scalars = scalars_at + ((static_cast<size_t>(stage) * H + h) * BLOCKS + block) * W::SCALARS;
    const float* dots = totals[block];
    float decay[L], step[L], passed[L];  // passed[j]: G_j / G_m
    float upto = 1.f, lost = 0.f, rest = 1.f;
#pragma unroll
    for (int j = 0; j < L; ++j) {
      const bool is = block * L + j < cn;
      const size_t at = static_cast<size_t>(start + block * L + j) * H + h;
      decay[j] = 1.f;
      if (is && MODE == 0) decay[j] = head_decay[h];
      if (is && MODE == 2) decay[j] = beta[at];
      if (is && MODE == 5) decay[j] = put[at];
      step[j] = is && DELTA ? beta[at] : 0.f;
      const float next = upto * decay[j];
      lost = fmaf(lost, decay[j], fmaf(upto, decay[j], -next));
      upto = next;
      if (j == m) scalars[W::AT_UPTO + m] = upto;
      if (j > m) rest *= decay[j];
      passed[j] = rest;
    }
    scalars[W::AT_REST + m] = rest;
    if (m == 0) scalars[W::AT_ALL] = upto, scalars[W::AT_ALL + 1] = lost;
#pragma unroll
    for (int j = 0; j < L; ++j) scalars[L * j + m] = j >= m ? dots[L * j + m] * passed[j] : 0.f;
    if (DELTA) {  // column m of T, by substitution; C_jn of two later tokens needs G_j / G_n
      float column[L];
#pragma unroll
      for (int j = 0; j < L; ++j) {
        float sum = 0.f;
        if (j > m) {
#pragma unroll
          for (int n = 0; n < j; ++n) {
            float between = 1.f;
#pragma unroll
            for (int x = n + 1; x <= j; ++x) between *= decay[x];
            if (n >= m) sum = fmaf(dots[L * n + j] * between, column[n], sum);
          }
        }
        column[j] = j == m ? step[j] : j > m ? -step[j] * sum : 0.f;
        scalars[W::AT_T + L * j + m] = column[j];
      }
    }
  }
}

__device__ __forceinline__ void walk_fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long walk_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long walk_pair(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 walk_parts(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// Thread (group of C columns, part p of P) holds rows 4 P a + 4 p + e, a < NQ, e < 4, of its columns.
template <int NQ, int C, int DP, int MODE, int L>
struct Walk {
  using W = WalkShape<DP, MODE, L>;
  static constexpr int P = DP / (4 * NQ), GROUPS = 32 / P, COLS = 4 * GROUPS * C, VALUES = L * C;
  static constexpr int SPARE = P / VALUES;  // lanes that end with the same sum
  static_assert(P <= 32 && SPARE >= 1, "a lane ends with one sum at most");
  static constexpr int BUFFER = W::STAGE + W::BLOCKS * W::SCALARS + kWalkStage * COLS;  // vectors | numbers | v
  static constexpr int BUFFERS = DP > 128 ? 2 : 3;
  static constexpr size_t BYTES = sizeof(float) * BUFFERS * BUFFER;
};

// ALL: of a step in one piece whose tokens let every sequence walk, sequence z; else the z-th that walks, and what of it the
// piece holds. (Finding them in the plain case too cost up to 12 % by the code around it: 16 heads of 128 with a bonus, 2,048
// tokens, 274 us against 245.)
template <int NQ, int C, int DP, int MODE, int L, bool ALL>
__global__ __launch_bounds__(128) void walk_scan_kernel(
    const float* __restrict__ vectors_at, const float* __restrict__ scalars_at, const float* __restrict__ v,
    float* __restrict__ state, float* __restrict__ out, const int* __restrict__ cu_seqlens, const int* __restrict__ slots,
    int seqs, int H, int KH, int d, int dv, long long v_stride, int wide, int least, WalkPiece piece) {
  using W = WalkShape<DP, MODE, L>;
  using K = Walk<NQ, C, DP, MODE, L>;
  constexpr int P = K::P, COLS = K::COLS, BLOCKS = W::BLOCKS, SCALARS = W::SCALARS, SPARE = K::SPARE;
  constexpr bool DELTA = W::DELTA, ROW_DECAY = W::ROW_DECAY;
  extern __shared__ __align__(16) float smem[];
  const int h = blockIdx.y, b = ALL ? blockIdx.z : walking_sequence(cu_seqlens, seqs, least, blockIdx.z);
  const int vh = ROW_DECAY ? h : h / (H / KH), VH = ROW_DECAY ? H : KH, col0 = blockIdx.x * COLS;
  if (!ALL && b < 0) return;
  int start = cu_seqlens[b], n = cu_seqlens[b + 1] - start, base_stage = walk_base(cu_seqlens, b);
  const int slot = slots[b];
  if (n < least) return;
  if (!ALL) {  // the part of the sequence in this launch, as a sequence of its own whose first stage lies at base_stage
    const int skipped = max(0, piece.first - base_stage) * kWalkStage;
    base_stage = max(0, base_stage - piece.first), start += skipped;
    n = min(n - skipped, (piece.count - base_stage) * kWalkStage);
    if (n <= 0 || (!piece.whole && slot < 0)) return;
  }
  const int stages = (n + kWalkStage - 1) / kWalkStage;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  auto issue = [&](int stage) {
    if (stage < stages) {
      float* to = smem + stage % K::BUFFERS * K::BUFFER;
      const float* from = vectors_at + (static_cast<size_t>(base_stage + stage) * VH + vh) * W::STAGE;
#pragma unroll 4
      for (int i = tid * 4; i < W::STAGE; i += 512) scan_cp_async(to + i, from + i, true, true);
      from = scalars_at + (static_cast<size_t>(base_stage + stage) * H + h) * BLOCKS * SCALARS;
      to += W::STAGE;
      if (tid * 4 < BLOCKS * SCALARS) scan_cp_async(to + tid * 4, from + tid * 4, true, true);
      to += BLOCKS * SCALARS;
      const int step = wide ? 4 : 1, per_v = COLS / step;
      for (int i = tid; i < kWalkStage * per_v; i += 128) {  // zeros for tokens and columns that are not there
        const int c = i / per_v, j = i % per_v * step;
        const bool in = stage * kWalkStage + c < n && col0 + j < dv;
        const size_t tok = static_cast<size_t>(start + (in ? stage * kWalkStage + c : 0));
        scan_cp_async(to + c * COLS + j, v + tok * v_stride + h * dv + (in ? col0 + j : 0), in, wide != 0);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  static_assert(BLOCKS * SCALARS <= 512, "a thread copies at most one piece of the numbers");

  const int p = lane % P, col = (warp * K::GROUPS + lane / P) * C;  // first of the thread's columns in the tile
  unsigned long long S[NQ][2][C];                                   // [quad of rows][pair of them][column]
  float* mine = slot >= 0 ? state + (static_cast<size_t>(slot) * H + h) * d * dv : nullptr;
#pragma unroll
  for (int i = 0; i < K::BUFFERS - 1; ++i) issue(i);
#pragma unroll
  for (int a = 0; a < NQ; ++a)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int row = 4 * P * a + 4 * p + 2 * e, j = col0 + col + c;
        const bool in = mine != nullptr && j < dv;
        S[a][e][c] = walk_pair(in && row < d ? mine[static_cast<size_t>(row) * dv + j] : 0.f,
                               in && row + 1 < d ? mine[static_cast<size_t>(row + 1) * dv + j] : 0.f);
      }
  // The sums over the parts of column c, token j end in the lanes with p / SPARE == c * L + j.
  const int my_col = p / SPARE / L, my_token = p / SPARE % L;
  auto add_parts = [&](const unsigned long long (&x)[C][L]) {
    float y[K::VALUES];
#pragma unroll
    for (int i = 0; i < K::VALUES; ++i) {
      const float2 parts = walk_parts(x[i / L][i % L]);
      y[i] = parts.x + parts.y;
    }
#pragma unroll
    for (int half = K::VALUES / 2, bit = P / 2; half > 0; half >>= 1, bit >>= 1) {
      const bool high = (p & bit) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float keep = high ? y[i + half] : y[i], give = high ? y[i] : y[i + half];
        y[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
      }
    }
#pragma unroll
    for (int o = SPARE / 2; o > 0; o >>= 1) y[0] += __shfl_xor_sync(0xffffffffu, y[0], o);
    return y[0];
  };
  const bool writes = p % SPARE == 0 && col0 + col + my_col < dv;
  float* rows = out + (static_cast<size_t>(start) * H + h) * dv + col0 + col + my_col;

  for (int stage = 0; stage < stages; ++stage) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(K::BUFFERS - 2));
    __syncthreads();  // this stage is here for every thread, and everyone is done with the one before
    issue(stage + K::BUFFERS - 1);
    const int cn = min(kWalkStage, n - stage * kWalkStage);
    const float* from = smem + stage % K::BUFFERS * K::BUFFER;
#pragma unroll
    for (int block = 0; block < BLOCKS; ++block) {
      const float* vectors = from + block * W::VECTORS * DP;
      const float* scalars = from + W::STAGE + block * SCALARS;
      const float* values = from + W::STAGE + BLOCKS * SCALARS + block * L * COLS + col;
      auto pairs = [&](int at) { return *reinterpret_cast<const ulonglong2*>(vectors + at + 4 * p); };
      unsigned long long reads[C][L], reads_out[C][L];
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int j = 0; j < L; ++j) reads[c][j] = reads_out[c][j] = 0ull;
      if (DELTA) {
#pragma unroll
        for (int a = 0; a < NQ; ++a)
#pragma unroll
          for (int j = 0; j < L; ++j) {
            const ulonglong2 x = pairs(j * DP + 4 * P * a);
#pragma unroll
            for (int c = 0; c < C; ++c) walk_fma2(reads[c][j], x.x, S[a][0][c]), walk_fma2(reads[c][j], x.y, S[a][1][c]);
          }
      }
#pragma unroll
      for (int a = 0; a < NQ; ++a)
#pragma unroll
        for (int j = 0; j < L; ++j) {
          const ulonglong2 x = pairs(W::AT_Q + j * DP + 4 * P * a);
#pragma unroll
          for (int c = 0; c < C; ++c) walk_fma2(reads_out[c][j], x.x, S[a][0][c]), walk_fma2(reads_out[c][j], x.y, S[a][1][c]);
        }
      // what the tokens write: `own` in the column whose read-outs end in this thread; u in all, as the state takes it
      float own[L];
      unsigned long long u[L][C];
      float rest[L];
#pragma unroll
      for (int j = 0; j < L; ++j) rest[j] = ROW_DECAY ? 1.f : scalars[W::AT_REST + j];
      if (DELTA) {
        float r = add_parts(reads);  // of my_token
        if (!ROW_DECAY) r *= scalars[W::AT_UPTO + my_token];
        r = values[my_token * COLS + my_col] - r;
        float all[L];
#pragma unroll
        for (int j = 0; j < L; ++j) all[j] = __shfl_sync(0xffffffffu, r, lane - p + (my_col * L + j) * SPARE);
#pragma unroll
        for (int j = 0; j < L; ++j) {
          float sum = 0.f;
#pragma unroll
          for (int m = 0; m <= j; ++m) sum = fmaf(scalars[W::AT_T + L * j + m], all[m], sum);
          own[j] = sum;
        }
#pragma unroll
        for (int j = 0; j < L; ++j)
#pragma unroll
          for (int c = 0; c < C; ++c) {  // (lanes of a token hold the same numbers: any of them gives the column's)
            const float x = __shfl_sync(0xffffffffu, own[j], lane - p + c * L * SPARE + p % (L * SPARE)) * rest[j];
            u[j][c] = walk_pair(x, x);
          }
      } else {
#pragma unroll
        for (int j = 0; j < L; ++j) {
          float x[C];
#pragma unroll
          for (int c = 0; c < C; c += 2) {
            const float2 two = *reinterpret_cast<const float2*>(values + j * COLS + c);
            x[c] = two.x, x[c + 1] = two.y;
          }
          own[j] = x[0];
#pragma unroll
          for (int c = 1; c < C; ++c) own[j] = my_col == c ? x[c] : own[j];
#pragma unroll
          for (int c = 0; c < C; ++c) u[j][c] = walk_pair(x[c] * rest[j], x[c] * rest[j]);
        }
      }
      // A state that is not finite keeps no lost part (infinity times nothing is not a number); it shows in the read-outs, to
      // which every row of the thread's columns has been added.
      bool finite = true;
      if (!ROW_DECAY) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const float2 sums = walk_parts(reads_out[c][0]);
          finite &= isfinite(sums.x + sums.y);
        }
      }
#pragma unroll
      for (int a = 0; a < NQ; ++a) {
        unsigned long long next[2][C];
        ulonglong2 decay;
        if (ROW_DECAY) {
          decay = pairs(W::AT_G + 4 * P * a);
        } else {
          const unsigned long long lost = walk_pair(scalars[W::AT_ALL + 1], scalars[W::AT_ALL + 1]);
          decay.x = decay.y = walk_pair(scalars[W::AT_ALL], scalars[W::AT_ALL]);
#pragma unroll
          for (int c = 0; c < C; ++c) next[0][c] = walk_mul2(S[a][0][c], lost), next[1][c] = walk_mul2(S[a][1][c], lost);
          if (!finite) {
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
              for (int c = 0; c < C; ++c) {
                const float2 held = walk_parts(S[a][e][c]), part = walk_parts(next[e][c]);
                next[e][c] = walk_pair(isfinite(held.x) ? part.x : 0.f, isfinite(held.y) ? part.y : 0.f);
              }
          }
        }
#pragma unroll
        for (int m = 0; m < L; ++m) {
          const ulonglong2 x = pairs(W::AT_W + m * DP + 4 * P * a);
#pragma unroll
          for (int c = 0; c < C; ++c) {
            if (ROW_DECAY && m == 0) {
              next[0][c] = walk_mul2(x.x, u[0][c]), next[1][c] = walk_mul2(x.y, u[0][c]);
            } else {
              walk_fma2(next[0][c], x.x, u[m][c]), walk_fma2(next[1][c], x.y, u[m][c]);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
          walk_fma2(next[0][c], S[a][0][c], decay.x), walk_fma2(next[1][c], S[a][1][c], decay.y);
          S[a][0][c] = next[0][c], S[a][1][c] = next[1][c];
        }
      }
      float o = add_parts(reads_out);
      if (!ROW_DECAY) o *= scalars[W::AT_UPTO + my_token];
#pragma unroll
      for (int m = 0; m < L; ++m)  // (a token's read-out takes nothing from the tokens behind it, not even a NaN)
        o = m <= my_token ? fmaf(scalars[L * my_token + m], own[m], o) : o;
      if (writes && block * L + my_token < cn) rows[static_cast<size_t>(stage * kWalkStage + block * L + my_token) * H * dv] = o;
    }
  }
  if (mine != nullptr) {
#pragma unroll
    for (int a = 0; a < NQ; ++a)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int row = 4 * P * a + 4 * p + 2 * e, j = col0 + col + c;
          const float2 pair = walk_parts(S[a][e][c]);
          if (j < dv && row < d) mine[static_cast<size_t>(row) * dv + j] = pair.x;
          if (j < dv && row + 1 < d) mine[static_cast<size_t>(row + 1) * dv + j] = pair.y;
        }
  }
}

// Floats of a stage in the workspace: its vectors, and its numbers per head (behind the vectors of all stages).
template <int MODE, int L>
long long walk_vectors(int H, int KH, int d) {
  using W = WalkShape<64, MODE, L>;
  return static_cast<long long>(W::BLOCKS) * (W::ROW_DECAY ? H : KH) * W::VECTORS * walk_padded(d);
}
template <int MODE, int L>
long long walk_block_floats(int H, int KH, int d) {
  using W = WalkShape<64, MODE, L>;
  return walk_vectors<MODE, L>(H, KH, d) + static_cast<long long>(W::BLOCKS) * H * W::SCALARS;
}

template <int NQ, int C, int DP, int MODE, int L>
int launch_walk(const WalkArgs& a) {
  using K = Walk<NQ, C, DP, MODE, L>;
  const long long all = walk_stages(a.rows.tokens, a.seqs), room = a.workspace.floats / walk_block_floats<MODE, L>(a.H, a.KH, a.d);
  auto kernel = room >= all && a.walkers == a.seqs ? walk_scan_kernel<NQ, C, DP, MODE, L, true>
                                                 : walk_scan_kernel<NQ, C, DP, MODE, L, false>;
  if (K::BYTES > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(K::BYTES));
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  const long long q_stride = a.rows.q > 0 ? a.rows.q : static_cast<long long>(a.KH) * a.d;
  const long long v_stride = a.rows.v > 0 ? a.rows.v : static_cast<long long>(a.H) * a.dv;
  const int wide = a.dv % 4 == 0 && v_stride % 4 == 0 && reinterpret_cast<uintptr_t>(a.v) % 16 == 0;
  // launched behind the kernel before, not beside it: let in early its CTAs pile up on the SMs that kernel leaves first
  const long long pieces = (all + room - 1) / room, per = (all + pieces - 1) / pieces;
  float* scalars = a.workspace.at + per * walk_vectors<MODE, L>(a.H, a.KH, a.d);
  for (long long first = 0; first < all; first += per) {
    const WalkPiece piece{static_cast<int>(first), static_cast<int>(min(per, all - first)), pieces == 1};
    LRM_LAUNCH((walk_prepare_kernel<DP, MODE, L>), dim3(piece.count, K::W::ROW_DECAY ? a.H : a.KH), 128, 0, a.stream, a.q, a.k, a.g,
               a.head_decay, a.beta, a.look, a.put, a.workspace.at, scalars, a.cu_seqlens, a.seqs, a.H, a.KH, a.d, q_stride, a.least,
               piece);
    kernel<<<dim3((a.dv + K::COLS - 1) / K::COLS, a.H, a.walkers), 128, K::BYTES, a.stream>>>(
        a.workspace.at, scalars, a.v, a.state, a.out, a.cu_seqlens, a.slots, a.seqs, a.H, a.KH, a.d, a.dv, v_stride, wide, a.least, piece);
    LRM_LAUNCH_CHECK();
  }
  return 0;
}

template <int MODE>
constexpr int walk_block(int padded) {  // tokens of a block
  return padded == 256 && WalkShape<64, MODE, 4>::DELTA ? 8 : 4;
}
template <int MODE>
long long walk_stage_floats(int H, int KH, int d) {
  return walk_block<MODE>(walk_padded(d)) == 8 ? walk_block_floats<MODE, 8>(H, KH, d) : walk_block_floats<MODE, 4>(H, KH, d);
}
template <int MODE>
int launch_walk(const WalkArgs& a) {
  constexpr int LONG = walk_block<MODE>(256);
  if (a.d > 128) return launch_walk<(LONG == 8 ? 4 : 2), (LONG == 8 ? 2 : 4), 256, MODE, LONG>(a);
  if (a.d > 64) return launch_walk<2, 4, 128, MODE, 4>(a);
  return launch_walk<1, 4, 64, MODE, 4>(a);
}

}  // namespace
