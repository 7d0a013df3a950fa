// The state scan of recurrent_scan.cuh for long sequences (prompts), a block of 16 tokens at a time on the tensor cores.
//
// A sequence's tokens form a chain through its state. Here a block of tokens reads the state once. With G_j the product of
// the decays of the block's first j tokens (per row i of the state) and S the state ahead of the block,
//   p_j = sum_i k_ji G_ji S_i                              what token j reads, but for its block's own writes
//   u_j = b_j (v_j - p_j - sum_{m<j} C_jm u_m)             C_jm = sum_i k_ji (G_j / G_m)_i k_mi      (delta rules)
//   u_j = v_j                                                                                        (the others)
//   o_j = sum_i q_ji G_ji S_i + sum_{m<=j} D_jm u_m        D_jm = sum_i q_ji (G_j / G_m)_i k_mi
//   S_i <- G_Li S_i + sum_m k_mi (G_L / G_m)_i u_m
// (with a bonus m for the newest, read before the write: G_{j-1} for q_j's G_j, and D_jj = sum_i q_ji m_i k_ji.)
// Quotients of decays are made as products of the decays between, so nothing is divided by a small number. u is T (v - p)
// with the triangular T = (I + diag(b) C)^-1 diag(b).
//
// In the walk the rules with a delta use p'_j = sum_i (T k G)_ji S_i, u = T v - p', and the read-outs o = D T v + (q G - D T k G) S,
// so that nothing waits for T or D; the others o = D v + q G S.
//
// Precision: the sums over i and m are bfloat16 products of float32 numbers cut into three parts, each rounded, which hold every bit;
// of the nine products the lowest, below 2^-34, is left out. The tensor core cuts sums off where it should round (measured:
// at 2^-23 of the largest term, up to 2^-25 of it kept within a product), so each runs over at most 64 terms from zero, the
// small products apart from the large ones; what is longer than that, the state itself first of all, is added in float32 on the
// CUDA cores. A read of one number is rounded once, as an FMA is. Distance from 64 bits, relative, read-outs and state, 16 heads of
// 128 x 128 that forget at 1e-3 to 0.3 a token (in brackets float32 FMAs, blocks of 8 or 4): delta rule, 96 tokens 1.4e-7 and
// 1.3e-7 (1.5e-7, 1.4e-7), 1,500 2.0e-7 and 1.9e-7 (2.1e-7, 2.0e-7); a decay per token 1.1e-7 and 6.6e-8 (1.2e-7, 9.3e-8), 1.3e-7 and 1.1e-7
// (2.0e-7, 2.0e-7); of these the states of the heads that forget the fastest 7.3e-8 (6.5e-8) and 5.5e-8 (4.8e-8): few terms, cut off.
//
// Two launches (behind one for a step's sequences that go token by token). What does not depend on the column is made first,
// for all blocks at once, into a workspace, cut into its parts: the vectors T k G, q G - D T k G (or q G), k (G_L / G_m) and G_L
// per head where decays differ by row or a delta rule is on, else the bare k and q per key head (one decay a token then
// multiplies sums instead of vectors); beside them per head and tile of 16 columns T v (or v) and D T v (or D v). G_L of one
// decay comes with the rounding it lost: a decay that is the same for every token would lose it the same way in every block.
// Then a CTA per (sequence, head, tile) walks the blocks. Four warps share the rows of the state: a warp holds the transposed
// state of its rows as accumulators of m16n8k16 products, whose layout is that of the next products' first operand; the
// warps' shares of p' meet in shared memory, once a block. Four more warps bring the stages and make the read-outs from the
// state's parts, off the chain.
//
// What bounds it: the chain of a block (cut the state, p', its exchange, cut u, the update) is 1.15 us under a delta rule and
// 0.87 us without, with a CTA of eight warps per SM; the tensor pipe is 38 % busy meanwhile. us, in
// brackets float32 FMAs in blocks of 8 or 4 tokens: delta rule, 16 heads of 128 x 128, 2,048 tokens 200 (262), 8 heads 175 (231),
// 16 heads of 64 x 64 148 (229); a decay per token 146 (203), 143 (168), 100 (160); 32 heads of 128 x 64, 1,500 and 777 tokens 145
// (187). One sequence of 96 tokens is within 2 us of the FMAs on both rules (16 heads of 128 x 128), 256 8 us below. (With six products
// of parts cut off, less exact for reads of few numbers: 187, 163, 137; 136, 133, 94; 131.)
// The shares as a second product of all eight warps' halves of the rows, and tiles of 32 columns a CTA, gave nothing.
//
// Numbers that are not finite: a product with a zero would spread them to tokens ahead of them. They are taken out (zero
// instead), and the columns of the state that they reach are done once more with float32 FMAs from the token they come with
// (BlockAgain), so an infinity or a NaN shows where the formulas above let it and nowhere else. So do vectors' numbers of 2^24 and more
// and states' of 2^64, whose products, 2^32 fold, could leave the range.
//
// Which sequences walk is each one's own matter, but this way or with FMAs follows the step's size, and with it the order of the
// sums: the same sequence gives other bits, within float32 rounding, in another step. Who needs the bits goes without a
// workspace, token by token.
#pragma once
#include "recurrent_walk.cuh"

namespace {

constexpr int kBlockCols = 16;    // columns of a CTA

template <int DP, int MODE>
struct BlockShape {
  static constexpr bool DELTA = MODE == 1 || MODE == 5, BONUS = MODE == 4;
  static constexpr bool ROW_DECAY = MODE == 1 || MODE == 4;  // G_L differs by row of the state
  static constexpr bool BY_HEAD = DELTA || BONUS;            // vectors per head, decays within; else per key head, without
  static constexpr int L = kWalkStage;
  static constexpr int PLANE = L * DP;                       // bfloat16 numbers of a part of a block's vectors
  static constexpr int AT_K = 0, AT_Q = BONUS ? 0 : 1, AT_W = BY_HEAD ? AT_Q + 1 : 0, VECTORS = (BY_HEAD ? AT_W : AT_Q) + 1;
  static constexpr int AT_G = VECTORS * 3 * PLANE / 2, STAGE = AT_G + (ROW_DECAY ? DP : 0);  // in floats
  // numbers of a block and head: G_j [L] | G_L, what its rounding lost, whether a vector's number is out of range
  static constexpr int AT_ALL = L, AT_BAD = AT_ALL + 2, SCALARS = AT_ALL + 4;
  // and of a tile of columns, each in the order of block_lane_at: what the tokens write but for what they read of the state |
  // what their read-outs are but for that
  static constexpr int TILE = 2 * L * kBlockCols;
  static_assert(STAGE % 4 == 0 && SCALARS % 4 == 0, "pieces of 16 bytes");
};

// Numbers are cut 2^16 fold, so that parts of the smallest are not lost; products of parts are brought back by 2^-32. Vectors' and
// states' numbers beyond these lines could leave the range in a product's sum.
constexpr float kBlockVector = 16777216.f, kBlockState = 18446744073709551616.f;  // 2^24, 2^64
constexpr float kBlockBack = 2.3283064365386963e-10f;                             // 2^-32
__device__ __forceinline__ void block_most(float& most, float x) { asm("max.NaN.f32 %0, %0, %1;" : "+f"(most) : "f"(fabsf(x))); }
__device__ __forceinline__ bool block_out(float x, float line) { return !(fabsf(x) < line); }  // (a NaN is out)
// Two numbers as the sums of three pairs of bfloat16, each rounded, exact.
__device__ __forceinline__ void block_split(float x, float y, uint32_t& high, uint32_t& middle, uint32_t& low) {
  x *= 65536.f, y *= 65536.f;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(high) : "f"(y), "f"(x));
  const float rx = x - __uint_as_float(high << 16), ry = y - __uint_as_float(high & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(middle) : "f"(ry), "f"(rx));
  const float sx = rx - __uint_as_float(middle << 16), sy = ry - __uint_as_float(middle & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(low) : "f"(sy), "f"(sx));
}
// One number of a block that goes by FMAs: as above, or its own bits and a mark.
constexpr uint16_t kBlockWhole = 0x7fc0;
__device__ __forceinline__ void block_split_any(float x, uint16_t (&part)[3]) {
  uint32_t high, middle, low;
  block_split(x, 0.f, high, middle, low);
  const bool whole = block_out(x, kBlockVector);
  part[0] = whole ? __float_as_uint(x) >> 16 : high & 0xffff;
  part[1] = whole ? __float_as_uint(x) & 0xffff : middle & 0xffff;
  part[2] = whole ? kBlockWhole : low & 0xffff;
}
__device__ __forceinline__ float block_join(const uint16_t* at, int plane) {
  const uint32_t high = at[0], middle = at[plane], low = at[2 * plane];
  if (low == kBlockWhole) return __uint_as_float(high << 16 | middle);
  return (__uint_as_float(high << 16) + (__uint_as_float(middle << 16) + __uint_as_float(low << 16))) * (1.f / 65536.f);
}
// Where row r of token t's vector lies in a part's [L][DP]: pieces of 8 rows change places so that eight tokens' pieces lie in
// different banks.
template <int DP>
__device__ __forceinline__ int block_at(int t, int r) {
  return t * DP + ((((r >> 3) ^ (t & 7)) << 3) | (r & 7));
}

// Where a block's vectors are cut and stored: rows r and r + 1 of token t's vector `which` at a time. `most` collects the largest;
// what is out of range is stored once more at the end (block_store_again).
template <int DP, int MODE>
__device__ __forceinline__ void block_store(uint16_t* planes, int which, int t, int r, float x, float y, float& most) {
  using W = BlockShape<DP, MODE>;
  uint32_t part[3];
  block_split(x, y, part[0], part[1], part[2]);
  block_most(most, x), block_most(most, y);
  const int at = block_at<DP>(t, r);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(planes + (which * 3 + i) * W::PLANE + at) = part[i];
}
__device__ __noinline__ void block_store_again(uint16_t* at, int plane, float x, float y) {
  uint16_t a[3], b[3];
  block_split_any(x, a), block_split_any(y, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(at + i * plane) = a[i] | static_cast<uint32_t>(b[i]) << 16;
}
// Vector `which` of COUNT tokens from t0 on; -> whether all is in range.
template <int DP, int MODE, int COUNT, int SIZE>
__device__ __forceinline__ bool block_store_all(uint16_t* planes, int which, int t0, int r, const float2 (&x)[SIZE]) {
  using W = BlockShape<DP, MODE>;
  float most = 0.f;
#pragma unroll
  for (int t = 0; t < COUNT; ++t) block_store<DP, MODE>(planes, which, t0 + t, r, x[t].x, x[t].y, most);
  if (!block_out(most, kBlockVector)) return true;
#pragma unroll
  for (int t = 0; t < COUNT; ++t) block_store_again(planes + which * 3 * W::PLANE + block_at<DP>(t0 + t, r), W::PLANE, x[t].x, x[t].y);
  return false;
}
// The stage's sequence, its first token there and how many it has there.
struct BlockTokens {
  int start, count, all, sequence;
};
__device__ __forceinline__ BlockTokens block_tokens(const int* cu_seqlens, int seqs, int stage) {
  int b = 0;  // the last sequence whose stages begin no later
  for (int high = seqs; high - b > 1;) {
    const int middle = (b + high) >> 1;
    if (walk_base(cu_seqlens, middle) <= stage) b = middle;
    else high = middle;
  }
  const int first = (stage - walk_base(cu_seqlens, b)) * kWalkStage, start = cu_seqlens[b] + first;
  return {start, min(kWalkStage, cu_seqlens[b + 1] - start), cu_seqlens[b + 1] - cu_seqlens[b], b};
}
// Where token t, column c of a tile's 16 x 16 numbers lies, in the order the walk's lanes hold them.
__device__ __forceinline__ int block_lane_at(int t, int c) {
  return ((t >> 3) * 32 + (c & 7) * 4 + ((t & 7) >> 1)) * 4 + (c >> 3) * 2 + (t & 1);
}
__device__ __forceinline__ void block_copy(float* dst, const float* src) {  // 16 bytes, past L1
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src));
}
struct BlockPrepare {
  const float *q, *k, *v, *g, *head_decay, *beta, *look, *put;
  float *vectors, *scalars, *values;
  const int *cu_seqlens, *slots;
  int seqs, H, KH, d, dv;
  long long q_stride, v_stride;
  int aligned, least;
  WalkPiece piece;
};

__device__ __forceinline__ float2 block_fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 ra, rb, rc, rd; mov.b64 ra, {%2, %3}; mov.b64 rb, {%4, %5}; mov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc; mov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
// sum_{m <= j} square[j][m] x_m for all j; `square` holds every number twice, beside itself.
__device__ __forceinline__ void block_triangle(const float2 (*square)[kWalkStage], const float2 (&x)[kWalkStage], float2 (&y)[kWalkStage]) {
#pragma unroll
  for (int j = 0; j < kWalkStage; ++j) {
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 0; m <= j; m += 2) {
      const float4 two = *reinterpret_cast<const float4*>(&square[j][m]);
      sum = block_fma2(make_float2(two.x, two.y), x[m], sum);
      if (m + 1 <= j) sum = block_fma2(make_float2(two.z, two.w), x[m + 1], sum);
    }
    y[j] = sum;
  }
}
// Columns c and c + 1 of a stage's v.
__device__ __forceinline__ void block_values(const BlockPrepare& a, const BlockTokens& tokens, int h, int c, float2 (&x)[kWalkStage]) {
  const float* from = a.v + static_cast<size_t>(tokens.start) * a.v_stride + static_cast<size_t>(h) * a.dv + c;
#pragma unroll
  for (int j = 0; j < kWalkStage; ++j) {
    x[j].x = j < tokens.count && c < a.dv ? from[0] : 0.f;
    x[j].y = j < tokens.count && c + 1 < a.dv ? from[1] : 0.f;
    from += a.v_stride;
  }
}

// Two columns' numbers into a tile's part.
__device__ __forceinline__ void block_store_columns(float* to, int c, const float2 (&x)[kWalkStage]) {
#pragma unroll
  for (int j = 0; j < kWalkStage; j += 2) {
    *reinterpret_cast<float2*>(to + block_lane_at(j, c)) = make_float2(x[j].x, x[j + 1].x);
    *reinterpret_cast<float2*>(to + block_lane_at(j, c + 1)) = make_float2(x[j].y, x[j + 1].y);
  }
}

// Rules whose vectors are a head's own. A CTA per stage and head, a warp per eight tokens and part of the rows, RP rows a lane.
// What two tokens of different halves of a block have to do with one another is a product of the later's read (its decays from
// the ninth token on) and the earlier's write (up to it), so quotients of decays are made within the halves only. Bound by
// latency at some 10,000 warp instructions a CTA and four CTAs an SM: 2,064 CTAs of 128 x 128 54 us (a warp doing all of a stage and
// head alone 53 us with fewer instructions, but 14 us for a single one against 8).
template <int DP, int MODE>
struct BlockHead {
  using W = BlockShape<DP, MODE>;
  static constexpr int L = W::L, B = 8, PITCH = DP + 4, RP = DP > 128 ? 4 : 2, PARTS = DP / (32 * RP);
  float kx[W::DELTA ? L : 1][PITCH], qx[L][PITCH], wx[B][PITCH];  // each half's own reads; the first half's writes
  float own[2][DP];                                               // products of a half's decays
  float2 T[W::DELTA ? L : 1][L], D[L][L];                         // every number twice, beside itself
  float totals[L][L];                  // [later j][earlier m] the D of j on m, [m][j] the C of j on m
  float partials[2][PARTS][64], X[B][B], steps[L];
  int spoilt[4];
};
template <int DP, int MODE>
__global__ __launch_bounds__(128, DP > 128 ? 3 : 4) void block_prepare_head_kernel(BlockPrepare a) {
  using W = BlockShape<DP, MODE>;
  using S = BlockHead<DP, MODE>;
  constexpr bool DELTA = W::DELTA, BONUS = W::BONUS;
  constexpr int L = W::L, B = S::B, RP = S::RP, PARTS = S::PARTS;
  extern __shared__ __align__(16) unsigned char block_smem[];
  S& at_hand = *reinterpret_cast<S*>(block_smem);
  auto& totals = at_hand.totals;
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = tid >> 6, part = warp & 1;
  if (tid == 0) at_hand.spoilt[0] = 0;
  pdl_wait();
  const int stage = blockIdx.x, h = blockIdx.y, kh = h / (a.H / a.KH), d = a.d;
  const BlockTokens tokens = block_tokens(a.cu_seqlens, a.seqs, a.piece.first + stage);
  if (tokens.count <= 0 || tokens.all < a.least || (!a.piece.whole && a.slots[tokens.sequence] < 0)) return;
  float* to = a.vectors + (static_cast<size_t>(stage) * a.H + h) * W::STAGE;
  float* scalars = a.scalars + (static_cast<size_t>(stage) * a.H + h) * W::SCALARS;
  uint16_t* planes = reinterpret_cast<uint16_t*>(to);
  bool bad = false;
  float decay[B];  // MODE 5: of this half's tokens
#pragma unroll
  for (int j = 0; j < B; ++j) {
    const bool is = half * B + j < tokens.count;
    const size_t at = static_cast<size_t>(tokens.start + half * B + j) * a.H + h;
    decay[j] = MODE == 5 && is ? a.put[at] : 1.f;
    if (DELTA && part == 0 && lane == j) at_hand.steps[half * B + j] = is ? a.beta[at] : 0.f;
  }
  if (part < PARTS) {
    float sums[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) sums[i] = 0.f;
    const int r0 = (part * 32 + lane) * RP;
    const float *q_at = a.q + (tokens.start + half * B) * a.q_stride + static_cast<size_t>(kh) * d + r0, *k_at = a.k + (q_at - a.q);
    const float* g_at = MODE == 5 ? nullptr : a.g + (static_cast<size_t>(tokens.start + half * B) * a.H + h) * d + r0;
    float qr[B][RP], kr[B][RP], gr[B][RP];
#pragma unroll
    for (int j = 0; j < B; ++j) {  // a token the sequence does not have: nothing read or written, no decay
      const bool is = half * B + j < tokens.count;
      auto load = [&](const float* from, float other, float (&x)[RP]) {
        if (a.aligned) {
          const bool in = is && r0 < d;
          if (RP == 4) {
            const float4 y = in ? *reinterpret_cast<const float4*>(from) : make_float4(other, other, other, other);
            x[0] = y.x, x[1] = y.y, x[RP - 2] = y.z, x[RP - 1] = y.w;
          } else {
            const float2 y = in ? *reinterpret_cast<const float2*>(from) : make_float2(other, other);
            x[0] = y.x, x[1] = y.y;
          }
        } else {
#pragma unroll
          for (int e = 0; e < RP; ++e) x[e] = is && r0 + e < d ? from[e] : other;
        }
      };
      load(q_at, 0.f, qr[j]);
      load(k_at, 0.f, kr[j]);
      if (MODE != 5) load(g_at, 1.f, gr[j]);
      q_at += a.q_stride, k_at += a.q_stride, g_at += static_cast<size_t>(a.H) * d;
#pragma unroll
      for (int e = 0; e < RP; ++e)
        if (MODE == 5) gr[j][e] = decay[j];
    }
    float upto[RP], factor[RP];
#pragma unroll
    for (int e = 0; e < RP; ++e) upto[e] = 1.f, factor[e] = BONUS && r0 + e < d ? a.look[h * d + r0 + e] : 0.f;
#pragma unroll
    for (int j = 0; j < B; ++j)
#pragma unroll
      for (int e = 0; e < RP; e += 2) {
        const float2 before = make_float2(qr[j][e] * upto[e], qr[j][e + 1] * upto[e + 1]);
        upto[e] *= gr[j][e], upto[e + 1] *= gr[j][e + 1];
        *reinterpret_cast<float2*>(&at_hand.qx[half * B + j][r0 + e]) =
            BONUS ? before : make_float2(qr[j][e] * upto[e], qr[j][e + 1] * upto[e + 1]);
        if (DELTA) *reinterpret_cast<float2*>(&at_hand.kx[DELTA ? half * B + j : 0][r0 + e]) = make_float2(kr[j][e] * upto[e], kr[j][e + 1] * upto[e + 1]);
      }
#pragma unroll
    for (int e = 0; e < RP; e += 2) *reinterpret_cast<float2*>(&at_hand.own[half][r0 + e]) = make_float2(upto[e], upto[e + 1]);
#pragma unroll
    for (int e = 0; e < RP; ++e)
#pragma unroll
      for (int m = 0; m < B; ++m) {  // token m's write on its way through the tokens behind it
        float w = kr[m][e];
        sums[(B + 1) * m] += qr[m][e] * (BONUS ? factor[e] * w : w);
#pragma unroll
        for (int j = m + 1; j < B; ++j) {
          if (BONUS) sums[B * j + m] = fmaf(qr[j][e], w, sums[B * j + m]);
          w *= gr[j][e];
          if (!BONUS) sums[B * j + m] = fmaf(qr[j][e], w, sums[B * j + m]);
          if (DELTA) sums[B * m + j] = fmaf(kr[j][e], w, sums[B * m + j]);
        }
        kr[m][e] = w;
      }
#pragma unroll
    for (int e = 0; e < RP; e += 2) {
      float2 w[B];
#pragma unroll
      for (int m = 0; m < B; ++m) {
        w[m] = make_float2(kr[m][e], kr[m][e + 1]);
        if (half == 0) *reinterpret_cast<float2*>(&at_hand.wx[m][r0 + e]) = w[m];
      }
      if (half == 1) bad |= !block_store_all<DP, MODE, B>(planes, W::AT_W, B, r0 + e, w);
    }
    // sums over the rows: every exchange halves the sums a lane holds, down to two
#pragma unroll
    for (int n = 32, bit = 16; n >= 2; n >>= 1, bit >>= 1) {
      const bool high = (lane & bit) != 0;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float keep = high ? sums[i + n] : sums[i], give = high ? sums[i] : sums[i + n];
        sums[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
      }
    }
    *reinterpret_cast<float2*>(&at_hand.partials[half][part][lane * 2]) = make_float2(sums[0], sums[1]);
  }
  const int tiles = (a.dv + kBlockCols - 1) / kBlockCols;
  __syncthreads();
  {  // within the halves; and the last eight tokens (j) on the first eight (m)
    const int i = tid & 63, j = i / B, m = i % B;
    float total = at_hand.partials[half][0][i];
    if (PARTS > 1) total += at_hand.partials[half][PARTS - 1][i];
    totals[half * B + j][half * B + m] = total;
    if (DELTA || half == 0) {
      float2 sum = make_float2(0.f, 0.f), sum2 = sum;
      const float* reads = DELTA && half == 1 ? at_hand.kx[DELTA ? B + j : 0] : at_hand.qx[B + j];
#pragma unroll 8
      for (int r = 0; r < DP; r += 4) {
        const float4 w = *reinterpret_cast<const float4*>(&at_hand.wx[m][r]), z = *reinterpret_cast<const float4*>(reads + r);
        sum = block_fma2(make_float2(z.x, z.y), make_float2(w.x, w.y), sum), sum2 = block_fma2(make_float2(z.z, z.w), make_float2(w.z, w.w), sum2);
      }
      (half == 0 ? totals[B + j][m] : totals[m][B + j]) = (sum.x + sum.y) + (sum2.x + sum2.y);
    }
  }
  __syncthreads();
  auto& D = at_hand.D;
  if (DELTA && warp == 0) {
    auto& T = at_hand.T;
    if (lane < L) {  // column m of a half's T, by substitution
      const int m = lane % B, at = lane - m;
      float column[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        float sum = 0.f;
#pragma unroll
        for (int n = 0; n < j; ++n)
          if (n >= m) sum = fmaf(totals[at + n][at + j], column[n], sum);
        column[j] = j == m ? at_hand.steps[at + j] : j > m ? -at_hand.steps[at + j] * sum : 0.f;
        T[at + j][at + m] = make_float2(column[j], column[j]);
      }
    }
    __syncwarp();
    // the later half's T on the earlier half: -T_2 C T_1
#pragma unroll
    for (int i = lane; i < B * B; i += 32) {
      const int j = i / B, m = i % B;
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < B; ++n)
        if (n >= m) sum = fmaf(totals[n][B + j], T[n][m].x, sum);
      at_hand.X[j][m] = sum;
    }
    __syncwarp();
#pragma unroll
    for (int i = lane; i < B * B; i += 32) {
      const int j = i / B, m = i % B;
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < B; ++n)
        if (n <= j) sum = fmaf(T[B + j][B + n].x, at_hand.X[n][m], sum);
      T[B + j][m] = make_float2(-sum, -sum);
    }
  } else {  // meanwhile: D; the first half's writes as the block's end finds them; the block's decays
    constexpr int first = DELTA ? 32 : 0, threads = 128 - first;
    for (int i = tid - first; i < L * L; i += threads) {
      const float z = i % L <= i / L ? totals[i / L][i % L] : 0.f;
      D[i / L][i % L] = make_float2(z, z);
    }
    for (int i = tid - first; i < DP; i += threads) {  // two rows, half of the tokens
      const int r = i >> 1 << 1, m0 = (i & 1) * (B / 2);
      const float2 early = *reinterpret_cast<const float2*>(&at_hand.own[0][r]), late = *reinterpret_cast<const float2*>(&at_hand.own[1][r]);
      if (W::ROW_DECAY && m0 == 0) {
        const float2 both = make_float2(early.x * late.x, early.y * late.y);
        *reinterpret_cast<float2*>(to + W::AT_G + r) = both;
        bad |= fmaf(both.x, 0.f, both.y * 0.f) != 0.f;
      }
      float2 w[B / 2];
#pragma unroll
      for (int m = 0; m < B / 2; ++m) {
        w[m] = *reinterpret_cast<const float2*>(&at_hand.wx[m0 + m][r]);
        w[m].x *= late.x, w[m].y *= late.y;
      }
      bad |= !block_store_all<DP, MODE, B / 2>(planes, W::AT_W, m0, r, w);
    }
  }
  float2 x[L], y[L];  // two rows or columns: the first two warps have the rows, the others the columns
  const int mine = (tid & 63) * 2;
  if (half == 1) block_values(a, tokens, h, mine, x);
  __syncthreads();
  if (half == 0) {  // K' = T k G, Q' = q G - D K'
#pragma unroll 1
    for (int r = mine; r < DP; r += 128) {
      const float2 early = *reinterpret_cast<const float2*>(&at_hand.own[0][r]);
      if constexpr (DELTA) {
#pragma unroll
        for (int j = 0; j < L; ++j) {
          x[j] = *reinterpret_cast<const float2*>(&at_hand.kx[j][r]);
          if (j >= B) x[j].x *= early.x, x[j].y *= early.y;
        }
        block_triangle(at_hand.T, x, y);
        bad |= !block_store_all<DP, MODE, L>(planes, W::AT_K, 0, r, y);
        block_triangle(D, y, x);
      }
#pragma unroll
      for (int j = 0; j < L; ++j) {
        y[j] = *reinterpret_cast<const float2*>(&at_hand.qx[j][r]);
        if (j >= B) y[j].x *= early.x, y[j].y *= early.y;
        if (DELTA) y[j].x -= x[j].x, y[j].y -= x[j].y;
      }
      bad |= !block_store_all<DP, MODE, L>(planes, W::AT_Q, 0, r, y);
    }
  } else {  // T v (or v), and its product with D, which the read-outs begin with
#pragma unroll 1
    for (int c = mine; c < tiles * kBlockCols; c += 128) {
      float* tile = a.values + ((static_cast<size_t>(stage) * a.H + h) * tiles + c / kBlockCols) * W::TILE;
      if (c != mine) block_values(a, tokens, h, c, x);
      if constexpr (DELTA) {
        block_triangle(at_hand.T, x, y);
        block_store_columns(tile, c % kBlockCols, y);
        block_triangle(D, y, x);
        block_store_columns(tile + W::TILE / 2, c % kBlockCols, x);
      } else {
        block_store_columns(tile, c % kBlockCols, x);
        block_triangle(D, x, y);
        block_store_columns(tile + W::TILE / 2, c % kBlockCols, y);
      }
    }
  }
  if (bad) at_hand.spoilt[0] = 1;
  __syncthreads();
  if (tid < L) scalars[tid] = 1.f;  // (in the vectors already)
  if (tid == 0) {
    float upto = 1.f, lost = 0.f;
    if (MODE == 5) {
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const float z = j < tokens.count ? a.put[static_cast<size_t>(tokens.start + j) * a.H + h] : 1.f, next = upto * z;
        lost = fmaf(lost, z, fmaf(upto, z, -next)), upto = next;
      }
    }
    scalars[W::AT_ALL] = upto, scalars[W::AT_ALL + 1] = lost;
    scalars[W::AT_BAD] = at_hand.spoilt[0] || !isfinite(upto) ? 1.f : 0.f, scalars[W::AT_BAD + 1] = 0.f;
  }
}

// One decay a token, and nothing read before it is written: the bare keys and queries are shared by a key head's heads. A CTA
// per stage, key head and kBlockHeads heads.
constexpr int kBlockHeads = 4;
template <int DP, int MODE>
__global__ __launch_bounds__(128) void block_prepare_shared_kernel(BlockPrepare a) {
  using W = BlockShape<DP, MODE>;
  constexpr int L = W::L, PITCH = DP + 4, PAIRS = DP / 2;
  __shared__ __align__(16) float rows[2 * L][PITCH];  // the keys, the queries
  __shared__ __align__(16) float2 D[kBlockHeads][L][L];
  __shared__ float totals[L][L], rests[kBlockHeads][L];
  __shared__ int spoilt;
  pdl_trigger();
  if (threadIdx.x == 0) spoilt = 0;
  pdl_wait();
  const int stage = blockIdx.x, kh = blockIdx.y, per_key = a.H / a.KH, d = a.d, tid = threadIdx.x;
  const BlockTokens tokens = block_tokens(a.cu_seqlens, a.seqs, a.piece.first + stage);
  if (tokens.count <= 0 || tokens.all < a.least || (!a.piece.whole && a.slots[tokens.sequence] < 0)) return;
  __syncthreads();
  const int head0 = blockIdx.z * kBlockHeads, heads = min(kBlockHeads, per_key - head0);
  float decay[L];  // of the thread's head (a thread per head and earlier token m)
  const int m = tid % L, hh = tid / L, h = kh * per_key + head0 + min(hh, heads - 1);
#pragma unroll
  for (int j = 0; j < L; ++j)
    decay[j] = j < tokens.count ? (MODE == 0 ? a.head_decay[h] : a.beta[static_cast<size_t>(tokens.start + j) * a.H + h]) : 1.f;
  uint16_t* planes = reinterpret_cast<uint16_t*>(a.vectors + (static_cast<size_t>(stage) * a.KH + kh) * W::STAGE);
  float most = 0.f;
  constexpr int PER = 2 * L * PAIRS / 128;
  float2 both[PER];
#pragma unroll
  for (int n = 0; n < PER; ++n) {
    const int i = tid + n * 128, row = i / PAIRS, j = row % L, r = i % PAIRS * 2;
    const float* from = (row < L ? a.k : a.q) + static_cast<size_t>(tokens.start + j) * a.q_stride + static_cast<size_t>(kh) * d + r;
    both[n] = make_float2(0.f, 0.f);
    if (j < tokens.count && a.aligned) {
      if (r < d) both[n] = *reinterpret_cast<const float2*>(from);
    } else if (j < tokens.count) {
      both[n] = make_float2(r < d ? from[0] : 0.f, r + 1 < d ? from[1] : 0.f);
    }
  }
#pragma unroll
  for (int n = 0; n < PER; ++n) {
    const int i = tid + n * 128, row = i / PAIRS, j = row % L, r = i % PAIRS * 2, which = row < L ? W::AT_K : W::AT_Q;
    *reinterpret_cast<float2*>(&rows[row][r]) = both[n];
    if (blockIdx.z == 0) block_store<DP, MODE>(planes, which, j, r, both[n].x, both[n].y, most);
    else block_most(most, both[n].x), block_most(most, both[n].y);
  }
  if (block_out(most, kBlockVector)) {
    spoilt = 1;
    if (blockIdx.z == 0) {
#pragma unroll
      for (int n = 0; n < PER; ++n) {
        const int i = tid + n * 128, row = i / PAIRS, which = row < L ? W::AT_K : W::AT_Q;
        block_store_again(planes + which * 3 * W::PLANE + block_at<DP>(row % L, i % PAIRS * 2), W::PLANE, both[n].x, both[n].y);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const int j = tid / L + 8 * n;
    float2 sum = make_float2(0.f, 0.f), sum2 = sum;
    if (m <= j) {
#pragma unroll 8
      for (int i = 0; i < DP; i += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&rows[L + j][i]), w = *reinterpret_cast<const float4*>(&rows[m][i]);
        sum = block_fma2(make_float2(x.x, x.y), make_float2(w.x, w.y), sum), sum2 = block_fma2(make_float2(x.z, x.w), make_float2(w.z, w.w), sum2);
      }
    }
    totals[j][m] = (sum.x + sum.y) + (sum2.x + sum2.y);
  }
  __syncthreads();
  if (hh < heads) {
    float upto = 1.f, lost = 0.f, behind = 1.f, gone = 0.f, rest = 1.f, mine = 1.f;  // products with what their rounding lost
#pragma unroll
    for (int j = 0; j < L; ++j) {
      const float x = decay[j], next = upto * x;
      lost = fmaf(lost, x, fmaf(upto, x, -next)), upto = next;
      if (j == m) mine = isfinite(lost) ? upto + lost : upto;
      if (j > m) {
        const float more = behind * x;
        gone = fmaf(gone, x, fmaf(behind, x, -more)), behind = more;
        rest = isfinite(gone) ? behind + gone : behind;
      }
      const float value = j >= m ? totals[j][m] * rest : 0.f;
      D[hh][j][m] = make_float2(value, value);
    }
    rests[hh][m] = rest;
    float* scalars = a.scalars + (static_cast<size_t>(stage) * a.H + h) * W::SCALARS;
    scalars[m] = mine;
    if (m == 0) {
      scalars[W::AT_ALL] = upto, scalars[W::AT_ALL + 1] = lost;
      scalars[W::AT_BAD] = spoilt || !isfinite(upto) ? 1.f : 0.f, scalars[W::AT_BAD + 1] = 0.f;
    }
  }
  __syncthreads();
  const int tiles = (a.dv + kBlockCols - 1) / kBlockCols, pairs = tiles * kBlockCols / 2;
#pragma unroll 1
  for (int i = tid; i < heads * pairs; i += 128) {
    const int head = i / pairs, c = i % pairs * 2;
    float* tile = a.values + ((static_cast<size_t>(stage) * a.H + kh * per_key + head0 + head) * tiles + c / kBlockCols) * W::TILE;
    float2 x[L], y[L];
    block_values(a, tokens, kh * per_key + head0 + head, c, x);
    block_triangle(D[head], x, y);
    block_store_columns(tile + W::TILE / 2, c % kBlockCols, y);
#pragma unroll
    for (int j = 0; j < L; ++j) x[j].x *= rests[head][j], x[j].y *= rests[head][j];  // as the block's end finds it
    block_store_columns(tile, c % kBlockCols, x);
  }
}

// c (+)= a b; the first product of a sum begins from zero.
template <bool FIRST>
__device__ __forceinline__ void block_mma(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  if (FIRST)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
template <bool TRANSPOSED>
__device__ __forceinline__ void block_ldmatrix(uint32_t (&r)[4], const uint16_t* at) {
  const uint32_t from = static_cast<uint32_t>(__cvta_generic_to_shared(at));
  if (TRANSPOSED)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(from) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(from) : "memory");
}

// A 16 x 16 operand's three parts, from the accumulators of two 16 x 8 products.
struct BlockParts {
  uint4 part[3];
  __device__ __forceinline__ void cut(const float (&x)[4], const float (&y)[4]) {
    block_split(x[0], x[1], part[0].x, part[1].x, part[2].x);
    block_split(x[2], x[3], part[0].y, part[1].y, part[2].y);
    block_split(y[0], y[1], part[0].z, part[1].z, part[2].z);
    block_split(y[2], y[3], part[0].w, part[1].w, part[2].w);
  }
};

// COUNT (1 or 2) 16 x 8 products of a 16 x 16 operand x, side by side, all products of parts but the two low ones: the large one
// into `large`, the small ones into `small`. `b`: the second operand's parts, for the products in turn, from `at` on.
template <bool FIRST, int COUNT>
__device__ __forceinline__ void block_products(float (&large)[COUNT][4], float (&small)[COUNT][4], const BlockParts& x, const uint32_t (&b)[3][4],
                                               int at = 0) {
  constexpr int of_x[7] = {1, 2, 2, 0, 1, 1, 0}, of_b[7] = {2, 1, 0, 2, 1, 0, 1};
#pragma unroll
  for (int p = 0; p < 7; ++p) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
      if (FIRST && p == 0) block_mma<true>(small[i], x.part[of_x[p]], b[of_b[p]][at + 2 * i], b[of_b[p]][at + 2 * i + 1]);
      else block_mma<false>(small[i], x.part[of_x[p]], b[of_b[p]][at + 2 * i], b[of_b[p]][at + 2 * i + 1]);
    }
    if (p == 0) {
#pragma unroll
      for (int i = 0; i < COUNT; ++i) block_mma<FIRST>(large[i], x.part[0], b[0][at + 2 * i], b[0][at + 2 * i + 1]);
    }
  }
}

template <int DP, int MODE>
struct BlockWalk {
  using W = BlockShape<DP, MODE>;
  static constexpr int AT_TILE = W::STAGE + W::SCALARS, BUFFER = AT_TILE + W::TILE;  // a stage's vectors | numbers | tile
  static constexpr int STATE = 3 * DP * kBlockCols / 2;                              // the state's parts
  static constexpr int SHARES = 2 * 4 * 256, HALVES = 2 * 32 * 4;                   // of p; of the read-outs
  static constexpr size_t bytes(int buffers) {
    return sizeof(float) * (static_cast<size_t>(buffers) * BUFFER + 2 * STATE + (W::DELTA ? SHARES : 512) + HALVES + 4);
  }
  static_assert(STATE >= kBlockCols * (DP + 4), "room for the state as it is, for columns that are done once more");
};

// What eight neighbouring threads of a column do with float32 FMAs where a number is out of range.
template <int DP, int MODE>
struct BlockAgain {
  using W = BlockShape<DP, MODE>;
  const float *vectors, *scalars;
  __device__ __forceinline__ float vector(int which, int t, int r) const {
    return block_join(reinterpret_cast<const uint16_t*>(vectors) + which * 3 * W::PLANE + block_at<DP>(t, r), W::PLANE);
  }
  // Token t's read of the state `held` through vector `which`.
  __device__ __noinline__ float read(int which, int t, const float* held) const {
    float sum = 0.f;
    for (int r = threadIdx.x & 7; r < DP; r += 8) sum = fmaf(vector(which, t, r), held[r], sum);
    const unsigned lanes = 0xffu << (threadIdx.x & 24);
    for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(lanes, sum, o);
    return W::BY_HEAD ? sum : sum * scalars[t];
  }
  // The state behind a block of `count` tokens that write u.
  __device__ __noinline__ void move(float* held, const float* u, int count) const {
    for (int r = threadIdx.x & 7; r < DP; r += 8) {
      float next = !W::ROW_DECAY && isfinite(held[r]) ? held[r] * scalars[W::AT_ALL + 1] : 0.f;
      for (int m = 0; m < count; ++m) next = fmaf(vector(W::AT_W, m, r), u[m], next);
      held[r] = fmaf(held[r], W::ROW_DECAY ? vectors[W::AT_G + r] : scalars[W::AT_ALL], next);
    }
  }
};

// ALL: of a step in one piece whose tokens let every sequence walk, sequence z; else the z-th that walks, and what of it the
// piece holds. BUFFERS: stages in shared memory; with three the next one has arrived at the barrier in the middle of a block,
// with two a second barrier at its beginning waits for it.
template <int DP, int MODE, bool ALL, int BUFFERS>
__global__ __launch_bounds__(256, DP > 128 ? 1 : 2) void block_scan_kernel(
    const float* vectors_at, const float* scalars_at, const float* values_at, float* __restrict__ state, float* __restrict__ out,
    const int* __restrict__ cu_seqlens, const int* __restrict__ slots, int seqs, int H, int KH, int d, int dv, int least, WalkPiece piece) {
  using W = BlockShape<DP, MODE>;
  using K = BlockWalk<DP, MODE>;
  constexpr int L = W::L, STEPS = DP / 64, ROWS = DP / 4, HP = DP + 4;  // products along a state warp's rows; its rows
  constexpr bool DELTA = W::DELTA, ROW_DECAY = W::ROW_DECAY, BY_HEAD = W::BY_HEAD;
  extern __shared__ __align__(16) float smem[];
  float* parts_at = smem + BUFFERS * K::BUFFER;             // [2][16 rows of the state each][3][32 lanes][4 pairs]
  float* shares = parts_at + 2 * K::STATE;                  // [2][4 warps][2][32 lanes][4]
  float* halves = shares + (DELTA ? K::SHARES : 512);       // [2][32 lanes][4]
  int* state_bad = reinterpret_cast<int*>(halves + K::HALVES);  // [2] the block whose state is out of range
  const int h = blockIdx.y, b = ALL ? blockIdx.z : walking_sequence(cu_seqlens, seqs, least, blockIdx.z);
  const int vh = BY_HEAD ? h : h / (H / KH), VH = BY_HEAD ? H : KH, col0 = blockIdx.x * kBlockCols;
  if (!ALL && b < 0) return;
  int start = cu_seqlens[b], n = cu_seqlens[b + 1] - start, base_stage = walk_base(cu_seqlens, b);
  const int slot = slots[b];
  if (n < least || n <= 0) return;
  if (!ALL) {  // the part of the sequence in this launch, as a sequence of its own whose first stage lies at base_stage
    const int skipped = max(0, piece.first - base_stage) * L;
    base_stage = max(0, base_stage - piece.first), start += skipped;
    n = min(n - skipped, (piece.count - base_stage) * L);
    if (n <= 0 || (!piece.whole && slot < 0)) return;
  }
  const int stages = (n + L - 1) / L;
  const int tid = threadIdx.x & 127, lane = threadIdx.x & 31, warp = tid >> 5, gid = lane >> 2, tig = lane & 3;
  const bool reader = threadIdx.x >= 128;
  if (threadIdx.x < 2) state_bad[threadIdx.x] = -1;

  // The readers bring the stages.
  const float* next_vectors = vectors_at + (static_cast<size_t>(base_stage) * VH + vh) * W::STAGE + tid * 4;
  const float* next_scalars = scalars_at + (static_cast<size_t>(base_stage) * H + h) * W::SCALARS + tid * 4;
  const float* next_tile = values_at + ((static_cast<size_t>(base_stage) * H + h) * gridDim.x + blockIdx.x) * W::TILE + tid * 4;
  float *next_to = smem, *const end_to = smem + BUFFERS * K::BUFFER;
  int left = stages;
  auto issue = [&]() {
    if (left > 0) {
      constexpr int WHOLE = W::STAGE / 512;
#pragma unroll
      for (int i = 0; i < WHOLE; ++i) block_copy(next_to + tid * 4 + i * 512, next_vectors + i * 512);
      if (W::STAGE % 512 && tid * 4 < W::STAGE % 512) block_copy(next_to + tid * 4 + WHOLE * 512, next_vectors + WHOLE * 512);
      if (tid * 4 < W::SCALARS) block_copy(next_to + W::STAGE + tid * 4, next_scalars);
      block_copy(next_to + K::AT_TILE + tid * 4, next_tile);
      static_assert(W::TILE == 512, "a piece a thread");
      next_tile += static_cast<size_t>(H) * gridDim.x * W::TILE;
      next_vectors += static_cast<size_t>(VH) * W::STAGE, next_scalars += static_cast<size_t>(H) * W::SCALARS;
      next_to += K::BUFFER;
      if (next_to == end_to) next_to = smem;
    }
    --left;
    asm volatile("cp.async.commit_group;\n" ::);
  };
  const float* at_stage = smem;  // this block's stage
  auto advance = [&]() {
    at_stage += K::BUFFER;
    if (at_stage == end_to) at_stage = smem;
  };

  if (reader) {
#pragma unroll
    for (int i = 0; i < BUFFERS - 1; ++i) issue();
    if (BUFFERS > 2) asm volatile("cp.async.wait_group %0;\n" ::"n"(BUFFERS - 2));
    if (BUFFERS > 2) __syncthreads();
    // warp: one of two 8 tokens, one of two halves of the state's rows
    const int eight = warp & 1, half = warp >> 1, token = eight * 8 + (lane & 7);
    float* mine = out + (static_cast<size_t>(start + eight * 8 + 2 * tig) * H + h) * dv + col0 + gid;  // [token of two][column of two]
    const size_t token_step = static_cast<size_t>(H) * dv;
    for (int block = 0; block < stages; ++block, mine += L * token_step) {
      if (BUFFERS == 2) {
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();  // this stage is here for every thread
      } else {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(BUFFERS - 3));
      }
      __syncthreads();  // the state's parts are here, and the stage of the block before is free
      issue();
      const float* scalars = at_stage + W::STAGE;
      const int t0 = block * L + eight * 8 + 2 * tig;
      if (scalars[W::AT_BAD] != 0.f || state_bad[block & 1] == block) {
        const float* held = parts_at + ((block + 1) & 1) * K::STATE + (tid >> 3) * HP;
        __syncthreads();  // the state as it is
        const BlockAgain<DP, MODE> again{at_stage, scalars};
        const int c = col0 + (tid >> 3);
        for (int t = 0; t < min(L, n - block * L); ++t) {
          const float sum = again.read(W::AT_Q, t, held);
          if ((tid & 7) == 0 && c < dv) out[(static_cast<size_t>(start + block * L + t) * H + h) * dv + c] =
              sum + at_stage[K::AT_TILE + W::TILE / 2 + block_lane_at(t, tid >> 3)];
        }
        __syncthreads();  // (before the state moves on)
        advance();
        continue;
      }
      const uint16_t* planes = reinterpret_cast<const uint16_t*>(at_stage) + W::AT_Q * 3 * W::PLANE + token * DP;
      const uint4* parts = reinterpret_cast<const uint4*>(parts_at + (block & 1) * K::STATE) + lane;
      float large[2][4], small[2][4];
#pragma unroll
      for (int s = 0; s < 2 * STEPS; s += 2) {
        const int step = half * 2 * STEPS + s;
        uint32_t operand[3][4];
        const int at = ((2 * step + (lane >> 3)) ^ (token & 7)) << 3;
#pragma unroll
        for (int i = 0; i < 3; ++i) block_ldmatrix<false>(operand[i], planes + i * W::PLANE + at);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          BlockParts x;
#pragma unroll
          for (int i = 0; i < 3; ++i) x.part[i] = parts[((step + e) * 3 + i) * 32];
          float(&l)[1][4] = reinterpret_cast<float(&)[1][4]>(large[e]), (&m)[1][4] = reinterpret_cast<float(&)[1][4]>(small[e]);
          if (s == 0) block_products<true, 1>(l, m, x, operand, 2 * e);
          else block_products<false, 1>(l, m, x, operand, 2 * e);
        }
      }
      float sum[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) sum[e] = ((large[0][e] + large[1][e]) + (small[0][e] + small[1][e])) * kBlockBack;
      float4* meet = reinterpret_cast<float4*>(halves) + eight * 32 + lane;
      if (half == 1) *meet = make_float4(sum[0], sum[1], sum[2], sum[3]);
      asm volatile("bar.sync %0, 64;" ::"r"(1 + eight) : "memory");
      if (half == 0) {
        const float4 other = *meet, begun = *reinterpret_cast<const float4*>(at_stage + K::AT_TILE + W::TILE / 2 + (eight * 32 + lane) * 4);
        const float all[4] = {begun.x, begun.y, begun.z, begun.w};
        sum[0] += other.x, sum[1] += other.y, sum[2] += other.z, sum[3] += other.w;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (!BY_HEAD) sum[e] *= scalars[eight * 8 + 2 * tig + (e & 1)];
          if (t0 + (e & 1) < n && col0 + gid + (e >> 1) * 8 < dv) mine[(e & 1) * token_step + (e >> 1) * 8] = all[e] + sum[e];
        }
      }
      advance();
    }
    return;
  }

  // S[t][e]: columns gid (e < 2) and gid + 8 of rows warp * ROWS + 8 t + 2 tig + (e & 1)
  float S[2 * STEPS][4];
  float* mine = slot >= 0 ? state + (static_cast<size_t>(slot) * H + h) * d * dv : nullptr;
#pragma unroll
  for (int t = 0; t < 2 * STEPS; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = warp * ROWS + 8 * t + 2 * tig + (e & 1), j = col0 + gid + (e >> 1) * 8;
      S[t][e] = mine != nullptr && row < d && j < dv ? mine[static_cast<size_t>(row) * dv + j] : 0.f;
    }
  const int along_t = (lane >> 4) * 8 + (lane & 7), along_c = warp * ROWS / 8 + ((lane >> 3) & 1);
  const int across_t = ((lane >> 3) & 1) * 8 + (lane & 7), across_c = warp * ROWS / 8 + (lane >> 4);
  // The state's parts, ahead of `block`, for its readers; whether it is in range; and under the delta rules the share of this
  // warp's rows in what the block's tokens read.
  auto present = [&](int block) {
    uint4* to = reinterpret_cast<uint4*>(parts_at + (block & 1) * K::STATE) + warp * STEPS * 3 * 32 + lane;
    const uint16_t* planes = reinterpret_cast<const uint16_t*>(at_stage) + along_t * DP;
    float large[2][4], small[2][4];
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      BlockParts x;
      x.cut(S[2 * s], S[2 * s + 1]);
#pragma unroll
      for (int i = 0; i < 3; ++i) to[(s * 3 + i) * 32] = x.part[i];
      if (DELTA) {
        uint32_t operand[3][4];
        const int at = ((along_c + 2 * s) ^ (along_t & 7)) << 3;
#pragma unroll
        for (int i = 0; i < 3; ++i) block_ldmatrix<false>(operand[i], planes + i * W::PLANE + at);
        if (s == 0) block_products<true, 2>(large, small, x, operand);
        else block_products<false, 2>(large, small, x, operand);
      }
    }
    float most[2] = {0.f, 0.f};
#pragma unroll
    for (int t = 0; t < 2 * STEPS; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) block_most(most[e & 1], S[t][e]);
    if (block_out(most[0], kBlockState) || block_out(most[1], kBlockState)) state_bad[block & 1] = block;
    if (DELTA) {
      float4* share = reinterpret_cast<float4*>(shares + ((block & 1) * 4 + warp) * 256) + lane;
#pragma unroll
      for (int i = 0; i < 2; ++i)
        share[i * 32] = make_float4((large[i][0] + small[i][0]) * kBlockBack, (large[i][1] + small[i][1]) * kBlockBack,
                                    (large[i][2] + small[i][2]) * kBlockBack, (large[i][3] + small[i][3]) * kBlockBack);
    }
  };
  auto again_state = [&](float* held) {
#pragma unroll
    for (int t = 0; t < 2 * STEPS; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) held[(gid + (e >> 1) * 8) * HP + warp * ROWS + 8 * t + 2 * tig + (e & 1)] = S[t][e];
  };
  auto take_state = [&](const float* held) {
#pragma unroll
    for (int t = 0; t < 2 * STEPS; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[t][e] = held[(gid + (e >> 1) * 8) * HP + warp * ROWS + 8 * t + 2 * tig + (e & 1)];
  };
  auto states_meet = []() { asm volatile("bar.sync 3, 128;" ::: "memory"); };
  const int again_c = tid >> 3;  // the column this thread helps to do once more

  if (BUFFERS > 2) __syncthreads();  // the first stage is here
  for (int block = 0; block < stages; ++block) {
    if (BUFFERS == 2) __syncthreads();
    present(block);
    __syncthreads();
    const float* scalars = at_stage + W::STAGE;
    float* held = parts_at + ((block + 1) & 1) * K::STATE;
    const int count = min(L, n - block * L);
    if (scalars[W::AT_BAD] != 0.f || state_bad[block & 1] == block) {
      again_state(held);
      __syncthreads();
      const BlockAgain<DP, MODE> again{at_stage, scalars};
      float writes[L];
#pragma unroll 1
      for (int t = 0; t < L; ++t) {
        writes[t] = at_stage[K::AT_TILE + block_lane_at(t, again_c)];
        if (DELTA) writes[t] -= again.read(W::AT_K, t, held + again_c * HP);
      }
      __syncthreads();
      again.move(held + again_c * HP, writes, count);
      states_meet();
      take_state(held);
      states_meet();
    } else {
      float u[2][4];  // u[i][e]: column gid (e < 2) or gid + 8, token 8 i + 2 tig + (e & 1)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(at_stage + K::AT_TILE + (i * 32 + lane) * 4);
        u[i][0] = x.x, u[i][1] = x.y, u[i][2] = x.z, u[i][3] = x.w;
      }
      if (DELTA) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4* from = reinterpret_cast<const float4*>(shares + (block & 1) * 4 * 256) + i * 32 + lane;
          const float4 x = from[0], y = from[64], z = from[128], w = from[192];
          u[i][0] -= (x.x + y.x) + (z.x + w.x), u[i][1] -= (x.y + y.y) + (z.y + w.y);
          u[i][2] -= (x.z + y.z) + (z.z + w.z), u[i][3] -= (x.w + y.w) + (z.w + w.w);
        }
      }
      float most = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) block_most(most, u[0][e]), block_most(most, u[1][e]);
      const bool spoilt = __any_sync(0xffffffffu, block_out(most, kBlockState));  // the same in all four warps
      float* writes = shares + ((block + 1) & 1) * (DELTA ? 4 * 256 : 256);
      if (spoilt) {
        again_state(held);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (warp == 0) writes[(gid + (e >> 1) * 8) * L + 8 * i + 2 * tig + (e & 1)] = u[i][e];
            if (block_out(u[i][e], kBlockState)) u[i][e] = 0.f;
          }
        states_meet();
        bool mine_spoilt = false;
        for (int t = 0; t < count; ++t) mine_spoilt = mine_spoilt || block_out(writes[again_c * L + t], kBlockState);
        const BlockAgain<DP, MODE> again{at_stage, scalars};
        if (mine_spoilt) again.move(held + again_c * HP, writes + again_c * L, count);
        states_meet();
      }
      BlockParts x;
      x.cut(u[0], u[1]);
      const uint16_t* planes = reinterpret_cast<const uint16_t*>(at_stage) + W::AT_W * 3 * W::PLANE + across_t * DP;
#pragma unroll
      for (int s = 0; s < STEPS; ++s) {
        uint32_t operand[3][4];
        const int at = ((across_c + 2 * s) ^ (across_t & 7)) << 3;
#pragma unroll
        for (int i = 0; i < 3; ++i) block_ldmatrix<true>(operand[i], planes + i * W::PLANE + at);
        float large[2][4], small[2][4];
        block_products<true, 2>(large, small, x, operand);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float2 decay;
          if (ROW_DECAY) decay = *reinterpret_cast<const float2*>(at_stage + W::AT_G + warp * ROWS + 16 * s + 8 * i + 2 * tig);
          else decay.x = decay.y = scalars[W::AT_ALL];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float& y = S[2 * s + i][e];
            float more = (large[i][e] + small[i][e]) * kBlockBack;
            if (!ROW_DECAY) more = fmaf(y, scalars[W::AT_ALL + 1], more);
            y = fmaf(y, e & 1 ? decay.y : decay.x, more);
          }
        }
      }
      if (spoilt) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          bool lost = false;
          for (int t = 0; t < count; ++t) lost = lost || block_out(writes[(gid + 8 * c) * L + t], kBlockState);
          if (lost) {
#pragma unroll
            for (int t = 0; t < 2 * STEPS; ++t)
#pragma unroll
              for (int e = 0; e < 2; ++e) S[t][2 * c + e] = held[(gid + 8 * c) * HP + warp * ROWS + 8 * t + 2 * tig + e];
          }
        }
        states_meet();
      }
    }
    advance();
  }
  if (mine != nullptr) {
#pragma unroll
    for (int t = 0; t < 2 * STEPS; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = warp * ROWS + 8 * t + 2 * tig + (e & 1), j = col0 + gid + (e >> 1) * 8;
        if (row < d && j < dv) mine[static_cast<size_t>(row) * dv + j] = S[t][e];
      }
  }
}

// Whether a step may hold sequences that go this way: heads of up to 256. Which ones do is decided by each sequence's own
// tokens, in the kernels, so that its bits do not hang on the lengths of the others.
inline bool takes_walk(int d, int tokens) { return tokens >= kWalkTokens && d <= 256; }
inline int walking(int seqs, int tokens) { return seqs < tokens / kWalkTokens ? seqs : tokens / kWalkTokens; }  // at most
// CTAs of the step's walks, for the choice of the way and its layout: as many whole walks as its tokens would make of the longest
// one, which is what the step waits for. Where that is not known: all sequences where they bring kWalkTokens on average, else one.
// us, counted so and by how many sequences could walk at most: 2,048 tokens beside 31 sequences of one, delta rule, 8 heads of 128 x 128
// 200 and 361 (alone 181), head decay with a delta, 16 heads 241 and 544 (210), a bonus 206 and 329 (165); 297 beside three of one 52 and 95.
inline long long walk_ctas(int seqs, int H, int dv, int tokens, int longest) {
  const long long one = static_cast<long long>((dv + kBlockCols - 1) / kBlockCols) * H;
  if (longest > 0) return longest < tokens ? one * tokens / longest : one;
  return tokens >= static_cast<long long>(seqs) * kWalkTokens ? one * seqs : one;
}

// Floats of a stage in the workspace: its vectors, its numbers per head, and its tiles' (each behind those of all stages).
template <int MODE>
long long block_vectors(int H, int KH, int d) {
  const int padded = walk_padded(d);
  const int stage = padded == 256 ? BlockShape<256, MODE>::STAGE : padded == 128 ? BlockShape<128, MODE>::STAGE : BlockShape<64, MODE>::STAGE;
  return static_cast<long long>(BlockShape<64, MODE>::BY_HEAD ? H : KH) * stage;
}
template <int MODE>
long long block_stage_floats(int H, int KH, int d, int dv) {
  const long long tiles = (dv + kBlockCols - 1) / kBlockCols;
  return block_vectors<MODE>(H, KH, d) + H * (BlockShape<64, MODE>::SCALARS + tiles * BlockShape<64, MODE>::TILE);
}

// Whether the step goes with float32 FMAs (recurrent_walk.cuh): once its CTAs pass what the SMs hold at once the preparation per
// head weighs more. us, tensor cores and FMAs, n sequences of so many tokens (CTAs): delta rule, 16 heads of 128 x 128, two of 600 (256)
// 126 and 122, three of 1,024 (384) 304 and 310, four (512) 361 and 318; head decay with a delta 126 and 167, 306 and 335, 372 and
// 341; a bonus, 32 heads of 64 x 64, three of 600 (384) 110 and 103, four (512) 134 and 110; one decay a token, 16 heads of 128 x 128, four of
// 1,024 (512) 263 and 249, five of 600 (640) 210 and 230, eight of 600 (1,024) 294 and 292, eight of 1,024 521 and 472 (the FMAs' CTAs have 32
// columns, two to an SM, and fill the SMs once at 592 of 16; sequences whose longest is not known are seldom equal, and then
// the tensor cores are ahead: 1,000, 700, 400 and 300 tokens 167 and 187), 32 heads of 64 x 64
// 384 CTAs 161 and 167, 512 194 and 173, 1,024 384 and 325. Heads of 256 x 64, 16 of them, three of 1,024 (192) delta rule 404 and 456, head
// decay with a delta 394 and 345, a decay per token 292 and 280; four (256) 457 and 476, 448 and 359, 314 and 290.
template <int MODE>
bool block_takes_fma(int seqs, int H, int d, int dv, int tokens, int longest) {
  const long long ctas = walk_ctas(seqs, H, dv, tokens, longest);
  if (d > 128) return 2 * ctas > 3 * kSmCount;
  if (BlockShape<64, MODE>::DELTA) return 2 * ctas > 5 * kSmCount;
  if (BlockShape<64, MODE>::BONUS || d <= 64) return ctas > 3 * kSmCount;
  return (longest > 0 && ctas > 3 * kSmCount && ctas <= 4 * kSmCount) || ctas > 6 * kSmCount;
}

template <int MODE>
long long floats_per_stage(int seqs, int H, int KH, int d, int dv, int tokens, int longest) {
  return block_takes_fma<MODE>(seqs, H, d, dv, tokens, longest) ? walk_stage_floats<MODE>(H, KH, d) : block_stage_floats<MODE>(H, KH, d, dv);
}

// Floats of a workspace that holds a step whole, 0 where the token-by-token kernel runs.
template <int MODE>
long long walk_floats(int seqs, int H, int KH, int d, int dv, int tokens, int longest) {
  return takes_walk(d, tokens) ? walk_stages(tokens, seqs) * floats_per_stage<MODE>(seqs, H, KH, d, dv, tokens, longest) : 0;
}

template <int DP, int MODE>
int launch_block(const WalkArgs& a) {
  using K = BlockWalk<DP, MODE>;
  const long long all = walk_stages(a.rows.tokens, a.seqs), room = a.workspace.floats / block_stage_floats<MODE>(a.H, a.KH, a.d, a.dv);
  const int walkers = a.walkers, tiles = (a.dv + kBlockCols - 1) / kBlockCols;
  const bool plain = room >= all && walkers == a.seqs;
  constexpr auto fit = [](int ctas) {
    int buffers = 2;
    while (buffers < 5 && ctas * (K::bytes(buffers + 1) + 1024) <= 228 * 1024) ++buffers;
    return buffers;
  };
  constexpr int ALONE = fit(1), BESIDE = fit(2);
  const bool alone = walk_ctas(a.seqs, a.H, a.dv, a.rows.tokens, a.rows.longest) <= kSmCount;
  auto kernel = alone ? (plain ? block_scan_kernel<DP, MODE, true, ALONE> : block_scan_kernel<DP, MODE, false, ALONE>)
                      : (plain ? block_scan_kernel<DP, MODE, true, BESIDE> : block_scan_kernel<DP, MODE, false, BESIDE>);
  const size_t bytes = K::bytes(alone ? ALONE : BESIDE);
  using Head = BlockHead<DP, MODE>;
  constexpr int HEAD_BYTES = sizeof(Head);
  if constexpr (K::W::BY_HEAD) {
    const cudaError_t e = cudaFuncSetAttribute(block_prepare_head_kernel<DP, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, HEAD_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e != cudaSuccess) return static_cast<int>(e);
  const long long q_stride = a.rows.q > 0 ? a.rows.q : static_cast<long long>(a.KH) * a.d;
  const long long v_stride = a.rows.v > 0 ? a.rows.v : static_cast<long long>(a.H) * a.dv;
  auto aligned = [](const float* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  // launched behind the kernel before, not beside it: let in early its CTAs pile up on the SMs that kernel leaves first
  const long long pieces = (all + room - 1) / room, per = (all + pieces - 1) / pieces;
  float* scalars = a.workspace.at + per * block_vectors<MODE>(a.H, a.KH, a.d);
  float* values = scalars + per * a.H * K::W::SCALARS;
  BlockPrepare prepare{a.q, a.k, a.v, a.g, a.head_decay, a.beta, a.look, a.put, a.workspace.at, scalars, values, a.cu_seqlens,
                      a.slots, a.seqs, a.H, a.KH, a.d, a.dv, q_stride, v_stride,
                      a.d % 4 == 0 && q_stride % 4 == 0 && aligned(a.q) && aligned(a.k) && aligned(a.g), a.least, {}};
  for (long long first = 0; first < all; first += per) {
    const WalkPiece piece{static_cast<int>(first), static_cast<int>(min(per, all - first)), pieces == 1};
    prepare.piece = piece;
    if constexpr (K::W::BY_HEAD)
      LRM_LAUNCH((block_prepare_head_kernel<DP, MODE>), dim3(piece.count, a.H), 128, HEAD_BYTES, a.stream, prepare);
    else
      LRM_LAUNCH((block_prepare_shared_kernel<DP, MODE>), dim3(piece.count, a.KH, (a.H / a.KH + kBlockHeads - 1) / kBlockHeads), 128, 0,
                 a.stream, prepare);
    kernel<<<dim3(tiles, a.H, walkers), 256, bytes, a.stream>>>(a.workspace.at, scalars, values, a.state, a.out, a.cu_seqlens, a.slots,
                                                                a.seqs, a.H, a.KH, a.d, a.dv, a.least, piece);
    LRM_LAUNCH_CHECK();
  }
  return 0;
}

// A step that the workspace does not hold whole goes in pieces, a run of stages at a time: a state is float32 on the way from
// piece to piece as it is within one, so the bits are the same. Padding has no state to go on from, so there it goes token by
// token. `workspace`: as many floats as a stage has at least.
template <int MODE>
int dispatch_walk(const float* q, const float* k, const float* v, const float* g, const float* head_decay, const float* beta,
                  const float* look, const float* put, float* state, float* out, const int* cu_seqlens, const int* slots, int seqs,
                  int H, int KH, int d, int dv, const Workspace& workspace, cudaStream_t stream, const Rows& rows) {
  WalkArgs a{q, k, v, g, head_decay, beta, look, put, state, out, cu_seqlens, slots, seqs, H, KH, d, dv, workspace, stream, rows, 0, walking(seqs, rows.tokens)};
  const long long stage = floats_per_stage<MODE>(seqs, H, KH, d, dv, rows.tokens, rows.longest);
  if (reinterpret_cast<uintptr_t>(workspace.at) % 16 || workspace.floats < stage) return LRM_BAD_ARGUMENT;
  const bool pieces = workspace.floats / stage < walk_stages(rows.tokens, seqs);
  if (seqs > 1 || pieces) {  // the sequences that bring fewer tokens, one after another
    a.least = seqs > 1 ? kWalkTokens : 0;
    Rows few = rows;
    few.below = a.least, few.below_padding = pieces ? INT_MAX : kWalkTokens;
    const int code = dispatch_scan<MODE>(q, k, v, g, head_decay, beta, look, put, state, out, cu_seqlens, slots, seqs, H, KH, d, dv,
                                         stream, few);
    if (code != 0) return code;
  }
  if (block_takes_fma<MODE>(seqs, H, d, dv, rows.tokens, rows.longest)) return launch_walk<MODE>(a);
  if (d > 128) return launch_block<256, MODE>(a);
  if (d > 64) return launch_block<128, MODE>(a);
  return launch_block<64, MODE>(a);
}

}  // namespace
