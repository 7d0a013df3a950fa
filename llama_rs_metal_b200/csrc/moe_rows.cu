// A mixture's experts for steps of few rows (decoding), bfloat16 matrices, every weight read once per step.
//
// Two launches, each a weight-streaming product per chosen expert in the manner of gemm_bf16_stream.cu: a CTA owns
// 16 weight rows of one expert, its warps split K, weights go from HBM straight into mma.sync fragments, and the
// columns are the (token, choice) pairs that chose the expert, gathered by index, 8 NT at a time.
//   up:    8 gate and the 8 matching up rows of an expert; the epilogue forms y = act(gate, up).
//   down:  16 rows of W_down; plane c of the result holds weight(t, c) * W_down y(t, c) for every token t.
// y is float32 between the two: it is handed over as three bfloat16 terms whose sum is y to 24 bits, so that the
// second product multiplies it exactly. The tensor cores' running sums truncate, so they run over 32 k at most and
// are added up in float32.
//
// blockIdx.y numbers the distinct experts of the step, found by every CTA from the ids, and the list of the expert's
// pairs is in ascending order, so a result depends on nothing else in the batch. Where there are twice as many pairs as experts (at
// least 86 % of the experts are then chosen, on average) blockIdx.y is the expert itself, so that the first product's CTAs ask for
// their weights while the router still runs: 8 rows, 2 of 8 experts of 3 x 1024 x 2048, router to sum 37.7 -> 35.0 us.
#include "common.cuh"

namespace {

constexpr int kMostPairs = 4096;   // pairs a step may have: a list of them in shared memory
constexpr int kMostExperts = 1024; // a word of the bitmap per lane
constexpr int kStep = 64, kPieces = kStep / 32;  // k values of a chunk, 16-byte pieces of a row per thread
constexpr int kDepth = 4;                        // chunks of weights a warp has under way

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ float activation(float g, float u, int act, float limit, float alpha) {
  if (act == 1) return g / (1.0f + expf(-g)) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
}

// For at most 32 pairs, by every warp for itself: the `nth` distinct expert among ids[0 .. n) (identity experts, >=
// experts, not counted; numbered by their first pair) and its pairs in ascending order; -1 when there are fewer.
__device__ __forceinline__ int chosen_expert_of_few(const int* ids, int n, int experts, int nth, int* list, int* count) {
  const int lane = threadIdx.x & 31;
  const int id = lane < n ? ids[lane] : -1;
  const unsigned same = __match_any_sync(0xffffffffu, id);
  unsigned first = __ballot_sync(0xffffffffu, id >= 0 && id < experts && __ffs(same) - 1 == lane);
  for (int i = 0; i < nth; ++i) first &= first - 1;
  if (first == 0) return -1;
  const int e = __shfl_sync(0xffffffffu, id, __ffs(first) - 1);
  const unsigned mine = __ballot_sync(0xffffffffu, id == e);
  if (id == e) list[__popc(mine & ((1u << lane) - 1u))] = lane;  // every warp writes the same
  *count = __popc(mine);
  __syncwarp();
  return e;
}

// The same expert for any number of pairs, by the whole block (experts numbered by their ids). words: [32] shared.
__device__ int chosen_expert(const int* ids, int n, int experts, int nth, unsigned* words, int* picked) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 32) words[tid] = 0u;
  __syncthreads();
  for (int i = tid; i < n; i += blockDim.x) {
    const int e = ids[i];
    if (e >= 0 && e < experts) atomicOr(words + (e >> 5), 1u << (e & 31));
  }
  __syncthreads();
  if (warp == 0) {
    const unsigned word = words[lane];
    int upto = __popc(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += other;
    }
    const int before = upto - __popc(word);
    if (lane == 31 && nth >= upto) *picked = -1;
    if (nth >= before && nth < upto) {
      unsigned rest = word;
      for (int i = before; i < nth; ++i) rest &= rest - 1;
      *picked = lane * 32 + __ffs(rest) - 1;
    }
  }
  __syncthreads();
  const int e = *picked;
  if (e < 0) return -1;
  return e;
}

// The pairs of ids [0 .. n) that chose expert e, in ascending order, by the whole block; `list` [n] shared.
__device__ __forceinline__ int pairs_of(const int* ids, int n, int e, int* list, int* count) {
  const int lane = threadIdx.x & 31;
  if (n <= 32) {  // every warp for itself, all writing the same
    const unsigned mine = __ballot_sync(0xffffffffu, lane < n && ids[lane] == e);
    if (mine >> lane & 1u) list[__popc(mine & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    return __popc(mine);
  }
  if (threadIdx.x < 32) {
    int held = 0;
    for (int i0 = 0; i0 < n; i0 += 128) {  // four loads under way together
      int id[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) id[s] = i0 + 32 * s + lane < n ? ids[i0 + 32 * s + lane] : -1;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const unsigned mine = __ballot_sync(0xffffffffu, id[s] == e);
        if (id[s] == e) list[held + __popc(mine & ((1u << lane) - 1u))] = i0 + 32 * s + lane;
        held += __popc(mine);
      }
    }
    if (lane == 0) *count = held;
  }
  __syncthreads();
  return *count;
}

// DOWN false: rows f (gate) and ff + f (up) of gate_up, right operand x rows [tokens, width], K = width;
// DOWN true: rows r and r + 8 of down, right operand the three terms of y [3][pairs, ff], K = ff.
// Only W is read ahead of the wait and through the read-only path; what the launches before write (x, x32, ids, weights, y3)
// is read through plain pointers, so that no load of it can be moved ahead of the wait.
template <int NT, int WARPS, bool DOWN>
__global__ __launch_bounds__(WARPS * 32, 16 / WARPS) void moe_grouped_kernel(
    const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ W, const int* ids, const float* weights, __nv_bfloat16* y3,
    float* planes, int tokens, int width, int ff, int experts, int top, float limit, float alpha, int act, const float* x32, int by_id) {
  extern __shared__ __align__(16) unsigned char shared[];
  __shared__ unsigned words[32];
  __shared__ int count_of, picked;
  float* red = reinterpret_cast<float*>(shared);                               // [WARPS][NT][32 lanes][4]
  int* list = reinterpret_cast<int*>(shared + sizeof(float) * WARPS * NT * 128);  // [pairs]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int pairs = tokens * top, row0 = blockIdx.x * (DOWN ? 16 : 8);
  // The second product's CTAs are let in when all of the first one's are past their wait, so the ids are there: they
  // find their expert and ask for its first weights before they wait for the first product. The first product's CTAs do
  // before they wait for the router where blockIdx.y is the expert.
  if (!DOWN && !by_id) pdl_wait();
  if (DOWN || !by_id) pdl_trigger();
  if (DOWN && blockIdx.y == gridDim.y - 1) {  // the identity experts: their output is their input
    pdl_wait();
    for (int p = warp; p < pairs; p += WARPS) {
      if (ids[p] < experts || lane >= 16 || row0 + lane >= width) continue;
      const size_t at = static_cast<size_t>(p / top) * width + row0 + lane;
      planes[static_cast<size_t>(p % top) * tokens * width + at] =
          weights[p] * (x32 != nullptr ? x32[at] : __bfloat162float(x[at]));
    }
    return;
  }
  int count = 0, e = blockIdx.y;
  if (!by_id) {
    if (pairs <= 32) {
      e = chosen_expert_of_few(ids, pairs, experts, blockIdx.y, list, &count);
    } else {
      e = chosen_expert(ids, pairs, experts, blockIdx.y, words, &picked);
      if (e >= 0) count = pairs_of(ids, pairs, e, list, &count_of);
    }
    if (e < 0) return;
  }
  const int K = DOWN ? ff : width, rows = DOWN ? width : ff;
  const int row_a = row0 + g, row_b = DOWN ? row0 + g + 8 : row0 + g;
  const bool ok_a = row_a < rows, ok_b = row_b < rows;
  const __nv_bfloat16 *wa, *wb;
  if (DOWN) {
    wa = W + (static_cast<size_t>(ok_a ? row_a : 0) * experts + e) * ff;
    wb = W + (static_cast<size_t>(ok_b ? row_b : 0) * experts + e) * ff;
  } else {
    wa = W + (static_cast<size_t>(e) * 2 * ff + (ok_a ? row_a : 0)) * width;
    wb = wa + static_cast<size_t>(ff) * width;
  }
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const int per_warp = ((K + WARPS - 1) / WARPS + kStep - 1) / kStep * kStep;
  const int k_begin = warp * per_warp, k_end = min(K, k_begin + per_warp);
  auto load_w = [&](int k0, uint4 (&a)[kPieces], uint4 (&b)[kPieces]) {
#pragma unroll
    for (int s = 0; s < kPieces; ++s) {
      const int k = k0 + 32 * s + 8 * t;
      const bool in = k < k_end;
      a[s] = in && ok_a ? ldg_stream(wa + k) : zero;
      b[s] = in && ok_b ? ldg_stream(wb + k) : zero;
    }
  };
  const size_t term = static_cast<size_t>(pairs) * ff;

  uint4 wa_at[kDepth][kPieces], wb_at[kDepth][kPieces];  // kDepth chunks of weights under way
#pragma unroll
  for (int i = 0; i < kDepth; ++i) load_w(k_begin + i * kStep, wa_at[i], wb_at[i]);
  if (!DOWN && by_id) {
    pdl_wait();
    pdl_trigger();
  }
  if (by_id) {
    count = pairs_of(ids, pairs, e, list, &count_of);
    if (count == 0) return;
  }
  if (DOWN) pdl_wait();
  for (int base = 0; base < count; base += 8 * NT) {
    int right[NT];  // element where this thread's column of every tile begins (-1: no pair)
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int at = base + 8 * j + g;
      right[j] = at < count ? (DOWN ? list[at] * ff : list[at] / top * width) : -1;
    }
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
    if (base > 0) {
#pragma unroll
      for (int i = 0; i < kDepth; ++i) load_w(k_begin + i * kStep, wa_at[i], wb_at[i]);
    }
    for (int k0 = k_begin; k0 < k_end; k0 += kDepth * kStep) {
#pragma unroll
      for (int i = 0; i < kDepth; ++i) {
#pragma unroll
        for (int s = 0; s < kPieces; ++s) {
          const int k = k0 + i * kStep + 32 * s + 8 * t;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            if (j > 0 && base + 8 * j >= count) break;  // no pair in this tile (the same for all threads)
            const bool in = right[j] >= 0 && k < k_end;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int part = DOWN ? 2 : 0; part >= 0; --part) {  // the smallest term of y first
              const __nv_bfloat16* from = DOWN ? y3 + part * term : x;
              const uint4 v = in ? *reinterpret_cast<const uint4*>(from + right[j] + k) : zero;
              mma16816(sum, wa_at[i][s].x, wb_at[i][s].x, wa_at[i][s].y, wb_at[i][s].y, v.x, v.y);
              mma16816(sum, wa_at[i][s].z, wb_at[i][s].z, wa_at[i][s].w, wb_at[i][s].w, v.z, v.w);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[j][c] += sum[c];
          }
        }
        load_w(k0 + (kDepth + i) * kStep, wa_at[i], wb_at[i]);
      }
    }
    if (base > 0) __syncthreads();  // the sums of the pairs before are read
#pragma unroll
    for (int j = 0; j < NT; ++j)
      *reinterpret_cast<float4*>(red + ((warp * NT + j) * 32 + lane) * 4) = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
    __syncthreads();
    for (int item = threadIdx.x; item < NT * 32; item += WARPS * 32) {
      const int j = item >> 5, ln = item & 31, gg = ln >> 2, tt = ln & 3;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {  // the warps' shares in warp order
        const float4 v = *reinterpret_cast<const float4*>(red + ((w * NT + j) * 32 + ln) * 4);
        sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
      }
      // .x, .y: weight row gg, pairs 8 j + 2 tt and the next; .z, .w: weight row gg + 8 (the up row)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int at = base + 8 * j + 2 * tt + i;
        if (at >= count) continue;
        const int p = list[at];
        const float first = i ? sum.y : sum.x, second = i ? sum.w : sum.z;
        if (DOWN) {
          const float weight = weights[p];
          float* dst = planes + (static_cast<size_t>(p % top) * tokens + p / top) * width + row0 + gg;
          if (row0 + gg < width) dst[0] = first * weight;
          if (row0 + gg + 8 < width) dst[8] = second * weight;
        } else if (row0 + gg < ff) {
          const float y = activation(first, second, act, limit, alpha);
          const __nv_bfloat16 high = __float2bfloat16_rn(y);
          const float rest = isfinite(__bfloat162float(high)) ? y - __bfloat162float(high) : 0.f;
          const __nv_bfloat16 middle = __float2bfloat16_rn(rest);
          __nv_bfloat16* dst = y3 + static_cast<size_t>(p) * ff + row0 + gg;
          dst[0] = high;
          dst[term] = middle;
          dst[2 * term] = __float2bfloat16_rn(rest - __bfloat162float(middle));
        }
      }
    }
  }
}

template <int NT, int WARPS, bool DOWN>
int launch_grouped(const void* x, const void* W, const int* ids, const float* weights, void* y3, float* planes, int tokens,
                   int width, int ff, int experts, int top, float limit, float alpha, int act, const float* x32,
                   cudaStream_t stream) {
  const int rows = DOWN ? width : ff, per = DOWN ? 16 : 8, pairs = tokens * top;
  const size_t bytes = sizeof(float) * WARPS * NT * 128 + sizeof(int) * (pairs < 32 ? 32 : pairs);
  const dim3 grid((rows + per - 1) / per, (experts < pairs ? experts : pairs) + (DOWN ? 1 : 0));
  // an expert a block row where nearly all are chosen: some choices are of identity experts where x32 is given
  const int by_id = pairs >= 2 * experts && x32 == nullptr;
  LRM_LAUNCH((moe_grouped_kernel<NT, WARPS, DOWN>), grid, WARPS * 32, bytes, stream, static_cast<const __nv_bfloat16*>(x),
             static_cast<const __nv_bfloat16*>(W), ids, weights, static_cast<__nv_bfloat16*>(y3), planes, tokens, width, ff,
             experts, top, limit, alpha, act, x32, by_id);
  return 0;
}

}  // namespace

// Steps this way of computing takes: rows of whole 16-byte pieces, at most kMostPairs (token, choice) pairs, experts of
// some size. Router, experts and the sum of the planes, us, against the pair-by-pair kernel of moe.cu, experts of 3 x 1024
// x 2048, 2 chosen: of 8 experts 1 row 24 (32), 8 rows 41 (80), 32 rows 55 (745), 63 rows 65 (1478); of 32 experts 8
// rows 61 (103); of 64 experts 300 rows 398 (1790). An expert of 72 x 40 is two launches for nothing: 6.5 (5.0) us.
LRM_API int lrm_moe_experts_grouped_supports(int tokens, int width, int ff, int experts, int top) {
  return tokens > 0 && top > 0 && static_cast<long long>(tokens) * top <= kMostPairs && width > 0 && width % 8 == 0 && ff > 0 &&
                 ff % 8 == 0 && experts > 0 && experts <= kMostExperts && width <= (1 << 18) && ff <= (1 << 18) &&
                 static_cast<long long>(width) * ff >= 65536
             ? 1 : 0;
}

// x bfloat16 [T, width]; gate_up [E, 2 ff, width] and down [width, E, ff] bfloat16; y3: scratch of 3 * T * top * ff
// bfloat16; planes float32 [top, T, width]. An id >= experts is an identity expert (x32 [T, width] where given, else x).
LRM_API int lrm_moe_experts_grouped(const void* x, const void* gate_up, const void* down, const int* ids, const float* weights,
                                    void* y3, float* planes, int tokens, int width, int ff, int experts, int top, float limit,
                                    float alpha, int act, const float* x32, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (!lrm_moe_experts_grouped_supports(tokens, width, ff, experts, top)) return LRM_UNSUPPORTED;
  if (act != 0 && act != 1) return LRM_BAD_ARGUMENT;
  for (const void* p : {x, gate_up, down, static_cast<const void*>(y3)})
    if (reinterpret_cast<uintptr_t>(p) % 16) return LRM_UNSUPPORTED;
  int code = 0;
#define LRM_GROUPED(NT)                                                                                                      \
  do {                                                                                                                       \
    code = launch_grouped<NT, 4, false>(x, gate_up, ids, weights, y3, planes, tokens, width, ff, experts, top, limit, alpha,  \
                                        act, x32, stream);                                                                   \
    if (code == 0)                                                                                                           \
      code = launch_grouped<NT, 4, true>(x, down, ids, weights, y3, planes, tokens, width, ff, experts, top, limit, alpha, act, \
                                         x32, stream);                                                                       \
  } while (0)
  if (tokens <= 8) LRM_GROUPED(1);       // an expert has at most a pair per token (the choices are distinct)
  else if (tokens <= 16) LRM_GROUPED(2);
  else LRM_GROUPED(4);
#undef LRM_GROUPED
  return code;
}

LRM_API int lrm_moe_router(const void* x, int x_dtype, const float* w, const float* bias, int* ids, float* weights, float* logits,
                           int tokens, int width, int E, int top, int scored, const float* correction, int groups, int keep,
                           int renormalize, float mass_eps, float weight_scale, cudaStream_t stream);
LRM_API int lrm_add_planes(float* x, const float* planes, int count, long long n, cudaStream_t stream);

// Scratch that lrm_moe_rows_step wants, in floats: y's terms, the choices and their weights.
LRM_API long long lrm_moe_rows_step_floats(int tokens, int ff, int top) {
  const long long pairs = static_cast<long long>(tokens) * top;
  return (3 * pairs * ff + 7) / 8 * 4 + (pairs + 3) / 4 * 4 + pairs;
}

// The whole part for a step of few rows in one call: lrm_moe_router (w [outputs, width], its arguments from `scored` on), then
// lrm_moe_experts_grouped, then, with `sum`, all planes into the first one. `scratch`: on 16 bytes, lrm_moe_rows_step_floats floats.
LRM_API int lrm_moe_rows_step(const void* x, const float* w, const float* bias, const void* gate_up, const void* down, float* scratch,
                              float* planes, int tokens, int width, int ff, int experts, int outputs, int top, float limit, float alpha,
                              int act, const float* x32, int sum, int scored, const float* correction, int groups, int keep,
                              int renormalize, float mass_eps, float weight_scale, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (top <= 0 || scratch == nullptr || !lrm_moe_experts_grouped_supports(tokens, width, ff, experts, top)) return LRM_BAD_ARGUMENT;
  const long long pairs = static_cast<long long>(tokens) * top;
  int* ids = reinterpret_cast<int*>(scratch + (3 * pairs * ff + 7) / 8 * 4);
  float* weights = reinterpret_cast<float*>(ids + (pairs + 3) / 4 * 4);
  int code = lrm_moe_router(x, LRM_BF16, w, bias, ids, weights, nullptr, tokens, width, outputs, top, scored, correction, groups, keep,
                            renormalize, mass_eps, weight_scale, stream);
  if (code == 0)
    code = lrm_moe_experts_grouped(x, gate_up, down, ids, weights, scratch, planes, tokens, width, ff, experts, top, limit, alpha, act, x32,
                                   stream);
  const long long numbers = static_cast<long long>(tokens) * width;
  if (code == 0 && sum && top > 1) code = lrm_add_planes(planes, planes + numbers, top - 1, numbers, stream);
  return code;
}
