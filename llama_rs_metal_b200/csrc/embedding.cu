// Token embedding: hidden[t,:] = table[ids[t],:] * scale, widened to the float32
// residual stream (scale 1 is exact, so a model without an embedding scale pays nothing).
// An id outside the table writes zeros; the host rejects such
// ids before launch (reference: crates/metal-backend/src/shaders/matrix.metal:94-103).
#include "common.cuh"

int g_lrm_pdl = 1;

// Switch programmatic dependent launch on or off for every kernel of the library.
LRM_API void lrm_set_pdl(int enabled) { g_lrm_pdl = enabled ? 1 : 0; }

template <typename W>
__global__ void embed_rows_kernel(const W* __restrict__ table, const int* __restrict__ ids,
                                  float* __restrict__ out, int hidden, int vocab, float scale) {
  pdl_trigger();  // a small kernel: let the next one start (and prefetch its weights) right away
  pdl_wait();
  const int t = blockIdx.x;
  const int id = ids[t];
  const bool ok = id >= 0 && id < vocab;
  const W* row = table + static_cast<size_t>(ok ? id : 0) * hidden;
  float* dst = out + static_cast<size_t>(t) * hidden;
  for (int i = threadIdx.x; i < hidden; i += blockDim.x) dst[i] = ok ? to_f32(row[i]) * scale : 0.f;
}

// The same 16 bytes of a row at a time, a piece of the row per thread and `pieces` CTAs per token, so that all of a step's loads are
// under way together (a thread that walks the row four bytes at a time waits for HBM as often as it loads): 32 tokens of 4,096
// bfloat16 numbers 10.1 -> 2.2 us, one of 2,048 3.8 -> 1.7, 4,353 tokens of 3,072 30 -> 21 us (3.8 TB/s of rows read and written).
// Rows and both tensors lie on 16 bytes. (ids may be what a launch before chose: a plain pointer, or their load might move ahead of the wait.)
template <typename W>
__global__ __launch_bounds__(256) void embed_rows_vec_kernel(const W* __restrict__ table, const int* ids,
                                                             float* __restrict__ out, int hidden, int vocab, int pieces, float scale) {
  constexpr int PER = 16 / sizeof(W);
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x / pieces, i = ((blockIdx.x - t * pieces) * blockDim.x + threadIdx.x) * PER;
  if (i >= hidden) return;
  const int id = ids[t];
  const bool ok = id >= 0 && id < vocab;
  const uint4 raw = ok ? *reinterpret_cast<const uint4*>(table + static_cast<size_t>(id) * hidden + i) : make_uint4(0u, 0u, 0u, 0u);
  const W* from = reinterpret_cast<const W*>(&raw);
  float* to = out + static_cast<size_t>(t) * hidden + i;
#pragma unroll
  for (int e = 0; e < PER; e += 4)
    *reinterpret_cast<float4*>(to + e) = ok ? make_float4(to_f32(from[e]) * scale, to_f32(from[e + 1]) * scale, to_f32(from[e + 2]) * scale,
                                                          to_f32(from[e + 3]) * scale)
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
}

template <typename W>
static int launch_embed_vec(const void* table, const int* ids, float* out, int tokens, int hidden, int vocab, float scale,
                            cudaStream_t stream) {
  const int per_row = hidden / (16 / static_cast<int>(sizeof(W))), threads = per_row >= 256 ? 256 : (per_row + 31) / 32 * 32;
  const int pieces = (per_row + threads - 1) / threads;
  LRM_LAUNCH(embed_rows_vec_kernel<W>, dim3(static_cast<unsigned>(tokens) * pieces), threads, 0, stream, static_cast<const W*>(table),
             ids, out, hidden, vocab, pieces, scale);
  LRM_LAUNCH_CHECK();
  return 0;
}

LRM_API int lrm_embed_rows(const void* table, int table_dtype, const int* ids, float* out,
                           int tokens, int hidden, int vocab, float scale, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (hidden <= 0 || vocab <= 0) return LRM_BAD_ARGUMENT;
  const bool aligned = (reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
  if (aligned && table_dtype == LRM_F32 && hidden % 4 == 0)
    return launch_embed_vec<float>(table, ids, out, tokens, hidden, vocab, scale, stream);
  if (aligned && table_dtype == LRM_BF16 && hidden % 8 == 0)
    return launch_embed_vec<__nv_bfloat16>(table, ids, out, tokens, hidden, vocab, scale, stream);
  const int threads = hidden >= 256 ? 256 : 64;
  if (table_dtype == LRM_F32)
    LRM_LAUNCH(embed_rows_kernel<float>, tokens, threads, 0, stream, static_cast<const float*>(table), ids, out,
               hidden, vocab, scale);
  else if (table_dtype == LRM_BF16)
    LRM_LAUNCH(embed_rows_kernel<__nv_bfloat16>, tokens, threads, 0, stream,
               static_cast<const __nv_bfloat16*>(table), ids, out, hidden, vocab, scale);
  else
    return LRM_BAD_ARGUMENT;
  LRM_LAUNCH_CHECK();
  return 0;
}
