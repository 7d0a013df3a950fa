// Causal grouped-query attention, a warp per (query, head), with a streaming softmax in float32 over blocks of 32 keys (heads of up
// to 128) or single keys (wider ones):
//   s = (q.k) * scale;  m' = max(m, s);  l = l e^(m-m') + sum e^(s-m');
//   acc = acc e^(m-m') + sum e^(s-m') v;  out = acc / l
// (reference: crates/metal-backend/src/shaders/attention.metal:28-57).
//
// A block's keys lie at multiples of 32 of their positions, a lane per key for the scores and a lane per column for the values, both
// added in ascending order, so a row's sums depend on nothing but the row. A CTA has up to 16 rows of a key/value head (queries and
// the heads that share it) and brings a block's keys and values to shared memory once for all of them, the next block's on their way
// meanwhile. Bound by a CTA's chain of blocks. The 1B shape in float32, us: a prompt of 333 tokens 62 (160 key by key, each of which
// waited for the sum of its dot product over the warp), a decode step of two layers with 3,000 keys, four sequences, 593 (6,287),
// 300 tokens onto 1,000 1,207 (7,570). 32 rows a CTA 509 a layer's prompt against 495, 8 rows 494 and 1,247 for the portion.
// Heads that share no keys, a query per sequence, us, in brackets key by key, then four and sixteen sequences to a CTA one after
// another: 256 of 300 keys, 16 heads of 128 322 (339, 352, 774), 32 heads of 64 336 (625, 324, 762); 128 of 500 283 (522, 285, 1,146)
// and 266 (530, 330, 612); four of 3,000 keys 316 (2,929, 1,204) and 195 (2,903, 750).
//
// It is the attention of the float32 path for prompts and for decoding, and
// the bfloat16 path's fallback for sizes its tiled kernels refuse (head sizes up to 1024). The two
// entry points differ only in where keys come from (the step's packed k/v, or
// the paged cache), so a prompt, its token-by-token replay and its replay in
// chunks of any size do the same arithmetic in the same order. The paged entry
// takes any number of queries per sequence (a decoded token, or a portion of
// several tokens appended to a started sequence, whose own keys are already in
// the cache). A window w lets a query at position p see keys p-w+1 .. p; a negative w stands for
// chunks of -w positions (first_visible_key).
// Values may have another width than keys (dv against d). With `slopes` (one
// float32 per query head) a key at distance n = p - j behind the query loses
// slope_h * n from its score (a linear distance penalty, no rotation needed);
// `out_scale` multiplies the result before it is rounded (a mixer whose output
// enters a weighted sum of mixers). With `sinks` (one float32 per query head) the softmax's
// denominator also holds exp(sink_h): a key that is always seen, with no value, whose score is
// not scaled. With a query temperature (`temp_every` > 0) the query at position p counts
// 1 + temp_coef * ln(floor((p + 1) / temp_every) + 1) times (the factor goes into the score's
// scale, in float32). `v_stride` is the distance between two value rows in elements: values
// that are the first dv columns of the key rows are read from the keys' storage with the keys' d.
#include <climits>

#include "common.cuh"

constexpr int kWidest = 32;  // elements of a row one lane holds at most: head sizes up to 1024

struct PackedKeys {
  const void* k;
  const void* v;
  size_t base;  // index of the sequence's first packed token
  int kv_heads, d, vs;
  template <typename A> __device__ const A* key(int p, int kh) const {
    return static_cast<const A*>(k) + ((base + p) * kv_heads + kh) * d;
  }
  template <typename A> __device__ const A* value(int p, int kh) const {
    return static_cast<const A*>(v) + ((base + p) * kv_heads + kh) * vs;
  }
};

struct PagedKeys {
  const void* k;
  const void* v;
  const int* table;  // this slot's row of the page table
  int kv_heads, d, vs, page_size;
  template <typename A> __device__ const A* key(int p, int kh) const {
    const size_t page = table[p / page_size];
    return static_cast<const A*>(k) + ((page * kv_heads + kh) * page_size + p % page_size) * d;
  }
  template <typename A> __device__ const A* value(int p, int kh) const {
    const size_t page = table[p / page_size];
    return static_cast<const A*>(v) + ((page * kv_heads + kh) * page_size + p % page_size) * vs;
  }
};

// PER: elements of a query (and of the output) one lane keeps in registers; d, dv <= 32 * PER.
template <typename A, int PER, typename Keys>
__device__ void attend_row(const A* __restrict__ q, A* __restrict__ out, const Keys& keys, int kh,
                           int first, int last, int d, int dv, float scale, float slope,
                           float out_scale, float sink) {
  const int lane = threadIdx.x & 31;
  float qv[PER], acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int j = lane + 32 * i;
    qv[i] = j < d ? to_f32(q[j]) : 0.f;
    acc[i] = 0.f;
  }
  // a sink is a key met before all others: score `sink`, weight 1 at its own maximum, no value
  float m = sink, l = sink > -INFINITY ? 1.f : 0.f;
  for (int p = first; p <= last; ++p) {
    const A* kr = keys.template key<A>(p, kh);
    const A* vr = keys.template value<A>(p, kh);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int j = lane + 32 * i;
      if (j < d) dot = fmaf(qv[i], to_f32(kr[j]), dot);
    }
    float s = warp_sum(dot) * scale;
    if (slope != 0.f) s -= slope * static_cast<float>(last - p);
    const float nm = fmaxf(m, s);
    const float old = expf(m - nm), prob = expf(s - nm);
    l = fmaf(l, old, prob);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int j = lane + 32 * i;
      if (j < dv) acc[i] = fmaf(prob, to_f32(vr[j]), __fmul_rn(acc[i], old));
    }
    m = nm;
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int j = lane + 32 * i;
    if (j < dv) out[j] = from_f32<A>(out_scale == 1.0f ? acc[i] / l : (acc[i] / l) * out_scale);
  }
}

__device__ __forceinline__ float query_temperature(int pos, float coef, int every) {
  return every > 0 ? 1.0f + coef * logf(static_cast<float>((pos + 1) / every + 1)) : 1.0f;
}

template <typename A, int PER>
__global__ void attention_packed_kernel(const A* __restrict__ q, const A* __restrict__ k,
                                        const A* __restrict__ v, A* __restrict__ out,
                                        const int* __restrict__ cu_seqlens,
                                        const int* __restrict__ seq_of_token, int q_heads,
                                        int kv_heads, int d, int dv, float scale, int window,
                                        const float* __restrict__ slopes, float out_scale,
                                        const float* __restrict__ sinks, float temp_coef,
                                        int temp_every, int v_stride) {
  const int t = blockIdx.x, h = blockIdx.y;
  const int start = cu_seqlens[seq_of_token[t]];
  const int pos = t - start;
  const int first = first_visible_key(pos, window);
  PackedKeys keys{k, v, static_cast<size_t>(start), kv_heads, d, v_stride};
  const size_t row = static_cast<size_t>(t) * q_heads + h;
  attend_row<A, PER>(q + row * d, out + row * dv, keys, h / (q_heads / kv_heads), first, pos, d, dv,
                scale * query_temperature(pos, temp_coef, temp_every),
                slopes != nullptr ? slopes[h] : 0.f, out_scale, sinks != nullptr ? sinks[h] : -INFINITY);
}

template <typename A, int PER>
__global__ void attention_paged_kernel(const A* __restrict__ q, const A* __restrict__ k_pages,
                                       const A* __restrict__ v_pages, A* __restrict__ out,
                                       const int* __restrict__ page_table, int table_stride,
                                       const int* __restrict__ slots,
                                       const int* __restrict__ kv_lens,
                                       const int* __restrict__ seq_of_token,
                                       const int* __restrict__ positions, int q_heads, int kv_heads,
                                       int d, int dv, int page_size, float scale, int window,
                                       const float* __restrict__ slopes, float out_scale,
                                       const float* __restrict__ sinks, float temp_coef,
                                       int temp_every, int v_stride) {
  // query t of the step belongs to sequence b and stands at position pos; without the two
  // arrays there is one query per sequence, its newest token
  const int t = blockIdx.x, h = blockIdx.y;
  const int b = seq_of_token != nullptr ? seq_of_token[t] : t;
  const int pos = positions != nullptr ? positions[t] : kv_lens[b] - 1;
  const int first = first_visible_key(pos, window);
  PagedKeys keys{k_pages, v_pages, page_table + static_cast<size_t>(slots[b]) * table_stride,
                 kv_heads, d, v_stride, page_size};
  const size_t row = static_cast<size_t>(t) * q_heads + h;
  attend_row<A, PER>(q + row * d, out + row * dv, keys, h / (q_heads / kv_heads), first, pos, d, dv,
                scale * query_temperature(pos, temp_coef, temp_every),
                slopes != nullptr ? slopes[h] : 0.f, out_scale, sinks != nullptr ? sinks[h] : -INFINITY);
}

// --------------------------------------------------------------------------- blocks of 32 keys
constexpr int kKeys = 32, kBlocked = 128;  // keys of a block; widest head that goes so

struct RowsArgs {
  const void *q, *k, *v;
  void* out;
  const int *cu_seqlens, *seq_of_token, *page_table, *slots, *kv_lens, *positions;
  int queries, q_heads, kv_heads, d, dv, page_size, table_stride, window, temp_every, v_stride;
  float scale, out_scale, temp_coef;
  const float *slopes, *sinks;
  int aligned;    // rows of q, k and v begin on four elements
  int per_query;  // CTAs of a query and key/value head where no two queries share a sequence; 0: a CTA's rows run on over queries
};

template <typename A>
__device__ __forceinline__ float4 load_four(const A* from, int count, bool aligned) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (count >= 4 && aligned) {
    if constexpr (sizeof(A) == 4) {
      x = *reinterpret_cast<const float4*>(from);
    } else {
      const uint2 raw = *reinterpret_cast<const uint2*>(from);
      x.x = __uint_as_float(raw.x << 16), x.y = __uint_as_float(raw.x & 0xffff0000u);
      x.z = __uint_as_float(raw.y << 16), x.w = __uint_as_float(raw.y & 0xffff0000u);
    }
  } else {
    if (count > 0) x.x = to_f32(from[0]);
    if (count > 1) x.y = to_f32(from[1]);
    if (count > 2) x.z = to_f32(from[2]);
    if (count > 3) x.w = to_f32(from[3]);
  }
  return x;
}

// WARPS * RW rows of key/value head blockIdx.y, RW a warp, the last ones first (in a prompt they see the most keys); row i is query
// i / group, head i % group of the group. The next block's keys and values are on their way to registers under a block's work.
template <typename A, int DP, int RW, int WARPS, bool PAGED>
__global__ __launch_bounds__(WARPS * 32) void attention_rows_kernel(const RowsArgs a) {
  constexpr int ROWS = RW * WARPS, THREADS = WARPS * 32, PER = DP / 32, KP = DP + 4;
  static_assert(ROWS <= 32, "a lane per row");
  extern __shared__ __align__(16) float rows_smem[];
  float(*qs)[DP] = reinterpret_cast<float(*)[DP]>(rows_smem);
  float(*ks)[KP] = reinterpret_cast<float(*)[KP]>(rows_smem + ROWS * DP);
  float(*vs)[DP] = reinterpret_cast<float(*)[DP]>(rows_smem + ROWS * DP + kKeys * KP);
  float(*ps)[kKeys] = reinterpret_cast<float(*)[kKeys]>(rows_smem + ROWS * DP + kKeys * KP + kKeys * DP);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kh = blockIdx.y, group = a.q_heads / a.kv_heads;
  const int block_at = static_cast<int>(gridDim.x - 1 - blockIdx.x), of_query = a.per_query > 0 ? block_at % a.per_query * ROWS : 0;
  const int row0 = a.per_query > 0 ? block_at / a.per_query * group + of_query : block_at * ROWS;
  const int count = min(ROWS, a.per_query > 0 ? group - of_query : a.queries * group - row0);
  const bool aligned = a.aligned != 0;

  // Lane r of every warp knows row r: its sequence, position and first key.
  int seq = -1, pos = -1, first = 0;
  if (lane < count) {
    const int t = (row0 + lane) / group;
    seq = a.seq_of_token != nullptr ? a.seq_of_token[t] : t;
    pos = PAGED ? (a.positions != nullptr ? a.positions[t] : a.kv_lens[seq] - 1) : t - a.cu_seqlens[seq];
    first = first_visible_key(pos, a.window);
  }
  for (int i = tid; i < ROWS * (DP / 4); i += THREADS) {
    const int r = i / (DP / 4), c = i % (DP / 4) * 4, idx = row0 + r;
    const A* from = static_cast<const A*>(a.q) + (static_cast<size_t>(idx / group) * a.q_heads + kh * group + idx % group) * a.d + c;
    *reinterpret_cast<float4*>(&qs[r][c]) = load_four<A>(from, r < count ? a.d - c : 0, aligned);
  }
  float m[RW], l[RW], scale[RW], slope[RW], acc[RW][PER];
  int my_seq[RW], my_pos[RW], my_first[RW];
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    const int r = warp * RW + i, h = kh * group + (row0 + r) % group;
    my_seq[i] = __shfl_sync(0xffffffffu, seq, r), my_pos[i] = __shfl_sync(0xffffffffu, pos, r), my_first[i] = __shfl_sync(0xffffffffu, first, r);
    // a sink is a key met before all others: score `sink`, weight 1 at its own maximum, no value
    m[i] = a.sinks != nullptr && r < count ? a.sinks[h] : -INFINITY, l[i] = m[i] > -INFINITY ? 1.f : 0.f;
    scale[i] = a.scale * query_temperature(my_pos[i], a.temp_coef, a.temp_every), slope[i] = a.slopes != nullptr && r < count ? a.slopes[h] : 0.f;
#pragma unroll
    for (int e = 0; e < PER; ++e) acc[i][e] = 0.f;
  }

  for (int begin = 0; begin < count;) {  // the rows of one sequence after another
    const int b = __shfl_sync(0xffffffffu, seq, begin);
    const unsigned same = __ballot_sync(0xffffffffu, lane >= begin && lane < count && seq == b);
    const int end = begin + __popc(same);  // (a step's tokens lie sequence after sequence)
    const bool in = lane >= begin && lane < end;
    int low = in ? first : INT_MAX, high = in ? pos : -1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) low = min(low, __shfl_xor_sync(0xffffffffu, low, o)), high = max(high, __shfl_xor_sync(0xffffffffu, high, o));
    const size_t base = PAGED ? 0 : static_cast<size_t>(a.cu_seqlens[b]);
    const int* table = PAGED ? a.page_table + static_cast<size_t>(a.slots[b]) * a.table_stride : nullptr;
    constexpr int PIECES = kKeys * (DP / 4) / THREADS;
    float4 next_k[PIECES], next_v[PIECES];
    auto fetch = [&](int block) {
#pragma unroll
      for (int n = 0; n < PIECES; ++n) {
        const int i = tid + n * THREADS, c = i % (DP / 4) * 4, p = block + i / (DP / 4);
        const bool there = p >= low && p <= high;
        size_t line = 0;
        if (there && PAGED) line = (static_cast<size_t>(table[p / a.page_size]) * a.kv_heads + kh) * a.page_size + p % a.page_size;
        else if (there) line = (base + p) * a.kv_heads + kh;
        next_k[n] = load_four<A>(static_cast<const A*>(a.k) + line * a.d + c, there ? a.d - c : 0, aligned);
        next_v[n] = load_four<A>(static_cast<const A*>(a.v) + line * a.v_stride + c, there ? a.dv - c : 0, aligned);
      }
    };
    int block = low / kKeys * kKeys;
    fetch(block);
    for (; block <= high; block += kKeys) {
      __syncthreads();  // everyone is done with the block before (and the queries are here)
#pragma unroll
      for (int n = 0; n < PIECES; ++n) {
        const int i = tid + n * THREADS, r = i / (DP / 4), c = i % (DP / 4) * 4;
        *reinterpret_cast<float4*>(&ks[r][c]) = next_k[n], *reinterpret_cast<float4*>(&vs[r][c]) = next_v[n];
      }
      __syncthreads();
      if (block + kKeys <= high) fetch(block + kKeys);
      bool active[RW], any = false, whole = true;  // rows that see a key of the block; whether all see all of them
#pragma unroll
      for (int i = 0; i < RW; ++i) {
        active[i] = my_seq[i] == b && warp * RW + i < count && my_pos[i] >= block && my_first[i] < block + kKeys;
        any = any || active[i];
        whole = whole && (!active[i] || (my_first[i] <= block && my_pos[i] >= block + kKeys - 1));
      }
      if (!any) continue;
      float2 dot[RW][2];
#pragma unroll
      for (int i = 0; i < RW; ++i) dot[i][0] = dot[i][1] = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int c = 0; c < a.d; c += 4) {
        const float4 key = *reinterpret_cast<const float4*>(&ks[lane][c]);
#pragma unroll
        for (int i = 0; i < RW; ++i) {
          const float4 query = *reinterpret_cast<const float4*>(&qs[warp * RW + i][c]);
          dot[i][0].x = fmaf(query.x, key.x, dot[i][0].x), dot[i][0].y = fmaf(query.y, key.y, dot[i][0].y);
          dot[i][1].x = fmaf(query.z, key.z, dot[i][1].x), dot[i][1].y = fmaf(query.w, key.w, dot[i][1].y);
        }
      }
      const int p = block + lane;
#pragma unroll
      for (int i = 0; i < RW; ++i) {
        if (!active[i]) continue;
        float score = ((dot[i][0].x + dot[i][0].y) + (dot[i][1].x + dot[i][1].y)) * scale[i];
        if (slope[i] != 0.f) score -= slope[i] * static_cast<float>(my_pos[i] - p);
        const bool seen = p >= my_first[i] && p <= my_pos[i];
        const float nm = fmaxf(m[i], warp_max(seen ? score : -INFINITY)), old = expf(m[i] - nm), prob = seen ? expf(score - nm) : 0.f;
        l[i] = fmaf(l[i], old, warp_sum(prob)), m[i] = nm;
        ps[warp * RW + i][lane] = prob;
#pragma unroll
        for (int e = 0; e < PER; ++e) acc[i][e] *= old;
      }
      __syncwarp();
#pragma unroll 2
      for (int j = 0; j < kKeys; j += 4) {
        float prob[RW][4];
#pragma unroll
        for (int i = 0; i < RW; ++i) {
          const float4 x = *reinterpret_cast<const float4*>(&ps[warp * RW + i][j]);
          prob[i][0] = x.x, prob[i][1] = x.y, prob[i][2] = x.z, prob[i][3] = x.w;
        }
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          float value[PER];
#pragma unroll
          for (int e = 0; e < PER; ++e) value[e] = vs[j + n][lane + 32 * e];
#pragma unroll
          for (int i = 0; i < RW; ++i) {  // (what a row does not see adds nothing, not even a NaN)
            if (active[i] && (whole || (block + j + n >= my_first[i] && block + j + n <= my_pos[i]))) {
#pragma unroll
              for (int e = 0; e < PER; ++e) acc[i][e] = fmaf(prob[i][n], value[e], acc[i][e]);
            }
          }
        }
      }
      __syncwarp();
    }
    begin = end;
  }
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    const int r = warp * RW + i, idx = row0 + r;
    if (r >= count) continue;
    A* to = static_cast<A*>(a.out) + (static_cast<size_t>(idx / group) * a.q_heads + kh * group + idx % group) * a.dv;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int j = lane + 32 * e;
      if (j < a.dv) to[j] = from_f32<A>(a.out_scale == 1.0f ? acc[i][e] / l[i] : (acc[i][e] / l[i]) * a.out_scale);
    }
  }
}

template <typename A, int DP, int RW, int WARPS, bool PAGED>
int launch_rows(const RowsArgs& a, cudaStream_t stream) {
  constexpr int ROWS = RW * WARPS;
  constexpr size_t bytes = sizeof(float) * (ROWS * DP + kKeys * (DP + 4) + kKeys * DP + ROWS * kKeys);
  if (bytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<A, DP, RW, WARPS, PAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  const long long rows = static_cast<long long>(a.queries) * (a.q_heads / a.kv_heads);
  const long long ctas = a.per_query > 0 ? static_cast<long long>(a.queries) * a.per_query : (rows + ROWS - 1) / ROWS;
  attention_rows_kernel<A, DP, RW, WARPS, PAGED><<<dim3(static_cast<unsigned>(ctas), a.kv_heads), WARPS * 32, bytes, stream>>>(a);
  LRM_LAUNCH_CHECK();
  return 0;
}

// 16 rows a CTA for prompts, which share their keys; 4 where few may, and no two sequences in a CTA where every query is its
// sequence's only one: a CTA goes through its sequences one after another.
template <typename A, bool PAGED>
int dispatch_rows(RowsArgs a, int seqs, cudaStream_t stream) {
  const int group = a.q_heads / a.kv_heads;
  if (PAGED && seqs == a.queries) a.per_query = (group + 3) / 4;
  const bool many = PAGED ? a.queries >= 128 && a.per_query == 0 && static_cast<long long>(a.queries) * group >= 4ll * seqs : true;
  if (a.d <= 64 && a.dv <= 64)
    return many ? launch_rows<A, 64, 2, 8, PAGED>(a, stream) : launch_rows<A, 64, 1, 4, PAGED>(a, stream);
  return many ? launch_rows<A, 128, 2, 8, PAGED>(a, stream) : launch_rows<A, 128, 1, 4, PAGED>(a, stream);
}

static int rows_alignment(const RowsArgs& a, int dtype) {
  const uintptr_t bytes = dtype == LRM_F32 ? 16 : 8;
  return a.d % 4 == 0 && a.v_stride % 4 == 0 && a.dv % 4 == 0 && reinterpret_cast<uintptr_t>(a.q) % bytes == 0 &&
         reinterpret_cast<uintptr_t>(a.k) % bytes == 0 && reinterpret_cast<uintptr_t>(a.v) % bytes == 0;
}

static bool bad_geometry(int q_heads, int kv_heads, int d, int dv) {
  return q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0 || d <= 0 ||
         d > 32 * kWidest || dv <= 0 || dv > 32 * kWidest;
}

LRM_API int lrm_attention_packed_rowwise(const void* q, const void* k, const void* v, void* out,
                                         int dtype, const int* cu_seqlens, const int* seq_of_token,
                                         int tokens, int q_heads, int kv_heads, int d, int dv,
                                         float scale, int window, const float* slopes,
                                         float out_scale, const float* sinks, float temp_coef,
                                         int temp_every, int v_stride, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (v_stride <= 0) v_stride = dv;
  if (bad_geometry(q_heads, kv_heads, d, dv)) return LRM_BAD_ARGUMENT;
  if (q_heads > 65535) return LRM_UNSUPPORTED;
  const dim3 grid(tokens, q_heads);
  const int widest = d > dv ? d : dv;
  if (widest <= kBlocked) {
    RowsArgs a{q, k, v, out, cu_seqlens, seq_of_token, nullptr, nullptr, nullptr, nullptr, tokens, q_heads, kv_heads, d, dv, 1, 0, window,
               temp_every, v_stride, scale, out_scale, temp_coef, slopes, sinks, 0, 0};
    a.aligned = rows_alignment(a, dtype);
    return dtype == LRM_F32    ? dispatch_rows<float, false>(a, 0, stream)
           : dtype == LRM_BF16 ? dispatch_rows<__nv_bfloat16, false>(a, 0, stream)
                               : LRM_BAD_ARGUMENT;
  }
#define LRM_PACKED(AT, PER)                                                                                      \
  attention_packed_kernel<AT, PER><<<grid, 32, 0, stream>>>(                                                     \
      static_cast<const AT*>(q), static_cast<const AT*>(k), static_cast<const AT*>(v), static_cast<AT*>(out),    \
      cu_seqlens, seq_of_token, q_heads, kv_heads, d, dv, scale, window, slopes, out_scale, sinks, temp_coef,    \
      temp_every, v_stride)
#define LRM_PACKED_BY_WIDTH(AT)                  \
  do {                                           \
    if (widest <= 512) LRM_PACKED(AT, 16);  \
    else LRM_PACKED(AT, 32);                     \
  } while (0)
  if (dtype == LRM_F32)
    LRM_PACKED_BY_WIDTH(float);
  else if (dtype == LRM_BF16)
    LRM_PACKED_BY_WIDTH(__nv_bfloat16);
  else
    return LRM_BAD_ARGUMENT;
#undef LRM_PACKED_BY_WIDTH
#undef LRM_PACKED
  LRM_LAUNCH_CHECK();
  return 0;
}

// `queries` rows of q. With seq_of_token and positions (int32 [queries]) query t belongs to
// sequence seq_of_token[t] and sees keys up to positions[t]; with both null there is one query
// per sequence, at position kv_lens[b] - 1. `seqs`: sequences that bring queries (for the layout).
LRM_API int lrm_attention_paged_rowwise(const void* q, const void* k_pages, const void* v_pages,
                                        void* out, int dtype, const int* page_table,
                                        int table_stride, const int* slots, const int* kv_lens,
                                        const int* seq_of_token, const int* positions,
                                        int queries, int q_heads, int kv_heads, int d, int dv,
                                        int page_size, float scale, int window, const float* slopes,
                                        float out_scale, const float* sinks, float temp_coef,
                                        int temp_every, int v_stride, int seqs, cudaStream_t stream) {
  if (queries <= 0) return 0;
  if (v_stride <= 0) v_stride = dv;
  if (positions == nullptr) seqs = queries;
  if (bad_geometry(q_heads, kv_heads, d, dv) || page_size <= 0) return LRM_BAD_ARGUMENT;
  if ((seq_of_token == nullptr) != (positions == nullptr)) return LRM_BAD_ARGUMENT;
  if (positions == nullptr && kv_lens == nullptr) return LRM_BAD_ARGUMENT;
  if (q_heads > 65535) return LRM_UNSUPPORTED;
  const dim3 grid(queries, q_heads);
  const int widest = d > dv ? d : dv;
  if (widest <= kBlocked) {
    RowsArgs a{q, k_pages, v_pages, out, nullptr, seq_of_token, page_table, slots, kv_lens, positions, queries, q_heads, kv_heads, d, dv,
               page_size, table_stride, window, temp_every, v_stride, scale, out_scale, temp_coef, slopes, sinks, 0, 0};
    a.aligned = rows_alignment(a, dtype);
    return dtype == LRM_F32    ? dispatch_rows<float, true>(a, seqs, stream)
           : dtype == LRM_BF16 ? dispatch_rows<__nv_bfloat16, true>(a, seqs, stream)
                               : LRM_BAD_ARGUMENT;
  }
#define LRM_PAGED(AT, PER)                                                                                       \
  attention_paged_kernel<AT, PER><<<grid, 32, 0, stream>>>(                                                      \
      static_cast<const AT*>(q), static_cast<const AT*>(k_pages), static_cast<const AT*>(v_pages),               \
      static_cast<AT*>(out), page_table, table_stride, slots, kv_lens, seq_of_token, positions, q_heads,         \
      kv_heads, d, dv, page_size, scale, window, slopes, out_scale, sinks, temp_coef, temp_every, v_stride)
#define LRM_PAGED_BY_WIDTH(AT)                  \
  do {                                          \
    if (widest <= 512) LRM_PAGED(AT, 16);  \
    else LRM_PAGED(AT, 32);                     \
  } while (0)
  if (dtype == LRM_F32)
    LRM_PAGED_BY_WIDTH(float);
  else if (dtype == LRM_BF16)
    LRM_PAGED_BY_WIDTH(__nv_bfloat16);
  else
    return LRM_BAD_ARGUMENT;
#undef LRM_PAGED_BY_WIDTH
#undef LRM_PAGED
  LRM_LAUNCH_CHECK();
  return 0;
}
