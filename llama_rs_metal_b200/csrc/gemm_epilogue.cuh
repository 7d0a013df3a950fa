// The epilogues of the tensor-core products, applied to 32 columns of one accumulator row at a time
// (shared by the single-CTA kernel and the kernel that runs pairs of CTAs):
//   0 store bfloat16, 1 store float32, 2 add into float32 in place (residual stream),
//   3 SiLU gate over alternating blocks of 8 gate / 8 up columns, 4 store float32 (a K slice's plane),
//   6 columns below a split as 1, the columns from it on as 3, each into a tensor of its own (SplitArgs),
// and epilogue 5, which works on whole heads of a fused q|k|v projection (store_heads).
#pragma once
#include <type_traits>

#include "silu.cuh"
#include "umma.cuh"

namespace {

// What epilogue 6 needs: two products with the same input in one launch. Columns [0, split) are stored in
// float32 to `out` [M, split]; columns from `split` (a multiple of 32) on are gate and up rows, and the
// gated values go to `gated`, whose rows are `pitch` elements apart.
struct SplitArgs {
  __nv_bfloat16* gated;
  long long pitch;
  int split;
};

// A warp's 32 accumulator rows on their way to memory. A thread that stores its own row touches 32 rows with every
// instruction, 16 bytes of each; through this piece of shared memory (2 KB per warp) the same bytes leave as runs of 64 bytes
// (32 for gated values): BYTES of every row, 16-byte pieces swapped about so that neither way meets a bank twice.
// us of a 128 x 256 tile's epilogue (1,536 x 9,472, K = 64: what a further round of tiles adds), in brackets each thread on its
// own row: bfloat16 2.4 (6.0), float32 4.1 (9.3), added 4.3 (8.7), gated 3.3 (5.6). It is not hidden behind the last tile, and
// only partly behind others: with K = 2048 the whole product is 42.3 (51.7), gated 45.7 (52.5).
constexpr int kStageBytes = 32 * 64;

template <int BYTES>
__device__ __forceinline__ void stage_row(unsigned char* stage, int lane, const uint32_t* v) {
  static_assert(BYTES == 32 || BYTES == 64, "");
#pragma unroll
  for (int c = 0; c < BYTES / 16; ++c) {
    const int at = BYTES == 64 ? c ^ ((lane >> 1) & 3) : c ^ ((lane >> 2) & 1);
    *reinterpret_cast<uint4*>(stage + lane * BYTES + at * 16) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  }
}

// f(row, byte of the row, 16 bytes) for all that the warp's lanes staged.
template <int BYTES, class F>
__device__ __forceinline__ void unstage(const unsigned char* stage, int lane, F f) {
  constexpr int PER = BYTES / 16, ROWS = 32 / PER;  // pieces of a row, rows per step
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 32 / ROWS; ++i) {
    const int row = i * ROWS + lane / PER, c = lane % PER;
    const int at = BYTES == 64 ? c ^ ((row >> 1) & 3) : c ^ ((row >> 2) & 1);
    f(row, c * 16, *reinterpret_cast<const uint4*>(stage + row * BYTES + at * 16));
  }
  __syncwarp();
}

// The epilogue of a 32-column piece of a warp's 32 accumulator rows (rows m0 .. of the product), a row per lane in registers.
// Every lane of the warp calls it.
__device__ __forceinline__ void store_piece(const uint32_t (&r)[32], unsigned char* stage, void* __restrict__ out, int m0,
                                            int lane, int n, int M, int N, int mode, const SplitArgs& parts) {
  if (n >= N) return;
  const int m = m0 + lane;
  size_t pitch = N >> 1;  // of the gated values
  if (mode == 6) {
    if (n < parts.split) {
      mode = 1;
      N = parts.split;
    } else {
      mode = 3;
      n -= parts.split;
      N -= parts.split;
      out = parts.gated;
      pitch = parts.pitch;
    }
  }
  const bool whole = n + 32 <= N;
  if (mode == 3) {
    // [8 gate | 8 up | 8 gate | 8 up] -> 16 gated values
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(out) + (n >> 1);
    float gate[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) gate[i] = __uint_as_float(r[(i >> 3) * 16 + (i & 7)]);
    silu_all(gate);
    uint32_t packed[8];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const int up = (i >> 3) * 16 + (i & 7) + 8;
      packed[i >> 1] = pack_bf16(gate[i] * __uint_as_float(r[up]), gate[i + 1] * __uint_as_float(r[up + 1]));
    }
    if (whole) {
      stage_row<32>(stage, lane, packed);
      unstage<32>(stage, lane, [&](int row, int byte, const uint4& v) {
        if (m0 + row < M) *reinterpret_cast<uint4*>(dst + static_cast<size_t>(m0 + row) * pitch + byte / 2) = v;
      });
    } else if (m < M) {
      __nv_bfloat16* mine = dst + static_cast<size_t>(m) * pitch;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t two = packed[i >> 1];
        const uint16_t bits = static_cast<uint16_t>((i & 1) ? two >> 16 : two);
        if (n + (i >> 3) * 16 + 8 + (i & 7) < N) mine[i] = __ushort_as_bfloat16(bits);
      }
    }
  } else if (mode == 0) {
    __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(out) + n;
    if (whole && (N & 7) == 0) {
      uint32_t packed[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) packed[i] = pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
      stage_row<64>(stage, lane, packed);
      unstage<64>(stage, lane, [&](int row, int byte, const uint4& v) {
        if (m0 + row < M) *reinterpret_cast<uint4*>(dst + static_cast<size_t>(m0 + row) * N + byte / 2) = v;
      });
    } else if (m < M) {
      __nv_bfloat16* mine = dst + static_cast<size_t>(m) * N;
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (n + i < N) mine[i] = __float2bfloat16_rn(__uint_as_float(r[i]));
    }
  } else {
    float* dst = static_cast<float*>(out) + n;
    if (whole && (N & 3) == 0) {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        stage_row<64>(stage, lane, r + 16 * half);
        unstage<64>(stage, lane, [&](int row, int byte, const uint4& raw) {
          if (m0 + row >= M) return;
          float4* to = reinterpret_cast<float4*>(dst + static_cast<size_t>(m0 + row) * N + 16 * half + byte / 4);
          const float4 v = make_float4(__uint_as_float(raw.x), __uint_as_float(raw.y), __uint_as_float(raw.z), __uint_as_float(raw.w));
          // Adding goes through a vector reduction in L2 (no value comes back, so the thread does
          // not wait for the old contents). Each element gets exactly one add per launch, so the
          // result is as deterministic as a read-modify-write.
          if (mode == 2) atomicAdd(to, v);
          else *to = v;
        });
      }
    } else if (m < M) {
      float* mine = dst + static_cast<size_t>(m) * N;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (n + i >= N) continue;
        if (mode == 2) atomicAdd(mine + i, __uint_as_float(r[i]));
        else mine[i] = __uint_as_float(r[i]);
      }
    }
  }
}

// 32 gate columns and the 32 up columns beside them, at these places of tensor memory, of a warp's 32 rows (m0 ..): weight *
// act(gate, up) to out [.., pitch]. Act 0: min(g, limit) sigmoid(alpha g) (clamp(u, -limit, limit) + 1); 1: silu(g) u.
__device__ __forceinline__ void store_gated(uint32_t gates, uint32_t ups, unsigned char* stage, __nv_bfloat16* out, int m0,
                                            int lane, float weight, int pitch, int act, float limit, float alpha) {
  uint32_t packed[16];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t raw[16], up[16];
    tmem_load16(gates + 16 * half, raw);
    tmem_load16(ups + 16 * half, up);
    float g[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) g[i] = act == 1 ? __uint_as_float(raw[i]) : fminf(__uint_as_float(raw[i]), limit);
    silu_all(g, act == 1 ? 1.f : alpha);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float u = __uint_as_float(up[i]);
      if (act != 1) u = fminf(fmaxf(u, -limit), limit) + 1.f;
      g[i] = weight != 0.f ? g[i] * u * weight : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) packed[8 * half + i] = pack_bf16(g[2 * i], g[2 * i + 1]);
  }
  stage_row<64>(stage, lane, packed);
  unstage<64>(stage, lane, [&](int row, int byte, const uint4& v) {
    *reinterpret_cast<uint4*>(out + static_cast<size_t>(m0 + row) * pitch + byte / 2) = v;
  });
}

// What epilogue 5 needs: the product is a prompt's fused q|k|v projection [T, (Hq + 2 Hk) d], and
// instead of storing it the epilogue rounds it to bfloat16, rotates q and k by their positions
// (split-half, the angles' cosines and sines from a table made once per step) and stores q, k
// and v packed for the prompt's own attention, and k and v into the paged cache as well: what
// rope_store.cu does in a launch of its own, with the same operations in the same order, so
// both ways give the same bits.
struct QkvArgs {
  __nv_bfloat16* q;          // [T, Hq, d]
  __nv_bfloat16* k;          // [T, Hk, d]
  __nv_bfloat16* v;          // [T, Hk, d]
  __nv_bfloat16* k_pages;    // [pages, Hk, page_size, d] or nullptr
  __nv_bfloat16* v_pages;
  const int* dest_rows;      // [T]: page * page_size + row of the token in the cache, < 0: not stored
  const float2* table;       // [T, d / 2] (cos, sin) of position * inverse frequency, or nullptr: no rotation
  int q_heads, kv_heads, head_dim, page_size;
};

// One warp's 32 accumulator rows (tokens m0 ..) of a tile whose first column n0 is the first of a head and whose
// width BN is a whole number of heads: `tmem_row` addresses the rows' first column in tensor
// memory. Every lane of the warp must call it; rows beyond M only load.
// Of the tile's heads this call takes those that begin in columns [first, last).
template <int BN>
__device__ __forceinline__ void store_heads(uint32_t tmem_row, unsigned char* stage, int m0, int lane, int n0, int M, int N,
                                            const QkvArgs& a, int first = 0, int last = BN) {
  const int d = a.head_dim, half = d >> 1;
  // where this lane's row goes in the cache (head 0); the lanes that store it ask for it
  uint32_t place = 0xffffffffu;  // in rows of d
  if (m0 + lane < M && a.k_pages != nullptr) {
    const int dest = a.dest_rows[m0 + lane];
    if (dest >= 0) place = static_cast<uint32_t>(dest / a.page_size) * a.kv_heads * a.page_size + dest % a.page_size;
  }
  for (int c0 = first; c0 < last && n0 + c0 < N; c0 += d) {
    const int head = (n0 + c0) / d;
    const bool is_q = head < a.q_heads, is_v = head >= a.q_heads + a.kv_heads;
    const int kh = is_q ? 0 : head - a.q_heads - (is_v ? a.kv_heads : 0);
    __nv_bfloat16* packed_dst = is_q ? a.q + static_cast<size_t>(head) * d : (is_v ? a.v : a.k) + static_cast<size_t>(kh) * d;
    const size_t pitch = static_cast<size_t>(is_q ? a.q_heads : a.kv_heads) * d;
    __nv_bfloat16* cache_dst = is_q || a.k_pages == nullptr ? nullptr
        : (is_v ? a.v_pages : a.k_pages) + static_cast<size_t>(kh) * a.page_size * d;
    const auto put = [&](auto bytes, int c, const uint32_t* packed) {  // columns c .. of the head
      stage_row<decltype(bytes)::value>(stage, lane, packed);
      unstage<decltype(bytes)::value>(stage, lane, [&](int row, int byte, const uint4& v) {
        const uint32_t at = __shfl_sync(0xffffffffu, place, row);
        if (m0 + row >= M) return;
        *reinterpret_cast<uint4*>(packed_dst + (m0 + row) * pitch + c + byte / 2) = v;
        if (cache_dst != nullptr && at != 0xffffffffu)
          *reinterpret_cast<uint4*>(cache_dst + static_cast<size_t>(at) * d + c + byte / 2) = v;
      });
    };
    if (is_v || a.table == nullptr) {
      for (int c = 0; c < d; c += 32) {
        uint32_t r[32];
        tmem_load32(tmem_row + c0 + c, r);
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) packed[i] = pack_bf16(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        put(std::integral_constant<int, 64>(), c, packed);
      }
      continue;
    }
    for (int c = 0; c < half; c += 16) {  // columns c.. pair with columns half + c..
      // The angles come as runs of 64 bytes of a row too and reach the rows' lanes through the staging area: every lane loading
      // its own row's cost as much as the stores.
      uint4 angles[2][4];
#pragma unroll
      for (int part = 0; part < 2; ++part)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = min(m0 + i * 8 + (lane >> 2), M - 1);
          angles[part][i] = __ldg(reinterpret_cast<const uint4*>(a.table + static_cast<size_t>(row) * half + c + part * 8) +
                                  (lane & 3));
        }
      uint32_t lo[16], hi[16], out_lo[8], out_hi[8];
      tmem_load16(tmem_row + c0 + c, lo);
      tmem_load16(tmem_row + c0 + half + c, hi);
#pragma unroll
      for (int part = 0; part < 2; ++part) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = i * 8 + (lane >> 2), at = (lane & 3) ^ ((row >> 1) & 3);
          *reinterpret_cast<uint4*>(stage + row * 64 + at * 16) = angles[part][i];
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // (cos, sin) of two columns
          const int i = part * 4 + u;
          const float4 t = *reinterpret_cast<const float4*>(stage + lane * 64 + (u ^ ((lane >> 1) & 3)) * 16);
          // the projection is rounded to bfloat16 first, as where it is stored before it is rotated
          const float xa0 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(lo[2 * i])));
          const float xa1 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(lo[2 * i + 1])));
          const float xb0 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(hi[2 * i])));
          const float xb1 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(hi[2 * i + 1])));
          out_lo[i] = pack_bf16(fmaf(xa0, t.x, -__fmul_rn(xb0, t.y)), fmaf(xa1, t.z, -__fmul_rn(xb1, t.w)));
          out_hi[i] = pack_bf16(fmaf(xa0, t.y, __fmul_rn(xb0, t.x)), fmaf(xa1, t.w, __fmul_rn(xb1, t.z)));
        }
        __syncwarp();
      }
      put(std::integral_constant<int, 32>(), c, out_lo);
      put(std::integral_constant<int, 32>(), half + c, out_hi);
    }
  }
}

}  // namespace
