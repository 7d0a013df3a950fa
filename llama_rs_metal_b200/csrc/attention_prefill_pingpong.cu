// Causal grouped-query flash attention for prompts on the 5th-generation tensor cores, with
// scores, probabilities and output in tensor memory and two chains of key tiles taking turns.
//
// Keys and values arrive in tiles through TMA (cp.async.bulk.tensor, 128-byte swizzle, a ring of
// stages). For a tile of 128 queries of one head and key tile j:
//   S = Q K_j^T    tcgen05.mma, M 128, K = head size, into tensor memory
//   softmax        four warps, one thread per query row: tcgen05.ld of the row, causal and window
//                  mask, running maximum and mass in float32 (log2 domain), P = 2^(s - m) rounded
//                  to bfloat16 and written back into tensor memory over the scores it came from
//                  (two values per column)
//   O += P V_j     tcgen05.mma with P read from tensor memory as the A operand and V from
//                  shared memory as an MN-major operand exactly as TMA laid it down; O stays
//                  in tensor memory for the whole row of key tiles
// Every step waits for the one before it, some 2,500 cycles per 64 keys (of a lone CTA: 310 until the issuer sees the
// probabilities, 180 and 175 to issue the two products, 285 until the scores are there, 120 for the load, 180 for the
// maximum, 400 for a rescaling, 740 for the probabilities, which the 2^x unit needs 512 for), so what bounds a prompt is
// how many such chains an SM has under way and how long the longest is. Three forms:
//   two chains per query tile   key tiles of 64, the even ones one chain and the odd ones the other,
//                               each with its own maximum, mass and O; at the end the two threads of a
//                               row exchange maximum and mass and each finishes half of the columns.
//                               Two CTAs per SM with head size 64, one with 128.
//   one chain                   key tiles of 64, twice the CTAs per SM: more of them begin and end under
//                               others, which short prompts by the dozen need.
//   two query tiles             head size 128, key tiles of 128: a chain each, sharing the keys and values.
// The issuing thread alternates between its two chains, so one's softmax runs under the other's products.
// A row's scores stay in registers from the maximum to the probabilities (except where four CTAs share an
// SM's), its maximum is taken as four, scale and mass two values an instruction.
//
// O is rescaled only when a row's maximum has moved by more than 2^rescale_step since the scale O was
// last brought to (the row's own thread multiplies its O row in tensor memory); P is formed against
// that older maximum meanwhile and stays below 2^8, and the division by the mass at the end makes
// the result exact regardless. With a step of 0 the largest probability is 1 and not rounded, which halves
// the error that rounding the probabilities gives (of 2,048 tokens: 0.00191 of the result, 0.00206 with a
// step of 8; the result's own rounding is 0.00180 of it), for a tenth more time.
//
// Rows and keys outside a sequence are zero-filled by TMA or belong to a neighbouring sequence
// of the packed batch; the causal mask hides such keys and such rows are never stored.
// PAGED: several queries per started sequence over its paged cache, which already holds the step's keys. A key tile is a
// page (64 keys, one piece of memory per head); the queries stand at the last positions of their sequence. The rows of a
// sequence's last page that hold no key of it are whatever an earlier owner left: their scores are masked, and their
// values are zeroed in shared memory before the tensor core may multiply them (0 x NaN).
//
// Every mbarrier wait is bounded; a wait that gives up records a code in `status`, and the CTA
// winds down and frees its tensor memory. No cluster multicast. Head sizes 64 and 128.
// (Reference: crates/metal-backend/src/shaders/attention.metal:28-57, the streaming softmax.)
#include <type_traits>

#include "umma.cuh"

namespace {

constexpr int BQ = 128, UMMA_K = 16;
// four softmax warps for each of the two chains, then the loader, then the issuer

enum : int { kStuckQ = 21, kStuckKV = 22, kStuckScores = 23, kStuckProbabilities = 24, kStuckOutput = 25,
             kStuckStage = 26, kMisaligned = 27 };

// NQ query tiles per CTA, CHAINS of dependent key tiles (equal to NQ with two query tiles).
template <int D, int NQ, int CHAINS> struct Shape {
  static constexpr int kThreads = (4 * CHAINS + 2) * 32;
  static constexpr int kStages = CHAINS == 2 && NQ == 1 ? 5 : 2;
  static constexpr int kCtasPerSm = NQ == 2 ? 1 : (D == 64 ? 4 : 2) / CHAINS;
  static constexpr int BKV = NQ == 2 ? 128 : 64;
  static constexpr bool kHold = kCtasPerSm < 4;  // registers for a row's scores
  static constexpr int kSmem = NQ * BQ * D * 2 + 2 * kStages * BKV * D * 2 + 256 + (CHAINS > NQ ? 2 * BQ * 8 : 0);
};

// The cache of a PAGED launch.
struct Pages {
  const int* table;    // [slots][stride]
  int stride;
  const int* slots;    // per sequence
  const int* kv_lens;  // keys per sequence, the step's own included
};

// Item u of the packed prompts' row tiles of `rows` queries, the last tiles (the longest rows of work under the causal mask)
// first: its sequence and its tile there, or -1. A warp per call, all with the same u; up to 32 sequences.
__device__ __forceinline__ int2 find_tile(int u, const int* __restrict__ cu_seqlens, int seqs, int rows) {
  const int lane = threadIdx.x & 31;
  const int mine = lane < seqs ? (cu_seqlens[lane + 1] - cu_seqlens[lane] + rows - 1) / rows : 0;  // tiles of a sequence
  auto behind = [&](int z) { return __reduce_add_sync(0xffffffffu, max(0, mine - 1 - z)); };       // items of tiles after z
  int low = 0, high = __reduce_max_sync(0xffffffffu, mine) - 1;
  if (u >= behind(-1)) return make_int2(-1, -1);
  while (low < high) {  // the first z with no more than u items behind it
    const int z = (low + high) >> 1;
    if (behind(z) <= u) high = z;
    else low = z + 1;
  }
  unsigned which = __ballot_sync(0xffffffffu, mine > low);
  for (int skip = u - behind(low); skip > 0; --skip) which &= which - 1;
  return make_int2(__ffs(which) - 1, low);
}

template <int D, int NQ, int CHAINS, bool PAGED>
__global__ __launch_bounds__((Shape<D, NQ, CHAINS>::kThreads), (Shape<D, NQ, CHAINS>::kCtasPerSm))
void attention_prefill_pingpong_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
    const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
    const int* __restrict__ cu_seqlens, int q_heads, int kv_heads, float scale_log2, int window,
    int* __restrict__ status, Pages pages, int listed, float rescale_step) {
  constexpr int BKV = Shape<D, NQ, CHAINS>::BKV;
  constexpr bool HOLD = Shape<D, NQ, CHAINS>::kHold;
  constexpr uint32_t TILE = BQ * D * 2;       // bytes of one [128][D] query tile
  constexpr uint32_t BLOCK = BQ * 64 * 2;     // bytes of one [128][64] block of it
  constexpr uint32_t KV_TILE = BKV * D * 2;   // bytes of one [BKV][D] key or value tile
  constexpr uint32_t KV_BLOCK = BKV * 64 * 2; // bytes of one [BKV][64] block of it
  constexpr int DB = D / 64;                  // 64-column blocks per tile
  constexpr int STAGES = Shape<D, NQ, CHAINS>::kStages;
  static_assert(NQ == 1 || CHAINS == NQ, "a chain per query tile, or two for one");
  static_assert(!PAGED || BKV == 64, "a page has 64 keys");
  constexpr int kLoaderWarp = 4 * CHAINS, kIssuerWarp = kLoaderWarp + 1;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0) {  // the swizzled tiles need it; give up rather than compute nonsense
    if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0, kMisaligned);
    return;
  }
  // NQ query tiles [BQ][D], STAGES pairs of a key and a value tile [BKV][D], barriers. A tile with D = 128 is two blocks of 64
  // columns one after the other (a swizzle row is 128 bytes = 64 elements).
  unsigned char* q_tiles = smem_raw;
  unsigned char* kv_tiles = q_tiles + NQ * TILE;            // stage s: K at s * 2 * KV_TILE, V right after
  uint64_t* bars = reinterpret_cast<uint64_t*>(kv_tiles + STAGES * 2 * KV_TILE);
  uint64_t* q_full = bars;
  uint64_t* kv_full = bars + 1;               // [STAGES]
  uint64_t* kv_free = kv_full + STAGES;       // [STAGES]
  uint64_t* s_full = kv_free + STAGES;        // [2] scores of tile i written
  uint64_t* p_ready = s_full + 2;             // [2] probabilities of tile i written (4 warps arrive)
  uint64_t* o_done = p_ready + 2;             // [2] the last P V of tile i is complete
  uint64_t* tail = o_done + 2;                // PAGED: the last page has arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 1);
  volatile int* bail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float2* halves = reinterpret_cast<float2*>(bars + 32);  // CHAINS > NQ: [2][128] maximum and mass of a row in either chain

  // CTAs are handed out in the order x, y, z: all heads and sequences of the last pair of query
  // tiles (the longest rows of work under the causal mask) first. `listed`: sequences of a grid that has a CTA per head and
  // tile there is, in the same order. Tiles that some sequences do not have would otherwise each wait for a CTA's worth of
  // shared memory before they end.
  int pair, b, h;
  if (listed > 0) {
    h = blockIdx.x % q_heads;
    const int2 tile = find_tile(blockIdx.x / q_heads, cu_seqlens, listed, NQ * BQ);
    b = tile.x, pair = tile.y;
    if (b < 0) return;
  } else {
    pair = gridDim.z - 1 - blockIdx.z, h = blockIdx.x, b = blockIdx.y;
  }
  const int start = cu_seqlens[b], len = cu_seqlens[b + 1] - start;
  const int q0 = pair * NQ * BQ;
  if (q0 >= len) return;
  const int kh = h / (q_heads / kv_heads);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // position of the sequence's first query, and the keys there are (PAGED: no key tile beyond them exists)
  const int base = PAGED ? pages.kv_lens[b] - len : 0, keys = base + len;
  const int kt_first = window > 0 ? max(0, base + q0 - window + 1) / BKV : 0;
  // Key tiles of either chain: with two query tiles, each up to its diagonal tile (the second may not exist); with one,
  // all of its key tiles, or the even and the odd ones.
  const int in_all = (min(base + q0 + BQ, keys) - 1) / BKV - kt_first + 1;
  const int n0 = NQ == 2 ? (q0 + BQ - 1) / BKV - kt_first + 1 : (in_all + CHAINS - 1) / CHAINS;
  const int n1 = NQ == 1 ? (CHAINS == 2 ? in_all / 2 : 0) : q0 + BQ < len ? n0 + 1 : 0;
  const int n_tiles = NQ == 1 ? in_all : max(n0, n1);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_free + s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(s_full + i, 1);
      mbar_init(p_ready + i, 4);
      mbar_init(o_done + i, 1);
    }
    mbar_init(tail, 1);
    *bail = 0;
    mbar_fence_init();
  }
  constexpr uint32_t kUsed = CHAINS * (BKV + D), kTmemColumns = kUsed <= 128 ? 128 : kUsed <= 256 ? 256 : 512;  // a power of two
  if (warp == kIssuerWarp) {
    tmem_alloc(tmem_slot, kTmemColumns);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto tmem_s = [&](int i) { return tmem_base + i * BKV; };
  auto tmem_o = [&](int i) { return tmem_base + CHAINS * BKV + i * D; };
  // Barriers and tensor memory were set up while the kernel that produces q, k and v may still
  // have been running (sequence bounds are the step's own input); its results are read from here on.
  pdl_wait();

  if (warp == kLoaderWarp) {
    // ---- one thread brings the query tiles once and the key/value tiles through the ring
    if (lane == 0) {
      const int q_held = NQ == 2 && n1 > 0 ? 2 : 1;
      mbar_expect_tx(q_full, q_held * TILE);
      for (int i = 0; i < q_held; ++i)
#pragma unroll
        for (int db = 0; db < DB; ++db)
          tma_load_2d(q_tiles + i * TILE + db * BLOCK, &map_q, q_full, h * D + db * 64, start + q0 + i * BQ);
    }
    auto bring = [&](int j, uint64_t* arrives, int column, int row) {
      unsigned char* kdst = kv_tiles + j % STAGES * 2 * KV_TILE;
      mbar_expect_tx(arrives, 2 * KV_TILE);
#pragma unroll
      for (int db = 0; db < DB; ++db) {
        tma_load_2d(kdst + db * KV_BLOCK, &map_k, arrives, column + db * 64, row);
        tma_load_2d(kdst + KV_TILE + db * KV_BLOCK, &map_v, arrives, column + db * 64, row);
      }
    };
    if constexpr (!PAGED) {
      if (lane == 0) {
        for (int j = 0; j < n_tiles && !*bail; ++j) {
          const int s = j % STAGES;
          if (j >= STAGES && !mbar_wait(kv_free + s, ((j / STAGES) - 1) & 1, status, kStuckStage)) {
            *bail = 1;
            break;
          }
          bring(j, kv_full + s, kh * D, start + (kt_first + j) * BKV);
        }
      }
    } else {
      const int* table = pages.table + static_cast<size_t>(pages.slots[b]) * pages.stride;
      const int tail_tile = keys % BKV != 0 ? keys / BKV - kt_first : -1;  // the page with rows that hold no key
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % STAGES;
        bool ok = true;  // (every decision is lane 0's: the warp stays together)
        if (lane == 0) {
          ok = !*bail && (j < STAGES || mbar_wait(kv_free + s, ((j / STAGES) - 1) & 1, status, kStuckStage));
          if (ok) bring(j, j == tail_tile ? tail : kv_full + s, 0, (table[kt_first + j] * kv_heads + kh) * BKV);
          if (ok && j == tail_tile) ok = mbar_wait(tail, 0, status, kStuckKV);
          if (!ok) *bail = 1;
        }
        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        if (j != tail_tile) continue;
        mbar_wait(tail, 0, status, kStuckKV);  // (lane 0 saw it complete) makes the copies visible to every lane
        // whole rows of 128 bytes, so the swizzle within a row does not matter
        unsigned char* values = kv_tiles + s * 2 * KV_TILE + KV_TILE;
        const int first = keys % BKV;
        for (int i = lane; i < (BKV - first) * 8; i += 32)
#pragma unroll
          for (int db = 0; db < DB; ++db)
            *reinterpret_cast<uint4*>(values + db * KV_BLOCK + first * 128 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(kv_full + s);
      }
    }
  } else if (warp == kIssuerWarp) {
    // ---- one thread drives the tensor core. The warp stays together around it, so that descriptors are computed once per
    // warp: with a branch of one lane around the loop a product's four MMAs took 340 cycles to issue.
    constexpr uint32_t idesc_s = umma_idesc(BQ, BKV);            // both K-major
    constexpr uint32_t idesc_pv = umma_idesc(BQ, D, true);       // V is MN-major
    const uint32_t q_at = smem_u32(q_tiles), kv_at = smem_u32(kv_tiles);
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    const int tiles = __shfl_sync(0xffffffffu, n_tiles, 0), last0 = __shfl_sync(0xffffffffu, n0, 0) - 1,
              last1 = __shfl_sync(0xffffffffu, n1, 0) - 1;
    const bool leader = elect_one();
    auto wait = [&](uint64_t* bar, int parity, int where) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, status, where));
      tc_fence_after();
      return ok;
    };
    auto scores = [&](int i, int j) {  // S_i = Q_i K_j^T
      const uint32_t qa = q_at + (NQ == 2 ? i * TILE : 0), ka = kv_at + (j % STAGES) * 2 * KV_TILE;
      if (leader) {
#pragma unroll
        for (int k = 0; k < D / UMMA_K; ++k) {  // 64-column block, then 32 bytes per step
          const uint32_t step = (k % 4) * UMMA_K * 2;
          umma_bf16(tmem + i * BKV, smem_desc(qa + (k / 4) * BLOCK + step), smem_desc(ka + (k / 4) * KV_BLOCK + step),
                    idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(s_full + i);
      }
    };
    // O_i (+)= P_i V_j, P from tensor memory (8 columns per 16 keys). `frees`: the last product that reads stage j; `ends`: the
    // chain's last. The commits stand in the elected lane's block of products, like that of the scores: one in an `if` of its own was
    // lost or came twice in a GEMM of this form (gemm_bf16_umma.cu). The one that is waited for before the CTA leaves is the last.
    auto weighted = [&](int i, int j, bool frees, bool ends) {
      const uint32_t va = kv_at + (j % STAGES) * 2 * KV_TILE + KV_TILE;
      if (leader) {
#pragma unroll
        for (int k = 0; k < BKV / UMMA_K; ++k)
          umma_bf16_a_tmem(tmem + CHAINS * BKV + i * D, tmem + i * BKV + k * (UMMA_K / 2),
                           smem_desc(va + k * UMMA_K * 128, KV_BLOCK), idesc_pv, (j >= CHAINS / NQ || k > 0) ? 1u : 0u);
        if (frees) umma_commit(kv_free + j % STAGES);
        if (ends) umma_commit(o_done + i);
      }
    };
    bool ok = wait(q_full, 0, kStuckQ) && wait(kv_full, 0, kStuckKV);
    if (ok) scores(0, 0);
    if constexpr (NQ == 1) {  // key tile t belongs to chain t % CHAINS
      if (CHAINS == 2 && ok && tiles > 1) {
        ok = wait(kv_full + 1, 0, kStuckKV);
        if (ok) scores(1, 1);
      }
      for (int t = 0; t < tiles && ok; ++t) {
        const int i = t % CHAINS, next = t + CHAINS;
        if (next < tiles) ok = wait(kv_full + next % STAGES, (next / STAGES) & 1, kStuckKV);
        ok = ok && wait(p_ready + i, (t / CHAINS) & 1, kStuckProbabilities);
        if (!ok) break;
        weighted(i, t, true, next >= tiles);
        if (next < tiles) scores(i, next);
      }
    } else {
      if (ok && last1 >= 0) scores(1, 0);
      for (int j = 0; j < tiles && ok; ++j) {
        if (j <= last0) {
          ok = wait(p_ready + 0, j & 1, kStuckProbabilities);
          if (!ok) break;
          weighted(0, j, j > last1, j == last0);
        }
        if (j < last0 || j < last1) {  // the next key tile has to be here for the next scores
          ok = wait(kv_full + (j + 1) % STAGES, ((j + 1) / STAGES) & 1, kStuckKV);
          if (!ok) break;
        }
        if (j < last0) scores(0, j + 1);
        if (j <= last1) {
          ok = wait(p_ready + 1, j & 1, kStuckProbabilities);
          if (!ok) break;
          weighted(1, j, true, j == last1);
        }
        if (j < last1) scores(1, j + 1);
      }
    }
    if (!ok) *bail = 1;
  } else {
    // ---- softmax and output: one thread per query row and chain. Warps 0-3 own chain 0, warps 4-7 chain 1;
    // a warp may touch the quarter of the tensor memory's lanes given by its index modulo 4.
    const int i = warp >> 2, quad = warp & 3;
    const int n_mine = i == 0 ? n0 : n1;
    const int query = q0 + (NQ == 2 ? i * BQ : 0) + quad * 32 + lane;  // of the sequence's queries
    const int row = base + query;                      // position in the sequence
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t my_s = tmem_s(i) + lane_base, my_o = tmem_o(i) + lane_base;
    float m_run = -INFINITY;   // the row's true running maximum (log2 domain)
    float m_ref = -INFINITY;   // the maximum O and the mass are scaled by
    float l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_mine; ++j) {
      if (*bail || !mbar_wait(s_full + i, j & 1, status, kStuckScores)) {
        *bail = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      const int key0 = (kt_first + (NQ == 2 ? j : CHAINS * j + i)) * BKV;
      const int first_row = base + q0 + (NQ == 2 ? i * BQ : 0);
      const bool edge = key0 + BKV - 1 > first_row || (window > 0 && key0 <= first_row + BQ - 1 - window);
      // the row comes into registers at once (all loads in flight, one wait) and stays there where they suffice; four running maxima, since
      // this is a chain of dependent steps (only tiles on the diagonal or the window's edge need the mask)
      constexpr int kChunks = BKV / 32;
      uint32_t sc[kChunks][32];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) tmem_load32_async(my_s + c * 32, sc[c]);
      tmem_load_wait();
#pragma unroll
      for (int c = 0; c < kChunks; ++c) tmem_pin(sc[c]);
      const int to = row - key0, from = window > 0 ? to - window : -1;  // keys from + 1 .. to of the tile count
      float most[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (edge) {
#pragma unroll
        for (int c = 0; c < kChunks; ++c)
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (c * 32 + e <= to && c * 32 + e > from) most[e & 3] = fmaxf(most[e & 3], __uint_as_float(sc[c][e]));
      } else {
#pragma unroll
        for (int c = 0; c < kChunks; ++c)
#pragma unroll
          for (int e = 0; e < 32; e += 8)
#pragma unroll
            for (int u = 0; u < 4; ++u)
              most[u] = fmaxf(fmaxf(most[u], __uint_as_float(sc[c][e + u])), __uint_as_float(sc[c][e + 4 + u]));
      }
      const float mx = fmaxf(fmaxf(most[0], most[1]), fmaxf(most[2], most[3]));
      m_run = fmaxf(m_run, mx * scale_log2);
      // bring O and the mass to the new maximum only when it has moved far (always for the first
      // tile, where O holds nothing yet and only the reference is set); here, since behind the probabilities it was slower
      // (8,192 tokens of head size 64 378 us, here 366)
      const bool far = m_run > m_ref + rescale_step;
      if (j == 0) {
        m_ref = m_run;
      } else if (__any_sync(0xffffffffu, far)) {
        const float alpha = far ? fast_exp2(m_ref - m_run) : 1.0f;  // m_ref = -inf gives 0, and O is 0 then
#pragma unroll 1
        for (int c = 0; c < D / 16; ++c) {  // (few at a time: the row's scores are in registers)
          uint32_t r[16];
          tmem_load16(my_o + c * 16, r);
#pragma unroll
          for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
          tmem_store16(my_o + c * 16, r);
        }
        tmem_store_wait();
        l *= alpha;
        if (far) m_ref = m_run;
      }
      const float m_use = m_ref == -INFINITY ? 0.f : m_ref;  // a row that has seen no key yet
      // probabilities against m_ref, rounded to bfloat16, written over the scores they came from: keys 16 c .. 16 c + 15
      // become columns 8 c .. 8 c + 7
      float2 sums[2] = {{0.f, 0.f}, {0.f, 0.f}};
      const float2 scale2{scale_log2, scale_log2}, less{-m_use, -m_use};
      auto probabilities = [&](auto masked) {
#pragma unroll
        for (int c = 0; c < 2 * kChunks; ++c) {
          if (!HOLD && c % 2 == 0) {  // the next 32 scores are on their way while these are worked on
            tmem_load_wait();
            tmem_pin(sc[c / 2]);
            if (c / 2 + 1 < kChunks) tmem_load32_async(my_s + (c / 2 + 1) * 32, sc[c / 2 + 1]);
          }
          uint32_t packed[8];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const int key = c * 16 + e;
            const float2 x = fma_f32x2(float2{__uint_as_float(sc[key / 32][key % 32]), __uint_as_float(sc[key / 32][key % 32 + 1])},
                                       scale2, less);
            float2 p{fast_exp2(x.x), fast_exp2(x.y)};
            if constexpr (decltype(masked)::value) {
              if (!(key <= to && key > from)) p.x = 0.f;
              if (!(key + 1 <= to && key + 1 > from)) p.y = 0.f;
            }
            sums[(e >> 1) & 1] = add_f32x2(sums[(e >> 1) & 1], p);
            packed[e >> 1] = pack_bf16(p.x, p.y);
          }
          tmem_store8(my_s + c * 8, packed);
        }
      };
      if (!HOLD) tmem_load32_async(my_s, sc[0]);
      if (edge) probabilities(std::true_type{});
      else probabilities(std::false_type{});
      const float sum = (sums[0].x + sums[0].y) + (sums[1].x + sums[1].y);
      tmem_store_wait();
      l += sum;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready + i);
    }
    if constexpr (CHAINS > NQ) {
      // Both chains' outputs lie in the lanes of this warp's quarter: the two threads of a row tell each other maximum and
      // mass, and each finishes half of the row's columns.
      ok = ok && mbar_wait(o_done, 0, status, kStuckOutput) && (n1 == 0 || mbar_wait(o_done + 1, 0, status, kStuckOutput));
      if (!ok) *bail = 1;
      halves[i * BQ + quad * 32 + lane] = make_float2(m_ref, l);
      asm volatile("bar.sync 1, 256;" ::: "memory");  // the softmax warps, whatever became of their waits
      tc_fence_after();
      if (ok) {
        const float2 other = halves[(i ^ 1) * BQ + quad * 32 + lane];
        const float top = fmaxf(m_ref, other.x), m_use = top == -INFINITY ? 0.f : top;
        const float mine = fast_exp2(m_ref - m_use), theirs = fast_exp2(other.x - m_use);
        const float inv = 1.0f / (l * mine + other.y * theirs);
        const float w0 = (i == 0 ? mine : theirs) * inv, w1 = (i == 0 ? theirs : mine) * inv;
        __nv_bfloat16* dst = out + (static_cast<size_t>(start + query) * q_heads + h) * D;
#pragma unroll 1
        for (int c = i * (D / 64); c < (i + 1) * (D / 64); ++c) {
          uint32_t r[32], r1[32];
          tmem_load32(tmem_o(0) + lane_base + c * 32, r);
          if (n1 > 0) {
            tmem_load32(tmem_o(1) + lane_base + c * 32, r1);
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(fmaf(__uint_as_float(r[e]), w0, __uint_as_float(r1[e]) * w1));
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * w0);
          }
          if (query < len) {
#pragma unroll
            for (int e = 0; e < 32; e += 8)
              *reinterpret_cast<uint4*>(dst + c * 32 + e) =
                  make_uint4(pack_bf16(__uint_as_float(r[e]), __uint_as_float(r[e + 1])),
                             pack_bf16(__uint_as_float(r[e + 2]), __uint_as_float(r[e + 3])),
                             pack_bf16(__uint_as_float(r[e + 4]), __uint_as_float(r[e + 5])),
                             pack_bf16(__uint_as_float(r[e + 6]), __uint_as_float(r[e + 7])));
          }
        }
      }
    }
    if (CHAINS == NQ && ok && n_mine > 0) {
      if (!mbar_wait(o_done + i, 0, status, kStuckOutput)) {
        *bail = 1;
        ok = false;
      }
      tc_fence_after();
    }
    if (CHAINS == NQ && ok && n_mine > 0) {
      // the mass belongs to m_ref, and so does O: their quotient is the row's attention output
      const float inv = 1.0f / l;
      __nv_bfloat16* dst = out + (static_cast<size_t>(start + query) * q_heads + h) * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_load32(my_o + c * 32, r);
        if (query < len) {
#pragma unroll
          for (int e = 0; e < 32; e += 8)
            *reinterpret_cast<uint4*>(dst + c * 32 + e) = make_uint4(
                pack_bf16(__uint_as_float(r[e]) * inv, __uint_as_float(r[e + 1]) * inv),
                pack_bf16(__uint_as_float(r[e + 2]) * inv, __uint_as_float(r[e + 3]) * inv),
                pack_bf16(__uint_as_float(r[e + 4]) * inv, __uint_as_float(r[e + 5]) * inv),
                pack_bf16(__uint_as_float(r[e + 6]) * inv, __uint_as_float(r[e + 7]) * inv));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kIssuerWarp) tmem_dealloc(tmem_base, kTmemColumns);
}

// Query tiles there are at most, all sequences together.
long long tiles_of(int seqs, int tokens, int max_seq_len) {
  const long long longest = (max_seq_len + BQ - 1) / BQ;
  return min(seqs * longest, tokens / BQ + static_cast<long long>(seqs));
}

// The grid, and the kernel's `listed`. Heads x sequences x tiles unless a third of it would be tiles that shorter sequences
// do not have: 32 heads of 64, prompts of 3,001, 517 and 1,200 tokens 93 us (112 with them in the grid), of 777, 300, 1,500,
// 31, 2,500, 64 and 900 100 us (132). Finding the tile costs each CTA about 0.5 us (16 prompts of 256 tokens 29.4 us
// against 26.1), and a warp looks at 32 sequences.
int choose_grid(int q_heads, int seqs, int tokens, int tiles, int rows, dim3& grid) {
  const long long all = static_cast<long long>(seqs) * tiles, there = min(all, tokens / rows + static_cast<long long>(seqs));
  if (seqs <= 32 && 2 * all > 3 * there && q_heads * there < (1ll << 31)) {
    grid = dim3(static_cast<unsigned>(q_heads * there));
    return seqs;
  }
  grid = dim3(q_heads, seqs, tiles);
  return 0;
}

template <int D, int NQ, int CHAINS>
int launch(const void* q, const void* k, const void* v, void* out, const int* cu_seqlens, int tokens,
           int seqs, int max_seq_len, int q_heads, int kv_heads, float scale, int window, int* status,
           float rescale_step, cudaStream_t stream) {
  using S = Shape<D, NQ, CHAINS>;
  constexpr int BKV = S::BKV, smem = S::kSmem;
  CUtensorMap map_q, map_k, map_v;
  if (!make_map_bf16(&map_q, q, tokens, static_cast<long long>(q_heads) * D, BQ) ||
      !make_map_bf16(&map_k, k, tokens, static_cast<long long>(kv_heads) * D, BKV) ||
      !make_map_bf16(&map_v, v, tokens, static_cast<long long>(kv_heads) * D, BKV))
    return LRM_UNSUPPORTED;

  auto kernel = attention_prefill_pingpong_kernel<D, NQ, CHAINS, false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int pairs = (max_seq_len + NQ * BQ - 1) / (NQ * BQ);
  if (seqs > 65535 || pairs > 65535) return LRM_UNSUPPORTED;
  dim3 grid;
  const int listed = choose_grid(q_heads, seqs, tokens, pairs, NQ * BQ, grid);
  LRM_LAUNCH(kernel, grid, dim3(S::kThreads), smem, stream, map_q, map_k, map_v,
             static_cast<__nv_bfloat16*>(out), cu_seqlens, q_heads, kv_heads, scale * 1.4426950408889634f, window,
             status, Pages{}, listed, rescale_step);
  return 0;
}

template <int D, int CHAINS>
int launch_paged(const void* q, const void* k_pages, const void* v_pages, long long page_rows, void* out, const int* cu_seqlens,
                 const Pages& pages, int tokens, int seqs, int max_seq_len, int q_heads, int kv_heads, float scale, int window,
                 int* status, cudaStream_t stream) {
  using S = Shape<D, 1, CHAINS>;
  constexpr int BKV = S::BKV, smem = S::kSmem;
  CUtensorMap map_q, map_k, map_v;
  if (!make_map_bf16(&map_q, q, tokens, static_cast<long long>(q_heads) * D, BQ) ||
      !make_map_bf16(&map_k, k_pages, page_rows, D, BKV) || !make_map_bf16(&map_v, v_pages, page_rows, D, BKV))
    return LRM_UNSUPPORTED;

  auto kernel = attention_prefill_pingpong_kernel<D, 1, CHAINS, true>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int tiles = (max_seq_len + BQ - 1) / BQ;
  if (seqs > 65535 || tiles > 65535) return LRM_UNSUPPORTED;
  dim3 grid;
  const int listed = choose_grid(q_heads, seqs, tokens, tiles, BQ, grid);
  LRM_LAUNCH(kernel, grid, dim3(S::kThreads), smem, stream, map_q, map_k, map_v,
             static_cast<__nv_bfloat16*>(out), cu_seqlens, q_heads, kv_heads, scale * 1.4426950408889634f, window, status, pages, listed, 0.f);
  return 0;
}

}  // namespace

LRM_API int lrm_attention_prefill_pingpong_supports(int head_dim) {
  return (head_dim == 64 || head_dim == 128) && encode_tiled() != nullptr ? 1 : 0;
}

// q [tokens, q_heads, d], k, v [tokens, kv_heads, d] packed bfloat16, 16-byte aligned; `status`: one
// int in device memory, 0 before the launch; a kernel that gave up on a wait writes a code there.
// `form`: 1 one chain, 2 two chains, 3 two query tiles (head size 128), 0 the rule below.
LRM_API int lrm_attention_prefill_pingpong(const void* q, const void* k, const void* v, void* out,
                                           const int* cu_seqlens, int tokens, int seqs, int max_seq_len,
                                           int q_heads, int kv_heads, int d, float scale, int window, int form,
                                           int* status, cudaStream_t stream) {
  if (seqs <= 0 || max_seq_len <= 0 || tokens <= 0) return 0;
  if (q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0 || status == nullptr) return LRM_BAD_ARGUMENT;
  if (form < 0 || form > 3 || (form == 3 && d != 128)) return LRM_BAD_ARGUMENT;
  if (q_heads > 65535 || seqs > 65535 || (d != 64 && d != 128)) return LRM_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(q) % 16 || reinterpret_cast<uintptr_t>(k) % 16 ||
      reinterpret_cast<uintptr_t>(v) % 16 || reinterpret_cast<uintptr_t>(out) % 16)
    return LRM_UNSUPPORTED;
  // (a short prompt filled up to whole rows with a few tokens of padding is one prompt)
  const bool single = 4ll * tokens < 5ll * max_seq_len;
  const long long ctas = q_heads * tiles_of(seqs, tokens, max_seq_len);
  const int reach = window > 0 && window < max_seq_len ? window : max_seq_len;
  // One prompt of moderate length: the exact maximum (see the header), the precision such prompts have always had.
  const float step = single && max_seq_len <= (d == 64 ? 2048 : 1535) ? 0.f : 8.f;
  if (form == 0) {
    if (d == 64) {
      // us, one chain and two, 32 heads: one prompt of 512 tokens 14.6 and 10.5, 2,048 51 and 41, 8,192 384 and 366; packed two of
      // 1,000 28.5 and 26.2, four of 768 32.3 and 31.1, four of 800 36.4 and 37.9, unequal ones the same within 3 %; but four of
      // 512 19.3 and 19.6, sixteen of 256 28.1 and 29.1, 32 of 128 22.9 and 26.7, eight of 700 53 and 56 (more than two CTAs per
      // SM, and short ones).
      form = !single && max_seq_len <= 768 && ctas > 2 * kSmCount ? 1 : 2;
    } else {
      // us, one chain, two, two query tiles, 24 heads: one prompt of 512 tokens 18, 14, 20, 1,024 28, 20, 30, 1,500 38, 31, 37,
      // 2,048 44, 50, 41, 8,192 450, 522, 374; packed two of 1,000 28, 35, 32, four of 512 23, 28, 28, sixteen of 256 33, 44, 39,
      // eight of 700 64, 81, 68; 700, 1,333, 64, 257 and 1,999 68, 85, 74, 3,001, 517 and 1,200 98, 121, 97; 2,048 within a window
      // of 512 37, 39, 41 (before the issuing warp stayed together).
      form = max_seq_len > 1535 && reach >= 1024 ? 3 : (single ? max_seq_len <= 1535 : ctas <= kSmCount) ? 2 : 1;
    }
  }
  const auto run = d == 64 ? (form == 1 ? launch<64, 1, 1> : launch<64, 1, 2>)
                           : (form == 1 ? launch<128, 1, 1> : form == 2 ? launch<128, 1, 2> : launch<128, 2, 2>);
  return run(q, k, v, out, cu_seqlens, tokens, seqs, max_seq_len, q_heads, kv_heads, scale, window, status, step, stream);
}

// Several queries per sequence over the paged cache: q [tokens, q_heads, d] packed by cu_seqlens, the queries of sequence b at
// its last positions of kv_lens[b]; pages [n_pages][kv_heads][64][d] of keys and of values, page_table [slots][table_stride].
LRM_API int lrm_attention_extend_umma(const void* q, const void* k_pages, const void* v_pages, int n_pages, void* out,
                                      const int* cu_seqlens, const int* page_table, int table_stride, const int* slots,
                                      const int* kv_lens, int tokens, int seqs, int max_seq_len, int q_heads, int kv_heads, int d,
                                      int page_size, float scale, int window, int* status, cudaStream_t stream) {
  if (seqs <= 0 || max_seq_len <= 0 || tokens <= 0) return 0;
  if (q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0 || n_pages <= 0 || status == nullptr) return LRM_BAD_ARGUMENT;
  const long long rows = static_cast<long long>(n_pages) * kv_heads * 64;
  if (page_size != 64 || window < 0 || q_heads > 65535 || rows >= (1ll << 31)) return LRM_UNSUPPORTED;
  for (const void* p : {q, k_pages, v_pages, static_cast<const void*>(out)})
    if (reinterpret_cast<uintptr_t>(p) % 16) return LRM_UNSUPPORTED;
  const Pages pages{page_table, table_stride, slots, kv_lens};
  if (d != 64 && d != 128) return LRM_UNSUPPORTED;
  // Two chains where one would leave SMs with a single CTA, us, one chain and two: head size 64 (32 heads) 400 and 129 tokens
  // onto 3,000 and 1,111 77 and 48, eight times 16 onto 3,000 72 and 46; head size 128, 128 onto 3,000 64 and 43, 400 and 129
  // 78 and 63, 1,000 onto 5,000 136 and 143, eight times 16 onto 3,000 75 and 84, 2,000 onto 16,000 742 and 814, of 24 heads
  // 717 and 616.
  const long long ctas = q_heads * max(static_cast<long long>(seqs), static_cast<long long>(tokens / BQ));
  const bool two = d == 64 || (ctas + kSmCount - 1) / kSmCount < 2 * ((ctas + 2 * kSmCount - 1) / (2 * kSmCount));
  const auto run = d == 64 ? launch_paged<64, 2> : two ? launch_paged<128, 2> : launch_paged<128, 1>;
  return run(q, k_pages, v_pages, rows, out, cu_seqlens, pages, tokens, seqs, max_seq_len, q_heads, kv_heads, scale, window,
             status, stream);
}
