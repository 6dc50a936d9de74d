// Ragged causal attention of prompt portions over the paged cache with the options of the designs beyond the dense one, on
// the 5th-generation tensor cores (tcgen05): bfloat16, key and value heads of 64 or 128 (-DHEAD_DIM), pages of a multiple
// of 16 tokens; a window that may keep the request's first keys, a penalty that grows with the distance, slopes, a soft
// cap, a sink in the denominator, a gate per head.  The mma.sync kernel of attention_tensor.cu computes the same for other
// sizes.
//
// A CTA takes 128 query rows of ONE request and ONE kv head (a row is a token and a query head of the group) over the key
// tiles of 128 that some row sees:
//
//   TMA warp          keys and values, two stages each: one copy per tile where the tile's pages follow each other in the
//                     pool, else one per 16 keys; tiles below the request's context before the dependency wait
//   MMA thread        S = Q K^T (128 x 128, float32, tensor memory, two buffers) and O += P V
//   2 x 4 softmax     one group takes the even tiles, the other the odd ones, each with a running maximum, a sum and an
//   warps             accumulator O of its own; a thread owns a row: it reads S, and writes P over it in tensor memory as
//                     TWO bfloat16 terms (the weight rounded, and what the rounding left), both multiplied with V from
//                     there.  Scores, maxima, sums and denominators are float32.  At the end the groups' halves join.
//
// What bounds it is the chain scores, softmax, values of a group (about 2 us a tile of 128 keys, 3 us with a penalty or a
// cap, whose logarithm or exponential and division come on top), which is why two groups take turns.  On mma.sync every warp
// loads a fragment of keys for 16 rows; here 128 rows meet a tile.  2,048 tokens, 16 heads of 128 on 2 kv heads, against
// the mma.sync kernel: 45 us with a sink (220 there), 57 with a window of 1,024 and a penalty (201), 61 with a cap (258);
// three portions of 500 over 1,500 keys 61 (389); 64 tokens over 4,000 keys 54 (431).
// Every wait is bounded.  A row's result depends on its own request's rows alone.
#include "blackwell.cuh"
#include "common.cuh"

#ifndef HEAD_DIM
#define HEAD_DIM 128
#endif

CIE_DEFINE_LAST_ERROR()

namespace cie {

using namespace bw;
using bf16 = __nv_bfloat16;
constexpr int D = HEAD_DIM;
static_assert(D == 64 || D == 128, "this kernel is built for head sizes 64 and 128");

constexpr int BM = 128, BN = 128;                   // query rows of a CTA, keys of a tile
constexpr int HALVES = D / 64;                      // 64-column pieces of a row
constexpr int SUB_BYTES = 128 * 128;                // 128 rows of 64 columns of Q
constexpr int Q_BYTES = HALVES * SUB_BYTES;
constexpr int GROUP_BYTES = HALVES * 1024;          // 8 keys of K or V: 8 x 64 left columns, then the right ones
constexpr int BLOCK_BYTES = 2 * GROUP_BYTES;        // 16 keys: what one copy of the second kind brings
constexpr int BLOCKS = BN / 16;
constexpr int TILE_BYTES = BLOCKS * BLOCK_BYTES;
constexpr int STAGES = 2;
constexpr int SMEM_BYTES = Q_BYTES + 2 * STAGES * TILE_BYTES + 1024;
constexpr int MMA_WARP = 8, TMA_WARP = 9, THREADS = 320;
constexpr int TMEM_COLS = 512;                      // S0 | S1 | O0 | O1, 128 columns each
constexpr uint32_t COL_S = 0, COL_O = 256;
constexpr int TABLE_SLOTS = 256;                    // block-table entries kept in shared memory (more are read from global memory)
constexpr float kGrow = 8.f;                        // rescale O when a maximum moved by more than this (log2 units)
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float fast_exp2(float x) {      // results below 2^-126 become 0; -inf gives 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&pair);
}
// Behind tcgen05.wait::ld: what is done with these registers stays behind it too.
__device__ __forceinline__ void pin(uint32_t (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));
}

struct Args {
  const bf16* q;
  int q_stride;
  bf16* out;
  int out_stride;
  const int* table;        // [requests][table_width]
  int table_width;
  int num_pages;
  int kv_heads;
  int page_size;
  const int* tile_request;
  const int* tile_q0;
  const int* context_lens;
  const int* query_lens;
  const int* query_start;
  int group, hpt, tpt, head_chunks;     // query heads per kv head, heads and tokens of a tile, tiles of a group's heads
  float scale_log2;
  int window, keep_first;
  const float* r1;         // the score (log2 units) is lowered by r1[h] log2(1 + r2[h] distance); nullptr: not
  const float* r2;
  const float* sinks;      // [query heads] or nullptr
  float cap;               // 0: none
  const float* slopes;     // [query heads] or nullptr
  const float* gates;      // head h of token t is multiplied by sigmoid(gates[t * gate_stride + h]); nullptr: not
  int gate_stride;
  int run_pages;           // pages of a tile whose pages follow each other (0: one copy per 16 keys always)
  int* err;
};

// What is done to a scaled score before the softmax, by build: a branch per score costs more than the arithmetic (one
// build for all of them took 105 us with the penalty and 119 with the cap).
enum Scores { kPlain, kPenalty, kCap, kSlopes, kAny };

// A score in units of log 2 (kAny: whatever the arguments name).  `gap`: distance between query and key, which is negative
// for keys that the mask takes out.
struct Row {
  float scale, cap, to_exponent, slope, r1, r2;
};
template <Scores kScores>
__device__ __forceinline__ float score_of(float product, float gap, const Row& row) {
  float s = product * row.scale;
  // cap * tanh(s / cap) = cap - 2 cap / (exp(2 s / cap) + 1)
  if (kScores == kCap || (kScores == kAny && row.cap > 0.f))
    s = fmaf(-2.f * row.cap, __fdividef(1.f, exp2f(s * row.to_exponent) + 1.f), row.cap);
  if (kScores == kSlopes || kScores == kAny) s = fmaf(-row.slope, gap, s);
  if (kScores == kPenalty || kScores == kAny) s = fmaf(-row.r1, __log2f(fmaf(row.r2, fmaxf(gap, 0.f), 1.f)), s);
  return s;
}

template <Scores kScores>
__global__ void __launch_bounds__(THREADS, 1)
prompt_options_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                      const __grid_constant__ CUtensorMap k_run_map, const __grid_constant__ CUtensorMap v_run_map,
                      const Args a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = smem;
  unsigned char* k_s = q_s + Q_BYTES;                  // [STAGES][TILE_BYTES]
  unsigned char* v_s = k_s + STAGES * TILE_BYTES;
  __shared__ __align__(8) uint64_t k_full[STAGES], k_empty[STAGES], v_full[STAGES], v_empty[STAGES];
  __shared__ __align__(8) uint64_t s_full[2], p_full[2], pv_done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int pages_s[TABLE_SLOTS];
  __shared__ float m_s[2][BM], l_s[2][BM];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the tile list puts the tiles with the most keys first; all heads of a tile follow each other
  const int columns = a.kv_heads * a.head_chunks, tile = blockIdx.x / columns, column = blockIdx.x % columns;
  const int kvh = column / a.head_chunks, h0 = (column % a.head_chunks) * a.hpt;
  const int request = a.tile_request[tile], q0 = a.tile_q0[tile];
  const int context = a.context_lens[request], q_len = a.query_lens[request];
  const int first_token = a.query_start[request] + q0;
  const int ntok = min(a.tpt, q_len - q0);
  const int* table_row = a.table + (size_t)request * a.table_width;
  const int pos_lo = context + q0, valid_hi = pos_lo + ntok;          // keys [.., valid_hi) are visible to some row
  const int valid_lo = a.window > 0 ? max(0, pos_lo - a.window + 1) : 0;
  // kept first keys below the window's range: whole tiles from key 0 come first (a tile that the kept keys share with the
  // window's range is taken once, with the window's)
  const int begin = valid_lo / BN;
  const int kept = a.window > 0 ? min(a.keep_first, valid_lo) : 0;
  const int pre = min((kept + BN - 1) / BN, begin);
  const int tiles = pre + (valid_hi + BN - 1) / BN - begin;
  auto tile_k0 = [&](int j) { return (j < pre ? j : begin + j - pre) * BN; };

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
    }
    for (int g = 0; g < 2; ++g) { mbar_init(&s_full[g], 1); mbar_init(&p_full[g], BM); mbar_init(&pv_done[g], 1); }
    mbar_init_fence();
  }
  {
    const int needed = min((valid_hi + a.page_size - 1) / a.page_size, min(a.table_width, TABLE_SLOTS));
    for (int idx = tid; idx < needed; idx += THREADS) pages_s[idx] = table_row[idx];
  }
  fence_async_smem();
  __syncthreads();
  bool alive = true;
  uint32_t tmem = 0;
  if (warp != TMA_WARP) {
    // everybody but the TMA warp: the Q tile, swizzled by hand (row r is token r / hpt, head h0 + r % hpt of the group).
    // Tensor memory is asked for behind the wait only: a CTA of an earlier kernel that is still to allocate its own on this
    // SM must never find it taken by a CTA that waits for that kernel.
    pdl_wait();
    pdl_trigger();
    if (warp == MMA_WARP) tmem_alloc<TMEM_COLS>(&tmem_slot);
    for (int idx = tid; idx < BM * (D / 8); idx += TMA_WARP * 32) {
      const int r = idx / (D / 8), c = idx % (D / 8);
      const int tok = r / a.hpt, hh = h0 + r % a.hpt;
      uint4 value = make_uint4(0u, 0u, 0u, 0u);
      if (tok < ntok && hh < a.group)
        value = *reinterpret_cast<const uint4*>(a.q + (size_t)(first_token + tok) * a.q_stride + (size_t)(kvh * a.group + hh) * D + c * 8);
      *reinterpret_cast<uint4*>(q_s + (c >> 3) * SUB_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = value;
    }
    fence_async_smem();
    tc_fence_before();
    asm volatile("bar.sync 2, %0;" ::"n"(TMA_WARP * 32) : "memory");
    tc_fence_after();
    tmem = tmem_slot;
  }

  if (warp == TMA_WARP) {
    bool waited = false;
    for (int j = 0; j < tiles && alive; ++j) {
      const int s = j % STAGES, k0 = tile_k0(j);
      // the blocks of 16 keys that some row sees (pages of the others may be gone): those of the window, and in a tile that
      // begins with kept keys those too
      const bool early = j < pre;
      const int b1 = min(BLOCKS, ((early ? kept : valid_hi) - k0 + 15) / 16);
      const int key = k0 + lane * 16;
      const bool mine = lane < b1 && (early || key + 16 > valid_lo || key < kept);
      if (!waited && k0 + BN > context) {      // a tile with keys of this step: the kernel before writes them
        pdl_wait();
        waited = true;
      }
      int page = 0;
      if (mine) {
        const int index = key / a.page_size;
        page = index >= a.table_width ? -1 : index < TABLE_SLOTS ? pages_s[index] : table_row[index];
      }
      // a whole tile with one copy, if it needs its first block and the pages follow each other
      const int first_page = __shfl_sync(0xffffffffu, page, 0);
      const bool follows = lane >= b1 || (mine && page == first_page + (lane * 16) / a.page_size);
      const bool run = __all_sync(0xffffffffu, follows) && a.run_pages > 0 && first_page >= 0 && first_page < a.num_pages;
      if (mine && (page < 0 || page >= a.num_pages)) {
        atomicOr(a.err, kErrBadPage);          // the copy must still happen: the barrier counts its bytes
        page = 0;
      }
      const int blocks = __popc(__ballot_sync(0xffffffffu, mine));
      const int row8 = ((page * a.kv_heads + kvh) * a.page_size + key % a.page_size) / 8;
      const int run_group = kvh * (a.page_size / 8) + (k0 % a.page_size) / 8;
      auto load = [&](unsigned char* stage, const CUtensorMap* map, const CUtensorMap* run_map, uint64_t* full) {
        // a whole box counts, also where it reaches past the keys in use or past the pool's end
        if (lane == 0) mbar_expect_tx(full, run ? (uint32_t)TILE_BYTES : (uint32_t)(blocks * BLOCK_BYTES));
        __syncwarp();
        if (run) {
          if (lane == 0) {
            if constexpr (HALVES == 2) tma_load_5d(stage, run_map, full, 0, 0, 0, run_group, first_page);
            else tma_load_4d(stage, run_map, full, 0, 0, run_group, first_page);
          }
        } else if (mine) {
          if constexpr (HALVES == 2) tma_load_4d(stage + lane * BLOCK_BYTES, map, full, 0, 0, 0, row8);
          else tma_load_3d(stage + lane * BLOCK_BYTES, map, full, 0, 0, row8);
        }
        __syncwarp();
      };
      const uint32_t before = ((j / STAGES) - 1) & 1;
      if (j >= STAGES) alive = mbar_wait(&k_empty[s], before, a.err);
      alive = __all_sync(0xffffffffu, alive);
      if (alive) {
        load(k_s + s * TILE_BYTES, &k_map, &k_run_map, &k_full[s]);
        if (j >= STAGES) alive = mbar_wait(&v_empty[s], before, a.err);
        alive = __all_sync(0xffffffffu, alive);
        if (alive) load(v_s + s * TILE_BYTES, &v_map, &v_run_map, &v_full[s]);
      }
    }
    if (!waited) pdl_wait();
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      constexpr uint32_t idesc_qk = idesc_bf16(BM, BN), idesc_pv = idesc_bf16(BM, D, true);
      const uint64_t q_desc = smem_desc_sw128(smem_u32(q_s));
      // keys: groups of 8 keys GROUP_BYTES apart, the right 64 columns 1 KB further; values the same memory order, read as
      // the operand whose N dimension is contiguous
      const uint64_t k_desc0 = smem_desc_sw128(smem_u32(k_s), 16, GROUP_BYTES);
      const uint64_t v_desc0 = smem_desc_sw128(smem_u32(v_s), 1024, GROUP_BYTES);
      auto values = [&](int j) -> bool {
        const int g = j & 1, s = j % STAGES;
        if (!mbar_wait(&p_full[g], (j >> 1) & 1, a.err) || !mbar_wait(&v_full[s], (j / STAGES) & 1, a.err)) return false;
        tc_fence_after();
        const uint64_t v_desc = v_desc0 + (uint64_t)((s * TILE_BYTES) >> 4);
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          // P lies over S: 32 columns hold 32 keys, 16 columns of first terms and then 16 of second ones
          const uint32_t p = tmem + COL_S + g * BN + (kk >> 1) * 32 + (kk & 1) * 8;
          const uint64_t v = v_desc + (uint64_t)((kk * BLOCK_BYTES) >> 4);
          umma_bf16_ta(tmem + COL_O + g * 128, p, v, idesc_pv, (j > 1 || kk > 0) ? 1u : 0u);
          umma_bf16_ta(tmem + COL_O + g * 128, p + 16, v, idesc_pv, 1u);
        }
        tc_commit(&v_empty[s]);
        tc_commit(&pv_done[g]);
        return true;
      };
      for (int j = 0; j < tiles && alive; ++j) {
        const int g = j & 1, s = j % STAGES;
        // the weights of tile j - 2, which lie in this buffer, have been used
        if (j > 1 && !mbar_wait(&pv_done[g], ((j >> 1) - 1) & 1, a.err)) { alive = false; break; }
        if (!mbar_wait(&k_full[s], (j / STAGES) & 1, a.err)) { alive = false; break; }
        tc_fence_after();
        const uint64_t k_desc = k_desc0 + (uint64_t)((s * TILE_BYTES) >> 4);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t q_off = ((kk >> 2) * SUB_BYTES + (kk & 3) * 32) >> 4, k_off = ((kk >> 2) * 1024 + (kk & 3) * 32) >> 4;
          umma_bf16(tmem + COL_S + g * BN, q_desc + q_off, k_desc + k_off, idesc_qk, kk > 0 ? 1u : 0u);
        }
        tc_commit(&s_full[g]);
        tc_commit(&k_empty[s]);
        if (j > 0) alive = values(j - 1);
      }
      if (alive) alive = values(tiles - 1);
    }
    __syncwarp();
  } else {
    // ---- softmax: group g takes tiles g, g + 2, ..; thread r of a group owns row r = tensor-memory lane r
    const int g = warp >> 2, r = tid & 127;
    const int tok = r / a.hpt, hh = h0 + r % a.hpt;
    const bool row_used = tok < ntok && hh < a.group;
    const int pos = row_used ? pos_lo + tok : -1, head = kvh * a.group + hh;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lane_base + COL_S + g * BN, o_addr = tmem + lane_base + COL_O;
    Row row{a.scale_log2, a.cap * kLog2e, a.cap > 0.f ? 2.f / a.cap : 0.f, 0.f, 0.f, 0.f};
    if (row_used) {
      if (a.r1) { row.r1 = a.r1[head]; row.r2 = a.r2[head]; }
      if (a.slopes) row.slope = a.slopes[head] * kLog2e;
    }
    const float scale = kScores != kPlain ? 1.f : a.scale_log2;      // of what the weights are made from
    float m_used = -INFINITY, l = 0.f;
    for (int j = g; j < tiles; j += 2) {
      const int k0 = tile_k0(j);
      if (k0 + BN > valid_hi || (k0 < valid_lo && k0 + BN > a.keep_first)) {
        // Values of keys that no row sees are cleared (a thread a key, its pieces in turn so that eight lanes meet all banks): a
        // weight of zero times what a page's former owner, or the owner of the page behind, left there need not be zero, nor
        // what lies in a stage where no copy went.  While the scores are worked out it costs little; by the TMA warp, beside
        // the softmax, the layer of 2,048 tokens took 2 us longer.
        if (!mbar_wait(&v_full[j % STAGES], (j / STAGES) & 1, a.err)) { alive = false; break; }
        const int key = k0 + r;
        if (key >= valid_hi || (key < valid_lo && key >= a.keep_first)) {
          unsigned char* row_v = v_s + (j % STAGES) * TILE_BYTES + (r >> 3) * GROUP_BYTES + (r & 7) * 128;
#pragma unroll
          for (int c = 0; c < HALVES * 8; ++c)
            *reinterpret_cast<uint4*>(row_v + (c >> 3) * 1024 + (((c + r) & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_async_smem();      // before the products, which this thread's arrival on p_full lets go, and later copies
      }
      if (!mbar_wait(&s_full[g], (j >> 1) & 1, a.err)) { alive = false; break; }
      tc_fence_after();
      // columns lo .. hi of this tile are visible, and those below `first`
      const int hi = pos - k0, lo = a.window > 0 ? hi - a.window + 1 : 0, first = a.window > 0 ? a.keep_first - k0 : 0;
      const bool masked = k0 + BN - 1 > pos_lo || (a.window > 0 && k0 < valid_hi - a.window);      // the same for the CTA
      auto hidden = [&](int i) { return i > hi || (i < lo && i >= first); };
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      // the row of S comes twice: for its maximum (scores that are more than products go back into tensor memory), and, 32
      // columns at a time, for the weights
      uint32_t raw[2][32];
      {
        uint32_t all[BN / 32][32];
#pragma unroll
        for (int c = 0; c < BN / 32; ++c) tmem_ld32(s_addr + c * 32, all[c]);
        tc_wait_ld();
        if constexpr (kScores != kPlain) {
          const float far = (float)hi;        // distance of column 0
#pragma unroll
          for (int i = 0; i < BN; ++i)
            all[i >> 5][i & 31] = __float_as_uint(score_of<kScores>(__uint_as_float(all[i >> 5][i & 31]), far - (float)i, row));
        }
        if (masked) {
#pragma unroll
          for (int i = 0; i < BN; ++i) {
            if (hidden(i)) all[i >> 5][i & 31] = 0xff800000u;      // -inf: out of the maximum
            mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(all[i >> 5][i & 31]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < BN; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(all[i >> 5][i & 31]));
        }
        if constexpr (kScores != kPlain) {
#pragma unroll
          for (int c = 1; c < BN / 32; ++c) tmem_st32(s_addr + c * 32, all[c]);
          tc_wait_st();
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) raw[0][i] = all[0][i];
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale;
      const bool grow = mx > m_used + kGrow;            // false while the row has seen no key
      if (__any_sync(0xffffffffu, grow)) {
        float alpha = 1.f;
        if (grow) {
          alpha = exp2f(m_used - mx);                   // 0 at the row's first keys
          m_used = mx;
          l *= alpha;
        }
        if (j > 1) {
          // S of this tile was asked for after O += P V of the group's tile before it had ended: O stands still
#pragma unroll 1
          for (int c = 0; c < D / 32; ++c) {
            uint32_t part[32];
            tmem_ld32(o_addr + g * 128 + c * 32, part);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) part[i] = __float_as_uint(__uint_as_float(part[i]) * alpha);
            tmem_st32(o_addr + g * 128 + c * 32, part);
          }
        }
      }
      const float m_eff = m_used == -INFINITY ? 0.f : m_used;
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t terms[32];
        uint32_t (&here)[32] = raw[c & 1];
        if (c > 0) {
          tc_wait_ld();
          pin(here);
          if (kScores == kPlain && masked) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (hidden(c * 32 + i)) here[i] = 0xff800000u;      // -inf: a weight of 0
          }
        }
        if (c + 1 < BN / 32) tmem_ld32(s_addr + (c + 1) * 32, raw[(c + 1) & 1]);     // on its way while this one is used
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(here[i]), scale, -m_eff));
          const float p1 = fast_exp2(fmaf(__uint_as_float(here[i + 1]), scale, -m_eff));
          l4[(i >> 1) & 3] += p0 + p1;
          const __nv_bfloat162 one = __floats2bfloat162_rn(p0, p1);
          const float2 back = __bfloat1622float2(one);
          const __nv_bfloat162 two = __floats2bfloat162_rn(p0 - back.x, p1 - back.y);
          terms[i >> 1] = *reinterpret_cast<const uint32_t*>(&one);
          terms[16 + (i >> 1)] = *reinterpret_cast<const uint32_t*>(&two);
        }
        tmem_st32(s_addr + c * 32, terms);
      }
      l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&p_full[g]);
    }
    // ---- the groups' halves: each group finishes half of the columns of every row
    const int mine = (tiles - g + 1) / 2;               // tiles of this group
    if (alive && mine > 0 && !mbar_wait(&pv_done[g], (mine - 1) & 1, a.err)) alive = false;
    tc_fence_after();
    m_s[g][r] = alive ? m_used : -INFINITY;
    l_s[g][r] = l;
    tc_fence_before();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    tc_fence_after();
    const float m0 = m_s[0][r], m1 = m_s[1][r];
    float top = fmaxf(m0, m1), sink = 0.f;
    if (a.sinks && row_used) {
      sink = a.sinks[head] * kLog2e;
      top = fmaxf(top, sink);
    }
    const float w0 = m0 == -INFINITY ? 0.f : exp2f(m0 - top), w1 = m1 == -INFINITY ? 0.f : exp2f(m1 - top);
    float total = l_s[0][r] * w0 + l_s[1][r] * w1;
    if (a.sinks && row_used) total += exp2f(sink - top);
    float inv = total > 0.f ? 1.f / total : 0.f;
    if (a.gates && row_used) inv /= 1.f + expf(-a.gates[(size_t)(first_token + tok) * a.gate_stride + head]);
    const bool both = tiles > 1;
    bf16* dst = a.out + (size_t)(first_token + tok) * a.out_stride + (size_t)head * D;
    for (int c = g; c < D / 32; c += 2) {
      uint32_t x0[32], x1[32];
      tmem_ld32(o_addr + c * 32, x0);
      if (both) tmem_ld32(o_addr + 128 + c * 32, x1);
      tc_wait_ld();
      if (row_used) {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float o[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            o[e] = __uint_as_float(x0[p * 8 + e]) * w0;
            if (both) o[e] = fmaf(__uint_as_float(x1[p * 8 + e]), w1, o[e]);
            o[e] *= inv;
          }
          *reinterpret_cast<uint4*>(dst + c * 32 + p * 8) = make_uint4(pack(o[0], o[1]), pack(o[2], o[3]), pack(o[4], o[5]), pack(o[6], o[7]));
        }
      }
      __syncwarp();
    }
  }
  if (!alive)      // a wait ran out: give copies and products that may still be in flight time to end before leaving
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_free<TMEM_COLS>(tmem);
}

}  // namespace cie

using namespace cie;

// The arguments are those of cie_attention_prefill_ex (attention_tensor.cu) for key and value heads of this build's size.
extern "C" int cie_attention_prompt_options(const void* q, int q_stride, void* out, int out_stride, const void* k_pool,
                                            const void* v_pool, const int* table, int table_width, int num_pages,
                                            const int* tile_request, const int* tile_q0, int num_tiles,
                                            const int* context_lens, const int* query_lens, const int* query_start,
                                            int q_heads, int kv_heads, int page_size, int hpt, float scale, int window,
                                            const float* r1, const float* r2, int keep_first, const float* sinks, float cap,
                                            const float* slopes, const float* gates, int gate_stride, int* err, void* stream) {
  if (num_tiles <= 0) return 0;
  if (kv_heads < 1 || q_heads % kv_heads) CIE_FAIL("attention_prompt_options: %d query heads over %d kv heads", q_heads, kv_heads);
  const int group = q_heads / kv_heads;
  if (hpt < 1 || hpt > BM || hpt > group) CIE_FAIL("attention_prompt_options: %d heads per tile with a group of %d", hpt, group);
  if (page_size < 16 || page_size % 16) CIE_FAIL("attention_prompt_options: pages of %d tokens (a multiple of 16 is needed)", page_size);
  if (q_stride % 8 || out_stride % 8) CIE_FAIL("attention_prompt_options: row strides must keep 16-byte alignment");
  if ((r1 == nullptr) != (r2 == nullptr)) CIE_FAIL("attention_prompt_options: a penalty needs both vectors");
  if (window < 0 || keep_first < 0 || cap < 0.f) CIE_FAIL("attention_prompt_options: window, kept keys and cap must not be negative");
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(k_pool) |
       reinterpret_cast<uintptr_t>(v_pool)) & 15)
    CIE_FAIL("attention_prompt_options: buffers must be 16-byte aligned");
  Args a;
  a.q = (const bf16*)q; a.q_stride = q_stride; a.out = (bf16*)out; a.out_stride = out_stride;
  a.table = table; a.table_width = table_width; a.num_pages = num_pages; a.kv_heads = kv_heads; a.page_size = page_size;
  a.tile_request = tile_request; a.tile_q0 = tile_q0; a.context_lens = context_lens; a.query_lens = query_lens;
  a.query_start = query_start; a.group = group; a.hpt = hpt; a.tpt = BM / hpt; a.head_chunks = (group + hpt - 1) / hpt;
  a.scale_log2 = scale * kLog2e; a.window = window; a.keep_first = keep_first; a.r1 = r1; a.r2 = r2; a.sinks = sinks;
  a.cap = cap; a.slopes = slopes; a.gates = gates; a.gate_stride = gate_stride; a.err = err;
  const long long ctas = (long long)num_tiles * kv_heads * a.head_chunks;
  if (ctas > 0x7fffffffll) CIE_FAIL("attention_prompt_options: too many tiles");
  CUtensorMap k_map, v_map;
  const long long rows = (long long)num_pages * kv_heads * page_size;
  if (!tensor_map_bf16_row_blocks(k_pool, rows, D, 16, &k_map) || !tensor_map_bf16_row_blocks(v_pool, rows, D, 16, &v_map))
    CIE_FAIL("attention_prompt_options: cuTensorMapEncodeTiled failed");
  CUtensorMap k_run = k_map, v_run = v_map;
  a.run_pages = 0;
  int run_pages = 0, groups = 0;
  // (two tiles of keys are few copies either way, and a map costs the host a quarter of a microsecond to encode)
  const bool many = (long long)table_width * page_size > 2 * BN;
  if (many && page_size <= BN && BN % page_size == 0) { run_pages = BN / page_size; groups = page_size / 8; }
  else if (many && page_size > BN && page_size % BN == 0) { run_pages = 1; groups = BN / 8; }
  if (run_pages > 0 && tensor_map_bf16_page_runs(k_pool, num_pages, kv_heads, page_size, D, groups, run_pages, &k_run) &&
      tensor_map_bf16_page_runs(v_pool, num_pages, kv_heads, page_size, D, groups, run_pages, &v_run))
    a.run_pages = run_pages;
  // (a scale that is not positive: the maximum of the products is not that of the scores)
  const bool distant = r1 != nullptr, sloped = slopes != nullptr, capped = cap > 0.f;
#define CIE_PROMPT_OPTIONS(kScores)                                                                                      \
  {                                                                                                                      \
    static const cudaError_t raised =                                                                                    \
        cudaFuncSetAttribute(prompt_options_kernel<kScores>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);   \
    if (raised != cudaSuccess) CIE_FAIL("attention_prompt_options: shared memory %d: %s", SMEM_BYTES, cudaGetErrorString(raised)); \
    CIE_LAUNCH("attention_prompt_options", prompt_options_kernel<kScores>, dim3((unsigned)ctas), dim3(THREADS),          \
               (size_t)SMEM_BYTES, (cudaStream_t)stream, k_map, v_map, k_run, v_run, a);                                 \
  }
  if (!(scale > 0.f) || distant + sloped + capped > 1) CIE_PROMPT_OPTIONS(kAny)
  else if (distant) CIE_PROMPT_OPTIONS(kPenalty)
  else if (capped) CIE_PROMPT_OPTIONS(kCap)
  else if (sloped) CIE_PROMPT_OPTIONS(kSlopes)
  else CIE_PROMPT_OPTIONS(kPlain)
#undef CIE_PROMPT_OPTIONS
  return 0;
}
