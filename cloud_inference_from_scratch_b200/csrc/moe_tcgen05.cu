// The grouped products of routed experts on the 5th-generation tensor cores.
//
// The (token, expert) pairs of a step are grouped by expert on the device (moe.cu: places, and tiles of up to 256 of them that
// belong to one expert and divide its rows evenly).  Weights are the left operand: a CTA an SM walks over tiles of 128
// weight rows and the tile's tokens, rounded up to 16, so that nothing is multiplied for tokens that an expert does
// not have.  Both come by TMA (128-byte swizzle) into a ring, one thread issues tcgen05.mma into float32 accumulators in
// tensor memory, and eight warps read a tile back with tcgen05.ld while the next one's products run; a lane holds a weight row, so that 32
// lanes write neighbouring columns of a token.  Rows must lie one after another for TMA, so the
// gate/up product first gathers the tokens' rows by place (one memory-bound kernel); the down
// product reads the activations, which the gate/up product wrote by place.
//
//   gate_up  W = [experts][2F][H], gate and up rows of an expert interleaved in blocks of 16 (16 gate
//            rows, their 16 up rows, ...): lanes exchange them, every lane works one SiLU(gate) * up out of
//            two tokens, act[place][channel] (bfloat16)
//   down     W = [experts][H][F]; the result goes, float32, to the row of the tile row's pair
//
// A tile's rows beyond the expert's last (they belong to the next expert, or lie outside the buffer and read as zero) are
// computed and never stored.  Every wait on an mbarrier is bounded.
// What bounds a large product: a stage's way through copy, products and back, 2 us of which four stages of 48 KB cover less
// than the products would use up (85 us of the 101 below without the epilogue, 70 without loads), and the epilogue's
// instructions.  2,048 tokens, 4 of 16 experts of 1,376 channels, 2,048 wide: 101 and 58 us, with token rows as the
// left operand in tiles of 128 by 256 119 and 66.  Tiles of 256 weight rows take up all of tensor memory, so that nothing hides
// their epilogue: 100 and 61.  Asking L2 for later weights: 3 us more.  The layer of 17 tokens 94 -> 88, 512 tokens 123 -> 103,
// 2,048 tokens of 32 experts of 2,048 channels, 4,096 wide, 689 -> 589.
#include "blackwell.cuh"
#include "common.cuh"
#include "glu.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

using namespace bw;
using bf16 = __nv_bfloat16;

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int TOKENS = 256, TOKEN_BOX = 64;      // tokens of a tile at most; of one copy
constexpr int WEIGHT_BYTES = BM * BK * 2, BOX_BYTES = TOKEN_BOX * BK * 2;
constexpr int STAGES = 4, STAGE_BYTES = WEIGHT_BYTES + TOKENS * BK * 2;
constexpr size_t GROUPED_SMEM = (size_t)STAGES * STAGE_BYTES + 1024;

// A warp a row, eight of its pieces asked for together: 8,192 rows of 2,048: 9 us cold, 11 with a division and a
// dependent load a piece (its bytes take 6)
__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(const bf16* __restrict__ x, bf16* __restrict__ sorted, const int* __restrict__ place_to_pair, int pairs,
                       int top, int hidden) {
  pdl_wait();
  pdl_trigger();
  const int pieces = hidden / 8, lane = threadIdx.x & 31, p = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (p >= pairs) return;
  const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)(place_to_pair[p] / top) * hidden);
  uint4* to = reinterpret_cast<uint4*>(sorted + (size_t)p * hidden);
  for (int c = lane; c < pieces; c += 256) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (c + 32 * u < pieces) v[u] = from[c + 32 * u];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (c + 32 * u < pieces) to[c + 32 * u] = v[u];
  }
}

struct GroupedArgs {
  void* out;
  const int* place_to_pair;
  const int* tiles;        // how many, then (expert, first place, rows) of each
  int rows_per_expert;     // weight rows of one expert (2F or H)
  int n;                   // output columns of a row (F or H)
  int k;
  int* err;
  GluAct glu_act;          // gate_up
};

// The results of 128 weight rows (a warp the 32 lanes whose first column is `from`) and every second 32 of a tile's tokens
// (from `first` on) to where they go.  pairs: those of the lane's tokens, which are read before the results are waited for.
constexpr int kTurns = TOKENS / 64;
template <bool kGateUp>
__device__ __forceinline__ void write_tile(const GroupedArgs& a, uint32_t from, int row0, int place0, int rows, int first,
                                           const int (&pairs)[kTurns]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int turn = 0; turn < kTurns; ++turn) {
    const int c0 = first + 64 * turn;
    if (c0 >= rows) break;
    uint32_t raw[32];
    tmem_ld32(from + c0, raw);                     // every lane of the warp takes part in the load
    const int pair = pairs[turn];
    const float weight = kGateUp && a.glu_act.weights ? a.glu_act.weights[pair] : 1.f;
    tc_wait_ld();
    if constexpr (kGateUp) {
      // lanes 0 .. 15 hold 16 gate rows, 16 .. 31 their up rows: the lower lanes take the even tokens, the upper the odd ones
      const bool upper = lane >= 16;
      const int channel = row0 / 2 + (lane & 15);
      bf16* dst = reinterpret_cast<bf16*>(a.out) + (size_t)(place0 + c0 + upper) * a.n + channel;
#pragma unroll
      for (int c = 0; c < 32; c += 2) {
        const float mine = __uint_as_float(upper ? raw[c + 1] : raw[c]);
        const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(upper ? raw[c] : raw[c + 1]), 16);
        const float w = __shfl_sync(0xffffffffu, weight, c + upper);
        if (c0 + c + upper < rows && channel < a.n)
          dst[(size_t)c * a.n] = __float2bfloat16_rn(glu_straight(a.glu_act, upper ? other : mine, upper ? mine : other, w));
      }
    } else {
      float* dst = reinterpret_cast<float*>(a.out) + row0 + lane;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const int to = __shfl_sync(0xffffffffu, pair, c);
        if (c0 + c < rows && row0 + lane < a.n) dst[(size_t)to * a.n] = __uint_as_float(raw[c]);
      }
    }
  }
}

// map_w: weight rows of all experts in boxes of 128, map_x: token rows in boxes of TOKEN_BOX.  Warps: copies, products, two
// groups of eight that write every second tile out.
constexpr int GROUPED_THREADS = 64 + 16 * 32;
template <bool kGateUp>
__global__ void __launch_bounds__(GROUPED_THREADS, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const GroupedArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 8);
    }
    mbar_init_fence();
  }
  pdl_wait();
  pdl_trigger();
  if (warp == 1) tmem_alloc<2 * TOKENS>(&tmem_base_s);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  const int row_tiles = (a.rows_per_expert + BM - 1) / BM, total = a.tiles[0] * row_tiles;
  const int k_tiles = (a.k + BK - 1) / BK;
  bool alive = true;
  // tile t: all weight rows of one tile of tokens after another, so that the CTAs of a moment share tokens and a few experts
  struct Tile { int expert, place0, rows, row0; };
  auto tile_at = [&](int t) {
    const int of_tokens = t / row_tiles;
    const int* at = a.tiles + 1 + 3 * of_tokens;
    return Tile{at[0], at[1], at[2], (t - of_tokens * row_tiles) * BM};
  };

  if (warp == 0) {
    if (lane == 0) {     // copies
      int s = 0;
      uint32_t phase = 1;
      for (int t = blockIdx.x; t < total && alive; t += gridDim.x) {
        const Tile tile = tile_at(t);
        const int boxes = (tile.rows + TOKEN_BOX - 1) / TOKEN_BOX, w_row = tile.expert * a.rows_per_expert + tile.row0;
        for (int kt = 0; kt < k_tiles; ++kt) {
          if (!mbar_wait(&empty_bar[s], phase, a.err)) { alive = false; break; }
          mbar_expect_tx(&full_bar[s], WEIGHT_BYTES + boxes * BOX_BYTES);
          unsigned char* dst = ring + (size_t)s * STAGE_BYTES;
          tma_load_2d(dst, &map_w, &full_bar[s], kt * BK, w_row);
          for (int b = 0; b < boxes; ++b)
            tma_load_2d(dst + WEIGHT_BYTES + b * BOX_BYTES, &map_x, &full_bar[s], kt * BK, tile.place0 + b * TOKEN_BOX);
          if (++s == STAGES) { s = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {     // products
      int s = 0, n = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < total && alive; t += gridDim.x, ++n) {
        const Tile tile = tile_at(t);
        const uint32_t idesc = idesc_bf16(BM, (tile.rows + 15) & ~15);
        // the accumulator's last results have been written out
        if (!mbar_wait(&acc_empty[n & 1], ((n >> 1) & 1) ^ 1, a.err)) { alive = false; break; }
        tc_fence_after();
        const uint32_t acc = tmem_base + (n & 1) * TOKENS;
        for (int kt = 0; kt < k_tiles; ++kt) {
          if (!mbar_wait(&full_bar[s], phase, a.err)) { alive = false; break; }
          tc_fence_after();
          const uint32_t at = smem_u32(ring + (size_t)s * STAGE_BYTES);
          const uint64_t w_desc = smem_desc_sw128(at), x_desc = smem_desc_sw128(at + WEIGHT_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk)
            umma_bf16(acc, w_desc + 2 * kk, x_desc + 2 * kk, idesc, (kt > 0 || kk > 0) ? 1u : 0u);
          tc_commit(&empty_bar[s]);
          if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        if (!alive) break;
        tc_commit(&acc_full[n & 1]);
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, group = (warp - 2) >> 3;      // the tensor-memory lanes a warp may read
    const int first = ((warp - 2) >> 2 & 1) * 32;
    int n = 0;
    for (int t = blockIdx.x; t < total && alive; t += gridDim.x, ++n) {
      if ((n & 1) != group) continue;
      const Tile tile = tile_at(t);
      int pairs[kTurns];
#pragma unroll
      for (int turn = 0; turn < kTurns; ++turn) {
        const int c = first + 64 * turn + lane;
        pairs[turn] = (!kGateUp || a.glu_act.weights) && c < tile.rows ? a.place_to_pair[tile.place0 + c] : 0;
      }
      alive = __all_sync(0xffffffffu, mbar_wait(&acc_full[group], (n >> 1) & 1, a.err));
      if (!alive) break;
      tc_fence_after();
      const int row0 = tile.row0 + quarter * 32;
      if (row0 < a.rows_per_expert)
        write_tile<kGateUp>(a, tmem_base + group * TOKENS + ((uint32_t)(quarter * 32) << 16), row0, tile.place0, tile.rows,
                            first, pairs);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[group]);
    }
  }
  if (!alive)      // a wait ran out: give copies and products that may still be in flight time to end before leaving
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_free<2 * TOKENS>(tmem_base);
}

template <bool kGateUp>
static int launch_grouped(const char* name, const void* x, const void* w, int pairs, int experts, const GroupedArgs& a, cudaStream_t stream) {
  CUtensorMap map_w, map_x;
  if (!tensor_map_bf16(x, pairs, a.k, TOKEN_BOX, &map_x) || !tensor_map_bf16(w, (long long)experts * a.rows_per_expert, a.k, BM, &map_w))
    CIE_FAIL("%s: cuTensorMapEncodeTiled failed", name);
  static const cudaError_t raised = cudaFuncSetAttribute(moe_grouped_kernel<kGateUp>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GROUPED_SMEM);
  if (raised != cudaSuccess) CIE_FAIL("%s: cannot set the kernel up: %s", name, cudaGetErrorString(raised));
  CIE_LAUNCH(name, moe_grouped_kernel<kGateUp>, dim3(device_sms()), dim3(GROUPED_THREADS), GROUPED_SMEM, stream, map_w, map_x, a);
  return 0;
}

// The list of tiles of up to TOKENS tokens, which moe.cu leaves behind the one of tiles of BM.
static const int* token_tiles(const int* tiles, int pairs, int experts) { return tiles + 3 * ((pairs + BM - 1) / BM + experts); }

}  // namespace cie

using namespace cie;

// x: [tokens][hidden]; sorted: scratch [tokens * top][hidden]; w_gate_up: [experts][2 ff][hidden], gate
// and up rows interleaved in blocks of 16; act: [tokens * top][ff], rows by place.  All bfloat16,
// 16-byte aligned; hidden a multiple of 8, ff a multiple of 16.  clamped, limit, slope, shift, input_weights: GluAct.
extern "C" int cie_moe_gate_up_tcgen05(const void* x, void* sorted, const void* w_gate_up, void* act,
                                       const int* place_to_pair, const int* tiles,
                                       int tokens, int top, int experts, int ff, int hidden, int row_tile, int clamped,
                                       float limit, float slope, float shift, const float* input_weights, int* err,
                                       void* stream) {
  if (tokens <= 0) return 0;
  if (hidden % 8 || ff % 16) CIE_FAIL("moe_gate_up_tcgen05: sizes %d / %d", hidden, ff);
  if (row_tile != BM) CIE_FAIL("moe_gate_up_tcgen05: tiles of %d rows, this kernel takes %d", row_tile, BM);
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(sorted) | reinterpret_cast<uintptr_t>(w_gate_up) |
       reinterpret_cast<uintptr_t>(act)) & 15)
    CIE_FAIL("moe_gate_up_tcgen05: operands must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const int pairs = tokens * top;
  CIE_LAUNCH("moe_gather_rows", moe_gather_rows_kernel, dim3((pairs + 7) / 8), dim3(256), 0, s, (const bf16*)x, (bf16*)sorted,
             place_to_pair, pairs, top, hidden);
  const GroupedArgs a = {act, place_to_pair, token_tiles(tiles, pairs, experts), 2 * ff, ff, hidden, err,
                         {clamped, limit, slope, shift, input_weights}};
  return launch_grouped<true>("moe_gate_up_tcgen05", sorted, w_gate_up, pairs, experts, a, s);
}

// act: [tokens * top][ff] by place; w_down: [experts][hidden][ff]; rows: float32 [tokens * top][hidden],
// the row of pair (t, j) at t * top + j.
extern "C" int cie_moe_down_tcgen05(const void* act, const void* w_down, float* rows, const int* place_to_pair,
                                    const int* tiles, int tokens, int top, int experts,
                                    int ff, int hidden, int row_tile, int* err, void* stream) {
  if (tokens <= 0) return 0;
  if (hidden % 8 || ff % 8) CIE_FAIL("moe_down_tcgen05: sizes %d / %d", hidden, ff);
  if (row_tile != BM) CIE_FAIL("moe_down_tcgen05: tiles of %d rows, this kernel takes %d", row_tile, BM);
  if ((reinterpret_cast<uintptr_t>(act) | reinterpret_cast<uintptr_t>(w_down) | reinterpret_cast<uintptr_t>(rows)) & 15)
    CIE_FAIL("moe_down_tcgen05: operands must be 16-byte aligned");
  const int pairs = tokens * top;
  const GroupedArgs a = {rows, place_to_pair, token_tiles(tiles, pairs, experts), hidden, hidden, ff, err, {}};
  return launch_grouped<false>("moe_down_tcgen05", act, w_down, pairs, experts, a, (cudaStream_t)stream);
}
