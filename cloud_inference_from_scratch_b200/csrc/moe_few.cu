// The products of routed experts for a step of few (token, expert) pairs, a decode step: what they cost is one pass over
// the chosen experts' weights.  A block takes units of 16 weight rows of an expert and up to eight of its pairs: the weights
// are the left operand of mma.sync, whose columns are the pairs, float32 sums; the eight warps share k and add their sums
// up in shared memory.  The order of k inside 32 columns is chosen so that a lane's pieces of 16 bytes, straight from memory,
// are its share of two products.  Every warp asks for the next 128 columns (or unit) before it multiplies the last.
// 8 tokens, 4 of 16 experts of 1,376 channels, 2,048 wide (162 + 81 MB of weights): 31 and 20 us, the layer 45; with the
// multiplications on the CUDA cores, which then were the bound, 44 and 34, 68.
//
//   gate_up  W = [experts][2F][H], gate and up rows of an expert interleaved in blocks of 16 (moe_tcgen05.cu);
//            act[pair][channel], bfloat16, with the gated activation of glu.cuh; a unit is eight channels
//   down     W = [experts][H][F]; rows[pair][column], float32; a unit is 16 columns
//
// A pair's result depends on the pair alone: every sum runs over k in one fixed order.
#include "common.cuh"
#include "glu.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

using bf16 = __nv_bfloat16;
constexpr int kFewPairs = 64;        // most pairs of a step
constexpr int kFewExperts = 1024;    // most experts
constexpr int kWarps = 8;
constexpr int kTokens = 8;           // pairs of a unit
constexpr int kBlocks = 4;           // 32-column blocks of a step of a warp

struct FewStep {
  uint4 low[kBlocks], high[kBlocks], x[kBlocks];      // columns 8 t .. 8 t + 7 of each block: of weight rows g and g + 8, of pair g
};

__device__ __forceinline__ void few_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// From zero: the tensor core cuts what it adds to an accumulator.  Results that stay float32 (the down product's) add products of
// 16 columns up in registers, where sums are rounded: 8.6e-8 of the rows' norm from 64 bits with 1,376 columns, 8.4e-8 as one
// FMA after the other, 1.31e-7 with accumulators.  Those of gate_up are rounded to 16 bits.
__device__ __forceinline__ void few_add(float (&sum)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  float d[4];
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
#pragma unroll
  for (int i = 0; i < 4; ++i) sum[i] += d[i];
}

// Two blocks an SM.  x: gate_up: token rows [tokens][k], the row of pair p is x[p / top]; down: rows by pair [pairs][k].  n:
// weight rows of an expert (2F or H, a multiple of 8).
template <bool kGateUp>
__global__ void __launch_bounds__(kWarps * 32, 2)
moe_few_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, void* __restrict__ out, const int* __restrict__ ids,
               int pairs, int top, int n, int k, GluAct act) {
  __shared__ __align__(16) float part_s[2][kWarps][16 * kTokens];      // [row][pair]
  __shared__ unsigned low_s[kFewExperts];              // of the first 32 pairs, those of an expert
  __shared__ int entry_s[kFewPairs], expert_s[kFewPairs], pair_s[kFewPairs][kTokens], here_s[kFewPairs], entries_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < kFewExperts; e += blockDim.x) low_s[e] = 0;
  if (threadIdx.x < kFewPairs) here_s[threadIdx.x] = 0;
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  if (warp == 0) {
    // Entries: an expert and up to eight of its pairs, in ascending order.  A pair's rank among its expert's pairs decides: every
    // eighth one leads an entry.
    const unsigned below = (1u << lane) - 1u;
    const int id[2] = {lane < pairs ? ids[lane] : -1, 32 + lane < pairs ? ids[32 + lane] : -1};
    unsigned same[2];
    int rank[2];
    same[0] = __match_any_sync(0xffffffffu, id[0]);
    same[1] = __match_any_sync(0xffffffffu, id[1]);
    rank[0] = __popc(same[0] & below);
    if (id[0] >= 0 && rank[0] == 0) low_s[id[0]] = same[0];
    __syncwarp();
    const unsigned low = id[1] >= 0 ? low_s[id[1]] : 0u;
    rank[1] = __popc(low) + __popc(same[1] & below);
    const unsigned lead0 = __ballot_sync(0xffffffffu, id[0] >= 0 && rank[0] % kTokens == 0);
    const unsigned lead1 = __ballot_sync(0xffffffffu, id[1] >= 0 && rank[1] % kTokens == 0);
    entry_s[lane] = __popc(lead0 & below);
    entry_s[32 + lane] = __popc(lead0) + __popc(lead1 & below);
    if (lane == 0) entries_s = __popc(lead0) + __popc(lead1);
    __syncwarp();
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      if (id[half] < 0) continue;
      const int place = rank[half] % kTokens;
      // the pair that leads: `place` pairs of the expert before this one
      unsigned before[2] = {half ? low : same[0] & below, half ? same[1] & below : 0u};
      int leader = 32 * half + lane;
      for (int back = 0; back < place; ++back) {
        const int word = before[1] ? 1 : 0, bit = 31 - __clz(before[word]);
        before[word] ^= 1u << bit;
        leader = 32 * word + bit;
      }
      const int entry = entry_s[leader];
      pair_s[entry][place] = 32 * half + lane;
      if (place == 0) expert_s[entry] = id[half];
      atomicMax(&here_s[entry], place + 1);
    }
  }
  __syncthreads();
  const int g = lane >> 2, t = lane & 3, pieces = k / 8, groups = (n + 15) / 16, units = groups * entries_s;
  // a warp's columns: 32-column blocks that follow each other, the same ones whatever the unit
  const int all_blocks = (k + 31) / 32, block0 = warp * all_blocks / kWarps, blocks = (warp + 1) * all_blocks / kWarps - block0;
  const int steps = ((all_blocks + kWarps - 1) / kWarps + kBlocks - 1) / kBlocks;
  const int first = (int)((long long)blockIdx.x * units / gridDim.x), last = (int)((long long)(blockIdx.x + 1) * units / gridDim.x);
  // rows g and g + 8 of a unit: of gate_up a gate row and its up row
  auto row_of = [&](int group, int high) {
    return kGateUp ? group / 2 * 32 + group % 2 * 8 + g + 16 * high : min(group * 16 + g + 8 * high, n - 1);
  };
  int ahead = first, ahead_step = 0;
  const uint4 *low = nullptr, *high = nullptr, *rows = nullptr;
  auto fetch = [&](FewStep& to) {
    if (ahead >= last) return;
    if (ahead_step == 0) {
      const int entry = ahead / groups, group = ahead - entry * groups;
      const bf16* base = w + (size_t)expert_s[entry] * n * k;
      const int pair = pair_s[entry][g < here_s[entry] ? g : 0];      // columns past the last pair repeat the first
      low = reinterpret_cast<const uint4*>(base + (size_t)row_of(group, 0) * k) + 4 * block0 + t;
      high = reinterpret_cast<const uint4*>(base + (size_t)row_of(group, 1) * k) + 4 * block0 + t;
      rows = reinterpret_cast<const uint4*>(x + (size_t)(kGateUp ? pair / top : pair) * k) + 4 * block0 + t;
    }
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {
      const int block = ahead_step * kBlocks + i;
      const bool in = block < blocks && 4 * (block0 + block) + t < pieces;
      const uint4 none = make_uint4(0u, 0u, 0u, 0u);
      to.low[i] = in ? __ldg(low + 4 * block) : none;
      to.high[i] = in ? __ldg(high + 4 * block) : none;
      to.x[i] = in ? rows[4 * block] : none;
    }
    if (++ahead_step == steps) {
      ahead_step = 0;
      ++ahead;
    }
  };
  int unit = first, step = 0;
  float sum[2][4] = {};      // the two products of a block each have one
  auto multiply = [&](const FewStep& s) {
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {
      if constexpr (kGateUp) {
        few_mma(sum[0], s.low[i].x, s.high[i].x, s.low[i].y, s.high[i].y, s.x[i].x, s.x[i].y);
        few_mma(sum[1], s.low[i].z, s.high[i].z, s.low[i].w, s.high[i].w, s.x[i].z, s.x[i].w);
      } else {
        few_add(sum[0], s.low[i].x, s.high[i].x, s.low[i].y, s.high[i].y, s.x[i].x, s.x[i].y);
        few_add(sum[1], s.low[i].z, s.high[i].z, s.low[i].w, s.high[i].w, s.x[i].z, s.x[i].w);
      }
    }
    if (++step < steps) return;
    step = 0;
    // rows g (0, 1) and g + 8 (2, 3), pairs 2 t and 2 t + 1
    float* part = part_s[unit & 1][warp] + g * kTokens + 2 * t;
    *reinterpret_cast<float2*>(part) = make_float2(sum[0][0] + sum[1][0], sum[0][1] + sum[1][1]);
    *reinterpret_cast<float2*>(part + 8 * kTokens) = make_float2(sum[0][2] + sum[1][2], sum[0][3] + sum[1][3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[0][e] = sum[1][e] = 0.f;
    __syncthreads();      // (the other set is free: whoever added it up has been here since)
    const int entry = unit / groups, group = unit - entry * groups, here = here_s[entry];
    if (kGateUp ? threadIdx.x < 64 : threadIdx.x < 128) {
      const int j = kGateUp ? threadIdx.x >> 3 : threadIdx.x >> 4, r = kGateUp ? threadIdx.x & 7 : threadIdx.x & 15;
      if (j < here) {
        const int pair = pair_s[entry][j];
        float one = 0.f, two = 0.f;
#pragma unroll
        for (int v = 0; v < kWarps; ++v) {
          one += part_s[unit & 1][v][r * kTokens + j];
          if (kGateUp) two += part_s[unit & 1][v][(r + 8) * kTokens + j];
        }
        if constexpr (kGateUp) {
          const float weight = act.weights ? act.weights[pair] : 1.f;
          reinterpret_cast<bf16*>(out)[(size_t)pair * (n / 2) + group * 8 + r] = __float2bfloat16_rn(glu(act, one, two, weight));
        } else if (group * 16 + r < n) {
          reinterpret_cast<float*>(out)[(size_t)pair * n + group * 16 + r] = one;
        }
      }
    }
    ++unit;
  };
  FewStep even, odd;
  fetch(even);
  for (int i = (last - first) * steps; i > 0; i -= 2) {
    fetch(odd);
    multiply(even);
    if (i == 1) break;
    fetch(even);
    multiply(odd);
  }
}

}  // namespace cie

using namespace cie;

extern "C" int cie_moe_few_pairs() { return kFewPairs; }

template <bool kGateUp>
static int launch_few(const void* x, const void* w, void* out, const int* ids, int pairs, int top, int experts, int n, int k,
                      const GluAct& act, void* stream) {
  if (pairs <= 0) return 0;
  if (pairs > kFewPairs) CIE_FAIL("moe_few: at most %d pairs, got %d", kFewPairs, pairs);
  if (k % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15))
    CIE_FAIL("moe_few: rows of %d elements must be 16-byte aligned", k);
  if (experts > kFewExperts) CIE_FAIL("moe_few: %d experts (at most %d)", experts, kFewExperts);
  CIE_LAUNCH("moe_few", moe_few_kernel<kGateUp>, dim3(2 * device_sms()), dim3(kWarps * 32), 0, (cudaStream_t)stream, (const bf16*)x,
             (const bf16*)w, out, ids, pairs, top, n, k, act);
  return 0;
}

// x: [tokens][hidden]; w_gate_up: [experts][2 ff][hidden] interleaved in blocks of 16; act: [tokens * top][ff] by pair; ids:
// [tokens * top].  hidden a multiple of 8, ff a multiple of 16 (clamped, limit, slope, shift, input_weights: GluAct).
extern "C" int cie_moe_gate_up_few(const void* x, const void* w_gate_up, void* act, const int* ids, int tokens, int top,
                                   int experts, int ff, int hidden, int clamped, float limit, float slope, float shift,
                                   const float* input_weights, void* stream) {
  if (ff % 16) CIE_FAIL("moe_gate_up_few: interleaved weights need a multiple of 16 channels, got %d", ff);
  return launch_few<true>(x, w_gate_up, act, ids, tokens * top, top, experts, 2 * ff, hidden,
                          GluAct{clamped, limit, slope, shift, input_weights}, stream);
}

extern "C" int cie_moe_down_few(const void* act, const void* w_down, float* rows, const int* ids, int tokens, int top,
                                int experts, int ff, int hidden, void* stream) {
  return launch_few<false>(act, w_down, rows, ids, tokens * top, top, experts, hidden, ff, GluAct{}, stream);
}
