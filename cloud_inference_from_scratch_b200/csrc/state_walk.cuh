// The walk of a recurrence with a matrix state over the chunks of its requests, on the tensor cores in float32 accuracy.
//
// A chunk of up to 32 tokens turns the state S [P keys][vdim values] into
//
//     U   = V - W S                     (kMode 1: the gated delta rule's writes; 0: U = V)
//     o_t = S^T q_t + sum_(s <= t) A_ts u_s
//     S  <- diag(d) S + sum_s k_s u_s^T
//
// where q, k, W, A and d (all decays multiplied in) come from a kernel per chunk and head, one `cell` each, and V are
// rows of the step's tokens.  kMode 2 (the generalized delta rule) writes both, with V2, k2 and A2 of the cell:
//
//     U   = V2 - W S,   o_t = S^T q_t + sum_(s <= t) A_ts v_s + A2_ts u_s,   S <- diag(d) S + sum_s k_s v_s^T + k2_s u_s^T
//
// grid (blocks of 16 MT value columns, heads, requests: those with the most chunks first).  A walk is a chain, and a prompt of one request has no more blocks
// than multiprocessors: what bounds it is the instructions of a chunk one after the other, so a block has many warps with
// little to do each.
//   * P / 16 warps own 16 keys of S^T each, in the layout in which mma.sync leaves a sum; with the keys of an operand named
//     in the same order that is also how it takes a left operand, so S never leaves the registers.  Their sums over keys
//     are left in shared memory, a share a warp; nobody waits for another (but for U).
//   * four warps take eight tokens each: what the chunk's own tokens add (A U), the shares, the outputs; U first.
//     One of them asks for the chunks to come.  (A bulk copy a row takes longer than the chunk: a cell is one.)
// Vector loads of operands from shared memory are free of bank conflicts: the order of keys inside a warp's 16 is chosen for
// that (lane 4 g + t reads keys 4 t .. 4 t + 3 of token g, and keys 2 g, 2 g + 1 of token t).
//
// Where an infinity, a NaN or a value near the largest one is met (in the cell, the warp's part of the state, or a sum), the
// same is worked out on the CUDA cores, where a token's outputs read nothing of later tokens (for all columns of the block, whose
// width follows the number of blocks: beside such a value, a finite one's last bits may depend on the company).
#pragma once

#include "blackwell.cuh"
#include "common.cuh"
#include "tf32x3.cuh"

namespace cie {

constexpr int kChunkTokens = 32;
constexpr int kRanked = 64;                   // requests whose walks are ordered by length at most
constexpr int kWalkHelpers = 4;               // warps of eight tokens each
constexpr int kWalkA = kChunkTokens + 4;      // row of A in shared memory

// A cell, as it lies in shared memory too, whose banks its rows are padded for: q [32][P + 16], (mode 1, 2: W [32][P + 16],) k
// [32][P + 8], (2: k2 [32][P + 8],) A [32][36] with row t, column s, (2: A2 [32][36],) decays [P], a flag (not 0: see above), and
// the chunk's tokens (an int).  Rows past the chunk's last token are zeros.  (2: behind it V2 [32][P].)
__host__ __device__ constexpr int walk_q_row(int P) { return P + 16; }
__host__ __device__ constexpr int walk_k_row(int P) { return P + 8; }
__host__ __device__ constexpr int walk_cell_w(int P) { return kChunkTokens * walk_q_row(P); }
__host__ __device__ constexpr int walk_cell_k(int P, int mode) { return (mode ? 2 : 1) * kChunkTokens * walk_q_row(P); }
__host__ __device__ constexpr int walk_cell_k2(int P) { return walk_cell_k(P, 2) + kChunkTokens * walk_k_row(P); }
__host__ __device__ constexpr int walk_cell_a(int P, int mode) { return walk_cell_k(P, mode) + (mode == 2 ? 2 : 1) * kChunkTokens * walk_k_row(P); }
__host__ __device__ constexpr int walk_cell_a2(int P) { return walk_cell_a(P, 2) + kChunkTokens * kWalkA; }
__host__ __device__ constexpr int walk_cell_decay(int P, int mode) { return walk_cell_a(P, mode) + (mode == 2 ? 2 : 1) * kChunkTokens * kWalkA; }
__host__ __device__ constexpr int walk_cell_v2(int P) { return walk_cell_decay(P, 2) + P + 4; }
// what a walk copies of a cell, and from one cell to the next
__host__ __device__ constexpr int walk_cell_copied(int P, int mode) { return walk_cell_decay(P, mode) + P + 4; }
__host__ __device__ constexpr int walk_cell_floats(int P, int mode) { return walk_cell_copied(P, mode) + (mode == 2 ? kChunkTokens * P : 0); }
__host__ __device__ constexpr int walk_pad(int dim) { return (dim + 31) & ~31; }

struct WalkArgs {
  const float* cells;      // [chunks][heads]
  const float* v;          // row of token t, head h, column c: v[t * v_stride + h * v_head + c]
  long long v_stride;
  int v_head;
  float* out;              // [tokens][out_stride], head h at column h * vdim
  int out_stride;
  float* state;            // [slots] of state_stride floats, head h at h * dim * vdim
  long long state_stride;
  const int *chunk_row, *chunk_count, *request_chunk_start, *slots, *request_active;
  int heads, dim, vdim, max_slots;
  int* err;
};

template <int P, int MT, int kMode>
struct WalkShape {
  static constexpr bool kWrites = kMode != 0, kBoth = kMode == 2;
  static constexpr int C = kChunkTokens, COLS = 16 * MT, KEY_WARPS = P / 16, THREADS = (KEY_WARPS + kWalkHelpers) * 32;
  static constexpr int VL = COLS + 8, PL = COLS + 4;
  static constexpr int V = walk_cell_copied(P, kMode), VALUES = C * VL;
  static constexpr int STAGE = V + (kBoth ? 2 : 1) * VALUES;      // a cell and the values (2: V, V2)
  static constexpr int PART = KEY_WARPS * C * PL;      // the warps' shares
  // Chunks ahead and sets of shares of o as shared memory holds them; one set of shares of W S, and U of two chunks
  static constexpr int STAGES = kBoth ? (P > 64 ? 1 : MT == 2 ? 2 : 3) : kWrites ? 2 : 3;
  static constexpr int PARTS = (kWrites && MT == 2 && P > 64) || (kBoth && P > 64) || (kMode == 1 && MT == 2) ? 1 : 2;
  static constexpr int KIND = 4 * MT * 32 * 8;         // V or U as the left operand of 8-token steps: hi and lo, four a lane
  static constexpr int FRAGS = (kBoth ? 2 : 1) * KIND;
  static constexpr int FLOATS = STAGES * STAGE + PARTS * PART + 2 * FRAGS + (kWrites ? PART + 2 * C * VL : 0);
  static_assert(FLOATS * 4 <= 226 * 1024, "shared memory of a multiprocessor");
};

__device__ __forceinline__ Tf32A walk_operand(const float* frag, int lane) {
  const uint4 hi = reinterpret_cast<const uint4*>(frag)[lane], lo = reinterpret_cast<const uint4*>(frag)[32 + lane];
  return Tf32A{{hi.x, hi.y, hi.z, hi.w}, {lo.x, lo.y, lo.z, lo.w}};
}

template <int P, int MT, int kMode>
__global__ void __launch_bounds__((WalkShape<P, MT, kMode>::THREADS), 1)
state_walk_kernel(WalkArgs a) {
  using namespace bw;
  using Shape = WalkShape<P, MT, kMode>;
  constexpr bool kWrites = Shape::kWrites, kBoth = Shape::kBoth;
  constexpr int C = kChunkTokens, COLS = Shape::COLS, QL = walk_q_row(P), KL = walk_k_row(P), VL = Shape::VL, PL = Shape::PL;
  constexpr int CELL = walk_cell_copied(P, kMode), A = walk_cell_a(P, kMode), D = walk_cell_decay(P, kMode);
  constexpr int KEY_WARPS = Shape::KEY_WARPS, STAGES = Shape::STAGES, PARTS = Shape::PARTS;
  extern __shared__ __align__(16) float walk_smem[];
  float* part_s = walk_smem + STAGES * Shape::STAGE;      // [PARTS][KEY_WARPS][C][PL]
  float* frag_both = part_s + PARTS * Shape::PART;        // [2][V, U: kMode 2][4][MT][hi, lo][32][4]
  float* ws_s = frag_both + 2 * Shape::FRAGS;             // [KEY_WARPS][C][PL]
  float* u_both = ws_s + Shape::PART;                     // [2][C][VL]
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], part_full[PARTS], part_empty[PARTS], ws_full, u_full[2], v_full[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1 + kWalkHelpers * 32); mbar_init(&empty_bar[s], KEY_WARPS + kWalkHelpers); }
    for (int s = 0; s < PARTS; ++s) { mbar_init(&part_full[s], KEY_WARPS); mbar_init(&part_empty[s], kWalkHelpers); }
    mbar_init(&ws_full, KEY_WARPS);
    for (int s = 0; s < 2; ++s) { mbar_init(&u_full[s], kWalkHelpers); mbar_init(&v_full[s], kWalkHelpers); }      // the tokens' warps may be a chunk ahead
    mbar_init_fence();
  }
  // The blocks that start first take the longest walks (ranked while the kernel before runs; more requests than kRanked, whose
  // blocks are many, come as they are): four portions of 7 to 15 chunks, 16 heads of 128, the layer 205 -> 188 us.
  __shared__ int chunks_s[kRanked], request_s;
  const int requests = gridDim.z;
  if (tid == 0) request_s = blockIdx.z;
  if (requests <= kRanked)
    for (int r = tid; r < requests; r += Shape::THREADS) chunks_s[r] = a.request_chunk_start[r + 1] - a.request_chunk_start[r];
  __syncthreads();
  if (requests <= kRanked)
    for (int r = tid; r < requests; r += Shape::THREADS) {
      int before = 0;
      for (int other = 0; other < requests; ++other) before += chunks_s[other] > chunks_s[r] || (chunks_s[other] == chunks_s[r] && other < r);
      if (before == (int)blockIdx.z) request_s = r;
    }
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const int request = request_s, head = blockIdx.y, col0 = blockIdx.x * COLS, columns = min(COLS, a.vdim - col0);
  const int slot = a.slots[request];
  if (slot < 0 || slot >= a.max_slots) {
    if (tid == 0) atomicOr(a.err, kErrBadRequest);
    return;
  }
  const int first = a.request_chunk_start[request], chunks = a.request_chunk_start[request + 1] - first;
  bool alive = true;

  if (warp >= KEY_WARPS) {
    // ---------------------------------------------------------------- eight tokens of every chunk
    const int tile = warp - KEY_WARPS;
    // a request's chunks follow each other, all but the last of them whole
    const int first_row = chunks > 0 ? a.chunk_row[first] : 0;
    const int end_row = chunks > 0 ? a.chunk_row[first + chunks - 1] + a.chunk_count[first + chunks - 1] : 0;
    // Every one asks for its tokens' values of the chunks to come (four columns of MT tokens a lane), the first for the cells,
    // each in one copy.  Addresses are carried along: a warp's chain of instructions counts here.
    constexpr int PIECES = COLS / 4;
    const int piece = lane % PIECES * 4, piece_row = 8 * tile + lane / PIECES;
    const bool pieces = a.v_stride % 4 == 0 && a.v_head % 4 == 0 && columns % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15) == 0;
    const float* v_at = a.v + (first_row + piece_row) * a.v_stride + (long long)head * a.v_head + col0 + piece;
    const long long v_step = (32 / PIECES) * a.v_stride;
    const float* cell_at = a.cells + ((size_t)first * a.heads + head) * walk_cell_floats(P, kMode);
    const uint32_t v_to = smem_u32(walk_smem + Shape::V + piece_row * VL + piece);
    int v_rows = end_row - first_row - piece_row, stage_to = 0;      // rows from the lane's on; the stage that is filled next
    uint32_t empty_phase = 1;                                        // (stages that were never filled are empty)
    auto load = [&]() {
      if (v_rows + piece_row <= 0) return;
      if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[stage_to], empty_phase, a.err))) { alive = false; return; }
      if (tile == 0 && lane == 0) {
        mbar_expect_tx(&full_bar[stage_to], CELL * 4);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(walk_smem + stage_to * Shape::STAGE)), "l"(cell_at), "r"(CELL * 4),
                       "r"(smem_u32(&full_bar[stage_to])) : "memory");
      }
      const uint32_t to = v_to + stage_to * (Shape::STAGE * 4);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const int row = i * (32 / PIECES);
        const bool in = row < v_rows && piece < columns;
        if (pieces) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + row * (VL * 4)), "l"(in ? v_at + i * v_step : a.v),
                       "r"(in ? 16 : 0) : "memory");
        } else {      // the stage's barrier waits for a thread's copies, not for its plain stores: copies here, too
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const bool here = in && piece + x < columns;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + row * (VL * 4) + 4 * x),
                         "l"(here ? v_at + i * v_step + x : a.v), "r"(here ? 4 : 0) : "memory");
          }
        }
        if (kBoth)      // whole rows of P columns, zeros where there is nothing
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + Shape::VALUES * 4 + row * (VL * 4)),
                       "l"(cell_at + walk_cell_v2(P) + (piece_row + row) * P + (col0 + piece < P ? col0 + piece : 0)),
                       "r"(col0 + piece < P ? 16 : 0) : "memory");
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full_bar[stage_to])) : "memory");
      v_at += C * a.v_stride;
      v_rows -= C;
      cell_at += (size_t)a.heads * walk_cell_floats(P, kMode);
      if (++stage_to == STAGES) {
        stage_to = 0;
        empty_phase ^= 1;
      }
    };
    float* out_at = a.out + (long long)(first_row + 8 * tile + 2 * t) * a.out_stride + head * a.vdim + col0 + g;
    int out_rows = end_row - first_row - 8 * tile - 2 * t;
    // The outputs of chunk i: its own tokens' part, o, and the shares.  Columns 16 m + g (elements 0, 1) and + 8 (2, 3) of tokens
    // 2 t (0, 2) and 2 t + 1 of the tile.
    auto finish = [&](int i, const float (&o)[MT][4]) {
      if (!__all_sync(0xffffffffu, mbar_wait(&part_full[i % PARTS], (i / PARTS) & 1, a.err))) { alive = false; return; }
      const float* at = part_s + i % PARTS * Shape::PART + (8 * tile + 2 * t) * PL + g;
      float x[MT][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) x[m][e] = at[(e & 1) * PL + 16 * m + 8 * (e >> 1)];
#pragma unroll
      for (int w = 1; w < KEY_WARPS; ++w)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) x[m][e] += at[w * C * PL + (e & 1) * PL + 16 * m + 8 * (e >> 1)];
      __syncwarp();
      if (lane == 0) mbar_arrive(&part_empty[i % PARTS]);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if ((e & 1) < out_rows && 16 * m + g + 8 * (e >> 1) < columns) (e & 1 ? out_at + a.out_stride : out_at)[16 * m + 8 * (e >> 1)] = x[m][e] + o[m][e];
      out_at += (long long)C * a.out_stride;
      out_rows -= C;
    };
    for (int i = 0; i < (STAGES > 1 ? STAGES - 1 : 1); ++i) load();
    float before[MT][4] = {};      // o of the chunk before
    int s = 0;
    uint32_t full_phase = 0;
    for (int i = 0; i < chunks; ++i) {
      const float* stage = walk_smem + s * Shape::STAGE;
      const float* a_s = stage + A;
      float* u_s = u_both + (i & 1) * C * VL;
      float* frag_s = frag_both + (i & 1) * Shape::FRAGS;
      if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[s], full_phase, a.err))) { alive = false; break; }
      bool plain = stage[D + P] != 0.f;
      // The tile's V (or U) as an operand.  Two chunks' lie side by side: whoever writes the next one has seen the end of the
      // one before this.
      auto operand = [&](const float* from, bool writes, float* frags) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          Tf32A u;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = 8 * tile + t + 4 * (e >> 1), c = 16 * m + g + 8 * (e & 1);
            float x = from[r * VL + c];
            if (writes) {
              float seen = 0.f;
#pragma unroll
              for (int w = 0; w < KEY_WARPS; ++w) seen += ws_s[(w * C + r) * PL + c];
              x -= seen;
              u_s[r * VL + c] = x;
            }
            u.set(e, x);
          }
          uint4* at = reinterpret_cast<uint4*>(frags + (tile * MT + m) * 256) + lane;
          at[0] = make_uint4(u.hi[0], u.hi[1], u.hi[2], u.hi[3]);
          at[32] = make_uint4(u.lo[0], u.lo[1], u.lo[2], u.lo[3]);
        }
        __syncwarp();
      };
      if (kBoth) {
        operand(stage + Shape::V, false, frag_s);
        if (lane == 0) mbar_arrive(&v_full[i & 1]);
      }
      if (kWrites && !__all_sync(0xffffffffu, mbar_wait(&ws_full, i & 1, a.err))) { alive = false; break; }
      operand(stage + Shape::V + (kBoth ? Shape::VALUES : 0), kWrites, frag_s + (kBoth ? Shape::KIND : 0));
      if (lane == 0) mbar_arrive(&u_full[i & 1]);
      if (kWrites && i > 0) finish(i - 1, before);      // the warps of the keys wait for the shares' place
      if (!alive) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&u_full[i & 1], (i >> 1) & 1, a.err))) { alive = false; break; }
      float o[MT][4];
      {
        Tf32Sum<!kBoth> sum[MT];
#pragma unroll
        for (int kind = 0; kind < (kBoth ? 2 : 1); ++kind)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            if (kk > tile) break;
            const float* w = a_s + kind * (C * kWalkA) + (8 * tile + g) * kWalkA + 8 * kk + t;
            const Tf32B b(w[0], w[4]);
#pragma unroll
            for (int m = 0; m < MT; ++m)
              sum[m].add(walk_operand(frag_s + kind * Shape::KIND + (kk * MT + m) * 256, lane), b, kind == 0 && kk == 0);
          }
        float all = 0.f;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            o[m][e] = sum[m].of(e);
            all += fabsf(o[m][e]);
          }
        plain |= tf32_unsafe(all);
      }
      if (__builtin_expect(plain, 0)) {      // in order, and nothing of later tokens: not even times zero
        const float* values = kMode == 1 ? u_s : stage + Shape::V;
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = 8 * tile + 2 * t + (e & 1), c = 16 * m + g + 8 * (e >> 1);
            float x = 0.f;
#pragma unroll 1
            for (int from = 0; from <= r; ++from) {
              x = fmaf(a_s[r * kWalkA + from], values[from * VL + c], x);
              if (kBoth) x = fmaf(a_s[(C + r) * kWalkA + from], u_s[from * VL + c], x);
            }
            o[m][e] = x;
          }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
      if (!kWrites && i > 0) finish(i - 1, before);
      if (alive) load();
      if (!alive) break;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) before[m][e] = o[m][e];
      if (++s == STAGES) {
        s = 0;
        full_phase ^= 1;
      }
    }
    if (alive && chunks > 0) finish(chunks - 1, before);
  } else {
    // ---------------------------------------------------------------- 16 keys of the state
    // element e of tile j: key 4 t + j + 2 (e & 1) of the warp's 16, column 16 m + g + 8 (e >> 1)
    float* s_base = a.state + (size_t)slot * a.state_stride + (size_t)head * a.dim * a.vdim + col0;
    auto key_of = [&](int j, int e) { return warp * 16 + 4 * t + j + 2 * (e & 1); };
    auto column_of = [&](int m, int e) { return 16 * m + g + 8 * (e >> 1); };
    float s[MT][2][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int key = key_of(j, e), c = column_of(m, e);
          s[m][j][e] = key < a.dim && c < columns ? s_base[(size_t)key * a.vdim + c] : 0.f;
        }
    int st = 0;
    uint32_t full_phase = 0;
    for (int i = 0; i < chunks; ++i) {
      const float* q_s = walk_smem + st * Shape::STAGE;
      const float* w_s = q_s + walk_cell_w(P);            // kWrites only
      const float* k_s = q_s + walk_cell_k(P, kMode);
      const float* u_s = u_both + (i & 1) * C * VL;          // kWrites only
      const float* d_s = q_s + D;
      const float* frag_s = frag_both + (i & 1) * Shape::FRAGS;
      float all = 0.f;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) all += fabsf(s[m][j][e]);
      // the left operand: k-step j takes keys 4 t + j and 4 t + j + 2
      Tf32A left[MT][2];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          left[m][j].set(0, s[m][j][0]);
          left[m][j].set(1, s[m][j][2]);
          left[m][j].set(2, s[m][j][1]);
          left[m][j].set(3, s[m][j][3]);
        }
      const bool torn = __any_sync(0xffffffffu, tf32_unsafe(all));
      if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[st], full_phase, a.err))) { alive = false; break; }
      const bool plain = torn || d_s[P] != 0.f;
      const int n = __float_as_int(d_s[P + 1]);
      // Sums over the warp's keys of S^T and rows of q or W, [columns][tokens].  The small terms first, then the large ones into
      // the same accumulator.
      float sum[4][MT][4];
      auto over_keys = [&](const float* rows) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          Tf32B b[2][2];
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            const float4 x = *reinterpret_cast<const float4*>(rows + (16 * half + 8 * y + g) * QL + warp * 16 + 4 * t);
            b[y][0] = Tf32B(x.x, x.z);
            b[y][1] = Tf32B(x.y, x.w);
          }
#pragma unroll
          for (int term = 0; term < 6; ++term)
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
              for (int m = 0; m < MT; ++m) {
                const int j = term & 1;
                float (&d)[4] = sum[2 * half + y][m];
                if (term == 0) mma_tf32_first(d, left[m][0].lo, b[y][0].hi);
                else mma_tf32(d, term < 2 ? left[m][j].lo : left[m][j].hi, term < 2 || term >= 4 ? b[y][j].hi : b[y][j].lo);
              }
        }
      };
      auto leave = [&](float* shares) {
        float* at = shares + (warp * C + 2 * t) * PL + g;
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) at[(8 * y + (e & 1)) * PL + 16 * m + 8 * (e >> 1)] = sum[y][m][e];
      };
      // the same on the CUDA cores: the four lanes of a column have four keys each
      auto over_keys_plain = [&](const float* rows, float* shares) {
#pragma unroll 1
        for (int r = 0; r < n; ++r)
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int high = 0; high < 2; ++high) {
              float x = 0.f;
#pragma unroll
              for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                  if (key_of(j, e) < a.dim) x = fmaf(rows[r * QL + key_of(j, e)], s[m][j][e + 2 * high], x);
              x += __shfl_xor_sync(0xffffffffu, x, 1);
              x += __shfl_xor_sync(0xffffffffu, x, 2);
              if (t == 0) shares[(warp * C + r) * PL + 16 * m + g + 8 * high] = x;
            }
      };
      if (kWrites) {      // the shares' place is free: the U that was made of the last ones has been waited for
        if (__builtin_expect(!plain, 1)) {
          over_keys(w_s);
          leave(ws_s);
        } else {
          over_keys_plain(w_s, ws_s);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ws_full);
      }
      float* shares = part_s + i % PARTS * Shape::PART;
      if (i >= PARTS && !__all_sync(0xffffffffu, mbar_wait(&part_empty[i % PARTS], (i / PARTS - 1) & 1, a.err))) { alive = false; break; }
      if (__builtin_expect(!plain, 1)) {
        over_keys(q_s);
        leave(shares);
      } else {
        over_keys_plain(q_s, shares);
      }
      float gained[MT][2][4];
      all = 0.f;
      auto gain_of = [&](const float* keys, const float* frags, bool more) {
        Tf32Sum<!kBoth> gain[2][MT];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const float* kt = keys + (8 * kk + t) * KL + warp * 16 + 2 * g;
          const float2 lo = *reinterpret_cast<const float2*>(kt), hi = *reinterpret_cast<const float2*>(kt + 4 * KL);
          const Tf32B b[2] = {Tf32B(lo.x, hi.x), Tf32B(lo.y, hi.y)};
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            const Tf32A u = walk_operand(frags + (kk * MT + m) * 256, lane);
#pragma unroll
            for (int j = 0; j < 2; ++j) gain[j][m].add(u, b[j], kk == 0);
          }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              gained[m][j][e] = more ? gained[m][j][e] + gain[j][m].of(e) : gain[j][m].of(e);
              all += fabsf(gained[m][j][e]);      // a value (or U) that is not fit shows here, too
            }
      };
      if (kBoth) {
        if (!__all_sync(0xffffffffu, mbar_wait(&v_full[i & 1], (i >> 1) & 1, a.err))) { alive = false; break; }
        if (__builtin_expect(!plain, 1)) gain_of(k_s, frag_s, false);
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&u_full[i & 1], (i >> 1) & 1, a.err))) { alive = false; break; }
      if (__builtin_expect(!plain, 1)) gain_of(kBoth ? q_s + walk_cell_k2(P) : k_s, frag_s + (kBoth ? Shape::KIND : 0), kBoth);
      if (__builtin_expect(__any_sync(0xffffffffu, plain || tf32_unsafe(all)), 0)) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int key = key_of(j, e), c = column_of(m, e);
              float x = 0.f;
              if (key < a.dim && c < columns)
#pragma unroll 1
                for (int r = 0; r < n; ++r) {
                  x = fmaf(k_s[r * KL + key], (kMode == 1 ? u_s : q_s + Shape::V)[r * VL + c], x);
                  if (kBoth) x = fmaf(k_s[(C + r) * KL + key], u_s[r * VL + c], x);
                }
              gained[m][j][e] = x;
            }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float d0 = d_s[key_of(j, 0)], d1 = d_s[key_of(j, 1)];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[m][j][e] = fmaf(e & 1 ? d1 : d0, s[m][j][e], gained[m][j][e]);
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&part_full[i % PARTS]);
        mbar_arrive(&empty_bar[st]);
      }
      if (++st == STAGES) {
        st = 0;
        full_phase ^= 1;
      }
    }
    if (alive && chunks > 0 && a.request_active[request]) {      // (whoever brings no tokens leaves the slot alone)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = key_of(j, e), c = column_of(m, e);
            if (key < a.dim && c < columns) s_base[(size_t)key * a.vdim + c] = s[m][j][e];
          }
    }
  }
  // a wait ran out: give copies that may still be in flight time to end before leaving
  if (!alive)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

// Narrow blocks (16 value columns) while each has a multiprocessor of its own: the chain of a chunk is shortest there.  More
// blocks than that are wide ones, which share the operands' loads and splits.
template <int kMode>
inline cudaError_t launch_state_walk(const WalkArgs& a, int P, int requests, cudaStream_t stream) {
  const bool narrow = (long long)requests * a.heads * ((a.vdim + 15) / 16) <= device_sms();
  auto go = [&](auto kernel, int MT, int threads, int floats) {
    const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, floats * (int)sizeof(float));
    if (status != cudaSuccess) return status;
    return launch(kernel, dim3((a.vdim + 16 * MT - 1) / (16 * MT), a.heads, requests), dim3(threads), (size_t)floats * sizeof(float), stream, a);
  };
#define CIE_WALK(p)                                                                                                        \
  if (P == p)                                                                                                              \
    return narrow ? go(state_walk_kernel<p, 1, kMode>, 1, WalkShape<p, 1, kMode>::THREADS, WalkShape<p, 1, kMode>::FLOATS) \
                  : go(state_walk_kernel<p, 2, kMode>, 2, WalkShape<p, 2, kMode>::THREADS, WalkShape<p, 2, kMode>::FLOATS)
  CIE_WALK(32);
  CIE_WALK(64);
  if constexpr (kMode != 2) {      // (whose heads are padded to powers of two)
    CIE_WALK(96);
  }
  CIE_WALK(128);
#undef CIE_WALK
  return cudaErrorInvalidValue;
}

}  // namespace cie
