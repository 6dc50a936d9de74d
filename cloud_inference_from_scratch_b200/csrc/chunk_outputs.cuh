// The last step of the recurrences that run in chunks of 32 tokens: a chunk's outputs from the state before it and from the
// chunk's own tokens,
//
//     o_t = S^T q_t + sum_(s <= t) a_ts v_s            t < 32, S: [dim][vdim], float32 on the CUDA cores
//
// by a block of 256 threads (dim and vdim up to 128).  What bounds it is the data shared memory returns (128 bytes a cycle,
// broadcast or not), so a thread takes 8 tokens and 4 columns: 12 cycles of loads for 32 products of a warp.  The warps form
// two halves that take every second 16 rows of S (and every second token s) and add their sums up at the end.  S comes
// once, 32 rows at a time, through two cp.async stages, which the callers lay over rows that they need no more: three blocks
// fit an SM, and their waits overlap.
#pragma once

#include "common.cuh"

namespace cie {

constexpr int kOutTokens = 32, kOutThreads = 256, kOutRows = 32;      // tokens of a chunk; rows of S of a stage
constexpr int kOutWeights = kOutTokens + 4;                           // row of the weights: a_s[s * kOutWeights + t]

__host__ __device__ __forceinline__ int pad4(int x) { return (x + 3) & ~3; }

// Calls load(row, piece) and then store(row, piece, value) for the 16-byte pieces of n rows, four loads a thread in flight;
// places by addition: a division a piece costs as much as the rest of the copy.
template <typename Load, typename Store>
__device__ __forceinline__ void each_piece(int n, int pieces, Load load, Store store) {
  int r = threadIdx.x / pieces, c = threadIdx.x - r * pieces;
  const int dr = blockDim.x / pieces, dc = blockDim.x - dr * pieces;
  while (r < n) {
    float4 v[4];
    int row[4], piece[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      row[u] = r;
      piece[u] = c;
      if (r < n) v[u] = load(r, c);
      r += dr;
      c += dc;
      if (c >= pieces) {
        c -= pieces;
        ++r;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (row[u] < n) store(row[u], piece[u], v[u]);
  }
}

// The stages of S: rows [dim][vdim] from global memory, vdim padded to whole 16-byte pieces, rows past dim zeros.
struct StateRing {
  float* first;           // the stages, kOutRows rows each
  float* second;
  const float* state;
  int dim, vdim;
  __device__ __forceinline__ int blocks() const { return (dim + kOutRows - 1) / kOutRows; }
  __device__ __forceinline__ float* stage(int block) const { return block & 1 ? second : first; }
  __device__ __forceinline__ void issue(int block) const {
    if (block < blocks()) {
      const int ld = pad4(vdim), first = block * kOutRows;
      float* dst = stage(block);
      if (vdim % 4 == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0) {
        const int pieces = vdim / 4, dr = kOutThreads / pieces, dc = (kOutThreads - dr * pieces) * 4;
        int r = threadIdx.x / pieces, c = (threadIdx.x - r * pieces) * 4;
        for (; r < kOutRows; r += dr, c += dc) {
          if (c >= vdim) {
            c -= vdim;
            if (++r >= kOutRows) break;
          }
          const bool in = first + r < dim;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * ld + c)),
                       "l"(state + (in ? (size_t)(first + r) * vdim + c : 0)), "r"(in ? 16 : 0));
        }
      } else {
        for (int e = threadIdx.x; e < kOutRows * ld; e += kOutThreads) {
          const int r = e / ld, c = e - r * ld;
          dst[e] = first + r < dim && c < vdim ? state[(size_t)(first + r) * vdim + c] : 0.f;
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  }
};

// q: [32][q_ld] in shared memory (q_ld and the padded dim multiples of 4, columns past dim zeros), v: [32][pad4(vdim)], a:
// the weights.  The ring's first block has been issued; the block meets here before anything is read.  write(t, c, o) gets
// the four columns c .. c + 3 of token t; tokens past the chunk's last one are worked out from whatever their rows hold.
template <typename Write>
__device__ __forceinline__ void chunk_outputs(const StateRing& s, const float* q, int q_ld, const float* a, const float* v, Write write) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (warp & 3) * 8, half = warp >> 2, c = lane * 4, ld = pad4(s.vdim);
  const bool live = c < ld;
  float4 acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int q_end = pad4(s.dim);
  for (int block = 0; block < s.blocks(); ++block) {
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();          // the block has landed; everybody is done with the one before, whose stage is filled next
    s.issue(block + 1);
    const float* rows = s.stage(block) + half * 16 * ld + c;
    const int x0 = block * kOutRows + half * 16, x1 = min(x0 + 16, q_end);
    if (live) {
      for (int x = x0; x < x1; x += 4) {
        float4 sv[4];
#pragma unroll
        for (int y = 0; y < 4; ++y) sv[y] = *reinterpret_cast<const float4*>(rows + (x - x0 + y) * ld);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 qv = *reinterpret_cast<const float4*>(q + (t0 + i) * q_ld + x);
          const float q4[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            acc[i].x = fmaf(q4[y], sv[y].x, acc[i].x);
            acc[i].y = fmaf(q4[y], sv[y].y, acc[i].y);
            acc[i].z = fmaf(q4[y], sv[y].z, acc[i].z);
            acc[i].w = fmaf(q4[y], sv[y].w, acc[i].w);
          }
        }
      }
    }
  }
  if (live) {
    for (int j = half; j < t0 + 8; j += 2) {
      const float4 vv = *reinterpret_cast<const float4*>(v + j * ld + c);
      const float4 lo = *reinterpret_cast<const float4*>(a + j * kOutWeights + t0), hi = *reinterpret_cast<const float4*>(a + j * kOutWeights + t0 + 4);
      const float w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (t0 + i < j) continue;      // a later token: not even times zero
        acc[i].x = fmaf(w[i], vv.x, acc[i].x);
        acc[i].y = fmaf(w[i], vv.y, acc[i].y);
        acc[i].z = fmaf(w[i], vv.z, acc[i].z);
        acc[i].w = fmaf(w[i], vv.w, acc[i].w);
      }
    }
  }
  __syncthreads();            // the ring is free: the second half's sums go through it
  if (half == 1 && live) {
#pragma unroll
    for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(s.first + (t0 + i) * ld + c) = acc[i];
  }
  __syncthreads();
  if (half == 0 && live) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 other = *reinterpret_cast<const float4*>(s.first + (t0 + i) * ld + c);
      write(t0 + i, c, make_float4(acc[i].x + other.x, acc[i].y + other.y, acc[i].z + other.z, acc[i].w + other.w));
    }
  }
}

// Four columns of a float32 row of `width` columns in all; `wide`: rows are 16-byte aligned whole pieces.
__device__ __forceinline__ void store4(float* row, int c, int width, const float4& o, bool wide) {
  if (wide) {
    *reinterpret_cast<float4*>(row + c) = o;
    return;
  }
  row[c] = o.x;
  if (c + 1 < width) row[c + 1] = o.y;
  if (c + 2 < width) row[c + 2] = o.z;
  if (c + 3 < width) row[c + 3] = o.w;
}

}  // namespace cie
