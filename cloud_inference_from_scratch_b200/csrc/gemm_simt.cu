// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) on the CUDA cores, float32 accumulation, any M, N, K.
//
// This is the 32-bit path's matrix product for rows that the tensor-core form (gemm_f32_tcgen05.cu: whole aligned pieces, 512
// columns and more) does not take, and the fallback of the bfloat16 path for shapes the tensor-core kernel refuses.  Each output element
// is the sum over k in ascending order with one fused multiply-add per k, so a row's result does
// not depend on how many other rows the call has or where the row sits in it, nor on the kernel and tile it is worked out in.
// The reference runs these products through cuBLAS (src/cloud_engine/model.py:100,134-136,217,227).
#include "common.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

constexpr int kTileM = 64, kTileN = 64, kTileK = 16;

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TIn* __restrict__ a, const TIn* __restrict__ w, const float* __restrict__ bias,
                 TOut* __restrict__ c, int m_total, int n_total, int k_total) {
  __shared__ float a_tile[kTileK][kTileM + 4];
  __shared__ float w_tile[kTileK][kTileN + 4];
  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < k_total; k0 += kTileK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256;      // 0..1023 over a 64 x 16 tile
      const int r = e / kTileK, kk = e % kTileK;
      const int gk = k0 + kk;
      const int gm = m0 + r, gn = n0 + r;
      a_tile[kk][r] = (gm < m_total && gk < k_total) ? to_float(a[(size_t)gm * k_total + gk]) : 0.f;
      w_tile[kk][r] = (gn < n_total && gk < k_total) ? to_float(w[(size_t)gn * k_total + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kTileK; ++kk) {
      float av[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = a_tile[kk][tm + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = w_tile[kk][tn + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + tm + i;
    if (gm >= m_total) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tn + j;
      if (gn >= n_total) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      c[(size_t)gm * n_total + gn] = from_float<TOut>(v);
    }
  }
}

// The 32-bit path's product: rows of A and W that are whole, aligned 16-byte pieces.  The same sums in the same order
// as above, whatever the tile.  A CTA's tile is BM x BN, a thread's TM x TN, a warp 4 x 8 threads whose rows and columns
// are interleaved.  Both operands come as they lie in memory, 32 columns at a time, through a ring of cp.async stages
// (the products of the 32-bit path are small: one or two CTAs an SM have to hide their own trips to memory), and are
// read from shared memory as 16-byte pieces along K: TM + TN loads for 4 TM TN products.
constexpr int kRingK = 32, kRingStages = 4, kRingRow = kRingK + 4;      // rows are padded: 8 of them side by side meet 32 banks

__device__ __forceinline__ void simt_cp_async16(void* dst, const void* src, bool whole) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(whole ? 16 : 0));       // 0 source bytes: zeros
}

template <int BM, int BN, int TM, int TN>
constexpr int gemm_f32_smem() { return kRingStages * (BM + BN) * kRingRow * (int)sizeof(float); }

template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(BM * BN / (TM * TN))
gemm_f32_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ c,
                int m_total, int n_total, int k_total) {
  constexpr int kThreads = BM * BN / (TM * TN), kWarpsM = BM / (4 * TM), kPieces = (BM + BN) * (kRingK / 4);
  extern __shared__ __align__(16) float ring[];
  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int row0 = (warp % kWarpsM) * 4 * TM + (lane >> 3), col0 = (warp / kWarpsM) * 8 * TN + (lane & 7);
  auto issue = [&](int step) {
    const int k0 = step * kRingK;
    if (k0 < k_total) {
      float* stage = ring + (step % kRingStages) * (BM + BN) * kRingRow;
      for (int e = tid; e < kPieces; e += kThreads) {
        const int r = e / (kRingK / 4), k = k0 + (e % (kRingK / 4)) * 4;
        const bool in_a = r < BM;
        const int row = in_a ? m0 + r : n0 + r - BM;
        const bool whole = row < (in_a ? m_total : n_total) && k < k_total;
        const float* src = in_a ? a : w;
        simt_cp_async16(stage + r * kRingRow + (k - k0), whole ? src + (size_t)row * k_total + k : src, whole);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  float acc[TM][TN] = {};
  const int steps = (k_total + kRingK - 1) / kRingK;
  for (int i = 0; i < kRingStages - 1; ++i) issue(i);
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kRingStages - 2));
    __syncthreads();               // the step has landed; everybody is done with the one before, whose place is filled next
    issue(step + kRingStages - 1);
    const float* a_s = ring + (step % kRingStages) * (BM + BN) * kRingRow + row0 * kRingRow;
    const float* w_s = ring + (step % kRingStages) * (BM + BN) * kRingRow + (BM + col0) * kRingRow;
#pragma unroll
    for (int kk = 0; kk < kRingK; kk += 4) {
      float4 av[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a_s + 4 * i * kRingRow + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 wv = *reinterpret_cast<const float4*>(w_s + 8 * j * kRingRow + kk);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].x, wv.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].y, wv.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].z, wv.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].w, wv.w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + row0 + 4 * i;
    if (gm >= m_total) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + col0 + 8 * j;
      if (gn >= n_total) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      c[(size_t)gm * n_total + gn] = v;
    }
  }
}

// The tiles, and what they cost for 2,048 columns of K (B200, us): one CTA an SM, and every further CTA of the SM.  A CTA
// alone waits for shared memory and its own products; several together are bound by what shared memory returns (128 bytes a
// cycle), which is why larger tiles win once there are enough of them.  Who comes here has few rows (logits) or short ones:
// logits of 151,936 x 2,048 take 313 us with 1 to 8 rows (8 x 128), 372 with 16 (16 x 128; 576 with 8 x 128), 665 with 17
// (32 x 32; 705 with 16 x 128) and 1,045 with 64 (64 x 128; 1,338 with 32 x 32); 300 rows of 2,048 x 508 33 (32 x 32; 36 with
// 16 x 128), 1,000 rows 59 (128 x 128; 73 with 32 x 32); 300 of 2,048 x 64 6, 1,000 10.
struct F32Tile {
  int rows, columns;
  float alone, further;
};
constexpr F32Tile kF32Tiles[] = {{8, 128, 46.f, 33.f}, {16, 128, 54.f, 39.f}, {32, 32, 52.f, 19.f},
                                 {64, 128, 183.f, 101.f}, {128, 128, 220.f, 221.f}};
constexpr int kF32TileCount = sizeof(kF32Tiles) / sizeof(kF32Tiles[0]);

int f32_tile(int m, int n) {
  const int sms = device_sms();
  int best = 0;
  float least = 0.f;
  for (int i = 0; i < kF32TileCount; ++i) {
    const F32Tile& tile = kF32Tiles[i];
    const long long tiles = (long long)((m + tile.rows - 1) / tile.rows) * ((n + tile.columns - 1) / tile.columns);
    const float cost = tile.alone + (float)((tiles + sms - 1) / sms - 1) * tile.further;
    if (i == 0 || cost < least) {
      best = i;
      least = cost;
    }
  }
  return best;
}

cudaError_t launch_f32(int tile, const float* a, const float* w, const float* bias, float* c, int m, int n, int k,
                       cudaStream_t stream) {
#define CIE_F32_TILE(BM, BN, TM, TN)                                                                                  \
  {                                                                                                                   \
    constexpr int smem = gemm_f32_smem<BM, BN, TM, TN>();                                                             \
    static const cudaError_t raised =                                                                                 \
        cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);     \
    if (raised != cudaSuccess) return raised;                                                                         \
    return launch(gemm_f32_kernel<BM, BN, TM, TN>, dim3((n + BN - 1) / BN, (m + BM - 1) / BM),                        \
                  dim3(BM * BN / (TM * TN)), smem, stream, a, w, bias, c, m, n, k);                                   \
  }
  switch (tile) {
    case 0: CIE_F32_TILE(8, 128, 2, 4)
    case 1: CIE_F32_TILE(16, 128, 4, 4)
    case 2: CIE_F32_TILE(32, 32, 4, 4)
    case 3: CIE_F32_TILE(64, 128, 8, 8)
    default: CIE_F32_TILE(128, 128, 8, 8)
  }
#undef CIE_F32_TILE
}

// Few rows (decode): one warp per output column, lanes stride over k; the per-lane partial sums
// are combined by a fixed shuffle tree, so the result still does not depend on M.
// Used only when m_total <= kSmallM.
constexpr int kSmallM = 8;
template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_small_m_kernel(const TIn* __restrict__ a, const TIn* __restrict__ w, const float* __restrict__ bias,
                    TOut* __restrict__ c, int m_total, int n_total, int k_total) {
  pdl_wait();
  pdl_trigger();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n_total) return;
  const TIn* wrow = w + (size_t)warp * k_total;
  float acc[kSmallM];
#pragma unroll
  for (int i = 0; i < kSmallM; ++i) acc[i] = 0.f;
  for (int k = lane; k < k_total; k += 32) {
    const float wv = to_float(wrow[k]);
#pragma unroll
    for (int i = 0; i < kSmallM; ++i)
      if (i < m_total) acc[i] = fmaf(to_float(a[(size_t)i * k_total + k]), wv, acc[i]);
  }
#pragma unroll
  for (int i = 0; i < kSmallM; ++i) {
    if (i >= m_total) break;
    float v = warp_sum(acc[i]);
    if (lane == 0) {
      if (bias) v += bias[warp];
      c[(size_t)i * n_total + warp] = from_float<TOut>(v);
    }
  }
}

}  // namespace cie

using namespace cie;

template <typename TIn, typename TOut>
static cudaError_t launch_simt(const void* a, const void* w, const float* bias, void* c, int m, int n,
                               int k, int allow_small, cudaStream_t stream) {
  if (allow_small && m <= kSmallM) {
    const int warps_per_block = 8;
    return cie::launch(gemm_small_m_kernel<TIn, TOut>, dim3((n + warps_per_block - 1) / warps_per_block),
                       dim3(256), 0, stream, (const TIn*)a, (const TIn*)w, bias, (TOut*)c, m, n, k);
  }
  dim3 grid((n + kTileN - 1) / kTileN, (m + kTileM - 1) / kTileM);
  return cie::launch(gemm_simt_kernel<TIn, TOut>, grid, dim3(256), 0, stream, (const TIn*)a,
                     (const TIn*)w, bias, (TOut*)c, m, n, k);
}

// in_dtype: element type of A and W; out_dtype: element type of C (float32 for logits).
// allow_small = 0 keeps one summation order for every M (the 32-bit check path uses that).
extern "C" int cie_gemm_simt(const void* a, const void* w, const float* bias, void* c, int m, int n,
                             int k, int in_dtype, int out_dtype, int allow_small, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0) CIE_FAIL("gemm_simt: K must be positive, got %d", k);
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t status;
  // 32-bit rows that are whole 16-byte pieces; operands that are not take the general kernel
  const bool pieces = k % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
  if (in_dtype == kFloat32 && out_dtype == kFloat32 && pieces && !(allow_small && m <= kSmallM))
    status = launch_f32(f32_tile(m, n), (const float*)a, (const float*)w, bias, (float*)c, m, n, k, s);
  else if (in_dtype == kFloat32 && out_dtype == kFloat32) status = launch_simt<float, float>(a, w, bias, c, m, n, k, allow_small, s);
  else if (in_dtype == kBFloat16 && out_dtype == kBFloat16) status = launch_simt<__nv_bfloat16, __nv_bfloat16>(a, w, bias, c, m, n, k, allow_small, s);
  else if (in_dtype == kBFloat16 && out_dtype == kFloat32) status = launch_simt<__nv_bfloat16, float>(a, w, bias, c, m, n, k, allow_small, s);
  else CIE_FAIL("gemm_simt: unsupported element types in=%d out=%d", in_dtype, out_dtype);
  if (status != cudaSuccess) CIE_FAIL("gemm_simt: launch failed: %s", cudaGetErrorString(status));
  return 0;
}
