// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) of float32 operands on the tensor cores, as accurate as float32 sums.
//
// Every value is the sum of three bfloat16 terms (8 + 8 + 8 bits of its mantissa: hi, mid, lo; exact from 2^-110 up, below
// that to 2^-134), and a product is worked out from the six of the nine pairs that matter: hi hi, hi mid, mid hi, hi lo,
// mid mid, lo hi.  What is left out is below 2^-26 of the product, half of what rounding it to float32 would cost.  The
// tensor core's own sums are the other half of the matter: it cuts what it adds, so a long sum in one accumulator would
// drift.  Here hi hi, the terms near 2^-8 and those near 2^-16 have an accumulator each, and every kInterval columns of K
// they are taken out and added up in registers, rounded to nearest.  Root mean
// square error of 300 x 2,048 results of normal operands, against sums in float32 along K: 1.3e-7 and 4.0e-7 at K = 512, 1.4e-7
// and 8.1e-7 at 2,048, 2.1e-7 and 1.9e-6 at 11,008.
//
// A row's result depends on neither the number of rows, nor its place among them, nor the tile (the additions of an element
// are the same ones in the same order).  A row of A or W that holds an infinity, a NaN or a value that bfloat16 rounds to
// infinity is found while it is split; its results are summed in float32 along K instead.
//
// What bounds it: shared memory, which the split terms are written to (3 x 2 bytes an element) and which the tensor core
// reads both operands from, and the trips of the 32-bit operands to memory.  300 rows,
// 2,048 x 2,048: 48 us against 125 on the CUDA cores; 22,016 x 2,048: 279 and 690; 2,048 x 11,008: 223 and 655; one row of
// 2,048 x 11,008: 139 and 239, of 2,048 x 2,048 28 and 46, of 22,016 x 2,048 108 and 73.
#include "blackwell.cuh"
#include "common.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

using namespace bw;

constexpr int kRows = 128, kStep = 64, kInterval = 128, kStages = 3;
constexpr int kSplitWarps = 16, kAddWarps = 8, kThreads = (kSplitWarps + 1 + kAddWarps) * 32;      // split, multiply, add up
constexpr int kMinK = 512;          // four intervals and more (see the flags below)

__host__ __device__ constexpr int stage_bytes(int columns) { return 3 * (kRows + columns) * kStep * 2; }

__device__ __forceinline__ void load_columns8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ uint32_t pair_of(float x, float y) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&pair);
}
// Two values to two bfloat16 and what is left of them.
__device__ __forceinline__ uint32_t take_term(float& x, float& y) {
  const uint32_t bits = pair_of(x, y);
  x -= __uint_as_float(bits << 16);
  y -= __uint_as_float(bits & 0xffff0000u);
  return bits;
}

__device__ __noinline__ float sum_of(const float* a, const float* w, int k_total) {
  float sum = 0.f;
  for (int k = 0; k < k_total; ++k) sum = fmaf(a[k], w[k], sum);
  return sum;
}

// Persistent: a CTA an SM, which walks over tiles of 128 rows of A and BN of W, row blocks of A fastest so that the CTAs that
// run at one time share rows of W in L2.  Warps 0..15 split: a step of kStep columns of K comes from memory into registers
// a step ahead and goes to shared memory as [A hi, mid, lo][W hi, mid, lo], 128-byte-swizzled.  Warp 16 multiplies: the W
// terms lie one after the other, so three instructions make the six products (hi by all three, mid by two, lo by one), each
// into the accumulator of its magnitude.  Warps 17..24 add up
// and write, half of the columns each four.
template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tc_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                   float* __restrict__ c, int m_total, int n_total, int k_total, int* err) {
  constexpr int STAGES = kStages, PASSES_A = kRows / 32, PASSES = (kRows + BN) / 32, TERM_A = kRows * kStep * 2, TERM_W = BN * kStep * 2;
  constexpr int COLUMNS = 6 * BN <= 256 ? 256 : 512;
  static_assert(6 * BN <= 512 && (3 * BN) % 16 == 0, "two sets of three accumulators in tensor memory");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int apart[2][kRows + BN];      // rows that are summed in float32: (number of the tile) + 1, every second tile's

  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_m = (m_total + kRows - 1) / kRows, tiles_n = (n_total + BN - 1) / BN, total = tiles_m * tiles_n;
  const int steps = (k_total + kStep - 1) / kStep, intervals = (steps + kInterval / kStep - 1) / (kInterval / kStep);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], kSplitWarps); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], kAddWarps); }
    mbar_init_fence();
  }
  for (int e = tid; e < 2 * (kRows + BN); e += kThreads) (&apart[0][0])[e] = 0;
  if (warp == kSplitWarps) tmem_alloc<COLUMNS>(&tmem_base_s);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  bool alive = true;

  if (warp < kSplitWarps) {
    const int sub = warp * 2 + (lane >> 4), kq = (lane & 15) * 4;      // rows sub, sub + 32, ..; four columns
    const uint32_t place = (uint32_t)(sub * 128 + ((((lane & 15) >> 1) ^ (sub & 7)) << 4) + (lane & 1) * 8);
    const float* row_at[PASSES];
    uint32_t inside = 0;              // which of the rows are the matrices'
    auto enter = [&](int tile) {
      const int row = tile % tiles_m * kRows + sub, col = tile / tiles_m * BN + sub;
      inside = 0;
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        const int r = i < PASSES_A ? row + i * 32 : col + (i - PASSES_A) * 32;
        const bool in = r < (i < PASSES_A ? m_total : n_total);
        inside |= (uint32_t)in << i;
        row_at[i] = (i < PASSES_A ? a : w) + (in ? (size_t)r * k_total : 0) + kq;
      }
    };
    auto fetch = [&](int i, bool in_k, int k0) {
      return (inside >> i & 1) && in_k ? __ldg(reinterpret_cast<const float4*>(row_at[i] + k0)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 next[PASSES];
    int tile = blockIdx.x;
    enter(tile);
#pragma unroll
    for (int i = 0; i < PASSES; ++i) next[i] = fetch(i, kq < k_total, 0);
    int count = 0, local = 0;
    for (; tile < total && alive; tile += gridDim.x, ++local) {
      for (int step = 0; step < steps; ++step, ++count) {
        const int s = count % STAGES;
        if (count >= STAGES && !__all_sync(0xffffffffu, mbar_wait(&empty_bar[s], (count / STAGES - 1) & 1, err))) { alive = false; break; }
        const uint32_t held = inside;
        int k0 = (step + 1) * kStep;
        if (step + 1 == steps) {
          k0 = 0;
          if (tile + (int)gridDim.x < total) enter(tile + gridDim.x);
        }
        const bool in_k = k0 + kq < k_total;
        unsigned char* stage = ring + (size_t)s * stage_bytes(BN) + place;
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
          constexpr int kRowBytes = 32 * 128;
          const bool in_a = i < PASSES_A;
          // rows behind the matrix are left as they are: what comes of them is not written
          if (held >> i & 1) {
            float4 x = next[i];
            unsigned char* dst = stage + (in_a ? i * kRowBytes : 3 * TERM_A + (i - PASSES_A) * kRowBytes);
            const int term = in_a ? TERM_A : TERM_W;
            uint32_t lo = take_term(x.x, x.y), hi = take_term(x.z, x.w);
            *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
            lo = take_term(x.x, x.y);
            hi = take_term(x.z, x.w);
            *reinterpret_cast<uint2*>(dst + term) = make_uint2(lo, hi);
            *reinterpret_cast<uint2*>(dst + 2 * term) = make_uint2(pair_of(x.x, x.y), pair_of(x.z, x.w));
            const float rest = (x.x + x.y) + (x.z + x.w);      // NaN where a term is not finite
            if (!(rest == rest)) apart[local & 1][in_a ? i * 32 + sub : kRows + (i - PASSES_A) * 32 + sub] = local + 1;
          }
          next[i] = fetch(i, in_k, k0);
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[s]);
      }
    }
  } else if (warp == kSplitWarps) {
    if (lane == 0) {
      const uint64_t desc0 = smem_desc_sw128(smem_u32(ring));
      int count = 0, part = 0;
      for (int tile = blockIdx.x; tile < total && alive; tile += gridDim.x) {
        for (int step = 0; step < steps; ++step, ++count) {
          const int s = count % STAGES, buf = part & 1;
          const bool first = step % (kInterval / kStep) == 0;
          if (first && part >= 2 && !mbar_wait(&acc_empty[buf], ((part >> 1) - 1) & 1, err)) { alive = false; break; }
          if (!mbar_wait(&full_bar[s], (count / STAGES) & 1, err)) { alive = false; break; }
          tc_fence_after();
          const uint64_t at = desc0 + (uint64_t)((s * stage_bytes(BN)) >> 4), wt = at + (uint64_t)((3 * TERM_A) >> 4);
          const uint32_t d = tmem_base + buf * 3 * BN;
#pragma unroll
          for (int kk = 0; kk < kStep / 16; ++kk) {
            umma_bf16(d, at + 2 * kk, wt + 2 * kk, idesc_bf16(kRows, 3 * BN), !first || kk > 0);
            umma_bf16(d + BN, at + (TERM_A >> 4) + 2 * kk, wt + 2 * kk, idesc_bf16(kRows, 2 * BN), 1);
            umma_bf16(d + 2 * BN, at + 2 * (TERM_A >> 4) + 2 * kk, wt + 2 * kk, idesc_bf16(kRows, BN), 1);
          }
          tc_commit(&empty_bar[s]);
          if (step + 1 == steps || (step + 1) % (kInterval / kStep) == 0) {
            tc_commit(&acc_full[buf]);
            ++part;
          }
        }
      }
    }
    __syncwarp();
  } else {
    constexpr int COLS = BN / 2;
    const int quarter = warp & 3, half = (warp - kSplitWarps - 1) >> 2;
    const uint32_t lane_base = ((uint32_t)(quarter * 32) << 16) + half * COLS;
    int part = 0, local = 0;
    for (int tile = blockIdx.x; tile < total && alive; tile += gridDim.x, ++local) {
      float acc[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
      for (int i = 0; i < intervals; ++i, ++part) {
        const int buf = part & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (part >> 1) & 1, err))) { alive = false; break; }
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < COLS; c0 += 8) {
          uint32_t big[8], middle[8], small[8];
          const uint32_t from = tmem_base + lane_base + buf * 3 * BN + c0;
          load_columns8(from, big);
          load_columns8(from + BN, middle);
          load_columns8(from + 2 * BN, small);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[c0 + j] += __uint_as_float(big[j]) + (__uint_as_float(middle[j]) + __uint_as_float(small[j]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      if (!alive) break;
      const int r = quarter * 32 + lane, row = tile % tiles_m * kRows + r, col0 = tile / tiles_m * BN + half * COLS;
      if (row < m_total) {
        // Flags are set before the step that they belong to is handed over.  The splitting warps are at most STAGES steps
        // ahead of the products, less than a tile of kMinK columns, and so never in the flags that are read here.
        const volatile int* flags = apart[local & 1];
        const bool whole_row = flags[r] == local + 1;
        float* dst = c + (size_t)row * n_total + col0;
        const bool wide = n_total % 4 == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
#pragma unroll
        for (int j = 0; j < COLS; j += 4) {
          if (col0 + j >= n_total) break;
#pragma unroll
          for (int x = j; x < j + 4; ++x) {
            const int col = min(col0 + x, n_total - 1);
            if (whole_row || flags[kRows + half * COLS + x] == local + 1)
              acc[x] = sum_of(a + (size_t)row * k_total, w + (size_t)col * k_total, k_total);
            if (bias) acc[x] += bias[col];
          }
          if (wide) {
            *reinterpret_cast<float4*>(dst + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
          } else {
#pragma unroll
            for (int x = j; x < j + 4; ++x)
              if (col0 + x < n_total) dst[x] = acc[x];
          }
        }
      }
      __syncwarp();
    }
  }
  // a wait ran out: give products that may still be in flight time to end before leaving
  if (!alive)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == kSplitWarps) tmem_free<COLUMNS>(tmem_base);
}

template <int BN>
cudaError_t launch_tiles(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int* err,
                         cudaStream_t stream) {
  constexpr int smem = kStages * stage_bytes(BN) + 1024;
  static const cudaError_t raised = cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (raised != cudaSuccess) return raised;
  const int sms = device_sms();
  const long long tiles = (long long)((m + kRows - 1) / kRows) * ((n + BN - 1) / BN);
  return launch(gemm_f32_tc_kernel<BN>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(kThreads), smem, stream, a, w, bias, c,
                m, n, k, err);
}

}  // namespace cie

using namespace cie;

// 1 if the operands can go to cie_gemm_f32_tc: rows of whole, aligned 16-byte pieces, long enough.
extern "C" int cie_gemm_f32_tc_takes(const void* a, const void* w, int k) {
  return k >= kMinK && k % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

extern "C" int cie_gemm_f32_tc(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int columns,
                               int* err, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (!cie_gemm_f32_tc_takes(a, w, k)) CIE_FAIL("gemm_f32_tc: K = %d (a multiple of 4 from %d on, operands on 16 bytes)", k, kMinK);
  if ((long long)((m + kRows - 1) / kRows) * ((n + 31) / 32) > 0x3fffffff) CIE_FAIL("gemm_f32_tc: %d x %d results", m, n);
  // narrow tiles while they do not make a second round: 64 x 2,048 results of 2,048 32 us against 37 with wide ones, 300 x
  // 2,048 (192 narrow tiles, 96 wide ones) 67 against 48
  const long long narrow = (long long)((m + kRows - 1) / kRows) * ((n + 31) / 32);
  if (columns != 32 && columns != 64) columns = narrow <= device_sms() ? 32 : 64;
  const cudaError_t status = columns == 32 ? launch_tiles<32>(a, w, bias, c, m, n, k, err, (cudaStream_t)stream)
                                           : launch_tiles<64>(a, w, bias, c, m, n, k, err, (cudaStream_t)stream);
  if (status != cudaSuccess) CIE_FAIL("gemm_f32_tc: launch failed: %s", cudaGetErrorString(status));
  return 0;
}
