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
// The rows of A are split once, by a kernel of their own, and come as terms by TMA; the rows of W, each of which one tile of
// columns reads, are split on their way to shared memory.  What bounds it: shared memory, which the terms are written to (3 x 2
// bytes an element) and which the tensor core reads both operands from (1,340 of the 1,870 cycles of a step), and the splitting
// warps' instructions.  300 rows, 2,048 x 2,048: 37 us against 47 where every tile split its rows of A itself and 124 on the CUDA
// cores; 22,016 x 2,048: 223, 282 and 692; 2,048 x 11,008: 168, 226 and 656; one row, the same three: 31, 33 and 46; 97, 116 and 77;
// 143, 157 and 240 (17 rows as one).  512 x 512 of one row: 12.0, 11.3 and 12.8.  Eight splitting warps, a step ahead: 16 warps, whose instructions get in each other's way, 233 (220 with eight),
// two steps ahead 244 and four 255.
#include "blackwell.cuh"
#include "common.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

using namespace bw;

constexpr int kRows = 128, kStep = 64, kInterval = 128, kStages = 3;
constexpr int kSplitWarps = 8, kAddWarps = 8, kThreads = (kSplitWarps + 1 + kAddWarps + 1) * 32;      // split, multiply, add up, copy
constexpr int kPassRows = 2 * kSplitWarps;      // rows of W that the splitting warps take at one time
constexpr int kMinK = 512;          // four intervals and more (see the flags below)
constexpr int kPart = 4096;         // columns of a row of A that a block splits
__host__ __device__ constexpr int padded_k(int k) { return (k + 7) & ~7; }
__host__ __device__ constexpr int parts_of(int k) { return (k + kPart - 1) / kPart; }

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

// terms: [3][m][padded_k(k)]: hi, mid and lo of every element, zeros behind the last; apart: [m][parts_of(k)]: 1 where a value of
// the part is not finite or rounds to infinity.  grid (m, parts_of(k))
__global__ void __launch_bounds__(256)
f32_terms_kernel(const float* __restrict__ a, __nv_bfloat16* __restrict__ terms, int* __restrict__ apart, int m, int k) {
  pdl_wait();
  pdl_trigger();
  const int row = blockIdx.x, kp = padded_k(k), k0 = blockIdx.y * kPart + threadIdx.x * 4;
  const float* from = a + (size_t)row * k;
  __nv_bfloat16* to = terms + (size_t)row * kp;
  float4 x[kPart / 1024];
#pragma unroll
  for (int i = 0; i < kPart / 1024; ++i)
    x[i] = k0 + 1024 * i < k ? *reinterpret_cast<const float4*>(from + k0 + 1024 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
  bool odd = false;
#pragma unroll
  for (int i = 0; i < kPart / 1024; ++i) {
    const int at = k0 + 1024 * i;
    if (at >= kp) break;
    const size_t term = (size_t)m * kp;
    uint32_t lo = take_term(x[i].x, x[i].y), hi = take_term(x[i].z, x[i].w);
    *reinterpret_cast<uint2*>(to + at) = make_uint2(lo, hi);
    lo = take_term(x[i].x, x[i].y);
    hi = take_term(x[i].z, x[i].w);
    *reinterpret_cast<uint2*>(to + term + at) = make_uint2(lo, hi);
    *reinterpret_cast<uint2*>(to + 2 * term + at) = make_uint2(pair_of(x[i].x, x[i].y), pair_of(x[i].z, x[i].w));
    const float rest = (x[i].x + x[i].y) + (x[i].z + x[i].w);      // NaN where a term is not finite
    odd |= !(rest == rest);
  }
  odd = __syncthreads_or(odd);
  if (threadIdx.x == 0) apart[row * gridDim.y + blockIdx.y] = odd;
}

// Persistent: a CTA an SM, which walks over tiles of 128 rows of A and BN of W, row blocks of A fastest so that the CTAs that
// run at one time share rows of W in L2.  Warps 0..7 split: a step of kStep columns of W comes from memory into registers
// a step ahead (the first before the kernels before have ended) and goes to shared memory as [A hi, mid, lo][W hi, mid, lo],
// 128-byte-swizzled; A's terms come there by TMA, asked for by warp 17 (three copies take the time of a step's splitting):
// map_a: rows of all three terms one after the other, a_rows a copy.  Warp 8 multiplies: the W terms lie one after the other, so
// three instructions make the six products (hi by all three, mid by two, lo by one), each into the accumulator of its
// magnitude.  Warps 9..16 add up and write, half of the columns each four.
template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, int a_rows, const int* __restrict__ a_apart,
                   const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                   float* __restrict__ c, int m_total, int n_total, int k_total, int* err) {
  constexpr int STAGES = kStages, PASSES = BN / kPassRows, TERM_A = kRows * kStep * 2, TERM_W = BN * kStep * 2;
  constexpr int COLUMNS = 6 * BN <= 256 ? 256 : 512;
  static_assert(6 * BN <= 512 && (3 * BN) % 16 == 0, "two sets of three accumulators in tensor memory");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ int apart[2][BN];      // rows of W that are summed in float32: (number of the tile) + 1, every second tile's

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_m = (m_total + kRows - 1) / kRows, tiles_n = (n_total + BN - 1) / BN, total = tiles_m * tiles_n;
  const int steps = (k_total + kStep - 1) / kStep, intervals = (steps + kInterval / kStep - 1) / (kInterval / kStep);
  // a splitting thread's place: rows sub, sub + kPassRows, .. of W; four columns
  const int sub = warp * 2 + (lane >> 4), kq = (lane & 15) * 4;
  struct Pieces {
    float4 x[PASSES];
    uint32_t inside;      // which of the rows are the matrix's
  };
  Pieces next;
  int ahead_tile = blockIdx.x, ahead_step = 0;
  const float* row_at[PASSES];      // where the next pieces lie
  uint32_t inside = 0;
  auto enter = [&]() {
    inside = 0;
    if (ahead_tile >= total) return;
    const int col = ahead_tile / tiles_m * BN + sub;
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const bool in = col + kPassRows * i < n_total;
      inside |= (uint32_t)in << i;
      row_at[i] = w + (in ? (size_t)(col + kPassRows * i) * k_total : 0) + kq;
    }
  };
  auto fetch = [&](Pieces& to) {
    to.inside = inside;
    const bool in_k = ahead_step * kStep + kq < k_total;
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      to.x[i] = (inside >> i & 1) && in_k ? __ldg(reinterpret_cast<const float4*>(row_at[i])) : make_float4(0.f, 0.f, 0.f, 0.f);
      row_at[i] += kStep;
    }
    if (++ahead_step == steps) {
      ahead_step = 0;
      ahead_tile += gridDim.x;
      enter();
    }
  };
  if (warp < kSplitWarps) {
    enter();
    fetch(next);
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], kSplitWarps + 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], kAddWarps); }
    mbar_init_fence();
  }
  for (int e = tid; e < 2 * BN; e += kThreads) (&apart[0][0])[e] = 0;
  pdl_wait();
  pdl_trigger();
  if (warp == kSplitWarps) tmem_alloc<COLUMNS>(&tmem_base_s);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;
  bool alive = true;

  if (warp < kSplitWarps) {
    const uint32_t place = (uint32_t)(3 * TERM_A + sub * 128 + ((((lane & 15) >> 1) ^ (sub & 7)) << 4) + (lane & 1) * 8);
    int s = 0, local = 0;
    uint32_t phase = 1;
    for (int tile = blockIdx.x; tile < total && alive; tile += gridDim.x, ++local) {
      for (int step = 0; step < steps; ++step) {
        const Pieces now = next;
        fetch(next);
        if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[s], phase, err))) { alive = false; break; }
        unsigned char* stage = ring + (size_t)s * stage_bytes(BN);
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
          // rows behind the matrix are left as they are: what comes of them is not written
          if (!(now.inside >> i & 1)) continue;
          float4 x = now.x[i];
          unsigned char* dst = stage + place + i * kPassRows * 128;
          uint32_t lo = take_term(x.x, x.y), hi = take_term(x.z, x.w);
          *reinterpret_cast<uint2*>(dst) = make_uint2(lo, hi);
          lo = take_term(x.x, x.y);
          hi = take_term(x.z, x.w);
          *reinterpret_cast<uint2*>(dst + TERM_W) = make_uint2(lo, hi);
          *reinterpret_cast<uint2*>(dst + 2 * TERM_W) = make_uint2(pair_of(x.x, x.y), pair_of(x.z, x.w));
          const float rest = (x.x + x.y) + (x.z + x.w);      // NaN where a term is not finite
          if (!(rest == rest)) apart[local & 1][i * kPassRows + sub] = local + 1;
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[s]);
        if (++s == STAGES) {
          s = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == kSplitWarps + 1 + kAddWarps) {
    if (lane == 0) {      // the terms of A
      int s = 0;
      uint32_t phase = 1;
      for (int tile = blockIdx.x; tile < total && alive; tile += gridDim.x) {
        const int row0 = tile % tiles_m * kRows;
        for (int step = 0; step < steps; ++step) {
          if (!mbar_wait(&empty_bar[s], phase, err)) { alive = false; break; }
          mbar_expect_tx(&full_bar[s], 3 * a_rows * kStep * 2);
#pragma unroll
          for (int term = 0; term < 3; ++term)
            tma_load_2d(ring + (size_t)s * stage_bytes(BN) + term * TERM_A, &map_a, &full_bar[s], step * kStep, term * m_total + row0);
          if (++s == STAGES) {
            s = 0;
            phase ^= 1;
          }
        }
      }
    }
    __syncwarp();
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
        bool whole_row = false;
        for (int p = 0; p < parts_of(k_total); ++p) whole_row |= a_apart[row * parts_of(k_total) + p] != 0;
        float* dst = c + (size_t)row * n_total + col0;
        const bool wide = n_total % 4 == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
#pragma unroll
        for (int j = 0; j < COLS; j += 4) {
          if (col0 + j >= n_total) break;
#pragma unroll
          for (int x = j; x < j + 4; ++x) {
            const int col = min(col0 + x, n_total - 1);
            if (whole_row || flags[half * COLS + x] == local + 1)
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
cudaError_t launch_tiles(const CUtensorMap& map_a, int a_rows, const int* apart, const float* a, const float* w, const float* bias,
                         float* c, int m, int n, int k, int* err, cudaStream_t stream) {
  constexpr int smem = kStages * stage_bytes(BN) + 1024;
  static const cudaError_t raised = cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (raised != cudaSuccess) return raised;
  const int sms = device_sms();
  const long long tiles = (long long)((m + kRows - 1) / kRows) * ((n + BN - 1) / BN);
  return launch(gemm_f32_tc_kernel<BN>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(kThreads), smem, stream, map_a, a_rows,
                apart, a, w, bias, c, m, n, k, err);
}

}  // namespace cie

using namespace cie;

// 1 if the operands can go to cie_gemm_f32_tc: rows of whole, aligned 16-byte pieces, long enough.
extern "C" int cie_gemm_f32_tc_takes(const void* a, const void* w, int k) {
  return k >= kMinK && k % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

// Floats of scratch memory for the terms of m rows.
extern "C" long long cie_gemm_f32_tc_floats(int m, int k) {
  return ((long long)m * 3 * padded_k(k) / 2 + 3) / 4 * 4 + (long long)m * parts_of(k);
}

// scratch: cie_gemm_f32_tc_floats(m, k) floats, on 16 bytes.
extern "C" int cie_gemm_f32_tc(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int columns,
                               float* scratch, int* err, void* stream) {
  if (m <= 0 || n <= 0) return 0;
  if (!cie_gemm_f32_tc_takes(a, w, k)) CIE_FAIL("gemm_f32_tc: K = %d (a multiple of 4 from %d on, operands on 16 bytes)", k, kMinK);
  if ((long long)((m + kRows - 1) / kRows) * ((n + 31) / 32) > 0x3fffffff || parts_of(k) > 65535)
    CIE_FAIL("gemm_f32_tc: %d x %d results of %d", m, n, k);
  __nv_bfloat16* terms = reinterpret_cast<__nv_bfloat16*>(scratch);
  int* apart = reinterpret_cast<int*>(scratch + ((long long)m * 3 * padded_k(k) / 2 + 3) / 4 * 4);
  const int a_rows = m < kRows ? (m + 7) & ~7 : kRows;      // few rows: no copy of what lies behind them
  CUtensorMap map_a;
  if (!tensor_map_bf16(terms, 3ll * m, padded_k(k), a_rows, &map_a)) CIE_FAIL("gemm_f32_tc: cuTensorMapEncodeTiled failed");
  CIE_LAUNCH("f32_terms", f32_terms_kernel, dim3(m, parts_of(k)), dim3(256), 0, (cudaStream_t)stream, a, terms, apart, m, k);
  // narrow tiles while they do not make a second round: 64 x 2,048 results of 2,048 31.5 us against 35 with wide ones, 300 x
  // 2,048 (192 narrow tiles, 96 wide ones) 59 against 37
  const long long narrow = (long long)((m + kRows - 1) / kRows) * ((n + 31) / 32);
  if (columns != 32 && columns != 64) columns = narrow <= device_sms() ? 32 : 64;
  const cudaError_t status =
      columns == 32 ? launch_tiles<32>(map_a, a_rows, apart, a, w, bias, c, m, n, k, err, (cudaStream_t)stream)
                    : launch_tiles<64>(map_a, a_rows, apart, a, w, bias, c, m, n, k, err, (cudaStream_t)stream);
  if (status != cudaSuccess) CIE_FAIL("gemm_f32_tc: launch failed: %s", cudaGetErrorString(status));
  return 0;
}
