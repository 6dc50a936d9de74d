// Gated linear attention: linear attention whose state decays by a factor of its own per key channel and token,
//
//     S_t = diag(alpha_t) S_(t-1) + k_t v_t^T          (S: [dim][vdim], float32, one per request and head)
//     o_t = S_t^T q_t,       alpha_t = sigmoid(z_t + bias)^(1 / tau)   (one number per head and key channel)
//
// over a ragged batch: every request brings one or more new tokens and continues from the state its slot holds.
// q, k and v arrive as columns of one float32 row per token (the projections' float32 results, never rounded
// again), z as a float32 row of its own [heads * dim]; q is multiplied by `q_scale` here.  The logarithm of the
// decay is log(alpha) = -softplus(-(z + bias)) / tau, worked out in float32; everything of the recurrence is
// float32: on the CUDA cores, or products on the tensor cores that are as accurate (tf32x3.cuh).
//
// Two forms.  `gla_scan_kernel` walks a request's tokens one by one (single tokens of a decode step, and key
// sizes above 128).  Prompt portions run in chunks of 32 tokens (key and value sizes up to 128): with
// b_i = sum_(s<=i) log(alpha_s) counted from the chunk's first token and S_0 the state before the chunk,
//
//     o_i = (q_i * exp(b_i))^T S_0 + sum_(j<=i) A_ij v_j        A_ij = sum_d q_i[d] k_j[d] exp(b_i[d] - b_j[d])
//     S_n = diag(exp(b_n)) S_0 + sum_j (k_j * exp(b_n - b_j)) v_j^T
//
// in which no exponent is above zero: (1) per (chunk, head) the sums b_i, the scaled rows of q and k, A and exp(b_n);
// (2) per (request, head, block of value columns) a walk over the request's chunks that works out the
// outputs and carries the state (state_walk.cuh).  Chunks come as a work list made on the host from the step's
// portion lengths (first token row and token count of each chunk; where every request's chunks start).  2,048 tokens of 16
// heads of 128 x 128: 39 and 92 us, 131 together; states of all chunks through memory (sums per chunk, a walk over them, outputs
// per chunk, on the CUDA cores) took 183.  Eight portions of 287 tokens, 32 heads: 223 against 457.
//
// A request's result depends on its own tokens and state only: the batch and the slot change nothing, the cut
// of a prompt into portions only the order of additions.
#include "state_walk.cuh"
#include "common.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

constexpr int kScanWarps = 8;        // warps of a block; in the scan warp w owns state rows w, w + 8, ...
constexpr int kScanColumns = 32;     // value columns of a scan block: one per lane
constexpr int kScanRows = 32;        // state rows a warp keeps in registers (dim <= 8 * 32)

// log(sigmoid(y)) / tau = -softplus(-y) / tau, without overflow for any y
__device__ __forceinline__ float log_decay(float y, float inv_tau) {
  return -(fmaxf(-y, 0.f) + log1pf(expf(-fabsf(y)))) * inv_tau;
}

struct GlaRows {
  const float* proj;     // [tokens][proj_stride]
  int proj_stride;
  int q_off, k_off, v_off;   // first column of q, k and v (heads side by side inside each)
  const float* z;        // [tokens][z_stride]: decay logits, heads x dim
  int z_stride;
  const float* z_bias;   // [heads * dim]
  float inv_tau;
  float q_scale;
};

// grid: (requests, heads, ceil(vdim / 32)).
__global__ void __launch_bounds__(kScanWarps * 32)
gla_scan_kernel(GlaRows in, float* __restrict__ out, int out_stride, float* __restrict__ state,
                const int* __restrict__ query_start, const int* __restrict__ slots,
                const int* __restrict__ request_active, int heads, int dim, int vdim, int max_slots, int* err) {
  __shared__ float q_s[2][kScanWarps * kScanRows], k_s[2][kScanWarps * kScanRows], a_s[2][kScanWarps * kScanRows];
  __shared__ float part_s[2][kScanWarps][kScanColumns];
  pdl_wait();
  pdl_trigger();
  const int request = blockIdx.x, head = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int column = blockIdx.z * kScanColumns + lane;
  const bool live = column < vdim;
  const int slot = slots[request];
  if (slot < 0 || slot >= max_slots) {
    if (threadIdx.x == 0) atomicOr(err, kErrBadRequest);
    return;
  }
  const int begin = query_start[request], end = query_start[request + 1];
  float* s_base = state + (((size_t)slot * heads + head) * dim) * vdim;
  float s[kScanRows];
#pragma unroll
  for (int r = 0; r < kScanRows; ++r) {
    const int i = warp + kScanWarps * r;
    s[r] = (i < dim && live) ? s_base[(size_t)i * vdim + column] : 0.f;
  }
  for (int t = begin; t < end; ++t) {
    const int buf = (t - begin) & 1;
    const float* row = in.proj + (size_t)t * in.proj_stride;
    const float* zr = in.z + (size_t)t * in.z_stride + head * dim;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
      q_s[buf][i] = row[in.q_off + head * dim + i] * in.q_scale;
      k_s[buf][i] = row[in.k_off + head * dim + i];
      a_s[buf][i] = expf(log_decay(zr[i] + in.z_bias[head * dim + i], in.inv_tau));
    }
    const float v = live ? row[in.v_off + head * vdim + column] : 0.f;
    __syncthreads();
    float o = 0.f;
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
      const int i = warp + kScanWarps * r;
      if (i < dim) {
        s[r] = fmaf(a_s[buf][i], s[r], k_s[buf][i] * v);
        o = fmaf(s[r], q_s[buf][i], o);
      }
    }
    part_s[buf][warp][lane] = o;
    __syncthreads();
    if (warp == 0 && live) {
      float total = 0.f;
#pragma unroll
      for (int w = 0; w < kScanWarps; ++w) total += part_s[buf][w][lane];
      out[(size_t)t * out_stride + head * vdim + column] = total;
    }
    // the buffers of token t are read again only after the first barrier of token t + 2
  }
  if (request_active[request] && live) {
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
      const int i = warp + kScanWarps * r;
      if (i < dim) s_base[(size_t)i * vdim + column] = s[r];
    }
  }
}

// ---------------------------------------------------------------- prompt portions in chunks
constexpr int kChunk = kChunkTokens;
constexpr int kChunkDim = 128;                          // largest key and value size of the chunked kernels
constexpr int kScoreThreads = 256;

// (1) grid (chunks, heads): the cell of a chunk and head (state_walk.cuh).  A thread takes a channel and, with its
// neighbours of the channel, all tokens in runs that follow each other.
template <int P>
__global__ void __launch_bounds__(kScoreThreads, 3)
gla_chunk_kernel(GlaRows in, float* __restrict__ cells, const int* __restrict__ chunk_row,
                 const int* __restrict__ chunk_count, int heads, int dim) {
  constexpr int C = kChunk, G = kScoreThreads / P, TG = C / G;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;                 // [C][P]
  float* k_s = q_s + C * P;          // [C][P]
  float* b_s = k_s + C * P;          // [C][P]: the sums in units of log 2, so that every exponential of A is one exp2
  float* part_s = b_s + C * P;       // [G][P]
  __shared__ int unsafe_s;
  pdl_wait();
  pdl_trigger();
  const int chunk = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = chunk_row[chunk], n = chunk_count[chunk];
  float* cell = cells + ((size_t)chunk * heads + head) * walk_cell_floats(P, 0);
  const int d = tid % P, group = tid / P, t0 = group * TG;
  if (group < G) {
    const bool live = d < dim;
    const float* row = in.proj + (size_t)(row0 + t0) * in.proj_stride + head * dim + d;
    const float* zr = in.z + (size_t)(row0 + t0) * in.z_stride + head * dim + d;
    const float bias = live ? in.z_bias[head * dim + d] : 0.f;
    float b[TG], q[TG], k[TG];
#pragma unroll
    for (int i = 0; i < TG; ++i) {
      const bool here = live && t0 + i < n;
      b[i] = here ? zr[(size_t)i * in.z_stride] : 0.f;
      q[i] = here ? row[(size_t)i * in.proj_stride + in.q_off] * in.q_scale : 0.f;
      k[i] = here ? row[(size_t)i * in.proj_stride + in.k_off] : 0.f;
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < TG; ++i) {
      if (live && t0 + i < n) sum += log_decay(b[i] + bias, in.inv_tau);
      b[i] = sum;
    }
    part_s[group * P + d] = sum;
    if (tid == 0) unsafe_s = 0;
    __syncthreads();
    float before = 0.f, after = 0.f;
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const float x = part_s[j * P + d];
      if (j < group) before += x;
      if (j > group) after += x;
    }
    bool unsafe = false;
#pragma unroll
    for (int i = 0; i < TG; ++i) {
      const int t = t0 + i;
      const float at = before + b[i];
      q_s[t * P + d] = q[i];
      k_s[t * P + d] = k[i];
      b_s[t * P + d] = at * 1.4426950408889634f;
      // what the carried state is read with, and what the token leaves in it
      const float from = q[i] * expf(at), left = k[i] * expf((sum - b[i]) + after);
      unsafe |= tf32_unsafe(from) || tf32_unsafe(left);
      cell[t * walk_q_row(P) + d] = from;
      cell[walk_cell_k(P, 0) + t * walk_k_row(P) + d] = left;
    }
    if (group == 0) cell[walk_cell_decay(P, 0) + d] = expf(sum + after);
    if (unsafe) unsafe_s = 1;
  } else {
    __syncthreads();
  }
  __syncthreads();
  // A in tiles of 4 x 4 that a warp takes together, a lane the 16-byte pieces lane, lane + 32, ..  Below the diagonal
  // the exponential is exp(b_i - b_r) exp(b_r - b_j) with r the last token of the columns' four: both exponents are at
  // most zero, and a factor vanishes only where the product does; 8 exponentials for 16 products instead of 16.  On the
  // diagonal every pair has its own.
  float* a_out = cell + walk_cell_a(P, 0);
  const int blocks = (n + 3) / 4;
  bool unsafe = false;
  for (int p = warp; p < blocks * (blocks + 1) / 2; p += kScoreThreads / 32) {
    int bi = (int)((sqrtf(8.f * (float)p + 1.f) - 1.f) * 0.5f);
    while (bi * (bi + 1) / 2 > p) --bi;
    while ((bi + 1) * (bi + 2) / 2 <= p) ++bi;
    const int bj = p - bi * (bi + 1) / 2, i0 = 4 * bi, j0 = 4 * bj;
    float dot[16] = {};      // [i][j]
    for (int x = lane * 4; x < P; x += 128) {
      float q[4][4], k[4][4];
      if (bi != bj) {
        float last[4];
        *reinterpret_cast<float4*>(last) = *reinterpret_cast<const float4*>(b_s + (j0 + 3) * P + x);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float b[4];
          *reinterpret_cast<float4*>(q[r]) = *reinterpret_cast<const float4*>(q_s + (i0 + r) * P + x);
          *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(b_s + (i0 + r) * P + x);
#pragma unroll
          for (int y = 0; y < 4; ++y) q[r][y] *= exp2f(b[y] - last[y]);
          *reinterpret_cast<float4*>(k[r]) = *reinterpret_cast<const float4*>(k_s + (j0 + r) * P + x);
          if (r == 3) continue;
          *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(b_s + (j0 + r) * P + x);
#pragma unroll
          for (int y = 0; y < 4; ++y) k[r][y] *= exp2f(last[y] - b[y]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int y = 0; y < 4; ++y) dot[4 * i + j] = fmaf(q[i][y], k[j][y], dot[4 * i + j]);
      } else {
        float b[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          *reinterpret_cast<float4*>(q[r]) = *reinterpret_cast<const float4*>(q_s + (i0 + r) * P + x);
          *reinterpret_cast<float4*>(k[r]) = *reinterpret_cast<const float4*>(k_s + (i0 + r) * P + x);
          *reinterpret_cast<float4*>(b[r]) = *reinterpret_cast<const float4*>(b_s + (i0 + r) * P + x);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j <= i; ++j)
#pragma unroll
            for (int y = 0; y < 4; ++y)
              dot[4 * i + j] = fmaf(q[i][y] * k[j][y], i == j ? 1.f : exp2f(b[i][y] - b[j][y]), dot[4 * i + j]);
      }
    }
    // the lanes' sums: every step a lane gives half of its cells away
#pragma unroll
    for (int half = 8; half >= 1; half >>= 1) {
      const bool upper = lane & (2 * half);
#pragma unroll
      for (int e = 0; e < half; ++e) {
        const float mine = upper ? dot[e + half] : dot[e], other = upper ? dot[e] : dot[e + half];
        dot[e] = mine + __shfl_xor_sync(0xffffffffu, other, 2 * half);
      }
    }
    const float total = dot[0] + __shfl_xor_sync(0xffffffffu, dot[0], 1);
    const int i = i0 + (lane >> 3), j = j0 + (lane >> 1 & 3);      // the cell that the steps left here
    if (!(lane & 1)) {
      a_out[i * kWalkA + j] = j <= i ? total : 0.f;
      if (j <= i) unsafe |= tf32_unsafe(total);
    }
  }
  // zeros above the tiles of the diagonal, and in the rows past the last token
  for (int e = tid; e < C * C; e += kScoreThreads) {
    const int i = e / C, j = e % C;
    if (j >= (i & ~3) + 4 || i >= 4 * blocks) a_out[i * kWalkA + j] = 0.f;
  }
  if (unsafe) unsafe_s = 1;
  __syncthreads();
  if (tid == 0) *reinterpret_cast<float2*>(cell + walk_cell_decay(P, 0) + P) = make_float2((float)unsafe_s, __int_as_float(n));
}

}  // namespace cie

using namespace cie;

static int check_rows(const char* name, const GlaRows& in, int heads, int dim, int vdim) {
  if (heads < 1 || dim < 1 || vdim < 1) CIE_FAIL("%s: %d heads of key size %d and value size %d", name, heads, dim, vdim);
  if (!(in.inv_tau > 0.f)) CIE_FAIL("%s: the decay's temperature must be positive", name);
  if (!in.proj || !in.z || !in.z_bias) CIE_FAIL("%s: q/k/v rows, decay logits and their bias are all needed", name);
  return 0;
}

extern "C" int cie_gla_scan_max_dim() { return kScanWarps * kScanRows; }
extern "C" int cie_gla_chunk_tokens() { return kChunk; }
extern "C" int cie_gla_chunk_max_dim() { return kChunkDim; }

// proj: float32 [tokens][proj_stride] with q, k, v at columns q_off, k_off, v_off (heads side by side); z: float32
// [tokens][z_stride] decay logits (heads x dim) still without z_bias [heads * dim]; out: float32
// [tokens][out_stride], head h at column h * vdim; state: float32 [max_slots][heads][dim][vdim].
extern "C" int cie_gla_scan(const float* proj, int proj_stride, int q_off, int k_off, int v_off, const float* z,
                            int z_stride, const float* z_bias, float inv_tau, float q_scale, float* out,
                            int out_stride, float* state, const int* query_start, const int* slots,
                            const int* request_active, int requests, int heads, int dim, int vdim, int max_slots,
                            int* err, void* stream) {
  if (requests <= 0) return 0;
  const GlaRows in{proj, proj_stride, q_off, k_off, v_off, z, z_stride, z_bias, inv_tau, q_scale};
  if (check_rows("gla_scan", in, heads, dim, vdim)) return 1;
  if (dim > kScanWarps * kScanRows) CIE_FAIL("gla_scan: key size %d is above %d", dim, kScanWarps * kScanRows);
  dim3 grid(requests, heads, (vdim + kScanColumns - 1) / kScanColumns);
  CIE_LAUNCH("gla_scan", gla_scan_kernel, grid, dim3(kScanWarps * 32), 0, (cudaStream_t)stream, in, out, out_stride,
             state, query_start, slots, request_active, heads, dim, vdim, max_slots, err);
  return 0;
}

// Floats of scratch memory that the chunked form wants.
extern "C" long long cie_gla_chunk_floats(int chunks, int heads, int dim) {
  return (long long)chunks * heads * walk_cell_floats(walk_pad(dim), 0);
}

// The chunked form.  cells: float32 scratch of cie_gla_chunk_floats, on 16 bytes.
extern "C" int cie_gla_chunked(const float* proj, int proj_stride, int q_off, int k_off, int v_off, const float* z,
                               int z_stride, const float* z_bias, float inv_tau, float q_scale, float* out,
                               int out_stride, float* state, float* cells, const int* chunk_row,
                               const int* chunk_count, const int* request_chunk_start, const int* slots,
                               const int* request_active, int chunks, int requests, int heads, int dim, int vdim,
                               int max_slots, int* err, void* stream) {
  if (chunks <= 0 || requests <= 0) return 0;
  const GlaRows in{proj, proj_stride, q_off, k_off, v_off, z, z_stride, z_bias, inv_tau, q_scale};
  if (check_rows("gla_chunked", in, heads, dim, vdim)) return 1;
  if (dim > kChunkDim || vdim > kChunkDim)
    CIE_FAIL("gla_chunked: key / value sizes %d / %d are above %d", dim, vdim, kChunkDim);
  cudaStream_t s = (cudaStream_t)stream;
  const int P = walk_pad(dim), groups = kScoreThreads / P;
  const size_t smem = (size_t)(3 * kChunk + groups) * P * sizeof(float);
  auto go = [&](auto kernel) {
    const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return status != cudaSuccess ? status
                                 : launch(kernel, dim3(chunks, heads), dim3(kScoreThreads), smem, s, in, cells, chunk_row, chunk_count, heads, dim);
  };
  const cudaError_t status = P == 32 ? go(gla_chunk_kernel<32>) : P == 64 ? go(gla_chunk_kernel<64>)
                             : P == 96 ? go(gla_chunk_kernel<96>) : go(gla_chunk_kernel<128>);
  if (status != cudaSuccess) CIE_FAIL("gla_chunk: launch failed: %s", cudaGetErrorString(status));
  const WalkArgs walk{cells, proj + v_off, proj_stride, vdim, out, out_stride, state, (long long)heads * dim * vdim, chunk_row, chunk_count,
                      request_chunk_start, slots, request_active, heads, dim, vdim, max_slots, err};
  const cudaError_t walked = launch_state_walk<0>(walk, P, requests, s);
  if (walked != cudaSuccess) CIE_FAIL("gla_walk: launch failed: %s", cudaGetErrorString(walked));
  return 0;
}
