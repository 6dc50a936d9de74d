// Generalized delta rule: per request and head a float32 state matrix S [dim keys][dim values] runs
// through the request's tokens,
//
//     u_t = k_t / sqrt(sum(k_t^2) + 1e-6)
//     S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T        (both first terms read S_(t-1))
//     o_t = S_t^T r_t
//
// with a decay w_t = exp(-exp(-1/2) * sigmoid(d_t + w0)) and a removal rate a_t = sigmoid(e_t + a0) per
// head and key channel.  r, k, v, e and d arrive as float32 projections of the token; everything from
// there on is float32.  A value column of S never meets another one, so eight lanes share a column
// (each an eighth of its rows, kept in registers) and join their sums by shuffles: what bounds the
// recurrence is the chain of dependent steps of one token, and more lanes a column shorten it.
//
// A second kernel divides every head of o by its own root mean square, multiplies by a gain vector and
// by sigmoid(gate), and rounds once.
//
// A request's result is worked out from its own tokens and state alone, whatever the batch and the slot.  The scan and the
// stream make the same additions in the same order.  The chunks group them (a chunk begins with its portion), and a step is
// run in chunks or not by what all of its requests together cost: so the cut of a prompt into portions and the requests
// beside it may change the order of a request's additions, as they may in other float32 sums of this framework, and with it
// the last bits; the difference stays within 1e-5 of the largest value.
#include "common.cuh"
#include "head_gate.cuh"
#include "state_walk.cuh"

CIE_DEFINE_LAST_ERROR()

namespace cie {

constexpr int kDeltaLanes = 8;         // lanes that share a value column
constexpr int kDeltaMaxDim = 256;       // largest head of the scan kernel
constexpr int kDeltaBlockColumns = 128;  // value columns of a block (heads above that take several blocks)
constexpr int kDeltaStreamMaxDim = 128; // largest head of the stream kernel (a column's rows are one thread's registers)

__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }

// out[t, i] = tanh(x[t * stride + i]) in the compute dtype, i < width
template <typename T>
__global__ void tanh_rows_kernel(const float* __restrict__ x, int stride, T* __restrict__ out, int width, long long total) {
  pdl_wait();
  pdl_trigger();
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  const long long t = e / width;
  const int i = (int)(e % width);
  out[e] = from_float<T>(tanhf(x[t * stride + i]));
}

// grid (requests, heads, blocks of kDeltaBlockColumns value columns); kDeltaLanes threads a column, rounded up
// to whole warps.  Every block stages all rows of k, r and the rates; it keeps only its own columns of S.
// proj: float32 rows [r | k | v | ... ] with heads side by side inside each part; `r_off`, `k_off`, `v_off`,
// `a_off` are the first columns of r, k, v and the removal projection; `decay` is its own tensor
// [T, heads * dim] (the decay projection, before its bias).  R = rows of a lane.
template <int R>
__global__ void __launch_bounds__(kDeltaLanes * kDeltaBlockColumns)
delta_scan_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                  const float* __restrict__ decay, int decay_stride, const float* __restrict__ decay_bias,
                  const float* __restrict__ removal_bias, float* __restrict__ out, int out_stride,
                  float* __restrict__ state, const int* __restrict__ query_start, const int* __restrict__ slots,
                  const int* __restrict__ request_active, int heads, int dim, int max_slots, int* err) {
  constexpr int kPad = kDeltaLanes * R;          // rows as the lanes see them (dim rounded up)
  __shared__ __align__(16) float w_s[2][kPad], au_s[2][kPad], u_s[2][kPad], k_s[2][kPad], r_s[2][kPad];
  pdl_wait();
  pdl_trigger();
  const int request = blockIdx.x, head = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31;
  const int column = blockIdx.z * kDeltaBlockColumns + tid / kDeltaLanes, part = tid % kDeltaLanes;
  const bool live = column < dim;
  const int slot = slots[request];
  if (slot < 0 || slot >= max_slots) {
    if (tid == 0) atomicOr(err, kErrBadRequest);
    return;
  }
  const int begin = query_start[request], end = query_start[request + 1];
  float* s_base = state + ((size_t)slot * heads + head) * dim * dim;
  float s[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = part * R + i;
    s[i] = (live && row < dim) ? s_base[(size_t)row * dim + column] : 0.f;
  }
  for (int i = tid; i < kPad; i += blockDim.x) {
#pragma unroll
    for (int b = 0; b < 2; ++b) w_s[b][i] = au_s[b][i] = u_s[b][i] = k_s[b][i] = r_s[b][i] = 0.f;
  }
  const int base = head * dim;
  const float w0 = tid < dim ? decay_bias[base + tid] : 0.f;
  const float a0 = tid < dim ? removal_bias[base + tid] : 0.f;
  const float decay_rate = -0.6065306597126334f;       // -exp(-1/2)
  const bool stager = tid < ((dim + 31) / 32) * 32;   // whole warps whose threads own an element i = tid

  // what token t needs from memory is asked for while token t - 1 is computed
  float kx = 0.f, rx = 0.f, ax = 0.f, dx = 0.f, vx = 0.f, ksq = 0.f;
  auto fetch = [&](int t) {
    const float* row = proj + (size_t)t * proj_stride;
    if (stager) {
      ksq = 0.f;
      for (int i = lane; i < dim; i += 32) {
        const float x = row[k_off + base + i];
        ksq = fmaf(x, x, ksq);
      }
      if (tid < dim) {
        kx = row[k_off + base + tid];
        rx = row[r_off + base + tid];
        ax = row[a_off + base + tid];
        dx = decay[(size_t)t * decay_stride + base + tid];
      }
    }
    if (live) vx = row[v_off + base + column];
  };
  if (begin < end) fetch(begin);
  for (int t = begin; t < end; ++t) {
    const int buf = (t - begin) & 1;
    if (stager) {
      const float total = warp_sum(ksq);
      if (tid < dim) {
        const float unit = kx * rsqrtf(total + 1e-6f);
        w_s[buf][tid] = expf(decay_rate * sigmoid_f(dx + w0));
        au_s[buf][tid] = sigmoid_f(ax + a0) * unit;
        u_s[buf][tid] = unit;
        k_s[buf][tid] = kx;
        r_s[buf][tid] = rx;
      }
    }
    const float v = vx;
    __syncthreads();
    if (t + 1 < end) fetch(t + 1);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) dot = fmaf(u_s[buf][part * R + i], s[i], dot);
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    dot += __shfl_xor_sync(0xffffffffu, dot, 4);
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = part * R + i;
      s[i] = fmaf(w_s[buf][row], s[i], fmaf(k_s[buf][row], v, -au_s[buf][row] * dot));
      o = fmaf(r_s[buf][row], s[i], o);
    }
    o += __shfl_xor_sync(0xffffffffu, o, 1);
    o += __shfl_xor_sync(0xffffffffu, o, 2);
    o += __shfl_xor_sync(0xffffffffu, o, 4);
    if (live && part == 0) out[(size_t)t * out_stride + base + column] = o;
    // the buffers of token t are written again for token t + 2, after the barrier of token t + 1
  }
  if (request_active[request] && live) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int row = part * R + i;
      if (row < dim) s_base[(size_t)row * dim + column] = s[i];
    }
  }
}

// ---------------------------------------------------------------- prompt portions: prepare, then stream
// For portions that the chunks further down do not serve (a few tokens each, or so many requests that a walk of each fills
// the device).  The scan above waits, token after token, for its own loads and for the
// exponentials of the rates.  Two kernels instead: `delta_prepare` computes, for all tokens at once,
// what the recurrence reads (w, a * u, u, k, r, v per head, float32, each padded with zeros to the rows
// the lanes keep) and `delta_stream` walks a request's tokens reading those rows through a ring of
// cp.async stages, several tokens ahead.  The arithmetic is that of the scan; the sums over a column's
// rows are added in another order (four chains a thread instead of a chain a lane).
constexpr int kDeltaStages = 3;      // stages of the ring
constexpr int kDeltaChunk = 4;       // tokens of a stage: the block meets once a stage, not once a token
constexpr int kDeltaFields = 6;      // w, a * u, u, k, r, v

// grid (tokens, heads), one warp or more; `pad` = rows as the stream kernel's lanes see them.
__global__ void __launch_bounds__(128)
delta_prepare_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                     const float* __restrict__ decay, int decay_stride, const float* __restrict__ decay_bias,
                     const float* __restrict__ removal_bias, float* __restrict__ packed, int tokens, int heads, int dim,
                     int pad) {
  __shared__ float scratch[33];
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, head = blockIdx.y, base = head * dim;
  const float* row = proj + (size_t)t * proj_stride;
  float sq = 0.f;
  for (int i = threadIdx.x; i < dim; i += blockDim.x) {     // the order of the scan: lane l adds l, l + 32, ...
    const float x = row[k_off + base + i];
    sq = fmaf(x, x, sq);
  }
  // the scan adds a warp's 32 partial sums; here a block of one warp does the same
  const float total = block_sum(sq, scratch);
  const float inv = rsqrtf(total + 1e-6f);
  float* dst = packed + ((size_t)head * tokens + t) * kDeltaFields * pad;     // head-major: a head's tokens follow each other
  for (int i = threadIdx.x; i < pad; i += blockDim.x) {
    float w = 0.f, au = 0.f, u = 0.f, k = 0.f, r = 0.f, v = 0.f;
    if (i < dim) {
      k = row[k_off + base + i];
      r = row[r_off + base + i];
      v = row[v_off + base + i];
      u = k * inv;
      au = sigmoid_f(row[a_off + base + i] + removal_bias[base + i]) * u;
      w = expf(-0.6065306597126334f * sigmoid_f(decay[(size_t)t * decay_stride + base + i] + decay_bias[base + i]));
    }
    dst[i] = w;
    dst[pad + i] = au;
    dst[2 * pad + i] = u;
    dst[3 * pad + i] = k;
    dst[4 * pad + i] = r;
    dst[5 * pad + i] = v;
  }
}

__device__ __forceinline__ void delta_cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}

// One thread a value column with ALL its rows in registers: every read of a token's row is then the
// same address for the whole warp (one shared-memory wavefront a load, where lanes that share a column
// read eight different places), and no sum crosses lanes.  P = rows as padded (32, 64 or 128).
template <int P>
__global__ void __launch_bounds__(kDeltaStreamMaxDim)
delta_stream_kernel(const float* __restrict__ packed, float* __restrict__ out, int out_stride, float* __restrict__ state,
                    const int* __restrict__ query_start, const int* __restrict__ slots,
                    const int* __restrict__ request_active, int tokens, int heads, int dim, int max_slots, int* err) {
  constexpr int kRow = kDeltaFields * P;             // floats of one token and head
  __shared__ __align__(16) float ring[kDeltaStages][kDeltaChunk * kRow];
  pdl_wait();
  pdl_trigger();
  const int request = blockIdx.x, head = blockIdx.y;
  const int tid = threadIdx.x;
  const int column = tid;
  const bool live = column < dim;
  const int slot = slots[request];
  if (slot < 0 || slot >= max_slots) {
    if (tid == 0) atomicOr(err, kErrBadRequest);
    return;
  }
  const int begin = query_start[request], end = query_start[request + 1];
  float* s_base = state + ((size_t)slot * heads + head) * dim * dim;
  float s[P];
#pragma unroll
  for (int i = 0; i < P; ++i) s[i] = (live && i < dim) ? s_base[(size_t)i * dim + column] : 0.f;
  const float* rows = packed + (size_t)head * tokens * kRow;
  auto issue = [&](int chunk) {
    const int first = begin + chunk * kDeltaChunk;
    if (first < end) {
      const int count = min(kDeltaChunk, end - first) * (kRow / 4);
      const float* src = rows + (size_t)first * kRow;
      float* dst = ring[chunk % kDeltaStages];
      for (int c = tid; c < count; c += blockDim.x) delta_cp_async16(dst + 4 * c, src + 4 * c);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  for (int i = 0; i < kDeltaStages - 1; ++i) issue(i);
  const int base = head * dim;
  for (int t = begin; t < end; ++t) {
    const int chunk = (t - begin) / kDeltaChunk, place = (t - begin) % kDeltaChunk;
    if (place == 0) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kDeltaStages - 2));
      __syncthreads();          // the chunk has landed; everybody is done with the chunk before, whose stage is filled next
      issue(chunk + kDeltaStages - 1);
    }
    const float* stage = ring[chunk % kDeltaStages] + place * kRow;
    const float4* w4 = reinterpret_cast<const float4*>(stage);
    const float4* au4 = reinterpret_cast<const float4*>(stage + P);
    const float4* u4 = reinterpret_cast<const float4*>(stage + 2 * P);
    const float4* k4 = reinterpret_cast<const float4*>(stage + 3 * P);
    const float4* r4 = reinterpret_cast<const float4*>(stage + 4 * P);
    const float v = stage[5 * P + (live ? column : 0)];
    float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;      // four chains, joined as (d0 + d1) + (d2 + d3)
#pragma unroll
    for (int i = 0; i < P / 4; ++i) {
      const float4 u = u4[i];
      d0 = fmaf(u.x, s[4 * i], d0);
      d1 = fmaf(u.y, s[4 * i + 1], d1);
      d2 = fmaf(u.z, s[4 * i + 2], d2);
      d3 = fmaf(u.w, s[4 * i + 3], d3);
    }
    const float dot = (d0 + d1) + (d2 + d3);
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int i = 0; i < P / 4; ++i) {
      const float4 w = w4[i], au = au4[i], k = k4[i], r = r4[i];
      s[4 * i] = fmaf(w.x, s[4 * i], fmaf(k.x, v, -au.x * dot));
      s[4 * i + 1] = fmaf(w.y, s[4 * i + 1], fmaf(k.y, v, -au.y * dot));
      s[4 * i + 2] = fmaf(w.z, s[4 * i + 2], fmaf(k.z, v, -au.z * dot));
      s[4 * i + 3] = fmaf(w.w, s[4 * i + 3], fmaf(k.w, v, -au.w * dot));
      o0 = fmaf(r.x, s[4 * i], o0);
      o1 = fmaf(r.y, s[4 * i + 1], o1);
      o2 = fmaf(r.z, s[4 * i + 2], o2);
      o3 = fmaf(r.w, s[4 * i + 3], o3);
    }
    if (live) out[(size_t)t * out_stride + base + column] = (o0 + o1) + (o2 + o3);
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (request_active[request] && live) {
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (i < dim) s_base[(size_t)i * dim + column] = s[i];
  }
}

// ---------------------------------------------------------------- prompt portions, in chunks
// Over a chunk of tokens 1..C that starts from S_0 let b_t be the decays multiplied from the chunk's first token to t
// (b_0 = 1; a decay is at least exp(-exp(-1/2)) > 0.54, so 1 / b_t stays below 3e8 for C = 32).  What a token reads back
// before its write, y_t = u_t^T S_(t-1), obeys a unit lower triangular system
//
//     y_t + sum_(s<t) A_ts y_s = (u_t b_(t-1))^T S_0 + sum_(s<t) B_ts v_s
//     A_ts = (u_t b_(t-1)) . (a_s u_s / b_s)      B_ts = (u_t b_(t-1)) . (k_s / b_s)
//
// so Y = Y' + W S_0 with the same elimination on both right-hand sides, and with C_ts, D_ts (s <= t) the same products of
// r_t b_t, and U = -Y:
//
//     U   = -Y' - W S_0
//     O   = diag-scaled r S_0 + D V + C U
//     S_C = b_C S_0 + sum_s (b_C k_s / b_s) v_s + (b_C a_s u_s / b_s) u'_s            (u'_s: row s of U)
//
//   1. delta_chunk (per chunk and head): A, B, C, D, W, Y' and the scaled rows
//   2. the walk of state_walk.cuh (per request, head and block of value columns)
//
// Float32: 1 on the CUDA cores, 2 as accurately on the tensor cores.  A token's results read rows of tokens up to its own
// alone (no weight of zero times a later row).  Against the stream below, whose chain of one token is 450 instructions long and
// which a prompt of one request and 32 heads runs on 32 SMs: 2,048 tokens, 32 heads of 64: 207 us in chunks, 1,790 as a stream (16
// heads of 128: 356 and 3,945).  What bounds delta_chunk is the data that shared memory
// can return (128 bytes a cycle: a 16-byte load of a warp is four cycles), hence tiles of 4 x 4 and more a thread.  With what a
// chunk does to any state as one matrix, [S; O] <- [M; Q] S + [N; O'], its products on the CUDA cores, the two kernels took
// 246 us (heads of 128: 515; eight portions of 287 tokens, 32 heads of 128: 1,143, now 635).
constexpr int kDeltaChunkTokens = 32;
constexpr int kDeltaMat = 2 * kDeltaChunkTokens + 4;      // row of the matrices [A C; B D], transposed

template <int P>
constexpr int delta_chunk_smem() {
  return (6 * kDeltaChunkTokens * (P + 4) + 2 * kDeltaChunkTokens * kDeltaMat + P + kDeltaChunkTokens + 256) * (int)sizeof(float);
}

// grid (chunks, heads), 256 threads
template <int P>
__global__ void __launch_bounds__(256)
delta_chunk_kernel(const float* __restrict__ proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                   const float* __restrict__ decay, int decay_stride, const float* __restrict__ decay_bias,
                   const float* __restrict__ removal_bias, float* __restrict__ cells, const int* __restrict__ chunk_row,
                   const int* __restrict__ chunk_count, int heads, int dim) {
  constexpr int C = kDeltaChunkTokens, LD = P + 4, ML = kDeltaMat, G = 256 / P, TG = C / G;
  extern __shared__ __align__(16) float delta_smem[];
  float* ub = delta_smem;           // u_t b_(t-1), then W
  float* rb = ub + C * LD;          // r_t b_t
  float* ai = rb + C * LD;          // a_s u_s / b_s
  float* ki = ai + C * LD;          // k_s / b_s
  float* vs = ki + C * LD;
  float* ys = vs + C * LD;          // B V, then Y'
  float* mat = ys + C * LD;         // [column: 32 of ai, 32 of ki][row: 32 of ub, 32 of rb]
  float* bn = mat + 2 * C * ML;
  float* inv = bn + P;
  float* part = inv + C;            // [G][P]
  pdl_wait();
  pdl_trigger();
  const int chunk = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = chunk_row[chunk], n = chunk_count[chunk], base = head * dim;
  for (int t = warp; t < C; t += 8) {
    float sq = 0.f;
    if (t < n) {
      const float* row = proj + (size_t)(row0 + t) * proj_stride + k_off + base;
      for (int i = lane; i < dim; i += 32) sq = fmaf(row[i], row[i], sq);
    }
    sq = warp_sum(sq);
    if (lane == 0) inv[t] = rsqrtf(sq + 1e-6f);
  }
  const int d = tid % P, g = tid / P;      // a column, and TG tokens of it
  {
    const bool live = d < dim;
    const float w0 = live ? decay_bias[base + d] : 0.f, a0 = live ? removal_bias[base + d] : 0.f;
    float product[TG], kx[TG], rx[TG], ax[TG], vx[TG];
#pragma unroll
    for (int i = 0; i < TG; ++i) {
      const bool in = live && g * TG + i < n;
      const size_t t = (size_t)(row0 + g * TG + i);
      const float* row = proj + t * proj_stride + base + d;
      product[i] = in ? decay[t * decay_stride + base + d] : 0.f;
      kx[i] = in ? row[k_off] : 0.f;
      rx[i] = in ? row[r_off] : 0.f;
      ax[i] = in ? row[a_off] : 0.f;
      vx[i] = in ? row[v_off] : 0.f;
    }
    float run = 1.f;
#pragma unroll
    for (int i = 0; i < TG; ++i) {
      if (live && g * TG + i < n) run *= expf(-0.6065306597126334f * sigmoid_f(product[i] + w0));      // -exp(-1/2)
      product[i] = run;
    }
    part[g * P + d] = run;
    __syncthreads();
    float before = 1.f;
    for (int j = 0; j < g; ++j) before *= part[j * P + d];
#pragma unroll
    for (int i = 0; i < TG; ++i) {
      const int t = g * TG + i;
      const float b = before * product[i], below = i > 0 ? before * product[i > 0 ? i - 1 : 0] : before, over = 1.f / b;
      const float u = kx[i] * inv[t];
      ub[t * LD + d] = u * below;
      rb[t * LD + d] = rx[i] * b;
      ai[t * LD + d] = sigmoid_f(ax[i] + a0) * u * over;
      ki[t * LD + d] = kx[i] * over;
      vs[t * LD + d] = vx[i];
    }
    if (g == G - 1) bn[d] = before * run;
  }
  __syncthreads();
  {
    // A, B, C, D: a warp takes 16 rows and 32 columns, a thread every fourth and every eighth; entries above the diagonal
    // are zeros that nothing reads
    const int wm = warp & 3, wn = warp >> 2, columns = wm & 1 ? 4 : 2;
    const int t0 = (wm & 1) * 16 + (lane >> 3), s0 = lane & 7;
    const float* rows = (wm < 2 ? ub : rb) + t0 * LD;
    const float* cols = (wn ? ki : ai) + s0 * LD;
    float acc[4][4] = {};
    for (int x = 0; x < P; x += 4) {
      float4 av[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const float4*>(rows + 4 * i * LD + x);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j >= columns) break;
        const float4 wv = *reinterpret_cast<const float4*>(cols + 8 * j * LD + x);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][j] = fmaf(av[i].x, wv.x, acc[i][j]);
          acc[i][j] = fmaf(av[i].y, wv.y, acc[i][j]);
          acc[i][j] = fmaf(av[i].z, wv.z, acc[i][j]);
          acc[i][j] = fmaf(av[i].w, wv.w, acc[i][j]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = t0 + 4 * i, s = s0 + 8 * j;
        mat[(wn * C + s) * ML + (wm >> 1) * C + t] = (wm < 2 ? s < t : s <= t) ? acc[i][j] : 0.f;
      }
  }
  __syncthreads();
  {
    // B V, a thread a column of its TG tokens
    float bv[TG] = {};
    const float* mat_row = mat + C * ML + g * TG;
    for (int s = 0; s < g * TG; ++s) {
      const float xv = vs[s * LD + d];
#pragma unroll
      for (int i = 0; i < TG; i += 4) {
        const float4 m = *reinterpret_cast<const float4*>(mat_row + s * ML + i);
        bv[i] = fmaf(m.x, xv, bv[i]);
        bv[i + 1] = fmaf(m.y, xv, bv[i + 1]);
        bv[i + 2] = fmaf(m.z, xv, bv[i + 2]);
        bv[i + 3] = fmaf(m.w, xv, bv[i + 3]);
      }
    }
#pragma unroll
    for (int q = 0; q < TG; ++q) {
      const float xv = vs[(g * TG + q) * LD + d];
#pragma unroll
      for (int i = q + 1; i < TG; ++i) bv[i] = fmaf(mat_row[(g * TG + q) * ML + i], xv, bv[i]);
    }
#pragma unroll
    for (int i = 0; i < TG; ++i) ys[(g * TG + i) * LD + d] = bv[i];
  }
  __syncthreads();
  if (tid < 2 * P) {       // a thread a column of [W, Y']: once a row is known it leaves all the rows below it
    float* column = tid < P ? ub + tid : ys + tid - P;
    float x[C];
#pragma unroll
    for (int t = 0; t < C; ++t) x[t] = column[t * LD];
#pragma unroll
    for (int s = 0; s < C - 1; ++s) {
#pragma unroll
      for (int t4 = (s + 1) / 4 * 4; t4 < C; t4 += 4) {
        const float4 m = *reinterpret_cast<const float4*>(mat + s * ML + t4);
        if (t4 > s) x[t4] = fmaf(-m.x, x[s], x[t4]);
        if (t4 + 1 > s) x[t4 + 1] = fmaf(-m.y, x[s], x[t4 + 1]);
        if (t4 + 2 > s) x[t4 + 2] = fmaf(-m.z, x[s], x[t4 + 2]);
        x[t4 + 3] = fmaf(-m.w, x[s], x[t4 + 3]);
      }
    }
#pragma unroll
    for (int t = 0; t < C; ++t) column[t * LD] = x[t];
  }
  __syncthreads();
  // the cell (tokens past the last one have rows of zeros)
  float* cell = cells + ((size_t)chunk * heads + head) * walk_cell_floats(P, 2);
  bool unsafe = false;
  const float kept = bn[d];
#pragma unroll
  for (int i = 0; i < TG; ++i) {
    const int t = g * TG + i;
    const float r = rb[t * LD + d], w = ub[t * LD + d], k = kept * ki[t * LD + d], removed = kept * ai[t * LD + d];
    unsafe |= tf32_unsafe(r) || tf32_unsafe(w) || tf32_unsafe(k) || tf32_unsafe(removed);
    cell[t * walk_q_row(P) + d] = r;
    cell[walk_cell_w(P) + t * walk_q_row(P) + d] = w;
    cell[walk_cell_k(P, 2) + t * walk_k_row(P) + d] = k;
    cell[walk_cell_k2(P) + t * walk_k_row(P) + d] = removed;
    cell[walk_cell_v2(P) + t * P + d] = -ys[t * LD + d];
  }
  if (g == 0) cell[walk_cell_decay(P, 2) + d] = kept;
  for (int e = tid; e < C * C; e += 256) {
    const int t = e / C, s = e % C;
    const float c = mat[s * ML + C + t], dv = mat[(C + s) * ML + C + t];
    unsafe |= tf32_unsafe(c) || tf32_unsafe(dv);
    cell[walk_cell_a(P, 2) + t * kWalkA + s] = dv;
    cell[walk_cell_a2(P) + t * kWalkA + s] = c;
  }
  const bool any = __syncthreads_or(unsafe);
  if (tid == 0)
    *reinterpret_cast<float2*>(cell + walk_cell_decay(P, 2) + P) = make_float2(any ? 1.f : 0.f, __int_as_float(n));
}

}  // namespace cie

#define DISPATCH_DTYPE(code, name, ...)                              \
  if ((code) == cie::kFloat32) { using T = float; __VA_ARGS__ }      \
  else if ((code) == cie::kBFloat16) { using T = __nv_bfloat16; __VA_ARGS__ } \
  else CIE_FAIL("%s: unknown dtype code %d", name, (code));

extern "C" int cie_delta_max_dim() { return cie::kDeltaMaxDim; }
extern "C" int cie_delta_stream_max_dim() { return cie::kDeltaStreamMaxDim; }

extern "C" int cie_tanh_rows(const float* x, int stride, void* out, int rows, int width, int dtype, void* stream) {
  using namespace cie;
  const long long total = (long long)rows * width;
  if (total <= 0) return 0;
  DISPATCH_DTYPE(dtype, "tanh_rows", {
    CIE_LAUNCH("tanh_rows", tanh_rows_kernel<T>, dim3((unsigned)((total + 255) / 256)), dim3(256), 0,
               (cudaStream_t)stream, x, stride, (T*)out, width, total);
  })
  return 0;
}

extern "C" int cie_delta_scan(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                              const float* decay, int decay_stride, const float* decay_bias,
                              const float* removal_bias, float* out, int out_stride, float* state,
                              const int* query_start, const int* slots, const int* request_active, int requests,
                              int heads, int dim, int max_slots, int* err, void* stream) {
  using namespace cie;
  if (requests <= 0) return 0;
  if (dim < 1 || dim > kDeltaMaxDim) CIE_FAIL("delta_scan: head size %d is outside 1..%d", dim, kDeltaMaxDim);
  const int columns = dim < kDeltaBlockColumns ? dim : kDeltaBlockColumns;
  const int threads = (kDeltaLanes * columns + 31) / 32 * 32;
  const dim3 grid(requests, heads, (dim + kDeltaBlockColumns - 1) / kDeltaBlockColumns);
#define CIE_DELTA_SCAN(R)                                                                                        \
  CIE_LAUNCH("delta_scan", delta_scan_kernel<R>, grid, dim3(threads), 0, (cudaStream_t)stream, proj, proj_stride, \
             r_off, k_off, v_off, a_off, decay, decay_stride, decay_bias, removal_bias, out, out_stride, state,  \
             query_start, slots, request_active, heads, dim, max_slots, err)
  if (dim <= 32) { CIE_DELTA_SCAN(4); }
  else if (dim <= 64) { CIE_DELTA_SCAN(8); }
  else if (dim <= 128) { CIE_DELTA_SCAN(16); }
  else { CIE_DELTA_SCAN(32); }
#undef CIE_DELTA_SCAN
  return 0;
}

// Floats of scratch memory the two-kernel form wants for `tokens` tokens.
extern "C" long long cie_delta_stream_floats(int tokens, int heads, int dim) {
  const int pad = dim <= 32 ? 32 : dim <= 64 ? 64 : 128;
  return (long long)tokens * heads * cie::kDeltaFields * pad;
}

extern "C" int cie_delta_stream(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                                const float* decay, int decay_stride, const float* decay_bias,
                                const float* removal_bias, float* packed, float* out, int out_stride, float* state,
                                const int* query_start, const int* slots, const int* request_active, int tokens,
                                int requests, int heads, int dim, int max_slots, int* err, void* stream) {
  using namespace cie;
  if (requests <= 0 || tokens <= 0) return 0;
  if (dim < 1 || dim > kDeltaStreamMaxDim) CIE_FAIL("delta_stream: head size %d is outside 1..%d", dim, kDeltaStreamMaxDim);
  const int pad = dim <= 32 ? 32 : dim <= 64 ? 64 : 128;
  CIE_LAUNCH("delta_prepare", delta_prepare_kernel, dim3(tokens, heads), dim3(32), 0, (cudaStream_t)stream, proj,
             proj_stride, r_off, k_off, v_off, a_off, decay, decay_stride, decay_bias, removal_bias, packed, tokens, heads,
             dim, pad);
  const int threads = (dim + 31) / 32 * 32;
  const dim3 grid(requests, heads);
#define CIE_DELTA_STREAM(P)                                                                                       \
  CIE_LAUNCH("delta_stream", delta_stream_kernel<P>, grid, dim3(threads), 0, (cudaStream_t)stream, packed, out,   \
             out_stride, state, query_start, slots, request_active, tokens, heads, dim, max_slots, err)
  if (pad == 32) { CIE_DELTA_STREAM(32); }
  else if (pad == 64) { CIE_DELTA_STREAM(64); }
  else { CIE_DELTA_STREAM(128); }
#undef CIE_DELTA_STREAM
  return 0;
}

extern "C" int cie_delta_chunk_tokens() { return cie::kDeltaChunkTokens; }

static int delta_pad(int dim) { return dim <= 32 ? 32 : dim <= 64 ? 64 : 128; }

// Floats of scratch memory the chunked form wants.
extern "C" long long cie_delta_chunk_floats(int chunks, int heads, int dim) {
  return (long long)chunks * heads * cie::walk_cell_floats(delta_pad(dim), 2);
}

// Portions in chunks of cie_delta_chunk_tokens() tokens: first token row and token count of every chunk, and where every
// request's chunks start.  Heads up to cie_delta_stream_max_dim().
extern "C" int cie_delta_chunked(const float* proj, int proj_stride, int r_off, int k_off, int v_off, int a_off,
                                 const float* decay, int decay_stride, const float* decay_bias, const float* removal_bias,
                                 float* cells, float* out, int out_stride, float* state, const int* chunk_row,
                                 const int* chunk_count, const int* request_chunk_start, const int* slots,
                                 const int* request_active, int chunks, int requests, int heads, int dim, int max_slots,
                                 int* err, void* stream) {
  using namespace cie;
  if (requests <= 0 || chunks <= 0) return 0;
  if (dim < 1 || dim > kDeltaStreamMaxDim) CIE_FAIL("delta_chunked: head size %d is outside 1..%d", dim, kDeltaStreamMaxDim);
  if (heads > 65535) CIE_FAIL("delta_chunked: too many heads");
  if (reinterpret_cast<uintptr_t>(cells) & 15) CIE_FAIL("delta_chunked: scratch memory must be 16-byte aligned");
  const cudaStream_t s = (cudaStream_t)stream;
  const int pad = delta_pad(dim);
  auto go = [&](auto kernel, int smem) {
    const cudaError_t raised = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return raised != cudaSuccess ? raised
                                 : launch(kernel, dim3(chunks, heads), dim3(256), (size_t)smem, s, proj, proj_stride, r_off, k_off, v_off,
                                          a_off, decay, decay_stride, decay_bias, removal_bias, cells, chunk_row, chunk_count, heads, dim);
  };
  const cudaError_t status = pad == 32   ? go(delta_chunk_kernel<32>, delta_chunk_smem<32>())
                             : pad == 64 ? go(delta_chunk_kernel<64>, delta_chunk_smem<64>())
                                         : go(delta_chunk_kernel<128>, delta_chunk_smem<128>());
  if (status != cudaSuccess) CIE_FAIL("delta_chunk: launch failed: %s", cudaGetErrorString(status));
  const WalkArgs walk{cells, proj + v_off, proj_stride, dim, out, out_stride, state, (long long)heads * dim * dim, chunk_row, chunk_count,
                      request_chunk_start, slots, request_active, heads, dim, dim, max_slots, err};
  const cudaError_t walked = launch_state_walk<2>(walk, pad, requests, s);
  if (walked != cudaSuccess) CIE_FAIL("delta_walk: launch failed: %s", cudaGetErrorString(walked));
  return 0;
}

extern "C" int cie_group_gate_norm(const float* o, int o_stride, const float* gate, int gate_stride,
                                   const float* gain, void* out, int out_stride, int tokens, int groups, int size,
                                   float eps, int dtype, void* stream) {
  using namespace cie;
  if (tokens <= 0 || groups <= 0) return 0;
  if (groups > 65535) CIE_FAIL("group_gate_norm: too many groups");
  const HeadGate a{o, o_stride, nullptr, gate, gate_stride, gain, 0, 0, out_stride, groups, size, eps};
  cudaError_t status;
  if (dtype == kFloat32) status = launch_head_gate(a, (float*)out, tokens, (cudaStream_t)stream);
  else if (dtype == kBFloat16) status = launch_head_gate(a, (__nv_bfloat16*)out, tokens, (cudaStream_t)stream);
  else CIE_FAIL("group_gate_norm: unknown dtype code %d", dtype);
  if (status != cudaSuccess) CIE_FAIL("group_gate_norm: launch failed: %s", cudaGetErrorString(status));
  return 0;
}
