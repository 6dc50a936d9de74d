// Every head of a token's float32 row divided by its own root mean square, times a gain, times sigmoid or SiLU of a gate,
// rounded once: what ends the recurrent mixers.
#pragma once

#include "common.cuh"

namespace cie {

struct HeadGate {
  const float* o;
  int o_stride;
  const float* denominators;      // [tokens][groups]: o is first divided by its token's and head's number; nullptr: not
  const float* gate;
  int gate_stride;
  const float* gain;
  int gain_shared;                // the gain's index is a head's element, or the row's column
  int silu;                       // the gate enters as z * sigmoid(z), or as sigmoid(z)
  int out_stride;
  int groups, size;
  float eps;
};

__device__ __forceinline__ float head_gate_of(float z, int silu) {
  const float s = 1.f / (1.f + expf(-z));
  return silu ? z * s : s;
}

// Heads of any size: a warp per (token, head).
template <typename T>
__global__ void __launch_bounds__(32) head_gate_any_kernel(HeadGate a, T* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, g = blockIdx.y, lane = threadIdx.x;
  const float* row = a.o + (size_t)t * a.o_stride + (size_t)g * a.size;
  const float below = a.denominators ? a.denominators[(size_t)t * a.groups + g] : 1.f;
  float sq = 0.f;
  for (int i = lane; i < a.size; i += 32) {
    const float x = row[i] / below;
    sq = fmaf(x, x, sq);
  }
  const float inv = rsqrtf(warp_sum(sq) / (float)a.size + a.eps);
  for (int i = lane; i < a.size; i += 32) {
    const int c = g * a.size + i;
    const float z = a.gate[(size_t)t * a.gate_stride + c];
    out[(size_t)t * a.out_stride + c] = from_float<T>(a.gain[a.gain_shared ? i : c] * ((row[i] / below) * inv) * head_gate_of(z, a.silu));
  }
}

__device__ __forceinline__ void head_gate_store(float* dst, const float (&v)[4]) {
  *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void head_gate_store(__nv_bfloat16* dst, const float (&v)[4]) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// Rows of whole, aligned 16-byte pieces and heads of up to 8 L elements: L lanes a head, both pieces a lane may have and
// the gate's asked for together.  What bounds it is memory; a block of one warp a head is bound by how fast
// blocks start (2,048 tokens: 32 heads of 64 69 us, 16 heads of 128 39 us; their bytes take 6.3).
template <typename T, int L>
__global__ void __launch_bounds__(256) head_gate_kernel(HeadGate a, T* __restrict__ out, int rows) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x % L, wanted = blockIdx.x * (256 / L) + threadIdx.x / L;
  const int row = min(wanted, rows - 1), t = row / a.groups, g = row - t * a.groups;      // all lanes reach the shuffles
  const float* src = a.o + (size_t)t * a.o_stride + (size_t)g * a.size;
  const float* gates = a.gate + (size_t)t * a.gate_stride + (size_t)g * a.size;
  float4 x[2], z[2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int i = (lane + p * L) * 4;
    if (i < a.size) {
      x[p] = *reinterpret_cast<const float4*>(src + i);
      z[p] = *reinterpret_cast<const float4*>(gates + i);
    } else {
      x[p] = z[p] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  if (a.denominators) {
    const float below = a.denominators[(size_t)t * a.groups + g];
#pragma unroll
    for (int p = 0; p < 2; ++p) { x[p].x /= below; x[p].y /= below; x[p].z /= below; x[p].w /= below; }
  }
  float sq = 0.f;
#pragma unroll
  for (int p = 0; p < 2; ++p) sq = fmaf(x[p].x, x[p].x, fmaf(x[p].y, x[p].y, fmaf(x[p].z, x[p].z, fmaf(x[p].w, x[p].w, sq))));
#pragma unroll
  for (int offset = L / 2; offset > 0; offset >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, offset);
  if (wanted >= rows) return;
  const float inv = rsqrtf(sq / (float)a.size + a.eps);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int i = (lane + p * L) * 4;
    if (i >= a.size) continue;
    const float4 gain = *reinterpret_cast<const float4*>(a.gain + (a.gain_shared ? 0 : g * a.size) + i);
    const float v[4] = {gain.x * (x[p].x * inv) * head_gate_of(z[p].x, a.silu), gain.y * (x[p].y * inv) * head_gate_of(z[p].y, a.silu),
                        gain.z * (x[p].z * inv) * head_gate_of(z[p].z, a.silu), gain.w * (x[p].w * inv) * head_gate_of(z[p].w, a.silu)};
    head_gate_store(out + (size_t)t * a.out_stride + (size_t)g * a.size + i, v);
  }
}

template <typename T>
inline cudaError_t launch_head_gate(const HeadGate& a, T* out, int tokens, cudaStream_t stream) {
  const bool pieces = a.size % 4 == 0 && a.size <= 256 && a.o_stride % 4 == 0 && a.gate_stride % 4 == 0 && a.out_stride % 4 == 0 &&
                      ((reinterpret_cast<uintptr_t>(a.o) | reinterpret_cast<uintptr_t>(a.gate) | reinterpret_cast<uintptr_t>(a.gain)) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(out) & (4 * sizeof(T) - 1)) == 0 && (long long)tokens * a.groups < (1ll << 31);
  if (!pieces) return launch(head_gate_any_kernel<T>, dim3(tokens, a.groups), dim3(32), 0, stream, a, out);
  const int rows = tokens * a.groups;
  // as many lanes as a head has pieces, or half as many (two pieces a lane)
  if (a.size <= 32) return launch(head_gate_kernel<T, 4>, dim3((rows + 63) / 64), dim3(256), 0, stream, a, out, rows);
  if (a.size <= 64) return launch(head_gate_kernel<T, 8>, dim3((rows + 31) / 32), dim3(256), 0, stream, a, out, rows);
  if (a.size <= 128) return launch(head_gate_kernel<T, 16>, dim3((rows + 15) / 16), dim3(256), 0, stream, a, out, rows);
  return launch(head_gate_kernel<T, 32>, dim3((rows + 7) / 8), dim3(256), 0, stream, a, out, rows);
}

}  // namespace cie
