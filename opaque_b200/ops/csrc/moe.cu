// Row kernels of the mixture of experts: combining the experts' outputs per token, the backward of that step, and the backward of
// the experts' gated activation.
//
// Rows are sorted by (expert, example); token t owns the k sorted rows pos[t * k .. t * k + k).  Both kernels touch every
// row once and are bound by memory:
//   combine    out[t] = sum_j w[t, j] * y[pos[t, j]]          k reads and one write per token, fp32 sum in slot order
//   row grad   dy[i] = w * dout[token(i)],  dw = <dout[token(i)], y[i]>      one pass over the rows
// The combine gathers, so it needs neither a zeroed output nor atomics and repeats bit for bit; a scatter-add into bf16
// rounded after every one of the k additions and ran at a tenth of the bandwidth.
// Measured with 8192 tokens, k = 4, H = 2048: combine 32 us, row gradients 59 us; the scatter-adds took 590 us each, and the
// element-wise chain around them (fp32 copies of [32768, 2816] operands among it) 2 ms per layer.
//
//   glu bwd    [dGate | dUp] of silu(gate) * up for packed [gate | up]       one pass: 3 I values in, 2 I out per row
// It rounds where the separate fp32 operations round (sigmoid by the accurate exponential and division, every product and sum
// for itself), so its results have their bits.  This file is compiled without fast math for its sake.
#include "common.cuh"
#include "api.h"

namespace ob {

__device__ __forceinline__ void unpack8(const uint4& q, float* v) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float2 f = __bfloat1622float2(h[t]);
    v[2 * t] = f.x;
    v[2 * t + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* v) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

// One thread per 8 columns of a token; four slots' rows are in flight before the first is added.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ w, const long long* __restrict__ pos,
                   __nv_bfloat16* __restrict__ out, long long tokens, int k, int H) {
  const int c8 = H >> 3;
  const long long total = tokens * c8;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const long long t = i / c8;
    const int col = static_cast<int>(i - t * c8) << 3;
    float acc[8] = {};
    for (int j0 = 0; j0 < k; j0 += 4) {
      uint4 q[4];
      float s[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j0 + j < k) {
          const long long r = __ldg(pos + t * k + j0 + j);
          q[j] = __ldg(reinterpret_cast<const uint4*>(y + r * H + col));
          s[j] = w ? __bfloat162float(__ldg(w + t * k + j0 + j)) : 1.f;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j0 + j < k) {
          float v[8];
          unpack8(q[j], v);
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[e] += s[j] * v[e];
        }
      }
    }
    *reinterpret_cast<uint4*>(out + t * H + col) = pack8(acc);
  }
}

// One warp per sorted row.
__global__ void __launch_bounds__(256)
moe_row_grad_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ y,
                    const __nv_bfloat16* __restrict__ w, const long long* __restrict__ token,
                    const long long* __restrict__ slot, __nv_bfloat16* __restrict__ dy, float* __restrict__ dw,
                    long long rows, int H) {
  const int lane = threadIdx.x & 31;
  for (long long i = blockIdx.x * 8LL + (threadIdx.x >> 5); i < rows; i += gridDim.x * 8LL) {
    const long long t = __ldg(token + i), sl = __ldg(slot + i);
    const float s = __bfloat162float(__ldg(w + sl));
    const uint4* g4 = reinterpret_cast<const uint4*>(dout + t * H);
    const uint4* y4 = reinterpret_cast<const uint4*>(y + i * H);
    uint4* o4 = reinterpret_cast<uint4*>(dy + i * H);
    float dot = 0.f;
#pragma unroll 4
    for (int c = lane; c < (H >> 3); c += 32) {
      float g[8], v[8];
      unpack8(__ldg(g4 + c), g);
      unpack8(__ldg(y4 + c), v);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        dot += g[e] * v[e];
        g[e] *= s;
      }
      o4[c] = pack8(g);
    }
    dot = warp_sum(dot);
    if (lane == 0) dw[sl] = dot;
  }
}

// Bound by memory (five values of 2 bytes per pair), with some 40 instructions a value for the exact exponential and division behind
// it.  Measured at 32768 x 1408: 92 us (71 at the copy rate), 83 with the approximate ones of elementwise.cu, which differ from
// the separate operations in 13 of a million results at gates around 3 and round 27 % more of them wrongly at gates around 30.
__global__ void __launch_bounds__(256)
moe_glu_bwd_kernel(const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ gate_up, __nv_bfloat16* __restrict__ dgate_up,
                   long long rows, int I) {
  const int c8 = I >> 3;
  const long long total = rows * c8;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const long long r = i / c8;
    const long long at = r * 2 * I + (static_cast<int>(i - r * c8) << 3);
    const uint4 qd = __ldg(reinterpret_cast<const uint4*>(dh) + i), qg = __ldg(reinterpret_cast<const uint4*>(gate_up + at)),
                qu = __ldg(reinterpret_cast<const uint4*>(gate_up + at + I));
    float d[8], g[8], u[8];
    unpack8(qd, d);
    unpack8(qg, g);
    unpack8(qu, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sig = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-g[e])));
      const float slope = __fadd_rn(1.f, __fmul_rn(g[e], __fsub_rn(1.f, sig)));
      u[e] = __fmul_rn(__fmul_rn(__fmul_rn(d[e], u[e]), sig), slope);
      d[e] = __fmul_rn(d[e], __fmul_rn(g[e], sig));
    }
    *reinterpret_cast<uint4*>(dgate_up + at) = pack8(u);
    *reinterpret_cast<uint4*>(dgate_up + at + I) = pack8(d);
  }
}

}  // namespace ob

static int moe_grid(long long blocks, int sms) {
  const long long cap = static_cast<long long>(sms) * 8;
  return static_cast<int>(blocks < cap ? blocks : cap);
}

extern "C" int ob_moe_combine(const void* y, const void* w, const long long* pos, void* out, long long tokens, int k, int H,
                              int sms, void* stream) {
  if (tokens <= 0 || H <= 0) return 0;
  if (k < 1 || (H & 7) || ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(out)) & 15)) return -2;
  ob::moe_combine_kernel<<<moe_grid((tokens * (H / 8) + 255) / 256, sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(w), pos, static_cast<__nv_bfloat16*>(out),
      tokens, k, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ob_moe_row_grad(const void* dout, const void* y, const void* w, const long long* token, const long long* slot,
                               void* dy, float* dw, long long rows, int H, int sms, void* stream) {
  if (rows <= 0 || H <= 0) return 0;
  if ((H & 7) || ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(dy)) & 15))
    return -2;
  ob::moe_row_grad_kernel<<<moe_grid((rows + 7) / 8, sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(w),
      token, slot, static_cast<__nv_bfloat16*>(dy), dw, rows, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ob_moe_glu_bwd(const void* dh, const void* gate_up, void* dgate_up, long long rows, int I, int sms, void* stream) {
  if (rows <= 0 || I <= 0) return 0;
  if ((I & 7) || ((reinterpret_cast<uintptr_t>(dh) | reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(dgate_up)) & 15))
    return -2;
  ob::moe_glu_bwd_kernel<<<moe_grid((rows * (I / 8) + 255) / 256, sms), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(dh), static_cast<const __nv_bfloat16*>(gate_up), static_cast<__nv_bfloat16*>(dgate_up), rows, I);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
