// LayerNorm forward / backward with per-example weight and bias gradients, per-example bias-gradient row sums and
// plain (ungated) activations for sm_100a.  These are the bandwidth-bound pieces of a GPT-2-style block under
// per-example clipping: the weight / bias gradients of LayerNorm and the bias gradients of linear layers are small
// enough to materialise per example ([B, H] each), so they are reduced over an example's T token rows by a kernel and
// added straight into that example's row of the per-example gradient buffer.
// bf16 storage, fp32 math, 16-byte vector accesses, one CTA per row for the normalisation passes.
#include "common.cuh"
#include "api.h"

namespace ob {

struct alignas(16) ln_bf16x8 {
  __nv_bfloat162 v[4];
};
__device__ __forceinline__ void ln_unpack8(const ln_bf16x8& p, float* f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ ln_bf16x8 ln_pack8(const float* f) {
  ln_bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

constexpr int LN_THREADS = 128;

// two simultaneous block-wide sums
__device__ __forceinline__ float2 ln_block_sum2(float a, float b, float2* red) {
  a = warp_sum(a);
  b = warp_sum(b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = make_float2(a, b);
  __syncthreads();
  float2 t = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < LN_THREADS / 32; ++i) {
    t.x += red[i].x;
    t.y += red[i].y;
  }
  return t;
}

__global__ void __launch_bounds__(LN_THREADS)
layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                     const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y, float* __restrict__ mean,
                     float* __restrict__ rstd, int H, float eps) {
  __shared__ float2 red[LN_THREADS / 32];
  const long long row = blockIdx.x;
  const ln_bf16x8* xr = reinterpret_cast<const ln_bf16x8*>(x + row * H);
  const int nv = H >> 3;
  float s = 0.f, ss = 0.f;
  for (int i = threadIdx.x; i < nv; i += LN_THREADS) {
    float f[8];
    ln_unpack8(xr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s += f[j];
      ss += f[j] * f[j];
    }
  }
  const float2 t = ln_block_sum2(s, ss, red);
  const float mu = t.x / H;
  const float var = fmaxf(t.y / H - mu * mu, 0.f);
  const float rs = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    mean[row] = mu;
    rstd[row] = rs;
  }
  const ln_bf16x8* wr = reinterpret_cast<const ln_bf16x8*>(w);
  const ln_bf16x8* br = reinterpret_cast<const ln_bf16x8*>(b);
  ln_bf16x8* yr = reinterpret_cast<ln_bf16x8*>(y + row * H);
  for (int i = threadIdx.x; i < nv; i += LN_THREADS) {
    float f[8], g[8], h[8];
    ln_unpack8(xr[i], f);
    ln_unpack8(wr[i], g);
    if (b != nullptr) ln_unpack8(br[i], h);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = (f[j] - mu) * rs * g[j] + (b != nullptr ? h[j] : 0.f);
    yr[i] = ln_pack8(f);
  }
}

__global__ void __launch_bounds__(LN_THREADS)
layernorm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                        const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean,
                        const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx, int H) {
  __shared__ float2 red[LN_THREADS / 32];
  const long long row = blockIdx.x;
  const ln_bf16x8* dyr = reinterpret_cast<const ln_bf16x8*>(dy + row * H);
  const ln_bf16x8* xr = reinterpret_cast<const ln_bf16x8*>(x + row * H);
  const ln_bf16x8* wr = reinterpret_cast<const ln_bf16x8*>(w);
  ln_bf16x8* dxr = reinterpret_cast<ln_bf16x8*>(dx + row * H);
  const int nv = H >> 3;
  const float mu = mean[row], rs = rstd[row];
  float s1 = 0.f, s2 = 0.f;
  for (int i = threadIdx.x; i < nv; i += LN_THREADS) {
    float a[8], f[8], g[8];
    ln_unpack8(dyr[i], a);
    ln_unpack8(xr[i], f);
    ln_unpack8(wr[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gw = a[j] * g[j];
      s1 += gw;
      s2 += gw * (f[j] - mu) * rs;
    }
  }
  const float2 t = ln_block_sum2(s1, s2, red);
  const float m1 = t.x / H, m2 = t.y / H;
  for (int i = threadIdx.x; i < nv; i += LN_THREADS) {
    float a[8], f[8], g[8];
    ln_unpack8(dyr[i], a);
    ln_unpack8(xr[i], f);
    ln_unpack8(wr[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = rs * (a[j] * g[j] - m1 - (f[j] - mu) * rs * m2);
    dxr[i] = ln_pack8(a);
  }
}

// Register-resident variants: 128 threads own one row (up to 128 * VPT 16-byte vectors, masked at the row end) and keep it
// in registers; two rows per CTA; one global read and one write per element.
constexpr int LN_ROW_THREADS = 128;

__device__ __forceinline__ float2 ln_row_group_sum2(float a, float b, float2* red) {     // red: 4 entries of this row group
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = (threadIdx.x & (LN_ROW_THREADS - 1)) >> 5;
  if ((threadIdx.x & 31) == 0) red[w] = make_float2(a, b);
  __syncthreads();
  const float2 t = make_float2(red[0].x + red[1].x + red[2].x + red[3].x, red[0].y + red[1].y + red[2].y + red[3].y);
  __syncthreads();
  return t;
}

template <int VPT>
__global__ void __launch_bounds__(2 * LN_ROW_THREADS)
layernorm_fwd_reg_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                         const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y, float* __restrict__ mean,
                         float* __restrict__ rstd, long long rows, int H, float eps) {
  __shared__ float2 red_all[2][4];
  const int grp = threadIdx.x / LN_ROW_THREADS, t = threadIdx.x % LN_ROW_THREADS;
  const long long row = static_cast<long long>(blockIdx.x) * 2 + grp;
  const bool live = row < rows;
  const long long r = live ? row : rows - 1;
  const int nv = H >> 3;
  float f[VPT][8];
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = t + v * LN_ROW_THREADS;
    if (i < nv) {
      ln_unpack8(reinterpret_cast<const ln_bf16x8*>(x + r * H)[i], f[v]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s += f[v][j];
        ss += f[v][j] * f[v][j];
      }
    }
  }
  const float2 tot = ln_row_group_sum2(s, ss, red_all[grp]);
  const float mu = tot.x / H;
  const float rs = rsqrtf(fmaxf(tot.y / H - mu * mu, 0.f) + eps);
  if (live && t == 0) {
    mean[row] = mu;
    rstd[row] = rs;
  }
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = t + v * LN_ROW_THREADS;
    if (i < nv) {
      float g[8], h[8];
      ln_unpack8(reinterpret_cast<const ln_bf16x8*>(w)[i], g);
      if (b != nullptr) ln_unpack8(reinterpret_cast<const ln_bf16x8*>(b)[i], h);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[v][j] = (f[v][j] - mu) * rs * g[j] + (b != nullptr ? h[j] : 0.f);
      if (live) reinterpret_cast<ln_bf16x8*>(y + r * H)[i] = ln_pack8(f[v]);
    }
  }
}

template <int VPT>
__global__ void __launch_bounds__(2 * LN_ROW_THREADS)
layernorm_bwd_dx_reg_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                            const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean,
                            const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx, long long rows, int H) {
  __shared__ float2 red_all[2][4];
  const int grp = threadIdx.x / LN_ROW_THREADS, t = threadIdx.x % LN_ROW_THREADS;
  const long long row = static_cast<long long>(blockIdx.x) * 2 + grp;
  const bool live = row < rows;
  const long long r = live ? row : rows - 1;
  const int nv = H >> 3;
  const float mu = mean[r], rs = rstd[r];
  float gw[VPT][8], xh[VPT][8];
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = t + v * LN_ROW_THREADS;
    if (i < nv) {
      float c[8];
      ln_unpack8(reinterpret_cast<const ln_bf16x8*>(dy + r * H)[i], gw[v]);
      ln_unpack8(reinterpret_cast<const ln_bf16x8*>(x + r * H)[i], xh[v]);
      ln_unpack8(reinterpret_cast<const ln_bf16x8*>(w)[i], c);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        gw[v][j] *= c[j];
        xh[v][j] = (xh[v][j] - mu) * rs;
        s1 += gw[v][j];
        s2 += gw[v][j] * xh[v][j];
      }
    }
  }
  const float2 tot = ln_row_group_sum2(s1, s2, red_all[grp]);
  const float m1 = tot.x / H, m2 = tot.y / H;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = t + v * LN_ROW_THREADS;
    if (i < nv) {
#pragma unroll
      for (int j = 0; j < 8; ++j) gw[v][j] = rs * (gw[v][j] - m1 - xh[v][j] * m2);
      if (live) reinterpret_cast<ln_bf16x8*>(dx + r * H)[i] = ln_pack8(gw[v]);
    }
  }
}

// Warp-per-row variants for narrow rows (H <= 1024).  A warp walks over rows (stride = warps in the grid) with the
// weight and bias vectors packed in registers for the whole walk, holds one row in registers (VPL 16-byte vectors per
// lane, masked at the row end) and reduces with shuffles only, so a CTA never synchronises.  The kernel is bound by
// the load/store unit's data pipe (a profile of the one-row-per-launch-warp version showed it at 91 % with DRAM at 39 %:
// per row the weight and bias re-reads cost as many wavefronts as the row itself), hence the register-resident
// parameters; two rows per warp in flight measured slower than one (3.0 vs 3.3 TB/s at H = 768).
constexpr int LN_WARPS = 8;
constexpr int LN_WALK_STAGES = 3;

// RES: the row is x + res (rounded to bf16 and stored to `sum`, the residual stream of the next block): the addition in front
// of a norm costs no pass of its own.  Measured at 16384 x 768: 27.8 us against 12.8 + 11.4 apart forward, 26.0 against
// 18.2 + 11.4 backward (below); with 256 rows the launch it saves is worth more than either.
template <int VPL, bool RES>
__global__ void __launch_bounds__(32 * LN_WARPS, VPL >= 3 ? 2 : 3)
layernorm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                          const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y, float* __restrict__ mean,
                          float* __restrict__ rstd, long long rows, int H, float eps, const __nv_bfloat16* __restrict__ res,
                          __nv_bfloat16* __restrict__ sum) {
  const int lane = threadIdx.x & 31;
  const long long stride = static_cast<long long>(gridDim.x) * LN_WARPS;
  long long row = static_cast<long long>(blockIdx.x) * LN_WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;                                   // whole warps leave together; nothing below synchronises
  const int nv = H >> 3;
  const float inv_h = 1.f / H;
  ln_bf16x8 wp[VPL], bp[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int i = lane + v * 32;
    if (i < nv) {
      wp[v] = reinterpret_cast<const ln_bf16x8*>(w)[i];
      if (b != nullptr) bp[v] = reinterpret_cast<const ln_bf16x8*>(b)[i];
    }
  }
  for (; row < rows; row += stride) {
    const ln_bf16x8* xr = reinterpret_cast<const ln_bf16x8*>(x + row * H);
    float f[VPL][8];
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      if (lane + v * 32 < nv) {
        ln_unpack8(xr[lane + v * 32], f[v]);
        if constexpr (RES) {
          float h[8];
          ln_unpack8(reinterpret_cast<const ln_bf16x8*>(res + row * H)[lane + v * 32], h);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[v][j] += h[j];
          const ln_bf16x8 q = ln_pack8(f[v]);
          reinterpret_cast<ln_bf16x8*>(sum + row * H)[lane + v * 32] = q;
          ln_unpack8(q, f[v]);
        }
      }
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      if (lane + v * 32 < nv) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s += f[v][j];
          ss += f[v][j] * f[v][j];
        }
      }
    s = warp_sum(s);
    ss = warp_sum(ss);
    const float mu = s * inv_h;
    const float rs = rsqrtf(fmaxf(ss * inv_h - mu * mu, 0.f) + eps);
    if (lane == 0) {
      mean[row] = mu;
      rstd[row] = rs;
    }
    ln_bf16x8* yr = reinterpret_cast<ln_bf16x8*>(y + row * H);
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const int i = lane + v * 32;
      if (i < nv) {
        float g[8], h[8];
        ln_unpack8(wp[v], g);
        if (b != nullptr) ln_unpack8(bp[v], h);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[v][j] = (f[v][j] - mu) * rs * g[j] + (b != nullptr ? h[j] : 0.f);
        yr[i] = ln_pack8(f[v]);
      }
    }
  }
}

// The backward kernel keeps one row per launched warp and re-reads the weight per row: the weight is a quarter of its
// wavefronts (dy, x in, dx out), and the registers for a resident copy cost more occupancy than the re-reads cost
// (measured inside the GPT-2 step: 17.0 us per launch this way, 19.2 us with the walking form of the forward kernel).
// RES: `ds`, the gradient that reaches the row past the norm (the residual branch), is added in.  The norm's own gradient is
// rounded to bf16 first and the sum after it, as two tensors of that type add up: where many rows' gradients nearly cancel (a
// bias of the first block), one rounding instead of two moved single sums by more than their root mean square.
template <int VPL, bool RES>
__global__ void __launch_bounds__(32 * LN_WARPS)
layernorm_bwd_dx_warp_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                             const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean,
                             const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx, long long rows, int H,
                             const __nv_bfloat16* __restrict__ ds) {
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * LN_WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int nv = H >> 3;
  const float mu = mean[row], rs = rstd[row];
  const ln_bf16x8* gr = reinterpret_cast<const ln_bf16x8*>(dy + row * H);
  const ln_bf16x8* xr = reinterpret_cast<const ln_bf16x8*>(x + row * H);
  float gw[VPL][8], xh[VPL][8];
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int i = lane + v * 32;
    if (i < nv) {
      float c[8];
      ln_unpack8(gr[i], gw[v]);
      ln_unpack8(xr[i], xh[v]);
      ln_unpack8(reinterpret_cast<const ln_bf16x8*>(w)[i], c);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        gw[v][j] *= c[j];
        xh[v][j] = (xh[v][j] - mu) * rs;
        s1 += gw[v][j];
        s2 += gw[v][j] * xh[v][j];
      }
    }
  }
  const float m1 = warp_sum(s1) / H, m2 = warp_sum(s2) / H;
  ln_bf16x8* or_ = reinterpret_cast<ln_bf16x8*>(dx + row * H);
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int i = lane + v * 32;
    if (i < nv) {
#pragma unroll
      for (int j = 0; j < 8; ++j) gw[v][j] = rs * (gw[v][j] - m1 - xh[v][j] * m2);
      if constexpr (RES) {
        float h[8];
        ln_unpack8(reinterpret_cast<const ln_bf16x8*>(ds + row * H)[i], h);
#pragma unroll
        for (int j = 0; j < 8; ++j) gw[v][j] = __bfloat162float(__float2bfloat16_rn(gw[v][j])) + h[j];
      }
      or_[i] = ln_pack8(gw[v]);
    }
  }
}

// Rows on their way through shared memory, one warp's: every lane copies the 16-byte vectors that IT will use into its own slots
// (cp.async; nothing to synchronise but the lane's own copies), STAGES - 1 rows ahead of the row being worked on.  A warp that walks
// over rows otherwise waits for memory once per row.
template <int VPL, int TENSORS, int STAGES>
struct LnRowRing {
  static constexpr int WARP_BYTES = STAGES * TENSORS * VPL * 512;
  static constexpr int BYTES = LN_WARPS * WARP_BYTES;
  const ln_bf16x8* at;      // this lane's slots: [STAGES][TENSORS][VPL] x 32 lanes
  __device__ __forceinline__ LnRowRing(uint8_t* smem, int warp, int lane) : at(reinterpret_cast<const ln_bf16x8*>(smem + warp * WARP_BYTES) + lane) {}
  __device__ __forceinline__ void fetch(int stage, int tensor, const __nv_bfloat16* row, int lane, int nv) const {
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      if (lane + v * 32 < nv)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(at + ((stage * TENSORS + tensor) * VPL + v) * 32)),
                     "l"(reinterpret_cast<const ln_bf16x8*>(row) + lane + v * 32) : "memory");
  }
  static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  static __device__ __forceinline__ void wait_row() { asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory"); }
  __device__ __forceinline__ const ln_bf16x8& get(int stage, int tensor, int v) const { return at[((stage * TENSORS + tensor) * VPL + v) * 32]; }
};

// layernorm_fwd_warp_kernel<VPL, true> for many rows: the same operations on rows that come through a ring.
template <int VPL>
__global__ void __launch_bounds__(32 * LN_WARPS, 2)
add_layernorm_fwd_walk_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                              __nv_bfloat16* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd, long long rows, int H, float eps,
                              const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ sum) {
  constexpr int STAGES = LN_WALK_STAGES;
  extern __shared__ uint8_t ln_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LnRowRing<VPL, 2, STAGES> ring(ln_smem, warp, lane);
  const long long stride = static_cast<long long>(gridDim.x) * LN_WARPS;
  long long row = static_cast<long long>(blockIdx.x) * LN_WARPS + warp;
  if (row >= rows) return;
  const int nv = H >> 3;
  const float inv_h = 1.f / H;
  auto fetch = [&](long long r, int stage) {
    if (r < rows) {
      ring.fetch(stage, 0, x + r * H, lane, nv);
      ring.fetch(stage, 1, res + r * H, lane, nv);
    }
    ring.commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(row + s * stride, s);
  ln_bf16x8 wp[VPL], bp[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int i = lane + v * 32;
    if (i < nv) {
      wp[v] = reinterpret_cast<const ln_bf16x8*>(w)[i];
      if (b != nullptr) bp[v] = reinterpret_cast<const ln_bf16x8*>(b)[i];
    }
  }
  int stage = 0;
  for (; row < rows; row += stride) {
    fetch(row + (STAGES - 1) * stride, stage == 0 ? STAGES - 1 : stage - 1);
    ring.wait_row();
    float f[VPL][8];
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      if (lane + v * 32 < nv) {
        float h[8];
        ln_unpack8(ring.get(stage, 0, v), f[v]);
        ln_unpack8(ring.get(stage, 1, v), h);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[v][j] += h[j];
        const ln_bf16x8 q = ln_pack8(f[v]);
        reinterpret_cast<ln_bf16x8*>(sum + row * H)[lane + v * 32] = q;
        ln_unpack8(q, f[v]);
      }
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      if (lane + v * 32 < nv) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s += f[v][j];
          ss += f[v][j] * f[v][j];
        }
      }
    s = warp_sum(s);
    ss = warp_sum(ss);
    const float mu = s * inv_h;
    const float rs = rsqrtf(fmaxf(ss * inv_h - mu * mu, 0.f) + eps);
    if (lane == 0) {
      mean[row] = mu;
      rstd[row] = rs;
    }
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const int i = lane + v * 32;
      if (i < nv) {
        float g[8], h[8];
        ln_unpack8(wp[v], g);
        if (b != nullptr) ln_unpack8(bp[v], h);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[v][j] = (f[v][j] - mu) * rs * g[j] + (b != nullptr ? h[j] : 0.f);
        reinterpret_cast<ln_bf16x8*>(y + row * H)[i] = ln_pack8(f[v]);
      }
    }
    if (++stage == STAGES) stage = 0;
  }
}

// layernorm_bwd_dx_warp_kernel with the per-example weight and bias sums (rows_group_sum_kernel's mode 1) of the same rows: dy and x are
// read once for both.  grid = examples x chunks of an example's rows; a warp walks over its chunk with its columns' sums in
// registers, the block adds its warps' up and adds them to the example's row with atomics.
// Bound by memory.  Measured in rotation over 300 MB of operands, against the data gradient's kernel and rows_group_sum_kernel: 32 x 512
// rows of 768 37.8 -> 23.9 us, 8 x 1024 22.3 -> 15.7, 16 x 1024 rows of 1024 55.6 -> 34.9; the copy rate allows 15.4, 7.7 and 20.5.
// The sums' error against 64 bits is no larger (7.0e-8 and 7.3e-8 of their size).  Which calls come here: _norm_sums in engine/blocks.py.
template <int VPL, bool RES>
__global__ void __launch_bounds__(32 * LN_WARPS, 2)
layernorm_bwd_sums_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                          const float* __restrict__ mean, const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ ds,
                          __nv_bfloat16* __restrict__ dx, int rows_per_example, int chunks, int H, float* __restrict__ out_w,
                          float* __restrict__ out_b, long long ld_out) {
  constexpr int TENSORS = RES ? 3 : 2, STAGES = LN_WALK_STAGES;
  extern __shared__ uint8_t ln_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LnRowRing<VPL, TENSORS, STAGES> ring(ln_smem, warp, lane);
  const int e = blockIdx.x / chunks, per = (rows_per_example + chunks - 1) / chunks;
  const long long r0 = static_cast<long long>(e) * rows_per_example + (blockIdx.x % chunks) * per;
  const long long r1 = min(r0 + per, static_cast<long long>(e + 1) * rows_per_example);
  const int nv = H >> 3;
  auto fetch = [&](long long r, int stage) {
    if (r < r1) {
      ring.fetch(stage, 0, dy + r * H, lane, nv);
      ring.fetch(stage, 1, x + r * H, lane, nv);
      if constexpr (RES) ring.fetch(stage, 2, ds + r * H, lane, nv);
    }
    ring.commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(r0 + warp + s * LN_WARPS, s);
  ln_bf16x8 wp[VPL];
  float aw[VPL][8] = {}, ab[VPL][8] = {};
#pragma unroll
  for (int v = 0; v < VPL; ++v)
    if (lane + v * 32 < nv) wp[v] = reinterpret_cast<const ln_bf16x8*>(w)[lane + v * 32];
  float mu_next = 0.f, rs_next = 0.f;
  if (r0 + warp < r1) {
    mu_next = mean[r0 + warp];
    rs_next = rstd[r0 + warp];
  }
  int stage = 0;
  for (long long row = r0 + warp; row < r1; row += LN_WARPS) {
    const float mu = mu_next, rs = rs_next;
    if (row + LN_WARPS < r1) {
      mu_next = mean[row + LN_WARPS];
      rs_next = rstd[row + LN_WARPS];
    }
    fetch(row + (STAGES - 1) * LN_WARPS, stage == 0 ? STAGES - 1 : stage - 1);
    ring.wait_row();
    // one vector of dy * w and of the normalised row, formed twice: kept from the first pass they would not fit the registers
    auto load = [&](int v, float* g, float* xh, float* gw) {
      ln_unpack8(ring.get(stage, 0, v), g);
      ln_unpack8(ring.get(stage, 1, v), xh);
      ln_unpack8(wp[v], gw);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[j] = (xh[j] - mu) * rs;
        gw[j] = g[j] * gw[j];
      }
    };
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      if (lane + v * 32 < nv) {
        float g[8], xh[8], gw[8];
        load(v, g, xh, gw);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          ab[v][j] += g[j];
          aw[v][j] += g[j] * xh[j];
          s1 += gw[j];
          s2 += gw[j] * xh[j];
        }
      }
    }
    const float m1 = warp_sum(s1) / H, m2 = warp_sum(s2) / H;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      if (lane + v * 32 < nv) {
        float g[8], xh[8], gw[8];
        load(v, g, xh, gw);
#pragma unroll
        for (int j = 0; j < 8; ++j) gw[j] = rs * (gw[j] - m1 - xh[j] * m2);
        if constexpr (RES) {
          float h[8];
          ln_unpack8(ring.get(stage, 2, v), h);
#pragma unroll
          for (int j = 0; j < 8; ++j) gw[j] = __bfloat162float(__float2bfloat16_rn(gw[j])) + h[j];
        }
        reinterpret_cast<ln_bf16x8*>(dx + row * H)[lane + v * 32] = ln_pack8(gw);
      }
    }
    if (++stage == STAGES) stage = 0;
  }
  // the block's sums, one of the two at a time through the ring's memory: [LN_WARPS][H]
  asm volatile("cp.async.wait_all;" ::: "memory");
  float* red = reinterpret_cast<float*>(ln_smem);
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    __syncthreads();
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      if (lane + v * 32 < nv) {
#pragma unroll
        for (int j = 0; j < 8; ++j) red[warp * H + (lane + v * 32) * 8 + j] = which == 0 ? aw[v][j] : ab[v][j];
      }
    __syncthreads();
    float* const out = which == 0 ? out_w : out_b;
    if (out != nullptr)
      for (int c = threadIdx.x; c < H; c += 32 * LN_WARPS) {
        const float* q = red + c;
        atomicAdd(out + e * ld_out + c, ((q[0] + q[H]) + (q[2 * H] + q[3 * H])) + ((q[4 * H] + q[5 * H]) + (q[6 * H] + q[7 * H])));
      }
  }
}

// Per-example reductions over the token rows of each example: out[e, col] += sum_r f(r, col).
//   mode 0: f = g                      (bias gradients: LayerNorm bias, linear bias)
//   mode 1: f = g * (x - mean) * rstd  (LayerNorm weight gradient)
//   mode 2: f = g * x * rstd           (RMSNorm weight gradient)
// grid = (examples, column blocks of 256, row splits).  A 256-thread block reads 8 rows x 256 columns per iteration
// with 16-byte loads (32 column groups x 8 row lanes), folds the row lanes through shared memory and adds the split's
// partial sums into that example's row of the fp32 per-example gradient buffer with atomics.
__global__ void __launch_bounds__(256)
rows_group_sum_kernel(const __nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ x,
                      const float* __restrict__ mean, const float* __restrict__ rstd, int rows_per_example, int N,
                      long long ldg, float* __restrict__ out, long long ld_out, int mode, float* __restrict__ out2,
                      long long ld_out2) {
  __shared__ float red[8][256 + 8];
  __shared__ float red2[8][256 + 8];
  const int e = blockIdx.x;
  const int cg = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int col = blockIdx.y * 256 + cg * 8;
  const int chunk = (rows_per_example + gridDim.z - 1) / gridDim.z;
  const int r0 = e * rows_per_example + blockIdx.z * chunk;
  const int r1 = min(r0 + chunk, (e + 1) * rows_per_example);
  float acc[8], acc2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = acc2[j] = 0.f;
  if (col < N) {
    for (int r = r0 + rl; r < r1; r += 8) {
      float gv[8];
      ln_unpack8(*reinterpret_cast<const ln_bf16x8*>(g + static_cast<long long>(r) * ldg + col), gv);
      if (mode != 0) {
        float xv[8];
        ln_unpack8(*reinterpret_cast<const ln_bf16x8*>(x + static_cast<long long>(r) * ldg + col), xv);
        const float mu = (mode == 1) ? __ldg(mean + r) : 0.f, rs = __ldg(rstd + r);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[j] += gv[j] * (xv[j] - mu) * rs;
          acc2[j] += gv[j];                      // the bias gradient of the same pass (used when out2 is given)
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += gv[j];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    red[rl][cg * 8 + j] = acc[j];
    if (out2 != nullptr) red2[rl][cg * 8 + j] = acc2[j];
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (blockIdx.y * 256 + c < N) {
    float t = 0.f, t2 = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += red[k][c];
    atomicAdd(out + static_cast<long long>(e) * ld_out + blockIdx.y * 256 + c, t);
    if (out2 != nullptr) {
#pragma unroll
      for (int k = 0; k < 8; ++k) t2 += red2[k][c];
      atomicAdd(out2 + static_cast<long long>(e) * ld_out2 + blockIdx.y * 256 + c, t2);
    }
  }
}

// The same sums for several matrices with the same rows in ONE launch: the bias and norm-weight gradients of a backward pass.  A
// block finds its (matrix, 256-column block) in the table; otherwise as above.  One launch per layer left most of the chip
// idle (a 768-column matrix has 3 column blocks) and cost a launch each.  Measured for the 48 biases of GPT-2 small: 0.71 -> 0.58
// ms with 32 x 512 tokens, 0.21 -> 0.01 with 2 x 64.
// Measured, all norm and bias sums of GPT-2 small: 26 launches and 152 us -> one of 11.5 us with 2 x 64 tokens, 345 -> 197 us
// with 11 x 333.  At 16,384 rows a launch per layer takes the operands while L2 still holds them (16.6 us each, 28 by HBM), so
// norm sums wait for one another up to 4,096 rows only.  Bias sums wait at any length (the 32 x 512 tokens above).
constexpr int RS_CAP = 128;
struct RowSumBatch {
  ob_rowsum_desc d[RS_CAP];
  int start[RS_CAP + 1];     // first column block
};

__global__ void __launch_bounds__(256)
rows_sum_batch_kernel(const __grid_constant__ RowSumBatch t, int rows_per_example) {
  __shared__ float red[8][256 + 8];
  __shared__ float red2[8][256 + 8];
  int i = 0;
  while (static_cast<int>(blockIdx.y) >= t.start[i + 1]) ++i;
  const int e = blockIdx.x;
  const int cg = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int col0 = (blockIdx.y - t.start[i]) * 256, col = col0 + cg * 8;
  const int N = t.d[i].N, mode = t.d[i].mode;
  const long long ldg = t.d[i].ldg;
  const int chunk = (rows_per_example + gridDim.z - 1) / gridDim.z;
  const int r0 = e * rows_per_example + blockIdx.z * chunk;
  const int r1 = min(r0 + chunk, (e + 1) * rows_per_example);
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(t.d[i].g) + col;
  float acc[8] = {}, acc2[8] = {};
  if (col < N && mode == 0) {
#pragma unroll 4
    for (int r = r0 + rl; r < r1; r += 8) {
      float gv[8];
      ln_unpack8(*reinterpret_cast<const ln_bf16x8*>(g + static_cast<long long>(r) * ldg), gv);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += gv[j];
    }
  } else if (col < N) {
    const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(t.d[i].x) + col;
    const float *mean = t.d[i].mean, *rstd = t.d[i].rstd;
#pragma unroll 2
    for (int r = r0 + rl; r < r1; r += 8) {
      float gv[8], xv[8];
      ln_unpack8(*reinterpret_cast<const ln_bf16x8*>(g + static_cast<long long>(r) * ldg), gv);
      ln_unpack8(*reinterpret_cast<const ln_bf16x8*>(x + static_cast<long long>(r) * ldg), xv);
      const float mu = mode == 1 ? __ldg(mean + r) : 0.f, rs = __ldg(rstd + r);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[j] += gv[j] * (xv[j] - mu) * rs;
        acc2[j] += gv[j];
      }
    }
  }
  float* const out2 = t.d[i].out2;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    red[rl][cg * 8 + j] = acc[j];
    if (out2 != nullptr) red2[rl][cg * 8 + j] = acc2[j];
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (col0 + c < N) {
    float s = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[k][c];
    atomicAdd(t.d[i].out + static_cast<long long>(e) * t.d[i].ld_out + col0 + c, s);
    if (out2 != nullptr) {
#pragma unroll
      for (int k = 0; k < 8; ++k) s2 += red2[k][c];
      atomicAdd(out2 + static_cast<long long>(e) * t.d[i].ld_out2 + col0 + c, s2);
    }
  }
}

// Gradients of the three attention inputs, each [B, heads, T, hd] with arbitrary (16-byte aligned) batch / head / token
// strides and contiguous head vectors, gathered into ONE [B*T, 3*heads*hd] buffer: the layout the fused q/k/v
// projection produced in the forward pass.  One thread moves one 16-byte vector; consecutive threads write
// consecutive destination vectors.
struct MergeHeadsSrc {
  const __nv_bfloat16* p;
  long long sb, sh, st;
};

// Idx is 32 bits wide where the vector count allows (three 64-bit divisions per 16 bytes moved bound it otherwise).  Measured on
// 16384 rows of 3 x 768: 39.5 -> 27.4 us (23 at the copy rate); 3663 rows 9.5 -> 7.3.
template <typename Idx>
__global__ void __launch_bounds__(256)
merge_heads3_kernel(MergeHeadsSrc s0, MergeHeadsSrc s1, MergeHeadsSrc s2, __nv_bfloat16* __restrict__ out, int T,
                    int heads, int hd, long long total_vec) {
  const unsigned vec_per_head = hd >> 3, vec_per_part = heads * vec_per_head;
  for (Idx i = static_cast<Idx>(blockIdx.x) * 256 + threadIdx.x; i < static_cast<Idx>(total_vec); i += static_cast<Idx>(gridDim.x) * 256) {
    const Idx rest = i / vec_per_part;                // (row, part)
    const unsigned within = static_cast<unsigned>(i - rest * vec_per_part);
    const Idx row = rest / 3u;
    const unsigned part = static_cast<unsigned>(rest - row * 3u);
    const long long h = within / vec_per_head, v = within % vec_per_head;
    const Idx b32 = row / static_cast<unsigned>(T);
    const long long b = b32, t = row - b32 * static_cast<unsigned>(T);
    const MergeHeadsSrc& s = part == 0 ? s0 : (part == 1 ? s1 : s2);
    reinterpret_cast<ln_bf16x8*>(out)[i] =
        *reinterpret_cast<const ln_bf16x8*>(s.p + b * s.sb + h * s.sh + t * s.st + v * 8);
  }
}

// Plain activations.  act: 0 silu, 1 gelu (erf), 2 gelu (tanh approximation), 3 relu.
__device__ __forceinline__ float pa_fwd(float e, int act) {
  if (act == 0) return e / (1.f + __expf(-e));
  if (act == 1) return 0.5f * e * (1.f + erff(e * 0.70710678118654752f));
  if (act == 3) return fmaxf(e, 0.f);
  const float u = 0.7978845608028654f * (e + 0.044715f * e * e * e);
  return 0.5f * e * (1.f + tanhf(u));
}
__device__ __forceinline__ float pa_bwd(float e, int act) {
  if (act == 0) {
    const float s = 1.f / (1.f + __expf(-e));
    return s * (1.f + e * (1.f - s));
  }
  if (act == 1) {
    const float cdf = 0.5f * (1.f + erff(e * 0.70710678118654752f));
    return cdf + e * 0.3989422804014327f * __expf(-0.5f * e * e);
  }
  if (act == 3) return e > 0.f ? 1.f : 0.f;
  const float u = 0.7978845608028654f * (e + 0.044715f * e * e * e);
  const float t = tanhf(u);
  return 0.5f * (1.f + t) + 0.5f * e * (1.f - t * t) * 0.7978845608028654f * (1.f + 0.134145f * e * e);
}

// BWD: out = dy * act'(x), else out = act(x).  The activation is a template parameter: chosen per element at run time, its
// branches cost more than the arithmetic of the one that is taken.
// Measured, tanh GELU at 16384 x 3072, mean of forward and backward inside a training step: 50.4 -> 48.9 us (38 at the copy rate).
template <int ACT, bool BWD>
__global__ void __launch_bounds__(256)
activation_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                  __nv_bfloat16* __restrict__ out, long long nvec) {
#pragma unroll 2
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < nvec; i += gridDim.x * 256LL) {
    float e[8], d[8];
    ln_unpack8(reinterpret_cast<const ln_bf16x8*>(x)[i], e);
    if constexpr (BWD) ln_unpack8(reinterpret_cast<const ln_bf16x8*>(dy)[i], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = BWD ? d[j] * pa_bwd(e[j], ACT) : pa_fwd(e[j], ACT);
    reinterpret_cast<ln_bf16x8*>(out)[i] = ln_pack8(e);
  }
}

}  // namespace ob

using namespace ob;

static int ln_sms() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int VPL>
static int add_layernorm_fwd_walk(const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* b, __nv_bfloat16* y, float* mean, float* rstd,
                                  long long rows, int H, float eps, const __nv_bfloat16* res, __nv_bfloat16* sum, cudaStream_t st) {
  constexpr int smem = ob::LnRowRing<VPL, 2, ob::LN_WALK_STAGES>::BYTES;
  static const cudaError_t configured = cudaFuncSetAttribute(add_layernorm_fwd_walk_kernel<VPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (configured != cudaSuccess) return -22;
  add_layernorm_fwd_walk_kernel<VPL><<<2 * ln_sms(), 32 * LN_WARPS, smem, st>>>(x, w, b, y, mean, rstd, rows, H, eps, res, sum);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

template <int VPL, bool RES>
static int layernorm_bwd_sums(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const float* mean, const float* rstd,
                              const __nv_bfloat16* ds, __nv_bfloat16* dx, int examples, int rows_per_example, int H, float* out_w, float* out_b,
                              long long ld_out, cudaStream_t st) {
  constexpr int ring = ob::LnRowRing<VPL, RES ? 3 : 2, ob::LN_WALK_STAGES>::BYTES;
  static_assert(ring >= ob::LN_WARPS * VPL * 256 * 4, "the block's sums fit the ring");
  static const cudaError_t configured =
      cudaFuncSetAttribute(layernorm_bwd_sums_kernel<VPL, RES>, cudaFuncAttributeMaxDynamicSharedMemorySize, ring);
  if (configured != cudaSuccess) return -22;
  // two blocks per SM where there are rows for them, at least a row per warp; 16 chunks at most, as rows_group_sum_kernel has: every
  // chunk is one more rounding of the example's sum (300 chunks: 2.4e-7 of the sum's size against 1.1e-7)
  const long long sms = ln_sms();
  long long chunks = 2 * sms / examples;
  if (chunks > 16) chunks = 16;
  if (chunks > (rows_per_example + LN_WARPS - 1) / LN_WARPS) chunks = (rows_per_example + LN_WARPS - 1) / LN_WARPS;
  if (chunks < 1) chunks = 1;
  // A few blocks too many share their SMs (half as long again where two fit), or are a second wave (above 768 columns with a residual,
  // where one fits): one block per SM with longer chunks where that is shorter.  10 examples of 1024 rows, us: 1024 columns 39.9 -> 25.5
  // with a residual, 29.2 -> 22.0 without, 768 columns 24.1 -> 18.0
  const long long one = sms / examples;
  const long long halves = 2 * ring <= 224 * 1024 ? 3 : 2 * ((examples * chunks + sms - 1) / sms);
  if (one >= 1 && one < chunks && halves * one > 2 * chunks) chunks = one;
  layernorm_bwd_sums_kernel<VPL, RES><<<static_cast<unsigned>(examples * chunks), 32 * LN_WARPS, ring, st>>>(
      dy, x, w, mean, rstd, ds, dx, rows_per_example, static_cast<int>(chunks), H, out_w, out_b, ld_out);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

// CTAs of the warp-per-row kernels: one warp per row while that fills fewer CTAs than are resident at once (two per SM
// for rows wider than 512, else three), else that many CTAs, whose warps walk over the rows
static unsigned ln_warp_grid(long long rows, int H) {
  const int sms = ln_sms();
  const long long want = (rows + ob::LN_WARPS - 1) / ob::LN_WARPS, cap = static_cast<long long>(sms) * (H > 512 ? 2 : 3);
  return static_cast<unsigned>(want < cap ? want : cap);
}

extern "C" int ob_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd,
                                long long rows, int H, float eps, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8 || !aligned16({x, w, b, y})) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *xp = static_cast<const __nv_bfloat16*>(x), *wp = static_cast<const __nv_bfloat16*>(w),
                      *bp = static_cast<const __nv_bfloat16*>(b);
  __nv_bfloat16* yp = static_cast<__nv_bfloat16*>(y);
  const unsigned pairs = static_cast<unsigned>((rows + 1) / 2);
  const unsigned octs = ln_warp_grid(rows, H);
  if (H <= 256) layernorm_fwd_warp_kernel<1, false><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, nullptr, nullptr);
  else if (H <= 512) layernorm_fwd_warp_kernel<2, false><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, nullptr, nullptr);
  else if (H <= 768) layernorm_fwd_warp_kernel<3, false><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, nullptr, nullptr);
  else if (H <= 1024) layernorm_fwd_warp_kernel<4, false><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, nullptr, nullptr);
  else if (H <= 2048) layernorm_fwd_reg_kernel<2><<<pairs, 2 * LN_ROW_THREADS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps);
  else if (H <= 4096) layernorm_fwd_reg_kernel<4><<<pairs, 2 * LN_ROW_THREADS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps);
  else layernorm_fwd_kernel<<<static_cast<unsigned>(rows), LN_THREADS, 0, st>>>(xp, wp, bp, yp, mean, rstd, H, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

// With the residual addition in front (H <= 1024): sum = x + res, y = layernorm(sum); and its backward, dx += ds.
extern "C" int ob_add_layernorm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* sum, float* mean,
                                    float* rstd, long long rows, int H, float eps, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8 || H > 1024 || !aligned16({x, res, w, b, y, sum})) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *xp = static_cast<const __nv_bfloat16*>(x), *wp = static_cast<const __nv_bfloat16*>(w),
                      *bp = static_cast<const __nv_bfloat16*>(b), *rp = static_cast<const __nv_bfloat16*>(res);
  __nv_bfloat16 *yp = static_cast<__nv_bfloat16*>(y), *sp = static_cast<__nv_bfloat16*>(sum);
  // Rows in flight pay once a warp has more than two rows (us with the operands in memory, hot in L2 in brackets: 16384 x 768 32.8 -> 24.6
  // (23.4 -> 16.7), 8192 x 768 22.5 -> 15.4 (10.8 -> 9.2), 5000 x 768 16.4 -> 12.3 (7.8 -> 5.9), 16384 x 1024 41.8 -> 31.6 (35.0 -> 26.3)).
  if (H > 512 && rows > 2 * 2 * static_cast<long long>(ln_sms()) * LN_WARPS)
    return H <= 768 ? add_layernorm_fwd_walk<3>(xp, wp, bp, yp, mean, rstd, rows, H, eps, rp, sp, st)
                    : add_layernorm_fwd_walk<4>(xp, wp, bp, yp, mean, rstd, rows, H, eps, rp, sp, st);
  const unsigned octs = ln_warp_grid(rows, H);
  if (H <= 256) layernorm_fwd_warp_kernel<1, true><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, rp, sp);
  else if (H <= 512) layernorm_fwd_warp_kernel<2, true><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, rp, sp);
  else if (H <= 768) layernorm_fwd_warp_kernel<3, true><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, rp, sp);
  else layernorm_fwd_warp_kernel<4, true><<<octs, 32 * LN_WARPS, 0, st>>>(xp, wp, bp, yp, mean, rstd, rows, H, eps, rp, sp);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ob_add_layernorm_bwd_dx(const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                                       const void* ds, void* dx, long long rows, int H, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8 || H > 1024 || !aligned16({dy, x, w, ds, dx})) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *gp = static_cast<const __nv_bfloat16*>(dy), *xp = static_cast<const __nv_bfloat16*>(x),
                      *wp = static_cast<const __nv_bfloat16*>(w), *dp = static_cast<const __nv_bfloat16*>(ds);
  __nv_bfloat16* op = static_cast<__nv_bfloat16*>(dx);
  const unsigned octs = static_cast<unsigned>((rows + LN_WARPS - 1) / LN_WARPS);
  if (H <= 256) layernorm_bwd_dx_warp_kernel<1, true><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, dp);
  else if (H <= 512) layernorm_bwd_dx_warp_kernel<2, true><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, dp);
  else if (H <= 768) layernorm_bwd_dx_warp_kernel<3, true><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, dp);
  else layernorm_bwd_dx_warp_kernel<4, true><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, dp);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

// Either backward (ds may be NULL) with the per-example sums: out_w[e] += sum over example e's rows of dy (x - mean) rstd, out_b[e] += of dy
// (fp32 rows of pitch ld_out; out_b may be NULL).  H <= 1024.
extern "C" int ob_layernorm_bwd_sums(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* ds,
                                     void* dx, int num_examples, int rows_per_example, int H, float* out_w, float* out_b, long long ld_out,
                                     void* stream) {
  if (num_examples <= 0 || rows_per_example <= 0) return 0;
  if (H % 8 || H > 1024 || out_w == nullptr || !aligned16({dy, x, w, ds, dx})) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *gp = static_cast<const __nv_bfloat16*>(dy), *xp = static_cast<const __nv_bfloat16*>(x),
                      *wp = static_cast<const __nv_bfloat16*>(w), *dp = static_cast<const __nv_bfloat16*>(ds);
  __nv_bfloat16* op = static_cast<__nv_bfloat16*>(dx);
#define OB_LN_SUMS(V)                                                                                                                        \
  return dp != nullptr ? layernorm_bwd_sums<V, true>(gp, xp, wp, mean, rstd, dp, op, num_examples, rows_per_example, H, out_w, out_b, ld_out, st) \
                       : layernorm_bwd_sums<V, false>(gp, xp, wp, mean, rstd, dp, op, num_examples, rows_per_example, H, out_w, out_b, ld_out, st)
  if (H <= 256) OB_LN_SUMS(1);
  if (H <= 512) OB_LN_SUMS(2);
  if (H <= 768) OB_LN_SUMS(3);
  OB_LN_SUMS(4);
#undef OB_LN_SUMS
}

extern "C" int ob_layernorm_bwd_dx(const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                                   void* dx, long long rows, int H, void* stream) {
  if (rows <= 0) return 0;
  if (H % 8 || !aligned16({dy, x, w, dx})) return -2;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *gp = static_cast<const __nv_bfloat16*>(dy), *xp = static_cast<const __nv_bfloat16*>(x),
                      *wp = static_cast<const __nv_bfloat16*>(w);
  __nv_bfloat16* op = static_cast<__nv_bfloat16*>(dx);
  const unsigned pairs = static_cast<unsigned>((rows + 1) / 2);
  const unsigned octs = static_cast<unsigned>((rows + LN_WARPS - 1) / LN_WARPS);
  if (H <= 256) layernorm_bwd_dx_warp_kernel<1, false><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, nullptr);
  else if (H <= 512) layernorm_bwd_dx_warp_kernel<2, false><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, nullptr);
  else if (H <= 768) layernorm_bwd_dx_warp_kernel<3, false><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, nullptr);
  else if (H <= 1024) layernorm_bwd_dx_warp_kernel<4, false><<<octs, 32 * LN_WARPS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H, nullptr);
  else if (H <= 2048) layernorm_bwd_dx_reg_kernel<2><<<pairs, 2 * LN_ROW_THREADS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H);
  else if (H <= 4096) layernorm_bwd_dx_reg_kernel<4><<<pairs, 2 * LN_ROW_THREADS, 0, st>>>(gp, xp, wp, mean, rstd, op, rows, H);
  else layernorm_bwd_dx_kernel<<<static_cast<unsigned>(rows), LN_THREADS, 0, st>>>(gp, xp, wp, mean, rstd, op, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ob_rows_group_sum(const void* g, const void* x, const float* mean, const float* rstd, int num_examples,
                                 int rows_per_example, int N, long long ldg, float* out, long long ld_out, int mode,
                                 float* out2, long long ld_out2, void* stream) {
  if (num_examples <= 0 || rows_per_example <= 0 || N <= 0) return 0;
  if ((N & 7) || (ldg & 7) || (reinterpret_cast<uintptr_t>(g) & 15) || (x != nullptr && (reinterpret_cast<uintptr_t>(x) & 15)))
    return -2;
  if ((mode == 1 && (x == nullptr || mean == nullptr || rstd == nullptr)) || (mode == 2 && (x == nullptr || rstd == nullptr)))
    return -3;
  int splits = rows_per_example / 64;
  splits = splits < 1 ? 1 : (splits > 16 ? 16 : splits);
  dim3 grid(num_examples, (N + 255) / 256, splits);
  rows_group_sum_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(g), static_cast<const __nv_bfloat16*>(x), mean, rstd, rows_per_example, N, ldg,
      out, ld_out, mode, mode == 0 ? nullptr : out2, ld_out2);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ob_rows_sum_batch(const ob_rowsum_desc* descs, int count, int num_examples, int rows_per_example, void* stream) {
  if (num_examples <= 0 || rows_per_example <= 0) return 0;
  int splits = rows_per_example / 64;
  splits = splits < 1 ? 1 : (splits > 16 ? 16 : splits);
  for (int first = 0; first < count; first += RS_CAP) {
    RowSumBatch t;
    const int n = count - first < RS_CAP ? count - first : RS_CAP;
    t.start[0] = 0;
    for (int i = 0; i < n; ++i) {
      const ob_rowsum_desc& d = descs[first + i];
      if (d.N <= 0 || (d.N & 7) || (d.ldg & 7) || (reinterpret_cast<uintptr_t>(d.g) & 15) || (reinterpret_cast<uintptr_t>(d.x) & 15)) return -2;
      if (d.mode < 0 || d.mode > 2 || (d.mode > 0 && (d.x == nullptr || d.rstd == nullptr)) || (d.mode == 1 && d.mean == nullptr) ||
          (d.mode == 0 && d.out2 != nullptr))
        return -3;
      t.d[i] = d;
      t.start[i + 1] = t.start[i] + (d.N + 255) / 256;
    }
    if (t.start[n] > 65535) return -4;
    rows_sum_batch_kernel<<<dim3(num_examples, t.start[n], splits), 256, 0, static_cast<cudaStream_t>(stream)>>>(t, rows_per_example);
    if (cudaGetLastError() != cudaSuccess) return -21;
  }
  return 0;
}

extern "C" int ob_merge_heads3(const void* q, const void* k, const void* v, const long long* strides, void* out,
                               long long B, int T, int heads, int hd, int sms, void* stream) {
  if (B <= 0 || T <= 0) return 0;
  if (hd % 8) return -2;
  const void* ptrs[3] = {q, k, v};
  MergeHeadsSrc src[3];
  for (int i = 0; i < 3; ++i) {
    src[i].p = static_cast<const __nv_bfloat16*>(ptrs[i]);
    src[i].sb = strides[3 * i];
    src[i].sh = strides[3 * i + 1];
    src[i].st = strides[3 * i + 2];
    if ((reinterpret_cast<uintptr_t>(ptrs[i]) & 15) || (src[i].sb & 7) || (src[i].sh & 7) || (src[i].st & 7)) return -2;
  }
  if (reinterpret_cast<uintptr_t>(out) & 15) return -2;
  const long long total_vec = B * T * 3 * heads * (hd / 8);
  long long grid = (total_vec + 255) / 256;
  const long long cap = static_cast<long long>(sms) * 16;
  if (grid > cap) grid = cap;
  const unsigned g = static_cast<unsigned>(grid);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  __nv_bfloat16* op = static_cast<__nv_bfloat16*>(out);
  if (total_vec < 0x7fffffffLL) merge_heads3_kernel<unsigned><<<g, 256, 0, st>>>(src[0], src[1], src[2], op, T, heads, hd, total_vec);
  else merge_heads3_kernel<unsigned long long><<<g, 256, 0, st>>>(src[0], src[1], src[2], op, T, heads, hd, total_vec);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int ob_activation(const void* x, const void* dy, void* out, long long numel, int act, int sms, void* stream) {
  if (numel <= 0) return 0;
  if (numel % 8 || !aligned16({x, dy, out})) return -2;
  const long long nvec = numel / 8;
  long long grid = (nvec + 255) / 256;
  const long long cap = static_cast<long long>(sms) * 16;
  if (grid > cap) grid = cap;
  const __nv_bfloat16 *xp = static_cast<const __nv_bfloat16*>(x), *gp = static_cast<const __nv_bfloat16*>(dy);
  __nv_bfloat16* op = static_cast<__nv_bfloat16*>(out);
  const unsigned g = static_cast<unsigned>(grid);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define OB_ACT(A)                                                          \
  do {                                                                     \
    if (gp != nullptr) activation_kernel<A, true><<<g, 256, 0, st>>>(xp, gp, op, nvec); \
    else activation_kernel<A, false><<<g, 256, 0, st>>>(xp, gp, op, nvec); \
  } while (0)
  if (act == 0) OB_ACT(0);
  else if (act == 1) OB_ACT(1);
  else if (act == 3) OB_ACT(3);
  else OB_ACT(2);
#undef OB_ACT
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
