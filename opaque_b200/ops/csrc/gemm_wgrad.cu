// Clip-weighted weight-gradient GEMM for sm_100a.
//
//   D[g][m, n]  (+)=  sum over rows t of segment g of   s[t] * A[t, m] * B[t, n]
//
// A = [T, M] and B = [T, N] are row-major bf16 (output gradients and layer inputs of a
// linear layer, rows = tokens).  The contraction runs over rows, so both operands are
// "MN-major" for the tensor core: TMA brings [64 rows x 64 cols] boxes (128-byte swizzle)
// and tcgen05.mma consumes them through MN-major shared-memory descriptors.  s[t] is the
// per-row clip factor c_example(t) (optional); it is applied to the A tile in shared memory
// by four "scaler" warps between the TMA arrival and the MMA issue, which also zero rows
// outside the segment so that grouped (per-example / per-expert) calls may have ragged ends.
//
// Warp roles (448 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner, warps 2-5
// epilogue (TMEM -> registers -> global), warps 6-13 scalers (two groups on alternate k-blocks).  The kernel is persistent: CTAs
// walk a work list of (segment, k-split, m-tile, n-tile); accumulators are double-buffered in
// TMEM so the epilogue of one item overlaps the main loop of the next.
//
// Epilogue: the fp32 tile is either stored or added (red.global.add) at
// flat index  out_offset + g_off + m*ldm + n*ldn.  When a peer table is given the flat index
// space is cut into equal contiguous shards, one per rank, and each element goes straight to
// the owning rank's buffer through its peer pointer: split-K accumulation, accumulation over
// microbatches and the cross-GPU reduce-scatter are the same instruction stream.
// Row-major output (ldn == 1) in this GPU's memory is reduced by the TMA engine: a warp lays 32 x 32 fp32 values out in
// shared memory and one lane issues cp.reduce.async.bulk.tensor.  With few rows per item (an expert's share of a short
// batch is one k-block) the kernel is all epilogue, and the load/store unit handled every value three times there.
// Measured, all weight gradients of a pass: one mixture-of-experts layer (60 experts) with 3 x 199 tokens 2.24 -> 1.52 ms, two
// with 4 x 2048 3.43 -> 2.01 ms; GPT-2 small with 2 x 64 tokens 0.30 -> 0.19 ms.
// Through a peer table the values are transposed in shared memory so that every warp-level reduction covers four 128-byte
// row segments (full NVLink packets / L2 lines).
//
// All waits are bounded (see common.cuh); on a timeout the CTA drains its TMA copies, frees
// TMEM and returns with a code in `status`.
#include <cstdio>
#include "common.cuh"
#include "api.h"

namespace ob {

constexpr int WG_BLOCK_M = 128;
constexpr int WG_BLOCK_K = 64;       // rows (tokens) per pipeline stage
constexpr int WG_UMMA_K = 16;
constexpr int WG_THREADS = 448;      // 2 + 4 epilogue + 2 x 4 scaler warps
constexpr int WG_STAGE_LD = 36;      // padded row length (floats) of the epilogue staging tile
constexpr int WG_EPI_WARP_BYTES = 8192;   // per epilogue warp: two 32 x 32 fp32 slabs, or one padded staging tile

struct WgradParams {
  int M, N, T;
  int num_groups;
  const int* seg_offsets;            // [num_groups + 1] or nullptr (one segment [0, T))
  int splits;
  const float* row_scale;            // [T] or nullptr
  float* out;                        // used when peer_out == nullptr
  float* const* peer_out;            // [world] base pointers of every rank's shard
  long long shard_elems;
  const long long* group_out_offset; // [num_groups] or nullptr (g * group_stride)
  long long group_stride;
  long long out_offset;
  long long ldm, ldn;
  int n_valid;                       // only columns n < n_valid are written
  int accumulate;
  int tma_out;                       // map_out describes the destination [groups, M, min(N, n_valid)] (accumulate only)
};

template <int BLOCK_N>
struct WgradSmem {
  static constexpr int A_BYTES = WG_BLOCK_K * WG_BLOCK_M * 2;
  static constexpr int B_BYTES = WG_BLOCK_K * BLOCK_N * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BLOCK_N == 256) ? 4 : 6;
  static constexpr int EPI_BYTES = 4 * WG_EPI_WARP_BYTES;
  static constexpr int BAR_BYTES = 256;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + EPI_BYTES + BAR_BYTES + 1024;
};

struct WorkItem {
  int g, m0, n0, row_begin, seg_end, num_kb;
  long long out_base;
};

__device__ __forceinline__ WorkItem decode_work(const WgradParams& p, int w, int block_n) {
  WorkItem it;
  const int tiles_m = (p.M + WG_BLOCK_M - 1) / WG_BLOCK_M, tiles_n = (p.N + block_n - 1) / block_n;
  const int mn = tiles_m * tiles_n;
  const int gs = w / mn, r = w % mn;
  it.g = gs / p.splits;
  const int split = gs % p.splits;
  it.m0 = (r / tiles_n) * WG_BLOCK_M;
  it.n0 = (r % tiles_n) * block_n;
  const int s0 = p.seg_offsets ? p.seg_offsets[it.g] : 0;
  const int e = p.seg_offsets ? p.seg_offsets[it.g + 1] : p.T;
  const int nkb = (e - s0 + WG_BLOCK_K - 1) / WG_BLOCK_K;
  const int kb0 = static_cast<int>(static_cast<long long>(nkb) * split / p.splits);
  const int kb1 = static_cast<int>(static_cast<long long>(nkb) * (split + 1) / p.splits);
  it.row_begin = s0 + kb0 * WG_BLOCK_K;
  it.seg_end = min(e, s0 + kb1 * WG_BLOCK_K);
  it.num_kb = kb1 - kb0;
  it.out_base = p.out_offset + (p.group_out_offset ? p.group_out_offset[it.g]
                                                   : static_cast<long long>(it.g) * p.group_stride);
  return it;
}

// Destination of flat index `idx`.  The fields are passed one by one: the callers keep them in registers for a whole item
// (re-reading a dynamically indexed problem's parameters for every 16 bytes stored cost the epilogue a quarter of its time).
__device__ __forceinline__ float* resolve_out(float* out, float* const* peer_out, long long shard_elems, long long idx) {
  if (peer_out == nullptr) return out + idx;
  const long long owner = idx / shard_elems;
  return peer_out[owner] + (idx - owner * shard_elems);
}

// TMA_OUT: every problem of the launch is reduced through its map_out; a template parameter because the two epilogues do not
// fit the 128 registers a thread of 14 warps has side by side.
template <int BLOCK_N, int CAP, bool TMA_OUT>
__global__ void __launch_bounds__(WG_THREADS, 1)
wgrad_clip_kernel(const __grid_constant__ TmaBatch<WgradParams, CAP> b) {
  using S = WgradSmem<BLOCK_N>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  float* epi = reinterpret_cast<float*>(smem + S::STAGES * S::STAGE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::STAGES * S::STAGE_BYTES + S::EPI_BYTES);
  uint64_t* full = bars;                     // [STAGES]  TMA bytes landed
  uint64_t* empty = bars + S::STAGES;        // [STAGES]  MMAs reading the stage retired
  uint64_t* scaled = bars + 2 * S::STAGES;   // [STAGES]  scaler warps done with the stage
  uint64_t* tmem_full = bars + 3 * S::STAGES;       // [2]
  uint64_t* tmem_empty = bars + 3 * S::STAGES + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * S::STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int total_work = b.total();
  const uint64_t budget = b.wait_budget_ns;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
      mbar_init(&scaled[s], 4);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&b.map_a[0]);
    tma_prefetch_desc(&b.map_b[0]);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BLOCK_N);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    int stage = 0;
    uint32_t phase = 0;
    uint32_t issued_mask = 0, issued_phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const WgradParams& p = b.p[cur];
      const WorkItem it = decode_work(p, w - b.start[cur], BLOCK_N);
      const int num_kb = uniform(it.num_kb), row_begin = uniform(it.row_begin);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, b.status, OB_ERR_WAIT_EMPTY, budget)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_expect_tx(&full[stage], S::STAGE_BYTES);
          uint8_t* a_dst = stage_base + stage * S::STAGE_BYTES;
          uint8_t* b_dst = a_dst + S::A_BYTES;
          const int row = row_begin + kb * WG_BLOCK_K;
#pragma unroll
          for (int j = 0; j < WG_BLOCK_M / 64; ++j)
            tma_load_2d(a_dst + j * (WG_BLOCK_K * 128), &b.map_a[cur], &full[stage], it.m0 + 64 * j, row);
#pragma unroll
          for (int j = 0; j < BLOCK_N / 64; ++j)
            tma_load_2d(b_dst + j * (WG_BLOCK_K * 128), &b.map_b[cur], &full[stage], it.n0 + 64 * j, row);
        }
        issued_mask |= 1u << stage;
        issued_phase = (issued_phase & ~(1u << stage)) | (phase << stage);
        if (++stage == S::STAGES) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok) {
      // unwind: let every copy this thread started land before the CTA's shared memory goes away
      for (int s = 0; s < S::STAGES; ++s)
        if (issued_mask & (1u << s)) {
          int dummy_abort = 0;
          mbar_wait(&full[s], (issued_phase >> s) & 1u, &dummy_abort, b.status, OB_ERR_DRAIN, budget);
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // One thread issues here: the MMAs follow the scalers, and issued by the whole warp (four times as fast) they only crowd the
    // scalers out of shared memory: 8192 x 2048 x 2048 72 us by the warp, 62 by the thread, 60 experts' 32768 x 1408 x 2048 288 and 293.
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(WG_BLOCK_M, BLOCK_N, 1, 1);
      int stage = 0;
      uint32_t phase = 0;
      int acc_iter = 0;
      bool ok = true;
      int cur = 0;
      for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
        cur = b.seek(w, cur);
        const WgradParams& p = b.p[cur];
        const WorkItem it = decode_work(p, w - b.start[cur], BLOCK_N);
        if (it.num_kb == 0) continue;
        const int as = acc_iter & 1;
        if (!mbar_wait(&tmem_empty[as], ((acc_iter >> 1) & 1) ^ 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_EMPTY,
                       budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * BLOCK_N;
        for (int kb = 0; kb < it.num_kb; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag, b.status, OB_ERR_WAIT_FULL, budget) ||
              !mbar_wait(&scaled[stage], phase, abort_flag, b.status, OB_ERR_WAIT_SCALED, budget)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(stage_base + stage * S::STAGE_BYTES);
          const uint32_t b_addr = a_addr + S::A_BYTES;
#pragma unroll
          for (int kk = 0; kk < WG_BLOCK_K / WG_UMMA_K; ++kk) {
            // MN-major, 128-byte swizzle: 8 rows = 1024 B (stride offset), next 64-column block =
            // BLOCK_K*128 B (leading offset); 16 rows per instruction = 2048 B per k-step.
            const uint64_t ad = make_smem_desc(a_addr + kk * (WG_UMMA_K * 128), WG_BLOCK_K * 128, 1024, 2);
            const uint64_t bd = make_smem_desc(b_addr + kk * (WG_UMMA_K * 128), WG_BLOCK_K * 128, 1024, 2);
            umma_bf16(d_tmem, ad, bd, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(&empty[stage]);
          if (++stage == S::STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(&tmem_full[as]);
        ++acc_iter;
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;                      // TMEM lane quadrant this warp may read
    float* st = epi + (warp - 2) * (WG_EPI_WARP_BYTES / 4);
    int slab = 0;
    int acc_iter = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const WgradParams& p = b.p[cur];
      const WorkItem it = decode_work(p, w - b.start[cur], BLOCK_N);
      const int n_lim = min(p.N, p.n_valid);
      if (it.num_kb == 0 && p.accumulate) continue;
      int as = 0;
      if (it.num_kb > 0) {
        as = acc_iter & 1;
        if (!mbar_wait(&tmem_full[as], (acc_iter >> 1) & 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_FULL, budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
      }
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * BLOCK_N;
      if constexpr (TMA_OUT) {
        const int rows0 = it.m0 + q * 32;
        if (rows0 < p.M) {                                   // rows past the matrix: nothing to add
          for (int c = 0; c < BLOCK_N / 32 && it.n0 + c * 32 < n_lim; ++c) {
            float v[32];
            tmem_ld32(t_row + c * 32, v);
            tmem_ld_wait();
            uint8_t* buf = reinterpret_cast<uint8_t*>(st) + slab * 4096;
            if (lane == 0) tma_store_wait_read1();           // the slab before last has been read
            __syncwarp();
            slab_row32(buf, v, lane);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_reduce_add_3d(&b.map_out[cur], buf, it.n0 + c * 32, rows0, it.g);
              tma_store_commit();
            }
            slab ^= 1;
          }
        }
      } else {
        const bool row_major = (p.ldn == 1) && ((n_lim & 3) == 0) && ((p.ldm & 3) == 0) && ((it.out_base & 3) == 0) &&
                               (p.peer_out == nullptr || (p.shard_elems & 3) == 0);
        float* const out = p.out;
        float* const* const peer_out = p.peer_out;
        const long long shard_elems = p.shard_elems, ldm = p.ldm, ldn = p.ldn;
        const int M = p.M;
        const bool accumulate = p.accumulate != 0;
        for (int c = 0; c < BLOCK_N / 32; ++c) {
          const int nc = it.n0 + c * 32;
          if (nc >= n_lim) break;
          float v[32];
          if (it.num_kb > 0) {
            tmem_ld32(t_row + c * 32, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
          }
          if (row_major) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              *reinterpret_cast<float4*>(st + lane * WG_STAGE_LD + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            __syncwarp();
#pragma unroll
            for (int rr = 0; rr < 8; ++rr) {
              const int r = rr * 4 + (lane >> 3), c4 = (lane & 7) * 4;
              const float4 x = *reinterpret_cast<const float4*>(st + r * WG_STAGE_LD + c4);
              const int m = it.m0 + q * 32 + r, n = nc + c4;
              if (m < M && n < n_lim) {
                float* dst = resolve_out(out, peer_out, shard_elems, it.out_base + static_cast<long long>(m) * ldm + n);
                if (accumulate) red_add_v4(dst, x);
                else *reinterpret_cast<float4*>(dst) = x;
              }
            }
            __syncwarp();
          } else {
            const int m = it.m0 + q * 32 + lane;
            if (m < M) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const int n = nc + j;
                if (n < n_lim) {
                  float* dst = resolve_out(out, peer_out, shard_elems, it.out_base + static_cast<long long>(m) * ldm + static_cast<long long>(n) * ldn);
                  if (accumulate) red_add_f32(dst, v[j]);
                  else *dst = v[j];
                }
              }
            }
          }
        }
      }
      if (it.num_kb > 0) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[as]);
        ++acc_iter;
      }
    }
    if constexpr (TMA_OUT) {
      if (lane == 0) tma_store_wait_all();                     // reductions done before shared memory is given back
    }
  } else {
    // ------------------------------------------------------------------ scalers
    // Two groups of four warps take alternate k-blocks, so the shared-memory round trip of one
    // block overlaps the other group's; the four row factors a thread needs for its NEXT block
    // are fetched before it waits for that block's TMA data.  The factor is rounded toward zero
    // to bf16 and applied with packed bf16x2 multiplies: |stored product| <= |s * g| (1 + 2^-9),
    // which the caller's guard on s absorbs.
    const int group = (warp - 6) >> 2;           // 0 or 1
    const int tid = (threadIdx.x - 6 * 32) & 127;
    const int my_row = tid >> 3;
    long long it_global = 0;                     // k-block counter over the whole work list
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const WgradParams& p = b.p[cur];
      const WorkItem it = decode_work(p, w - b.start[cur], BLOCK_N);
      // first k-block of this item that belongs to this group
      int kb = static_cast<int>((group - (it_global & 1) + 2) & 1);
      float sc[4];
      bool have = false;
      const float* const row_scale = p.row_scale;
      auto fetch = [&](int kblock) {
        const int row0 = it.row_begin + kblock * WG_BLOCK_K;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rg = row0 + my_row + 16 * i;
          sc[i] = (rg < it.seg_end) ? (row_scale ? __ldg(row_scale + rg) : 1.f) : 0.f;
        }
      };
      if (kb < it.num_kb) { fetch(kb); have = true; }
      for (; kb < it.num_kb; kb += 2) {
        const long long g_it = it_global + kb;
        const int stage = static_cast<int>(g_it % S::STAGES);
        const uint32_t phase = static_cast<uint32_t>((g_it / S::STAGES) & 1);
        const int row0 = it.row_begin + kb * WG_BLOCK_K;
        const bool touch = (row_scale != nullptr) || (row0 + WG_BLOCK_K > it.seg_end);
        __nv_bfloat162 s2[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat16 h = __float2bfloat16_rz(sc[i]);
          s2[i] = __halves2bfloat162(h, h);
        }
        if (kb + 2 < it.num_kb) fetch(kb + 2);   // prefetch for the next block of this group
        if (!mbar_wait(&full[stage], phase, abort_flag, b.status, OB_ERR_WAIT_FULL, budget)) {
          ok = false;
          break;
        }
        if (touch) {
          uint4* a_tile = reinterpret_cast<uint4*>(stage_base + stage * S::STAGE_BYTES);
          uint4 x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = a_tile[tid + 128 * i];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&x[i]);
#pragma unroll
            for (int e = 0; e < 4; ++e) h[e] = __hmul2(h[e], s2[i & 3]);
            a_tile[tid + 128 * i] = x[i];
          }
          fence_proxy_async_smem();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&scaled[stage]);
      }
      (void)have;
      it_global += it.num_kb;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BLOCK_N);
  }
}

// ---------------------------------------------------------------------------------------------
// Per-example variant: every example owns a whole number of 64-row k-blocks (uniform rows_per_example), so the clip
// factor is constant over an accumulation run.  The operand maps are [example][row][column], so the last k-block of an
// example whose length is no multiple of 64 is filled up with zeros, not with the next example's rows.  The MMA warp accumulates ONE example's A_e^T G_e per TMEM buffer and
// the epilogue warps fold it into fp32 register accumulators as  acc += c_e * P_e  while the tensor core already
// works on the next example in the other buffer.  Operands are never touched in shared memory (no scaling pass, no
// extra barrier in the TMA -> MMA chain) and c_e is applied in full fp32 precision.
constexpr int WP_THREADS = 320;      // TMA warp, MMA warp, 8 epilogue warps (2 per TMEM lane quadrant)
constexpr int WP_BLOCK_N = 256;
constexpr int WP_STAGES = 4;
constexpr int WP_A_BYTES = WG_BLOCK_K * WG_BLOCK_M * 2;
constexpr int WP_B_BYTES = WG_BLOCK_K * WP_BLOCK_N * 2;
constexpr int WP_STAGE_BYTES = WP_A_BYTES + WP_B_BYTES;
constexpr int WP_SMEM = WP_STAGES * WP_STAGE_BYTES + 8 * 4096 + 256 + 1024;    // + a 32 x 32 fp32 slab per epilogue warp

struct WgradPeParams {
  int M, N;
  int num_examples, ex_rows;
  int splits;                        // each split owns a contiguous range of examples
  const float* ex_scale;             // [num_examples] or nullptr (all ones)
  float* out;
  float* const* peer_out;
  long long shard_elems;
  long long out_offset;
  long long ldm;
  int accumulate;
  float* norm2_out;                  // NORM kernel: [num_examples] squared Frobenius norms are added here; nothing else is written
  int tma_out;                       // map_out describes the destination [1, M, N] (accumulate only)
};

// NORM = true: the direct form of a per-example gradient norm.  The same per-example products P_e = A_e^T G_e pass through
// tensor memory tile by tile, but the epilogue only sums their squares into norm2_out[e]; nothing is scaled, accumulated or
// stored.  Costs 2 T d_in d_out FLOPs per example against T^2 (d_in + d_out) for the Gram-matrix form, so it is the
// cheaper one for long sequences on small layers.
template <bool NORM, int CAP, bool TMA_OUT>
__global__ void __launch_bounds__(WP_THREADS, 1)
wgrad_clip_pe_kernel(const __grid_constant__ TmaBatch<WgradPeParams, CAP> b) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* slabs = smem + WP_STAGES * WP_STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(slabs + 8 * 4096);
  uint64_t* full = bars;
  uint64_t* empty = bars + WP_STAGES;
  uint64_t* tmem_full = bars + 2 * WP_STAGES;
  uint64_t* tmem_empty = bars + 2 * WP_STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * WP_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int total_work = b.total();
  const uint64_t budget = b.wait_budget_ns;

  if (threadIdx.x == 0) {
    for (int s = 0; s < WP_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full[a], 1);
      mbar_init(&tmem_empty[a], 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&b.map_a[0]);
    tma_prefetch_desc(&b.map_b[0]);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * WP_BLOCK_N);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);

  // work item w -> (split, m tile, n tile); split s owns examples [e0, e1)
  auto decode = [](const WgradPeParams& p, int w, int& m0, int& n0, int& e0, int& e1) {
    const int tiles_m = (p.M + WG_BLOCK_M - 1) / WG_BLOCK_M, tiles_n = (p.N + WP_BLOCK_N - 1) / WP_BLOCK_N;
    const int mn = tiles_m * tiles_n;
    const int split = w / mn, r = w % mn;
    m0 = (r / tiles_n) * WG_BLOCK_M;
    n0 = (r % tiles_n) * WP_BLOCK_N;
    e0 = static_cast<int>(static_cast<long long>(p.num_examples) * split / p.splits);
    e1 = static_cast<int>(static_cast<long long>(p.num_examples) * (split + 1) / p.splits);
  };

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0, issued_mask = 0, issued_phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const WgradPeParams& p = b.p[cur];
      const int kpe = (p.ex_rows + WG_BLOCK_K - 1) / WG_BLOCK_K;
      int m0, n0, e0, e1;
      decode(p, w - b.start[cur], m0, n0, e0, e1);
      const int nkb = (e1 - e0) * kpe;
      int ex = e0, row = 0;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, b.status, OB_ERR_WAIT_EMPTY, budget)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_expect_tx(&full[stage], WP_STAGE_BYTES);
          uint8_t* a_dst = smem + stage * WP_STAGE_BYTES;
          uint8_t* b_dst = a_dst + WP_A_BYTES;
#pragma unroll
          for (int j = 0; j < WG_BLOCK_M / 64; ++j)
            tma_load_3d(a_dst + j * (WG_BLOCK_K * 128), &b.map_a[cur], &full[stage], m0 + 64 * j, row, ex);
#pragma unroll
          for (int j = 0; j < WP_BLOCK_N / 64; ++j)
            tma_load_3d(b_dst + j * (WG_BLOCK_K * 128), &b.map_b[cur], &full[stage], n0 + 64 * j, row, ex);
        }
        row += WG_BLOCK_K;
        if (row >= kpe * WG_BLOCK_K) {
          row = 0;
          ++ex;
        }
        issued_mask |= 1u << stage;
        issued_phase = (issued_phase & ~(1u << stage)) | (phase << stage);
        if (++stage == WP_STAGES) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok) {
      for (int s = 0; s < WP_STAGES; ++s)
        if (issued_mask & (1u << s)) {
          int dummy_abort = 0;
          mbar_wait(&full[s], (issued_phase >> s) & 1u, &dummy_abort, b.status, OB_ERR_DRAIN, budget);
        }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(WG_BLOCK_M, WP_BLOCK_N, 1, 1);
    const uint32_t ring = smem_u32(smem);
    int stage = 0, acc_iter = 0;
    uint32_t phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const WgradPeParams& p = b.p[cur];
      const int kpe = (p.ex_rows + WG_BLOCK_K - 1) / WG_BLOCK_K;
      int m0, n0, e0, e1;
      decode(p, w - b.start[cur], m0, n0, e0, e1);
      for (int e = e0; ok && e < e1; ++e) {
        const int as = acc_iter & 1;
        if (!mbar_wait_warp(&tmem_empty[as], ((acc_iter >> 1) & 1) ^ 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_EMPTY, budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * WP_BLOCK_N;
        bool ready = false;
        for (int kb = 0; kb < kpe; ++kb) {
          if (!ready && !mbar_wait_warp(&full[stage], phase, abort_flag, b.status, OB_ERR_WAIT_FULL, budget)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = ring + stage * WP_STAGE_BYTES;
          const uint64_t ad = make_smem_desc(a_addr, WG_BLOCK_K * 128, 1024, 2);
          const uint64_t bd = make_smem_desc(a_addr + WP_A_BYTES, WG_BLOCK_K * 128, 1024, 2);
          const int next = stage + 1 == WP_STAGES ? 0 : stage + 1;
          const bool peek = kb + 1 < kpe && mbar_test_wait(&full[next], next == 0 ? phase ^ 1 : phase);
          if (elect_one()) umma_bf16_kblock<128, 128>(d_tmem, ad, bd, idesc, kb > 0, &empty[stage]);
          ready = __all_sync(0xffffffffu, peek);
          if (++stage == WP_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (elect_one()) umma_commit(&tmem_full[as]);
        ++acc_iter;
      }
    }
  } else {
    const int q = warp & 3;                      // TMEM lane quadrant this warp may read
    const int half = (warp - 2) >> 2;            // which 128 of the tile's 256 columns
    int acc_iter = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const WgradPeParams& p = b.p[cur];
      int m0, n0, e0, e1;
      decode(p, w - b.start[cur], m0, n0, e0, e1);
      float acc[128];
#pragma unroll
      for (int j = 0; j < 128; ++j) acc[j] = 0.f;
      for (int e = e0; e < e1; ++e) {
        const int as = acc_iter & 1;
        const float c = p.ex_scale ? __ldg(p.ex_scale + e) : 1.f;
        if (!mbar_wait(&tmem_full[as], (acc_iter >> 1) & 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_FULL, budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if constexpr (NORM) {
          // rows / columns outside the matrices were zero-filled by the tensor maps, so no masking is needed
          float ss = 0.f;
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            float v[32];
            tmem_ld32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * WP_BLOCK_N + half * 128 + ch * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) ss = fmaf(v[j], v[j], ss);
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          if (lane == 0) atomicAdd(p.norm2_out + e, ss);
        } else if (c != 0.f) {
        // an example with factor 0 (non-finite norm, padding) is skipped, not multiplied: 0 * NaN would poison the sum
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            float v[32];
            tmem_ld32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * WP_BLOCK_N + half * 128 + ch * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[ch * 32 + j] = fmaf(c, v[j], acc[ch * 32 + j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tmem_empty[as]);
        ++acc_iter;
      }
      if (!ok) break;
      if constexpr (NORM) continue;
      if (e1 <= e0 && p.accumulate) continue;
      const int m = m0 + q * 32 + lane;
      if constexpr (TMA_OUT) {
        uint8_t* buf = slabs + (warp - 2) * 4096;
        if (m0 + q * 32 < p.M) {
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            const int n = n0 + half * 128 + ch * 32;
            if (n < p.N) {
              if (lane == 0) tma_store_wait_read();
              __syncwarp();
              slab_row32(buf, acc + ch * 32, lane);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                tma_reduce_add_3d(&b.map_out[cur], buf, n, m0 + q * 32, 0);
                tma_store_commit();
              }
            }
          }
        }
      } else if (m < p.M) {
        const bool vec_ok = ((p.ldm & 3) == 0) && ((p.N & 3) == 0) && ((p.out_offset & 3) == 0) &&
                            (p.peer_out == nullptr || (p.shard_elems & 3) == 0);
        const long long row_base = p.out_offset + static_cast<long long>(m) * p.ldm;
        float* const out = p.out;
        float* const* const peer_out = p.peer_out;
        const long long shard_elems = p.shard_elems;
        const int N = p.N;
        const bool accumulate = p.accumulate != 0;
#pragma unroll
        for (int j4 = 0; j4 < 32; ++j4) {
          const int n = n0 + half * 128 + 4 * j4;
          if (n >= N) break;
          if (vec_ok) {
            float* dst = resolve_out(out, peer_out, shard_elems, row_base + n);
            const float4 x = make_float4(acc[4 * j4], acc[4 * j4 + 1], acc[4 * j4 + 2], acc[4 * j4 + 3]);
            if (accumulate) red_add_v4(dst, x);
            else *reinterpret_cast<float4*>(dst) = x;
          } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
              if (n + t < N) {
                float* dst = resolve_out(out, peer_out, shard_elems, row_base + n + t);
                if (accumulate) red_add_f32(dst, acc[4 * j4 + t]);
                else *dst = acc[4 * j4 + t];
              }
          }
        }
      }
    }
    if constexpr (TMA_OUT) {
      if (lane == 0) tma_store_wait_all();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * WP_BLOCK_N);
  }
}

// ---------------------------------------------------------------------------------------------
// host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

static thread_local char g_map_detail[192] = {0};

// bf16 [examples][rows][cols] with row pitch ld, 64 x 64 boxes (a box never crosses into the next example)
static int make_bf16_map_3d(CUtensorMap* map, const void* base, long long examples, long long rows, long long cols, long long ld);

// 2-D bf16 tensor map over a row-major [rows, cols] matrix with row pitch `ld` elements.
int make_bf16_map_2d(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld,
                     int box_cols, int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return -10;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((ld * 2) & 15) != 0) {
    snprintf(g_map_detail, sizeof(g_map_detail), "operand not 16-byte aligned: base=%p ld=%lld", base, ld);
    return -11;
  }
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  // Driver entry points need a context bound to the calling thread; framework worker threads (autograd) may never
  // have made a runtime call of their own on the default device, so bind the primary context once per thread.
  static thread_local bool bound = false;
  if (!bound) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) bound = true;
  }
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    snprintf(g_map_detail, sizeof(g_map_detail), "tensor map rejected (CUresult %d): base=%p rows=%lld cols=%lld ld=%lld box=%dx%d",
             static_cast<int>(r), base, rows, cols, ld, box_cols, box_rows);
  return r == CUDA_SUCCESS ? 0 : -12;
}
static int make_bf16_map_3d(CUtensorMap* map, const void* base, long long examples, long long rows, long long cols, long long ld) {
  CUtensorMap whole;                     // the checks (alignment, pitch) and the thread's context of the 2-D form
  const int rc = make_bf16_map_2d(&whole, base, examples * rows, cols, ld, 64, WG_BLOCK_K);
  if (rc) return rc;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(examples)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2, static_cast<cuuint64_t>(ld) * 2 * rows};
  cuuint32_t box[3] = {64, WG_BLOCK_K, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = get_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    snprintf(g_map_detail, sizeof(g_map_detail), "tensor map rejected (CUresult %d): base=%p examples=%lld rows=%lld cols=%lld ld=%lld",
             static_cast<int>(r), base, examples, rows, cols, ld);
  return r == CUDA_SUCCESS ? 0 : -12;
}

// Tensor map of an fp32 destination [groups][m][n] with row pitch ldm and group pitch gstride (elements), 32 x 32 boxes in the
// 128-byte-swizzled layout of slab_row32; false when its alignment rules it out.
static bool make_out_map(CUtensorMap* map, float* base, long long n, long long m, long long groups, long long ldm, long long gstride) {
  EncodeTiledFn enc = get_encode_fn();
  if (groups == 1) gstride = ldm * m;
  if (enc == nullptr || (reinterpret_cast<uintptr_t>(base) & 15) || (ldm & 3) || (gstride & 3) || n <= 0 || m <= 0 || ldm < n) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(n), static_cast<cuuint64_t>(m), static_cast<cuuint64_t>(groups)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ldm) * 4, static_cast<cuuint64_t>(gstride) * 4};
  if (strides[1] >= (1ull << 40)) return false;
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static_assert(sizeof(TmaBatch<WgradParams, BATCH_CAP>) <= 32764 && sizeof(TmaBatch<WgradPeParams, BATCH_CAP>) <= 32764,
              "a launch's parameters");

template <class P, int CAP>
static bool all_tma_out(const TmaBatch<P, CAP>& b) {
  for (int i = 0; i < b.count; ++i)
    if (!b.p[i].tma_out) return false;
  return true;
}

template <int BLOCK_N, bool TMA_OUT, int CAP>
static int launch_wgrad_as(const TmaBatch<WgradParams, CAP>& b, int sms, cudaStream_t stream) {
  using S = WgradSmem<BLOCK_N>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(wgrad_clip_kernel<BLOCK_N, CAP, TMA_OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL) !=
        cudaSuccess)
      return -20;
    configured = true;
  }
  const int total = b.start[b.count];
  if (total <= 0) return 0;
  const int grid = total < sms ? total : sms;
  wgrad_clip_kernel<BLOCK_N, CAP, TMA_OUT><<<grid, WG_THREADS, S::TOTAL, stream>>>(b);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

template <int BLOCK_N, int CAP>
static int launch_wgrad(const TmaBatch<WgradParams, CAP>& b, int sms, cudaStream_t stream) {
  return all_tma_out(b) ? launch_wgrad_as<BLOCK_N, true>(b, sms, stream) : launch_wgrad_as<BLOCK_N, false>(b, sms, stream);
}

template <int CAP>
static int launch_wgrad_bn(const TmaBatch<WgradParams, CAP>& b, int block_n, int sms, cudaStream_t st) {
  if (block_n == 256) return launch_wgrad<256>(b, sms, st);
  if (block_n == 128) return launch_wgrad<128>(b, sms, st);
  if (block_n == 64) return launch_wgrad<64>(b, sms, st);
  return -1;
}

// Appends one problem to the batch; 0 on success (also when it has no work).
template <int CAP>
static int wgrad_append(TmaBatch<WgradParams, CAP>& b, const ob_wgrad_desc& d, float* out, float* const* peer_out,
                        long long shard_elems, int block_n) {
  if (d.T <= 0 || d.M <= 0 || d.N <= 0 || d.num_groups <= 0) return 0;
  const int i = b.count;
  int rc = make_bf16_map_2d(&b.map_a[i], d.a, d.T, d.M, d.lda, 64, WG_BLOCK_K);
  if (rc) return rc;
  rc = make_bf16_map_2d(&b.map_b[i], d.b, d.T, d.N, d.ldb, 64, WG_BLOCK_K);
  if (rc) return rc;
  WgradParams& p = b.p[i];
  p.M = d.M; p.N = d.N; p.T = d.T;
  p.num_groups = d.num_groups;
  p.seg_offsets = d.seg_offsets;
  p.splits = d.splits < 1 ? 1 : d.splits;
  p.row_scale = d.row_scale;
  p.out = out;
  p.peer_out = peer_out;
  p.shard_elems = shard_elems;
  p.group_out_offset = d.group_out_offset;
  p.group_stride = d.group_stride;
  p.out_offset = d.out_offset;
  p.ldm = d.ldm; p.ldn = d.ldn;
  p.n_valid = d.n_valid > 0 ? d.n_valid : d.N;
  p.accumulate = d.accumulate;
  p.tma_out = d.accumulate && out != nullptr && peer_out == nullptr && d.ldn == 1 && d.group_out_offset == nullptr &&
              make_out_map(&b.map_out[i], out + d.out_offset, d.N < p.n_valid ? d.N : p.n_valid, d.M, d.num_groups, d.ldm, d.group_stride);
  const long long tiles = static_cast<long long>((d.M + WG_BLOCK_M - 1) / WG_BLOCK_M) * ((d.N + block_n - 1) / block_n);
  const long long end = b.start[i] + tiles * d.num_groups * p.splits;
  if (end > 0x7fffffffLL - (1 << 16)) return -5;
  b.start[i + 1] = static_cast<int>(end);
  ++b.count;
  return 0;
}

template <bool NORM, bool TMA_OUT, int CAP>
static int launch_wgrad_pe_as(const TmaBatch<WgradPeParams, CAP>& b, int sms, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(wgrad_clip_pe_kernel<NORM, CAP, TMA_OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, WP_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  const int total = b.start[b.count];
  if (total <= 0) return 0;
  const int grid = total < sms ? total : sms;
  wgrad_clip_pe_kernel<NORM, CAP, TMA_OUT><<<grid, WP_THREADS, WP_SMEM, stream>>>(b);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

template <bool NORM, int CAP>
static int launch_wgrad_pe(const TmaBatch<WgradPeParams, CAP>& b, int sms, cudaStream_t stream) {
  if constexpr (NORM) return launch_wgrad_pe_as<true, false>(b, sms, stream);
  else return all_tma_out(b) ? launch_wgrad_pe_as<false, true>(b, sms, stream) : launch_wgrad_pe_as<false, false>(b, sms, stream);
}

template <int CAP>
static int wgrad_pe_append(TmaBatch<WgradPeParams, CAP>& b, const ob_wgrad_pe_desc& d, float* out, float* const* peer_out,
                           long long shard_elems) {
  if (d.num_examples <= 0 || d.ex_rows <= 0 || d.M <= 0 || d.N <= 0) return 0;
  int splits = d.splits < 1 ? 1 : d.splits;
  if (splits > d.num_examples) splits = d.num_examples;
  if (splits > 1 && !d.accumulate && d.norm2 == nullptr) return -4;   // split partial sums must be reduced into the destination
  const long long T = static_cast<long long>(d.num_examples) * d.ex_rows;
  if (T > 0x7fffffffLL) return -5;
  const int i = b.count;
  int rc = make_bf16_map_3d(&b.map_a[i], d.a, d.num_examples, d.ex_rows, d.M, d.lda);
  if (rc) return rc;
  rc = make_bf16_map_3d(&b.map_b[i], d.b, d.num_examples, d.ex_rows, d.N, d.ldb);
  if (rc) return rc;
  WgradPeParams& p = b.p[i];
  p.M = d.M; p.N = d.N;
  p.num_examples = d.num_examples; p.ex_rows = d.ex_rows;
  p.splits = splits;
  p.ex_scale = d.ex_scale;
  p.out = out;
  p.peer_out = peer_out;
  p.shard_elems = shard_elems;
  p.out_offset = d.out_offset;
  p.ldm = d.ldm;
  p.accumulate = d.accumulate;
  p.norm2_out = d.norm2;
  p.tma_out = d.accumulate && out != nullptr && peer_out == nullptr && d.norm2 == nullptr &&
              make_out_map(&b.map_out[i], out + d.out_offset, d.N, d.M, 1, d.ldm, 0);
  const long long tiles = static_cast<long long>((d.M + WG_BLOCK_M - 1) / WG_BLOCK_M) * ((d.N + WP_BLOCK_N - 1) / WP_BLOCK_N);
  const long long end = b.start[i] + tiles * splits;
  if (end > 0x7fffffffLL - (1 << 16)) return -5;
  b.start[i + 1] = static_cast<int>(end);
  ++b.count;
  return 0;
}

template <class P, int CAP>
static void batch_begin(TmaBatch<P, CAP>& b, int* status, double wait_budget_s) {
  b.count = 0;
  b.start[0] = b.start[1] = 0;
  b.status = status;
  b.wait_budget_ns = static_cast<unsigned long long>(wait_budget_s * 1e9);
}

}  // namespace ob

extern "C" int ob_wgrad_clip(const void* a, const void* b, int T, int M, int N, long long lda, long long ldb,
                             const float* row_scale, const int* seg_offsets, int num_groups, int splits,
                             float* out, float* const* peer_out, long long shard_elems,
                             const long long* group_out_offset, long long group_stride, long long out_offset,
                             long long ldm, long long ldn, int n_valid, int accumulate, int block_n, int* status,
                             double wait_budget_s, int num_sms, void* stream) {
  using namespace ob;
  const ob_wgrad_desc d = {a, b, row_scale, seg_offsets, group_out_offset, lda, ldb, group_stride, out_offset, ldm, ldn,
                           T, M, N, num_groups, splits, n_valid, accumulate};
  TmaBatch<WgradParams, 1> w;
  batch_begin(w, status, wait_budget_s);
  if (block_n != 64 && block_n != 128 && block_n != 256) return -1;
  const int rc = wgrad_append(w, d, out, peer_out, shard_elems, block_n);
  return rc ? rc : launch_wgrad_bn(w, block_n, num_sms, static_cast<cudaStream_t>(stream));
}

extern "C" int ob_wgrad_clip_batch(const ob_wgrad_desc* descs, int count, float* out, float* const* peer_out,
                                   long long shard_elems, int block_n, int* status, double wait_budget_s, int num_sms,
                                   void* stream) {
  using namespace ob;
  if (block_n != 64 && block_n != 256) return -1;
  TmaBatch<WgradParams, BATCH_CAP> w;
  for (int i = 0; i < count;) {
    batch_begin(w, status, wait_budget_s);
    for (; i < count && w.count < BATCH_CAP; ++i) {
      const int rc = wgrad_append(w, descs[i], out, peer_out, shard_elems, block_n);
      if (rc) return rc;
    }
    const int rc = block_n == 256 ? launch_wgrad<256>(w, num_sms, static_cast<cudaStream_t>(stream))
                                  : launch_wgrad<64>(w, num_sms, static_cast<cudaStream_t>(stream));
    if (rc) return rc;
  }
  return 0;
}

extern "C" int ob_wgrad_clip_pe_batch(const ob_wgrad_pe_desc* descs, int count, float* out, float* const* peer_out,
                                      long long shard_elems, int* status, double wait_budget_s, int num_sms, void* stream) {
  using namespace ob;
  TmaBatch<WgradPeParams, BATCH_CAP> w;
  for (int i = 0; i < count;) {
    batch_begin(w, status, wait_budget_s);
    const bool norm = descs[i].norm2 != nullptr;
    for (; i < count && w.count < BATCH_CAP && (descs[i].norm2 != nullptr) == norm; ++i) {
      const int rc = wgrad_pe_append(w, descs[i], out, peer_out, shard_elems);
      if (rc) return rc;
    }
    const int rc = norm ? launch_wgrad_pe<true>(w, num_sms, static_cast<cudaStream_t>(stream))
                        : launch_wgrad_pe<false>(w, num_sms, static_cast<cudaStream_t>(stream));
    if (rc) return rc;
  }
  return 0;
}

extern "C" int ob_last_detail(char* buf, int len) {
  int i = 0;
  for (; ob::g_map_detail[i] && i < len - 1; ++i) buf[i] = ob::g_map_detail[i];
  buf[i] = 0;
  return 0;
}
