// Ghost per-example gradient norms of a linear layer on sm_100a.
//
// For example i with token rows A_i [T, Da] (layer inputs) and G_i [T, Dg] (output
// gradients) the weight gradient is A_i^T G_i and its squared Frobenius norm equals
//     sum over (t, t') of (A_i A_i^T)[t, t'] * (G_i G_i^T)[t, t'],
// so it can be computed without ever forming the [Da, Dg] per-example gradient.  One work
// item is (example, 128 x 128 tile of the T x T Gram matrices, upper triangle only): the two
// Gram tiles are accumulated side by side in TMEM by tcgen05.mma (K-major operands, 128-byte
// swizzle, TMA-fed), and the epilogue multiplies them element-wise, masks rows / columns that
// fall outside the example, doubles off-diagonal tiles and adds the tile's sum to norm2[i].
// A diagonal tile multiplies a row block with itself, so its producer loads that block once and both operand
// descriptors point at it (the kernel is bound by the L2 -> shared-memory feed, not by the tensor pipe).
//
// With `ids` given (embedding layers) the first Gram matrix is replaced by the indicator
// [ids_t == ids_t'], which is the Gram matrix of one-hot rows.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer / TMEM owner, warps 2-5 epilogue; persistent
// CTAs, double-buffered accumulators, bounded waits (see common.cuh).
#include "common.cuh"
#include "api.h"

namespace ob {

int make_bf16_map_2d(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld,
                     int box_cols, int box_rows);

constexpr int GH_TILE = 128;
constexpr int GH_BLOCK_K = 64;
constexpr int GH_STAGES = 6;
constexpr int GH_TILE_BYTES = GH_TILE * GH_BLOCK_K * 2;    // 16 KB
constexpr int GH_STAGE_BYTES = 2 * GH_TILE_BYTES;
constexpr int GH_THREADS = 192;
constexpr int GH_SMEM = GH_STAGES * GH_STAGE_BYTES + 256 + 1024;

struct GhostParams {
  int B, T, Da, Dg;      // B segments of (at most) T rows
  const int* ids;        // [rows] or nullptr
  const int* seg;        // [B + 1] row offsets of ragged segments, or nullptr (segment b = rows [b*T, (b+1)*T))
  const int* seg_out;    // [B] accumulator index of every segment, or nullptr (identity)
  float* norm2;          // accumulated with atomics
};

// tile counts of one problem
struct GhostShape {
  int nt, ncb, pairs, wide_items, ka, num_kb;
  __host__ __device__ __forceinline__ explicit GhostShape(const GhostParams& p) {
    nt = (p.T + GH_TILE - 1) / GH_TILE;
    ncb = (nt + 1) / 2;
    pairs = nt * (nt + 1) / 2;
    wide_items = nt * ncb - (nt / 2) * (nt / 2) + ((nt & 1) ? 0 : nt / 2);   // sum over row blocks tb of ncb - tb / 2
    ka = p.ids ? 0 : (p.Da + GH_BLOCK_K - 1) / GH_BLOCK_K;
    num_kb = ka + (p.Dg + GH_BLOCK_K - 1) / GH_BLOCK_K;
  }
};

struct GhostItem {
  int ex, tb, tb2;
};

__device__ __forceinline__ GhostItem ghost_decode(int w, int pairs, int nt) {
  GhostItem it;
  it.ex = w / pairs;
  int r = w % pairs;
  int tb = 0;
  while (r >= nt - tb) {
    r -= nt - tb;
    ++tb;
  }
  it.tb = tb;
  it.tb2 = tb + r;
  return it;
}

template <int CAP>
__global__ void __launch_bounds__(GH_THREADS, 1)
ghost_norm_kernel(const __grid_constant__ TmaBatch<GhostParams, CAP> b) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GH_STAGES * GH_STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + GH_STAGES;
  uint64_t* tmem_full = bars + 2 * GH_STAGES;
  uint64_t* tmem_empty = bars + 2 * GH_STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * GH_STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int total_work = b.total();
  const uint64_t budget = b.wait_budget_ns;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GH_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
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
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0, issued_mask = 0, issued_phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const GhostParams& p = b.p[cur];
      const GhostShape sh(p);
      const GhostItem it = ghost_decode(w - b.start[cur], sh.pairs, sh.nt);
      const int s0 = p.seg ? uniform(p.seg[it.ex]) : it.ex * p.T;
      const int len = p.seg ? uniform(p.seg[it.ex + 1]) - s0 : p.T;
      if (it.tb2 * GH_TILE >= len) continue;                 // tile pair lies outside this (ragged) segment
      const int r1 = s0 + it.tb * GH_TILE, r2 = s0 + it.tb2 * GH_TILE;
      const bool diag = it.tb == it.tb2;
      for (int kb = 0; kb < sh.num_kb; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, b.status, OB_ERR_WAIT_EMPTY, budget)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          // a diagonal tile multiplies a row block with itself: one load serves both operands
          mbar_expect_tx(&full[stage], diag ? GH_TILE_BYTES : GH_STAGE_BYTES);
          uint8_t* dst = smem + stage * GH_STAGE_BYTES;
          const CUtensorMap* map = kb < sh.ka ? &b.map_a[cur] : &b.map_b[cur];
          const int col = (kb < sh.ka ? kb : kb - sh.ka) * GH_BLOCK_K;
          tma_load_2d(dst, map, &full[stage], col, r1);
          if (!diag) tma_load_2d(dst + GH_TILE_BYTES, map, &full[stage], col, r2);
        }
        issued_mask |= 1u << stage;
        issued_phase = (issued_phase & ~(1u << stage)) | (phase << stage);
        if (++stage == GH_STAGES) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok) {
      for (int s = 0; s < GH_STAGES; ++s)
        if (issued_mask & (1u << s)) {
          int dummy_abort = 0;
          mbar_wait(&full[s], (issued_phase >> s) & 1u, &dummy_abort, b.status, OB_ERR_DRAIN, budget);
        }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(GH_TILE, GH_TILE, 0, 0);
    const uint32_t ring = smem_u32(smem);
    int stage = 0, acc_iter = 0;
    uint32_t phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const GhostParams& p = b.p[cur];
      const GhostShape sh(p);
      const GhostItem it = ghost_decode(w - b.start[cur], sh.pairs, sh.nt);
      if (p.seg && it.tb2 * GH_TILE >= uniform(p.seg[it.ex + 1] - p.seg[it.ex])) continue;
      const uint32_t b_off = it.tb == it.tb2 ? 0u : static_cast<uint32_t>(GH_TILE_BYTES);
      const int as = acc_iter & 1;
      if (!mbar_wait_warp(&tmem_empty[as], ((acc_iter >> 1) & 1) ^ 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_EMPTY, budget)) {
        ok = false;
        break;
      }
      tc_fence_after();
      bool ready = false;
      for (int kb = 0; kb < sh.num_kb; ++kb) {
        if (!ready && !mbar_wait_warp(&full[stage], phase, abort_flag, b.status, OB_ERR_WAIT_FULL, budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // K-major, 128-byte swizzle: rows are 128 B apart, 8-row groups 1024 B apart; a k-step of 16 elements moves the start
        // address by 32 B inside the swizzled row.
        const uint32_t t1 = ring + stage * GH_STAGE_BYTES;
        const uint64_t ad = make_smem_desc(t1, 16, 1024, 2), bd = make_smem_desc(t1 + b_off, 16, 1024, 2);
        const uint32_t d_tmem = tmem_base + as * 256 + (kb < sh.ka ? 0 : 128);
        const int next = stage + 1 == GH_STAGES ? 0 : stage + 1;
        const bool peek = kb + 1 < sh.num_kb && mbar_test_wait(&full[next], next == 0 ? phase ^ 1 : phase);
        const bool first = (kb == 0) || (kb == sh.ka);
        if (elect_one()) umma_bf16_kblock<2, 2>(d_tmem, ad, bd, idesc, !first, &empty[stage]);
        ready = __all_sync(0xffffffffu, peek);
        if (++stage == GH_STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (elect_one()) umma_commit(&tmem_full[as]);
      ++acc_iter;
    }
  } else {
    const int q = warp & 3;
    int acc_iter = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const GhostParams& p = b.p[cur];
      const GhostShape sh(p);
      const GhostItem it = ghost_decode(w - b.start[cur], sh.pairs, sh.nt);
      const int s0 = p.seg ? p.seg[it.ex] : it.ex * p.T;
      const int len = p.seg ? p.seg[it.ex + 1] - s0 : p.T;
      if (it.tb2 * GH_TILE >= len) continue;
      const int as = acc_iter & 1;
      if (!mbar_wait(&tmem_full[as], (acc_iter >> 1) & 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_FULL, budget)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int t = it.tb * GH_TILE + q * 32 + lane;
      const int my_id = (p.ids && t < len) ? p.ids[s0 + t] : -1;
      float acc = 0.f;
      for (int c = 0; c < GH_TILE / 32; ++c) {
        float sg[32], sa[32];
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * 256 + c * 32;
        tmem_ld32(taddr + 128, sg);
        if (!p.ids) tmem_ld32(taddr, sa);
        tmem_ld_wait();
        const int tc0 = it.tb2 * GH_TILE + c * 32;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int t2 = tc0 + j;
          float a;
          if (p.ids) {
            const int other = (t2 < len) ? __ldg(p.ids + s0 + t2) : -2;
            a = (other == my_id) ? 1.f : 0.f;
          } else {
            a = sa[j];
          }
          if (t < len && t2 < len) acc += a * sg[j];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[as]);
      ++acc_iter;
      acc = warp_sum(acc);
      if (lane == 0) atomicAdd(p.norm2 + (p.seg_out ? p.seg_out[it.ex] : it.ex), (it.tb == it.tb2 ? 1.f : 2.f) * acc);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------
// Wide variant: one work item is a 128 x 256 block of the T x T Gram matrices (row block tb, column blocks 2cb and
// 2cb+1).  Per k-block the tensor core reads 48 KB of shared memory for 4.2 MFLOP instead of 32 KB for 2.1 MFLOP, which
// lifts the shared-memory bound of the 128 x 128 tiles.  The two Gram tiles fill TMEM (2 x 256 columns), so
// accumulators are single-buffered: the next item's MMAs start when the 8 epilogue warps have drained both tiles.
// Column blocks below the diagonal inside a super-block get weight 0, the diagonal block 1, blocks above it 2.
constexpr int GW_TILE_N = 256;
constexpr int GW_STAGES = 4;
constexpr int GW_A_BYTES = GH_TILE * GH_BLOCK_K * 2;       // 16 KB: rows of the row block
constexpr int GW_B_BYTES = GW_TILE_N * GH_BLOCK_K * 2;     // 32 KB: rows of the two column blocks
constexpr int GW_STAGE_BYTES = GW_A_BYTES + GW_B_BYTES;
constexpr int GW_THREADS = 320;                            // TMA, MMA, 8 epilogue warps
constexpr int GW_SMEM = GW_STAGES * GW_STAGE_BYTES + 256 + 1024;

struct GhostWideItem {
  int ex, tb, cb;
};

// items of one example, ordered by row block: row block tb owns super-blocks cb = tb/2 .. ncb-1
__device__ __forceinline__ GhostWideItem ghost_wide_decode(int w, int per_example, int nt, int ncb) {
  GhostWideItem it;
  it.ex = w / per_example;
  int r = w % per_example;
  int tb = 0;
  while (r >= ncb - (tb >> 1)) {
    r -= ncb - (tb >> 1);
    ++tb;
  }
  it.tb = tb;
  it.cb = (tb >> 1) + r;
  (void)nt;
  return it;
}

template <int CAP>
__global__ void __launch_bounds__(GW_THREADS, 1)
ghost_norm_wide_kernel(const __grid_constant__ TmaBatch<GhostParams, CAP> b) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GW_STAGES * GW_STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + GW_STAGES;
  uint64_t* tmem_full = bars + 2 * GW_STAGES;
  uint64_t* tmem_empty = bars + 2 * GW_STAGES + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * GW_STAGES + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform(static_cast<int>(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int total_work = b.total();
  const uint64_t budget = b.wait_budget_ns;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GW_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(tmem_empty, 8);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&b.map_a[0]);
    tma_prefetch_desc(&b.map_b[0]);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*tmem_slot);

  // segment of example `ex`: first row and length; an item is skipped when its column blocks start past the end
  auto segment = [](const GhostParams& p, int ex, int& s0, int& len) {
    s0 = p.seg ? p.seg[ex] : ex * p.T;
    len = p.seg ? p.seg[ex + 1] - s0 : p.T;
  };

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0, issued_mask = 0, issued_phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const GhostParams& p = b.p[cur];
      const GhostShape sh(p);
      const GhostWideItem it = ghost_wide_decode(w - b.start[cur], sh.wide_items, sh.nt, sh.ncb);
      int s0, len;
      segment(p, it.ex, s0, len);
      s0 = uniform(s0);
      len = uniform(len);
      if (it.tb * GH_TILE >= len || it.cb * GW_TILE_N >= len) continue;
      const int r1 = s0 + it.tb * GH_TILE, r2 = s0 + it.cb * GW_TILE_N;
      const bool diag = (it.tb >> 1) == it.cb;              // the row block is one of the two column blocks
      for (int kb = 0; kb < sh.num_kb; ++kb) {
        if (!mbar_wait_warp(&empty[stage], phase ^ 1, abort_flag, b.status, OB_ERR_WAIT_EMPTY, budget)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_expect_tx(&full[stage], diag ? GW_B_BYTES : GW_STAGE_BYTES);
          uint8_t* dst = smem + stage * GW_STAGE_BYTES;
          const CUtensorMap* map = kb < sh.ka ? &b.map_a[cur] : &b.map_b[cur];
          const int col = (kb < sh.ka ? kb : kb - sh.ka) * GH_BLOCK_K;
          if (!diag) tma_load_2d(dst, map, &full[stage], col, r1);
          tma_load_2d(dst + GW_A_BYTES, map, &full[stage], col, r2);
          tma_load_2d(dst + GW_A_BYTES + GW_A_BYTES, map, &full[stage], col, r2 + GH_TILE);
        }
        issued_mask |= 1u << stage;
        issued_phase = (issued_phase & ~(1u << stage)) | (phase << stage);
        if (++stage == GW_STAGES) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok) {
      for (int s = 0; s < GW_STAGES; ++s)
        if (issued_mask & (1u << s)) {
          int dummy_abort = 0;
          mbar_wait(&full[s], (issued_phase >> s) & 1u, &dummy_abort, b.status, OB_ERR_DRAIN, budget);
        }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(GH_TILE, GW_TILE_N, 0, 0);
    const uint32_t ring = smem_u32(smem);
    int stage = 0, acc_iter = 0;
    uint32_t phase = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const GhostParams& p = b.p[cur];
      const GhostShape sh(p);
      const GhostWideItem it = ghost_wide_decode(w - b.start[cur], sh.wide_items, sh.nt, sh.ncb);
      int s0, len;
      segment(p, it.ex, s0, len);
      s0 = uniform(s0);
      len = uniform(len);
      if (it.tb * GH_TILE >= len || it.cb * GW_TILE_N >= len) continue;
      // on a diagonal super-block the A operand is read from the copy of that row block inside the B operand
      const uint32_t a_off = (it.tb >> 1) == it.cb ? static_cast<uint32_t>(GW_A_BYTES + (it.tb & 1) * GW_A_BYTES) : 0u;
      if (!mbar_wait_warp(tmem_empty, (acc_iter & 1) ^ 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_EMPTY, budget)) {
        ok = false;
        break;
      }
      tc_fence_after();
      bool ready = false;
      for (int kb = 0; kb < sh.num_kb; ++kb) {
        if (!ready && !mbar_wait_warp(&full[stage], phase, abort_flag, b.status, OB_ERR_WAIT_FULL, budget)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // K-major, 128-byte swizzle: rows are 128 B apart, 8-row groups 1024 B apart; a k-step of 16 elements moves the start
        // address by 32 B inside the swizzled row.
        const uint32_t st0 = ring + stage * GW_STAGE_BYTES;
        const uint64_t ad = make_smem_desc(st0 + a_off, 16, 1024, 2), bd = make_smem_desc(st0 + GW_A_BYTES, 16, 1024, 2);
        const uint32_t d_tmem = tmem_base + (kb < sh.ka ? 0 : GW_TILE_N);
        const int next = stage + 1 == GW_STAGES ? 0 : stage + 1;
        const bool peek = kb + 1 < sh.num_kb && mbar_test_wait(&full[next], next == 0 ? phase ^ 1 : phase);
        const bool first = (kb == 0) || (kb == sh.ka);
        if (elect_one()) umma_bf16_kblock<2, 2>(d_tmem, ad, bd, idesc, !first, &empty[stage]);
        ready = __all_sync(0xffffffffu, peek);
        if (++stage == GW_STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (elect_one()) umma_commit(tmem_full);
      ++acc_iter;
    }
  } else {
    const int q = warp & 3;                  // TMEM lane quadrant
    const int half = (warp - 2) >> 2;        // which of the two 128-column blocks
    int acc_iter = 0;
    bool ok = true;
    int cur = 0;
    for (int w = blockIdx.x; ok && w < total_work; w += gridDim.x) {
      cur = b.seek(w, cur);
      const GhostParams& p = b.p[cur];
      const GhostShape sh(p);
      const GhostWideItem it = ghost_wide_decode(w - b.start[cur], sh.wide_items, sh.nt, sh.ncb);
      int s0, len;
      segment(p, it.ex, s0, len);
      if (it.tb * GH_TILE >= len || it.cb * GW_TILE_N >= len) continue;
      if (!mbar_wait(tmem_full, acc_iter & 1, abort_flag, b.status, OB_ERR_WAIT_TMEM_FULL, budget)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int cblk = 2 * it.cb + half;
      const float weight = cblk < it.tb ? 0.f : (cblk == it.tb ? 1.f : 2.f);
      const int t = it.tb * GH_TILE + q * 32 + lane;
      float acc = 0.f;
      if (weight != 0.f && cblk * GH_TILE < len) {
        const int my_id = (p.ids && t < len) ? p.ids[s0 + t] : -1;
        for (int c = 0; c < GH_TILE / 32; ++c) {
          float sg[32], sa[32];
          const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * GH_TILE + c * 32;
          tmem_ld32(taddr + GW_TILE_N, sg);
          if (!p.ids) tmem_ld32(taddr, sa);
          tmem_ld_wait();
          const int tc0 = cblk * GH_TILE + c * 32;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int t2 = tc0 + j;
            float a;
            if (p.ids) {
              const int other = (t2 < len) ? __ldg(p.ids + s0 + t2) : -2;
              a = (other == my_id) ? 1.f : 0.f;
            } else {
              a = sa[j];
            }
            if (t < len && t2 < len) acc += a * sg[j];
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty);
      ++acc_iter;
      acc = warp_sum(acc);
      if (lane == 0 && acc != 0.f) atomicAdd(p.norm2 + (p.seg_out ? p.seg_out[it.ex] : it.ex), weight * acc);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace ob

// 1 (default): 128 x 256 Gram blocks for examples of >= 1024 rows; 2: whenever an example spans two row blocks;
// 0: always 128 x 128 blocks
static int wide_enabled = 1;
extern "C" int ob_ghost_set_wide(int enabled) {
  const int old = wide_enabled;
  wide_enabled = enabled;
  return old;
}

namespace ob {

template <int CAP>
static int launch_ghost(const TmaBatch<GhostParams, CAP>& b, bool wide, int num_sms, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(ghost_norm_kernel<CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, GH_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(ghost_norm_wide_kernel<CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, GW_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  const int total = b.start[b.count];
  if (total <= 0) return 0;
  const int grid = total < num_sms ? total : num_sms;
  if (wide) ghost_norm_wide_kernel<CAP><<<grid, GW_THREADS, GW_SMEM, stream>>>(b);
  else ghost_norm_kernel<CAP><<<grid, GH_THREADS, GH_SMEM, stream>>>(b);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

// The line was drawn where the wide blocks won while one thread issued copies and MMAs (from about 1024 rows per example).  Issued by
// whole warps, the 128 x 128 blocks with their double-buffered accumulators win at 1024 rows as well, and the two are even from about 2048
// on (us, 128 x 128 / 128 x 256: 8 x 1024 x 2048 x 2048 33.7 / 50.5, 8 x 1024 x 2048 x 8192 79 / 116, 4 x 1300 x 2048 x 2048 32 / 50,
// 4 x 2048 x 2048 x 1408 52 / 52, 2 x 4096 x 768 x 3072 114 / 109).
static bool ghost_use_wide(int T) {
  const int nt = (T + GH_TILE - 1) / GH_TILE;
  return wide_enabled == 2 ? nt >= 2 : (wide_enabled == 1 && nt >= 8);
}

// Appends one problem to the batch; 0 on success (also when it has no work).
template <int CAP>
static int ghost_append(TmaBatch<GhostParams, CAP>& b, const ob_ghost_desc& d, bool wide) {
  if (d.B <= 0 || d.T <= 0 || d.Dg <= 0) return 0;
  const long long rows = d.seg ? d.total_rows : static_cast<long long>(d.B) * d.T;
  if (rows <= 0) return 0;
  const int i = b.count;
  int rc = make_bf16_map_2d(&b.map_b[i], d.g, rows, d.Dg, d.ldg, GH_BLOCK_K, GH_TILE);
  if (rc) return rc;
  if (d.ids == nullptr) {
    rc = make_bf16_map_2d(&b.map_a[i], d.a, rows, d.Da, d.lda, GH_BLOCK_K, GH_TILE);
    if (rc) return rc;
  } else {
    b.map_a[i] = b.map_b[i];
  }
  GhostParams& p = b.p[i];
  p.B = d.B; p.T = d.T; p.Da = d.Da; p.Dg = d.Dg;
  p.ids = d.ids; p.seg = d.seg; p.seg_out = d.seg_out; p.norm2 = d.norm2;
  const GhostShape sh(p);
  const long long end = b.start[i] + static_cast<long long>(d.B) * (wide ? sh.wide_items : sh.pairs);
  if (end > 0x7fffffffLL - (1 << 16)) return -23;
  b.start[i + 1] = static_cast<int>(end);
  ++b.count;
  return 0;
}

}  // namespace ob

extern "C" int ob_ghost_norm_batch(const ob_ghost_desc* descs, int count, int* status, double wait_budget_s, int num_sms,
                                   void* stream) {
  using namespace ob;
  // two groups by block shape, each in launches of up to BATCH_CAP problems
  for (int wide = 0; wide < 2; ++wide) {
    TmaBatch<GhostParams, BATCH_CAP> b;
    b.status = status;
    b.wait_budget_ns = static_cast<unsigned long long>(wait_budget_s * 1e9);
    int i = 0;
    while (i < count) {
      b.count = 0;
      b.start[0] = 0;
      for (; i < count && b.count < BATCH_CAP; ++i) {
        if (ghost_use_wide(descs[i].T) != (wide != 0)) continue;
        const int rc = ghost_append(b, descs[i], wide != 0);
        if (rc) return rc;
      }
      if (b.count == 0) continue;
      const int rc = launch_ghost(b, wide != 0, num_sms, static_cast<cudaStream_t>(stream));
      if (rc) return rc;
    }
  }
  return 0;
}
