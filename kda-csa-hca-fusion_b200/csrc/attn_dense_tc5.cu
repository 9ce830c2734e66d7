// Attention core on tcgen05 over contiguous key rows: every visible compressed block, or the subset that a selection list
// names, plus the sliding window (naive_hca, ops_hca.py:139-192; naive_csa, ops_csa.py:1126-1155: joint softmax over
// [compressed entries | window] with the sink logit in the denominator; single KV head, the attended row is key and value
// at once).
//
// Nothing is gathered here, so the products can be real tiles: 128 / HP consecutive queries of a sequence (HP = heads
// padded to 8 or 16) are one item, their heads the 128 rows of the MMA, and the entries they can see are walked in tiles
// of 64 keys.  Two persistent CTAs per SM take the items in turn, the longest first:
//   * Q tile [128 rows x 128 channels] by two TMA copies through a 3-D view {channel, head, token} of the projection
//     output (un-normalised bf16 as stored; 1 / ||q|| is applied to the score row in fp32 -- closer to the reference's
//     fp32 normalisation than a rounded normalised copy); the next item's copy starts as soon as the last score product
//     of this one has read it;
//   * key tiles [64 x 128] by TMA (128-byte swizzle, no multicast) through a 4-stage ring that runs on across items:
//     ceil(ns / 64) tiles of compressed rows, then the window rows of the queries (at most win + 15) in tiles of their own;
//   * S = Q K^T (M = 128, N = 64, K = 128) into one of two tensor-memory buffers; eight softmax warps (two per row
//     quarter, 32 keys of one row per thread) apply the mask of the row -- causal / window range, or the bits of the
//     query's selection list -- and exp(s * scale / ||q|| - shift) with the fixed shift max(|scale|, sink_h) (|s| <=
//     |scale| for unit rows, so partial sums simply add), keep the row sum and write P as bf16 over the scores;
//   * O += P V (M = 128, N = 128, K = 64) with P read from tensor memory and the SAME shared-memory key tile read as an
//     MN-major B operand;
//   * the epilogue divides by the row sum (+ the sink term) and stores 128 contiguous bytes per thread, while the next
//     item's first scores are computed.
// A selection list costs its bit mask (about 6.5 ns an index of a query tile), and a masked entry is computed and dropped.
// That is worth it because a gathered row (attn_mma.cu) is bound by the L2 -> shared-memory path at 256 bytes per (query,
// entry), while here a key tile is read once for 8 or 16 queries; the caller weighs the two (am_mask_us, am_gather_us).
// Bound: the chain of a tile (score product, hand-over, softmax, hand-over, value product), of which two CTAs keep two under
// way on an SM: about 1300 cycles a tile and SM, no unit at its limit (CSA, 16384 tokens, top-k 1024: tensor pipe active
// 43 %, issue slots 49 %).  The score product's N = 64 steps run at the rate of N = 128 ones (62 cycles each, the 128 rows
// of A are read from shared memory either way), the value product at its own (67 cycles, A in tensor memory), so the
// pipe's own limit would be 780 cycles a tile; ex2 needs 512 and the issue slots of the softmax warps ~600.  It was 2200
// with four softmax warps, P in shared memory, one item per CTA and MMAs issued from a branch on the lane number.
// CSA core, 2 x 10007 tokens, top-k 1024: 1132 us gathered -> 327; 4096 tokens, 8 heads, top-k 512: 164 -> 34; HCA core,
// 2 x 32768 tokens: 354 -> 288.
// A masked key multiplies its value row by p = 0, which is no mask for an infinity or a NaN; O shows it (it is not finite
// then), and the CTA redoes the item entry by entry, reading only what each row attends (dt_slow_row).
// Every wait is bounded (status word, see kch_device_status).
#include <cuda.h>
#include <math.h>
#include <stdlib.h>

#include "kch_common.cuh"
#include "tc5_utils.cuh"

#define DT_C 128
#define DT_KT 64                       // keys per tile
#define DT_KSTAGES 4
#define DT_SOFT 256                    // softmax threads
#define DT_THREADS (DT_SOFT + 64)      // + producer warp, MMA warp
#define DT_SPIN (1u << 24)

struct DtArgs {
  int B, T, nh;
  int qtiles;                          // query tiles of a sequence that this launch covers, from token 0
  int n_comp, m, nvis_fixed;
  int64_t t0;
  int64_t comp_batch_rows, win_batch_rows;
  int win_size, win_t0;
  int has_comp, has_win;
  const int32_t* sel; int topk, mask_words;      // selection lists [B*T, topk]; 32-bit mask words per query in shared memory
  const bf16 *q, *comp, *win; int64_t q_ld, win_ld;      // what lies behind the tensor maps (non-finite keys only)
  const void* sink; int sink_dtype;
  float scale;
  bf16* out;
  unsigned int* status;
};

struct DtSmem {
  alignas(1024) bf16 q[2][128 * 64];                 // two 64-channel panels of [128 rows][64]
  alignas(1024) bf16 k[DT_KSTAGES][2][DT_KT * 64];   // per stage: two 64-channel panels of [64 keys][64]
  float part[2][2][128];                             // halves of ||q||^2, and of the row sums
  alignas(8) uint64_t q_full, q_empty;
  uint64_t k_full[DT_KSTAGES], k_empty[DT_KSTAGES];
  uint64_t s_full[2], p_full[2], pv_done;
  uint64_t o_full, o_empty;
  uint32_t tmem;
  uint32_t odd_rows;                                 // 1 + the item in which a row of O was not finite
};

__device__ __forceinline__ void dt_tma_load_3d(void* dst, const void* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_addr_u32(dst)), "l"(map), "r"(smem_addr_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void dt_soft_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DT_SOFT) : "memory"); }
// pairs of fp32 values: one issue slot for two of them (the softmax loop is close to the issue limit)
__device__ __forceinline__ uint64_t dt_pack(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void dt_unpack(uint64_t v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ uint64_t dt_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t dt_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// bits [lo, hi) of a 32-bit word (any lo, hi)
__device__ __forceinline__ uint32_t dt_range(int lo, int hi) {
  lo = max(lo, 0);
  hi = min(hi, 32);
  return hi > lo ? (0xFFFFFFFFu >> (32 - (hi - lo))) << lo : 0u;
}

// One (query, head) row on one warp, reading only the entries it attends: lane l holds channels 4l .. 4l + 3.
__device__ __noinline__ void dt_slow_row(const DtArgs& a, int b, int t, int h, int n, const uint32_t* mask, int lane) {
  auto load4 = [&](const bf16* p, float (&x)[4]) {
    const uint2 v = *reinterpret_cast<const uint2*>(p + 4 * lane);
    x[0] = __uint_as_float(v.x << 16); x[1] = __uint_as_float(v.x & 0xFFFF0000u);
    x[2] = __uint_as_float(v.y << 16); x[3] = __uint_as_float(v.y & 0xFFFF0000u);
  };
  float q[4], o[4] = {0.f, 0.f, 0.f, 0.f}, l = 0.f;
  load4(a.q + ((int64_t)b * a.T + t) * a.q_ld + h * DT_C, q);
  const float nn = warp_sum(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
  const float sink = a.sink ? ld_any(a.sink, h, a.sink_dtype) : -INFINITY, shift = fmaxf(fabsf(a.scale), sink);
  const float qs2 = a.scale / fmaxf(sqrtf(nn), 1e-12f) * 1.4426950408889634f, sh2 = shift * 1.4426950408889634f;
  auto add = [&](const bf16* row) {
    float k[4];
    load4(row, k);
    const float s = warp_sum(q[0] * k[0] + q[1] * k[1] + q[2] * k[2] + q[3] * k[3]);
    const float p = ex2_fast(fmaf(s, qs2, -sh2)), pr = __bfloat162float(__float2bfloat16_rn(p));
    l += p;
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c] = fmaf(pr, k[c], o[c]);
  };
  for (int j = 0; j < n; ++j)
    if (!mask || ((mask[j >> 5] >> (j & 31)) & 1u)) add(a.comp + ((int64_t)b * a.comp_batch_rows + j) * DT_C);
  if (a.has_win)
    for (int j = max(t + a.win_t0 - a.win_size + 1, 0); j <= t + a.win_t0; ++j)
      add(a.win + ((int64_t)b * a.win_batch_rows + j) * a.win_ld);
  const float inv = l > 0.f ? 1.f / (l + (a.sink ? __expf(sink - shift) : 0.f)) : 0.f;
  *reinterpret_cast<uint2*>(a.out + ((int64_t)b * a.T + t) * ((int64_t)a.nh * DT_C) + h * DT_C + 4 * lane) =
      make_uint2(pack2_bf16(o[0] * inv, o[1] * inv), pack2_bf16(o[2] * inv, o[3] * inv));
}

// D [tensor memory] (+)= A [tensor memory: bf16 pairs of the contraction index in each column] x B [shared memory]
__device__ __forceinline__ void dt_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void dt_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

template <int HP, bool SEL>
__global__ void __launch_bounds__(DT_THREADS, 2)
attn_dense_tc5_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap cmap,
                      const __grid_constant__ CUtensorMap wmap, DtArgs a) {
  constexpr int NQ = 128 / HP;                       // queries per tile
  extern __shared__ uint8_t dt_raw[];
  DtSmem& sm = *reinterpret_cast<DtSmem*>(((uintptr_t)dt_raw + 1023) & ~(uintptr_t)1023);
  uint32_t* smask = reinterpret_cast<uint32_t*>(&sm + 1);          // [NQ][mask_words]
  const int tid = threadIdx.x, warp = t5_warp_index(), lane = tid & 31;
  auto nvis_of = [&](int tt) -> int {
    int64_t nv64 = a.nvis_fixed >= 0 ? a.nvis_fixed : (a.m > 0 ? (a.t0 + tt + 1) / a.m : a.n_comp);
    return (int)(nv64 < a.n_comp ? nv64 : a.n_comp);
  };
  struct Item { int b, tq0, nct, ntiles, wrow0; };
  const int items = a.B * a.qtiles;
  auto item_of = [&](int it) -> Item {               // the longest first
    Item x;
    x.b = it % a.B;
    x.tq0 = (a.qtiles - 1 - it / a.B) * NQ;
    const int t_last = min(x.tq0 + NQ, a.T) - 1;
    const int ns = a.has_comp ? nvis_of(t_last) : 0;               // compressed rows to walk: [0, ns)
    int nw = 0;                                                    // window rows to walk: [wrow0, wrow0 + nw)
    x.wrow0 = 0;
    if (a.has_win) { x.wrow0 = max(x.tq0 + a.win_t0 - a.win_size + 1, 0); nw = t_last + a.win_t0 - x.wrow0 + 1; }
    x.nct = (ns + DT_KT - 1) / DT_KT;
    x.ntiles = x.nct + (nw + DT_KT - 1) / DT_KT;
    return x;
  };

  if (tid == 0) {
    mbarrier_init(&sm.q_full, 1);
    mbarrier_init(&sm.q_empty, 1 + DT_SOFT / 32);
    for (int s = 0; s < DT_KSTAGES; ++s) { mbarrier_init(&sm.k_full[s], 1); mbarrier_init(&sm.k_empty[s], 1); }
    for (int i = 0; i < 2; ++i) { mbarrier_init(&sm.s_full[i], 1); mbarrier_init(&sm.p_full[i], DT_SOFT / 32); }
    mbarrier_init(&sm.pv_done, 1);
    mbarrier_init(&sm.o_full, 1);
    mbarrier_init(&sm.o_empty, DT_SOFT / 32);
    sm.odd_rows = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr_u32(&sm.tmem)), "r"(256) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  __syncthreads();
  t5_fence_after();
  const uint32_t tmem = sm.tmem;
  // S buffers at columns 0 and 64 (P of the same tile over their columns 0..15 and 32..47), O at 128..255
  const uint32_t tS = tmem, tO = tmem + 128;
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbarrier_wait_bounded(bar, parity & 1, KCH_STATUS_ATTEND_TILES, DT_SPIN, a.status); };

  if (warp == 8) {
    // ------------------------------ producer: the query tile, then the key tiles -----------------------------------
    if (t5_elect()) {
      bool ok = true;
      int g = 0, c = 0;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++c) {
        const Item x = item_of(it);
        if (c) ok = wait(&sm.q_empty, c - 1);
        if (!ok) break;
        mbarrier_expect_tx(&sm.q_full, 2 * 128 * 64 * 2);
        dt_tma_load_3d(sm.q[0], &qmap, 0, 0, x.b * a.T + x.tq0, &sm.q_full);
        dt_tma_load_3d(sm.q[1], &qmap, 64, 0, x.b * a.T + x.tq0, &sm.q_full);
        for (int i = 0; i < x.ntiles; ++i, ++g) {
          const int st = g % DT_KSTAGES;
          if (g >= DT_KSTAGES) ok = wait(&sm.k_empty[st], g / DT_KSTAGES - 1);
          if (!ok) break;
          mbarrier_expect_tx(&sm.k_full[st], 2 * DT_KT * 64 * 2);
          if (i < x.nct) {
            const int row = (int)((int64_t)x.b * a.comp_batch_rows) + i * DT_KT;
            t5_tma_load_2d(sm.k[st][0], &cmap, 0, row, &sm.k_full[st]);
            t5_tma_load_2d(sm.k[st][1], &cmap, 64, row, &sm.k_full[st]);
          } else {
            const int row = (int)((int64_t)x.b * a.win_batch_rows) + x.wrow0 + (i - x.nct) * DT_KT;
            t5_tma_load_2d(sm.k[st][0], &wmap, 0, row, &sm.k_full[st]);
            t5_tma_load_2d(sm.k[st][1], &wmap, 64, row, &sm.k_full[st]);
          }
        }
      }
    }
  } else if (warp == 9) {
    // ------------------------------ MMA issuer ----------------------------------------------------------------------
    // (issued from a branch on the lane number, the MMAs took 1400 cycles a tile)
    if (t5_elect()) {
      const uint32_t id_s = t5_idesc(DT_KT), id_o = t5_idesc(128) | (1u << 16);
      const uint64_t dq = t5_desc(smem_addr_u32(sm.q[0])), dk = t5_desc(smem_addr_u32(sm.k[0][0]));
      const uint64_t dv = t5_desc_mn(smem_addr_u32(sm.k[0][0]), 8192u);
      bool ok = true;
      int g = 0, c = 0;
      auto issue_pv = [&](int gi, bool first) {        // O (+)= P V of tile gi; frees its key stage and its S / P buffer
        t5_fence_after();
        const uint32_t pa = tS + 64u * (gi & 1);
        const uint64_t vd = dv + (uint64_t)((gi % DT_KSTAGES) * (2 * DT_KT * 64 * 2 >> 4));
#pragma unroll
        for (int ks = 0; ks < DT_KT / 16; ++ks)
          dt_mma_ts(tO, pa + 32u * (ks >> 1) + 8u * (ks & 1), vd + ks * (2048 >> 4), id_o, first && ks == 0 ? 0u : 1u);
        t5_commit(&sm.pv_done);
        t5_commit(&sm.k_empty[gi % DT_KSTAGES]);
      };
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++c) {
        const Item x = item_of(it);
        ok = wait(&sm.q_full, c);
        for (int i = 0; i <= x.ntiles && ok; ++i) {
          if (i < x.ntiles) {
            ok = wait(&sm.k_full[g % DT_KSTAGES], g / DT_KSTAGES);
            // P of two tiles ago lies in this S buffer (at the start of an item the last PV has been issued as well: wait
            // for that one, so that the barrier is never more than one phase ahead)
            if (ok && g >= 2) ok = wait(&sm.pv_done, i ? g - 2 : g - 1);
            if (!ok) break;
            t5_fence_after();
            const uint64_t kd = dk + (uint64_t)((g % DT_KSTAGES) * (2 * DT_KT * 64 * 2 >> 4));
#pragma unroll
            for (int k = 0; k < 8; ++k)                // (a panel of 64 channels, four steps of 16)
              t5_mma(tS + 64u * (g & 1), dq + (k >> 2) * (128 * 64 * 2 >> 4) + 2 * (k & 3), kd + (k >> 2) * (DT_KT * 64 * 2 >> 4) + 2 * (k & 3),
                     id_s, k ? 1u : 0u);
            t5_commit(&sm.s_full[g & 1]);
            ++g;
          }
          if (i == x.ntiles - 1 || x.ntiles == 0) t5_commit(&sm.q_empty);      // the query tile has been read
          if (i == (x.ntiles ? 1 : 0) && c) ok = wait(&sm.o_empty, c - 1);     // the last item's O has been read
          if (i >= 1 && ok) {
            const int gp = i < x.ntiles ? g - 2 : g - 1;                       // tile i - 1 of this item
            ok = wait(&sm.p_full[gp & 1], gp >> 1);
            if (ok) issue_pv(gp, i == 1);
          }
        }
        if (ok) t5_commit(&sm.o_full);
      }
    }
  } else {
    // ------------------------------ softmax + epilogue: half a (query, head) row per thread --------------------------
    const int r = (warp & 3) * 32 + lane, half = warp >> 2, qi = r / HP, h = r % HP;
    const float ascale = fabsf(a.scale);
    float sink = -INFINITY;
    if (a.sink && h < a.nh) sink = ld_any(a.sink, h, a.sink_dtype);
    const float shift = fmaxf(ascale, sink), sh2 = shift * 1.4426950408889634f;
    const float sink_term = a.sink && h < a.nh ? __expf(sink - shift) : 0.f;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t* mrow = smask + qi * a.mask_words + half;
    const int per = (a.topk + 31) / 32;                // runs of 32 entries of a selection list
    bool ok = true;
    int g = 0, c = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++c) {      // (a failed wait keeps every thread in step)
      const Item x = item_of(it);
      const int t = x.tq0 + qi, tw = t + a.win_t0;
      const bool active = t < a.T && h < a.nh;
      const int nvis = (active && a.has_comp) ? nvis_of(t) : 0;
      if (SEL) {                                       // the selection lists of the queries as bit masks
        for (int i = tid; i < NQ * a.mask_words; i += DT_SOFT) smask[i] = 0u;
        dt_soft_sync();
        const int nq = min(NQ, a.T - x.tq0);
        const int32_t* list = a.sel + ((int64_t)x.b * a.T + x.tq0) * a.topk;
        for (int i0 = warp; i0 < nq * per; i0 += 8 * (DT_SOFT / 32)) {      // eight loads in flight per thread
          int id[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * (DT_SOFT / 32), q = i / per, e = (i - q * per) * 32 + lane;
            id[u] = q < nq && e < a.topk ? __ldg(list + (int64_t)q * a.topk + e) : -1;
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int q = (i0 + u * (DT_SOFT / 32)) / per;
            if (id[u] >= 0 && id[u] < nvis_of(x.tq0 + q)) atomicOr(&smask[q * a.mask_words + (id[u] >> 5)], 1u << (id[u] & 31));
          }
        }
      }
      if (ok) ok = wait(&sm.q_full, c);
      // ||q||^2 of this row from the staged tile, a panel per half (chunk k of row r sits at r * 128 + ((k ^ (r & 7)) << 4))
      float ss = 0.f;
      if (ok) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint4 v = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(sm.q[half]) + r * 128 + ((k ^ (r & 7)) << 4));
          const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float x0 = __uint_as_float(w4[e] << 16), x1 = __uint_as_float(w4[e] & 0xFFFF0000u);
            ss = fmaf(x0, x0, ss);
            ss = fmaf(x1, x1, ss);
          }
        }
        __syncwarp();
        if (lane == 0) mbarrier_arrive(&sm.q_empty);
      }
      sm.part[0][half][r] = ss;
      dt_soft_sync();
      ss = sm.part[0][0][r] + sm.part[0][1][r];
      // exp(s * scale / ||q|| - shift) = 2^(s * qs2 - sh2): one FMA and one ex2 per entry
      const float qs2 = a.scale / fmaxf(sqrtf(ss), 1e-12f) * 1.4426950408889634f;
      const uint64_t qs22 = dt_pack(qs2, qs2), sh22 = dt_pack(-sh2, -sh2);
      float l = 0.f;
      for (int i = 0; i < x.ntiles && ok; ++i, ++g) {
        // which of this thread's 32 keys its row attends
        uint32_t mk;
        if (i < x.nct) {
          if (SEL) mk = active ? mrow[2 * i] : 0u;
          else mk = dt_range(0, nvis - i * DT_KT - 32 * half);
        } else {
          const int w0 = x.wrow0 + (i - x.nct) * DT_KT + 32 * half;  // window row of the first of them
          mk = active ? dt_range(tw - a.win_size + 1 - w0, tw + 1 - w0) : 0u;
        }
        ok = wait(&sm.s_full[g & 1], g >> 1);
        if (!ok) break;
        t5_fence_after();
        uint32_t sv[32];
        t5_ld32(tS + 64u * (g & 1) + lane_base + 32u * half, sv);
        t5_wait_ld();
        const bool full = __all_sync(0xffffffffu, mk == 0xFFFFFFFFu);      // no entry of any row masked
        uint64_t sum2 = 0;                               // two partial row sums
        uint32_t o[16];
        if (full) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float x0, x1;
            dt_unpack(dt_fma2(dt_pack(__uint_as_float(sv[2 * e]), __uint_as_float(sv[2 * e + 1])), qs22, sh22), x0, x1);
            const float p0 = ex2_fast(x0), p1 = ex2_fast(x1);
            sum2 = dt_add2(sum2, dt_pack(p0, p1));
            o[e] = pack2_bf16(p0, p1);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float x0, x1;
            dt_unpack(dt_fma2(dt_pack(__uint_as_float(sv[2 * e]), __uint_as_float(sv[2 * e + 1])), qs22, sh22), x0, x1);
            const float p0 = mk & (1u << (2 * e)) ? ex2_fast(x0) : 0.f, p1 = mk & (2u << (2 * e)) ? ex2_fast(x1) : 0.f;
            sum2 = dt_add2(sum2, dt_pack(p0, p1));
            o[e] = pack2_bf16(p0, p1);
          }
        }
        float la, lb;
        dt_unpack(sum2, la, lb);
        l += la + lb;
        dt_st16(tS + 64u * (g & 1) + lane_base + 32u * half, o);       // over the scores this thread has read
        t5_wait_st();
        t5_fence_before();
        __syncwarp();
        if (lane == 0) mbarrier_arrive(&sm.p_full[g & 1]);
      }
      // ---- epilogue -------------------------------------------------------------------------------------------------
      sm.part[1][half][r] = l;
      if (ok) ok = wait(&sm.o_full, c);
      t5_fence_after();
      bf16* orow = a.out + ((int64_t)x.b * a.T + t) * ((int64_t)a.nh * DT_C) + h * DT_C;
      uint32_t ov[2][32];
      if (ok && x.ntiles > 0) {
        t5_ld32(tO + lane_base + 64 * half, ov[0]);
        t5_ld32(tO + lane_base + 64 * half + 32, ov[1]);
        t5_wait_ld();
      } else {
#pragma unroll
        for (int k = 0; k < 32; ++k) ov[0][k] = ov[1][k] = 0u;
      }
      t5_fence_before();
      __syncwarp();
      if (lane == 0) mbarrier_arrive(&sm.o_empty);
      float sum = 0.f;                                 // stays finite unless a value of the row is not
#pragma unroll
      for (int k = 0; k < 32; ++k) sum += __uint_as_float(ov[0][k]) * 0.f + __uint_as_float(ov[1][k]) * 0.f;
      if (active && sum != 0.f) sm.odd_rows = (uint32_t)c + 1u;
      dt_soft_sync();
      const bool odd = sm.odd_rows == (uint32_t)c + 1u;
      l = sm.part[1][0][r] + sm.part[1][1][r];
      // an entry in the row: its p is at least 2^(-2 |scale| log2 e) > 0 unless a large sink makes it vanish, and then
      // the row is 0 either way
      const float inv = l > 0.f ? 1.f / (l + sink_term) : 0.f;
      if (odd) {
        for (int row = warp; row < 128; row += DT_SOFT / 32) {
          const int tr = x.tq0 + row / HP, hr = row % HP;
          if (ok && tr < a.T && hr < a.nh)
            dt_slow_row(a, x.b, tr, hr, a.has_comp ? nvis_of(tr) : 0, SEL ? smask + (row / HP) * a.mask_words : nullptr, lane);
        }
        dt_soft_sync();                                // the masks are read until here
      } else if (active && ok) {
#pragma unroll
        for (int v4 = 0; v4 < 8; ++v4) {
          uint32_t o4[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            o4[e] = pack2_bf16(__uint_as_float(ov[v4 >> 2][8 * (v4 & 3) + 2 * e]) * inv, __uint_as_float(ov[v4 >> 2][8 * (v4 & 3) + 2 * e + 1]) * inv);
          *reinterpret_cast<uint4*>(orow + 64 * half + 8 * v4) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
        }
      }
    }
  }
  __syncthreads();
  if (warp == 8) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
  }
}

// ---- host ---------------------------------------------------------------------------------------------------------
typedef CUresult (*PFN_dt_encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int kch_make_tensor_map_2d_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld_elems,
                                uint32_t box_rows, uint32_t box_cols);
int kch_make_tensor_map_qtile_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint32_t nh, uint64_t ld_elems,
                                   uint32_t box_heads, uint32_t box_rows);

// KCH_OK when launched; -100 when the shape is not this kernel's.  `sel` (optional): selection lists [B*T, topk] of
// distinct indices.  With a list only the queries t < q_end are done (q_end rounded up to a query tile is returned in
// *q_done); the caller's gather kernel takes the rest.
int kch_attend_dense_tc5(const bf16* q, int64_t q_ld, int B, int T, int nh, const bf16* comp, int64_t comp_batch_rows,
                         int n_comp, int m, int64_t t0, int nvis_fixed, const bf16* win, int64_t win_ld,
                         int64_t win_batch_rows, int win_size, int win_t0, const void* sink, int sink_dtype, float scale,
                         bf16* out, const int32_t* sel, int topk, int q_end, int* q_done, cudaStream_t s) {
  if (nh < 1 || nh > 16 || T < 1 || B < 1) return -100;
  if ((q_ld % 8) != 0 || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) return -100;
  if (comp && ((uintptr_t)comp & 15)) return -100;
  if (win && (((uintptr_t)win & 15) || (win_ld % 8) != 0)) return -100;
  if ((int64_t)B * T > 0x7FFFFFF0LL || (int64_t)B * comp_batch_rows > 0x7FFFFFF0LL || (int64_t)B * win_batch_rows > 0x7FFFFFF0LL) return -100;
  const bool has_comp = comp != nullptr && n_comp > 0, has_win = win != nullptr && win_size > 0;
  if (!has_comp && !has_win) return -100;
  CUtensorMap qmap, cmap, wmap;
  const int HP = nh <= 8 ? 8 : 16, NQ = 128 / HP;
  if (kch_make_tensor_map_qtile_bf16(&qmap, q, (uint64_t)B * T, (uint32_t)nh, (uint64_t)q_ld, (uint32_t)HP, (uint32_t)NQ) != KCH_OK) return -100;
  // a map that is not used still has to be a valid object: point it at the other operand
  const bf16* cbase = has_comp ? comp : win;
  const uint64_t crows = has_comp ? (uint64_t)B * comp_batch_rows : (uint64_t)B * win_batch_rows;
  const uint64_t cld = has_comp ? DT_C : (uint64_t)win_ld;
  if (kch_make_tensor_map_2d_bf16(&cmap, cbase, crows, DT_C, cld, DT_KT, 64) != KCH_OK) return -100;
  const bf16* wbase = has_win ? win : comp;
  const uint64_t wrows = has_win ? (uint64_t)B * win_batch_rows : (uint64_t)B * comp_batch_rows;
  const uint64_t wld = has_win ? (uint64_t)win_ld : DT_C;
  if (kch_make_tensor_map_2d_bf16(&wmap, wbase, wrows, DT_C, wld, DT_KT, 64) != KCH_OK) return -100;
  DtArgs a;
  a.B = B; a.T = T; a.nh = nh; a.n_comp = has_comp ? n_comp : 0; a.m = m; a.nvis_fixed = nvis_fixed; a.t0 = t0;
  a.comp_batch_rows = comp_batch_rows; a.win_batch_rows = win_batch_rows; a.win_size = has_win ? win_size : 0; a.win_t0 = win_t0;
  a.has_comp = has_comp ? 1 : 0; a.has_win = has_win ? 1 : 0;
  a.sink = sink; a.sink_dtype = sink_dtype; a.scale = scale; a.out = out;
  a.status = kch_status_device_ptr();
  KCH_REQUIRE(a.status != nullptr, "kch_attend: cannot resolve the device status word");
  a.q = q; a.comp = comp; a.win = win; a.q_ld = q_ld; a.win_ld = win_ld;
  a.sel = has_comp ? sel : nullptr; a.topk = topk;
  if (sel && q_end < T) {
    a.qtiles = (q_end + NQ - 1) / NQ;
    if (a.qtiles * NQ < T) T = a.qtiles * NQ;                    // (only the count of tiles below uses it)
  }
  a.qtiles = (T + NQ - 1) / NQ;
  if (q_done) *q_done = T;
  // the mask covers the blocks that the last of these queries sees, in whole key tiles
  int64_t nv = nvis_fixed >= 0 ? nvis_fixed : (m > 0 ? (t0 + T) / m : n_comp);
  if (nv > n_comp) nv = n_comp;
  a.mask_words = a.sel ? 2 * (int)((nv + DT_KT - 1) / DT_KT) : 0;
  const size_t smem = sizeof(DtSmem) + 1024 + (size_t)NQ * a.mask_words * 4;
  if (smem > 113 * 1024) return -100;                            // two CTAs per SM, or the gather kernel
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    KCH_CUDA_OK(cudaGetDevice(&dev));
    KCH_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  const int64_t tiles = (int64_t)B * a.qtiles;
  const unsigned ctas = (unsigned)(tiles < 2 * sms ? tiles : 2 * sms);
#define DT_GO(HP_, SEL_)                                                                                                \
  do {                                                                                                                  \
    KCH_CUDA_OK(cudaFuncSetAttribute(attn_dense_tc5_kernel<HP_, SEL_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    attn_dense_tc5_kernel<HP_, SEL_><<<ctas, DT_THREADS, smem, s>>>(qmap, cmap, wmap, a);                               \
  } while (0)
  if (HP == 8) { if (a.sel) DT_GO(8, true); else DT_GO(8, false); }
  else { if (a.sel) DT_GO(16, true); else DT_GO(16, false); }
#undef DT_GO
  KCH_LAUNCH_OK();
  return KCH_OK;
}
