// Sequential stage of chunked KDA on the fifth-generation tensor cores (tcgen05), state resident in
// tensor memory.  Same arithmetic as kda_scan_mma_kernel (naive_chunk_kda, ops_kda.py:509-535):
//   vt^T = u^T - S^T w^T ;  o^T = S^T qg^T + vt^T Aqk^T ;  S^T <- S^T diag(dl) + vt^T kg
// with every product as hi*hi + lo*hi + hi*lo of two-term bf16 splits and fp32 accumulation.
//
// One CTA per (batch, value head); S^T [128 v x 128 k] fp32 is the accumulator of the update product and never leaves
// tensor memory between chunks; the bf16 hi / lo images of S^T and of vt^T are A operands there as well (an A operand in
// tensor memory needs no proxy fence, which cost 300 cycles at each of a chunk's four conversions, and frees the shared
// memory for a second [w; qg] stage).  Per chunk (the dependent chain is S -> D1w -> vt -> S):
//   vector warps : read S^T (tcgen05.ld, one row v per thread), write its hi / lo images, one 64-channel panel at a time,
//                  and S^T diag(dl) back
//   MMA thread   : [D1w | D1q] = S^T [w; qg]^T (N = 64 + 64 tokens, K = 128 channels), starting on a panel as soon as it
//                  is there (D1q apart, behind D1w, slowed the vector warps' own tensor-memory accesses by as much)
//   vector warps : vt^T = u^T - D1w -> hi / lo images, 16 tokens at a time
//   MMA thread   : S^T += vt^T kg (N = 128, kg read as an MN-major operand, i.e. in its natural [token][channel]
//                  layout), then D1q += vt^T Aqk^T (N = 64); K = 64 tokens
//   vector warps : o^T = D1q of the chunk before -> bf16 -> global, while the products of this one run (the [D1w | D1q]
//                  block is double-buffered)
// A producer warp streams the chunk's operand tiles (written by the prepare kernel in this layout) with 1-D bulk copies:
// [w; qg] into two stages, a chunk ahead; u^T with dl, and kg with Aqk, into one stage each, as the chunk before releases it.
// Every wait is a bounded mbarrier wait that records a status code and leaves the loops.
// Bound: the dependent chain, 4200 to 4400 cycles a chunk, the tensor pipe active for two thirds of them: 1540 of D1 and ~900
// of the update, the rest the two conversions and four hand-overs of ~250 cycles.  It was 5300 with the images in shared
// memory and o stored two bytes at a time ahead of vt (1 x 8192 tokens, 16 heads, both stages: 526 -> 433 us).
//
// Workspace record of a chunk in this layout (written by kda_prepare_mma_kernel when PrepArgs::umma is set):
//   0      [w; qg] hi: two 64-channel panels of [128 rows][64] bf16 (rows 0..63 w, 64..127 qg), 128-byte swizzle
//   32768  [w; qg] lo
//   65536  Aqk hi [64][64], lo
//   81920  kg hi: two 64-channel panels of [64 tokens][64] bf16;  98304 kg lo
//   114688 u^T fp32 as [token / 32][token / 4 % 8][v][token % 4], then dl [128] fp32
#include <math.h>
#include <stdlib.h>

#include "mma_utils.cuh"
#include "tc5_utils.cuh"

#define T5_THREADS 320
#define T5_SPIN (1u << 26)
// workspace record of one chunk (offsets shared with kda_mma.cu)
#define T5_OFF_WHI 0
#define T5_OFF_WLO 16384
#define T5_OFF_QHI 32768
#define T5_OFF_QLO 49152
#define T5_OFF_AQK 65536
#define T5_OFF_KHI 81920
#define T5_OFF_KLO 98304
#define T5_OFF_U 114688
#define T5_U_SLICE 16896
#define T5_CHUNK_BYTES (T5_OFF_U + 2 * T5_U_SLICE)

struct T5Args {
  const uint8_t* ws;
  const float* S0;
  bf16* o;
  float* S_out;
  unsigned int* status;
  int T, HV, NT;                     // T: tokens from the first chunk of this launch to the end of the sequence
  int Tb;                            // tokens between consecutive batch entries (the whole sequence length)
  int o_vec;                         // o is 8-byte aligned
  // A sequence in `nseg` segments of `per` chunks, scanned side by side (0: the whole sequence in one CTA, see the host part)
  int nseg, per, pass;
  float* starts;                     // [nseg][B * HV] states at the start of each segment, [k][v]
  float* trans;                      // [nseg][B * HV] transition of each segment, transposed: [k'][k]
  const uint32_t* serial;            // [B * HV] != 0: a transition expands, segments 1 .. nseg - 1 are one chain
};

// shared-memory map (bytes, 1024-aligned operand tiles)
#define T5_TW 0                      // two stages of [w; qg] hi panels, lo panels: 4 x 16384 each
#define T5_TK 131072                 // kg hi [64][128] (16384), lo (16384)
#define T5_TA (T5_TK + 32768)        // Aqk hi [64][64] (8192), lo (8192)
#define T5_TU (T5_TA + 16384)        // u^T and dl as in the record (straight from global memory they came 500 cycles too late)
#define T5_BARS (T5_TU + 32768 + 512)
#define T5_TOTAL (T5_BARS + 128)
// tensor-memory columns
#define T5_CS 0                      // S^T fp32
#define T5_CSA 128                   // S^T images: hi 64 columns (two channels each), lo 64
#define T5_CD 256                    // [D1w | D1q] of even chunks, of odd chunks; once a vector warp has read its 32 columns
                                     // of D1w, the images of the same tokens of vt^T lie there: hi 16, lo 16 columns
static_assert(T5_TOTAL + 1024 <= 232448, "shared memory of the KDA scan");

__device__ __forceinline__ void t5_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
template <int N>
__device__ __forceinline__ void t5_stn(uint32_t taddr, const uint32_t* r) {
  if constexpr (N == 16)
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
  else
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// SEG: segments of a sequence side by side (see the host part).  A kernel of its own: with the choices of a segment made at run
// time, the chain of a whole sequence took 1.5 us more before its first chunk and 1 % of both stages (64 heads: 2 chunks
// 29.8 us, 31.6 with them; 128 chunks 842, 850).
template <bool SEG>
__global__ void __launch_bounds__(T5_THREADS, 1) kda_scan_tc5_kernel(T5Args a) {
  extern __shared__ uint8_t t5_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>(((uintptr_t)t5_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + T5_BARS);
  uint64_t *sa_ready0 = bars + 0, *sa_ready1 = bars + 1, *va_ready0 = bars + 2, *va_ready1 = bars + 3, *d1_full = bars + 4,
           *s_full = bars + 5, *o_full = bars + 6;
  uint64_t *w_full = bars + 7, *w_empty = bars + 9, *k_full = bars + 11, *k_empty = bars + 12, *u_full = bars + 13, *u_empty = bars + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  const int hv = blockIdx.x, b = blockIdx.y;
  const int warp = t5_warp_index(), lane = threadIdx.x & 31;
  const int64_t bh = (int64_t)b * a.HV + hv;
  constexpr uint32_t TMEM_COLS = 512;
  // this CTA's run of chunks, what it starts from and what it leaves behind
  int n0 = 0, NT = a.NT;
  const float* S0 = a.S0 ? a.S0 + bh * (128 * 128) : nullptr;
  float* S_out = a.S_out ? a.S_out + bh * (128 * 128) : nullptr;
  bool out_wanted = true, values = true;
  if constexpr (SEG) {
    const int z = blockIdx.z, seg = a.pass == 1 ? (z + 1) / 2 : z + 1;
    const int64_t slot = (int64_t)gridDim.x * gridDim.y;
    n0 = seg * a.per;
    NT = min(a.per, a.NT - n0);
    if (a.pass == 1) {
      S_out = a.starts + ((int64_t)(seg + 1) * slot + bh) * (128 * 128);
      if (seg > 0) {
        S0 = nullptr;
        out_wanted = false;
        values = z & 1;
        if (!values) S_out = a.trans + ((int64_t)seg * slot + bh) * (128 * 128);
      }
    } else {
      const bool chain = a.serial[bh] != 0u;
      if (chain && seg > 1) return;
      S0 = a.starts + ((int64_t)seg * slot + bh) * (128 * 128);
      if (chain) NT = a.NT - n0;
      else if (seg + 1 < a.nseg) S_out = nullptr;
    }
  }
  // (constants where the sequence is one chain); with_u false: rows of the identity instead of values
  const bool with_o = !SEG || out_wanted, with_u = !SEG || values;
  const int T_left = a.T - n0 * 64;                              // tokens from this run's first chunk to the end of the sequence
  const uint8_t* wsb = a.ws + (bh * a.NT + n0) * (int64_t)T5_CHUNK_BYTES;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbarrier_init(w_full + i, 1); mbarrier_init(w_empty + i, 1); }
    mbarrier_init(k_full, 1); mbarrier_init(k_empty, 1); mbarrier_init(u_full, 1); mbarrier_init(u_empty, 8);
    mbarrier_init(sa_ready0, 8); mbarrier_init(sa_ready1, 8); mbarrier_init(d1_full, 1); mbarrier_init(va_ready0, 8); mbarrier_init(va_ready1, 8); mbarrier_init(s_full, 1); mbarrier_init(o_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  __syncthreads();
  t5_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem + T5_CS, tSA = tmem + T5_CSA, tDD = tmem + T5_CD;

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    if (t5_elect()) {
      for (int n = 0; n < NT; ++n) {
        const uint8_t* src = wsb + (int64_t)n * T5_CHUNK_BYTES;
        const int st = n & 1;
        const uint32_t ph = (uint32_t)n & 1;
        if (!mbarrier_wait_bounded(w_empty + st, ((uint32_t)(n >> 1) & 1) ^ 1, 41, T5_SPIN, a.status)) break;
        mbarrier_expect_tx(w_full + st, with_o ? 4 * 16384 : 4 * 8192);
        if (with_o) {
          bulk_copy_g2s(sm + T5_TW + st * 65536, src + T5_OFF_WHI, 4 * 16384, w_full + st);   // [w; qg] hi panels, then lo panels
        } else {                                                                              // w only
          for (int i = 0; i < 4; ++i) bulk_copy_g2s(sm + T5_TW + st * 65536 + i * 16384, src + T5_OFF_WHI + i * 16384, 8192, w_full + st);
        }
        if (!mbarrier_wait_bounded(u_empty, ph ^ 1, 54, T5_SPIN, a.status)) break;
        mbarrier_expect_tx(u_full, with_u ? 32768 + 512 : 512);                               // u^T, dl
        if (with_u) bulk_copy_g2s(sm + T5_TU, src + T5_OFF_U, 32768 + 512, u_full);
        else bulk_copy_g2s(sm + T5_TU + 32768, src + T5_OFF_U + 32768, 512, u_full);
        if (!mbarrier_wait_bounded(k_empty, ph ^ 1, 42, T5_SPIN, a.status)) break;
        mbarrier_expect_tx(k_full, with_o ? 2 * 16384 + 16384 : 2 * 16384);
        bulk_copy_g2s(sm + T5_TK, src + T5_OFF_KHI, 2 * 16384, k_full);                       // kg hi, lo
        if (with_o) bulk_copy_g2s(sm + T5_TA, src + T5_OFF_AQK, 16384, k_full);               // Aqk hi, lo
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (t5_elect()) {
      const uint32_t id64 = t5_idesc(64), id128 = t5_idesc(128), id128mn = t5_idesc(128) | (1u << 16);
      const uint64_t dw0 = t5_desc(smem_addr_u32(sm + T5_TW)), da0 = t5_desc(smem_addr_u32(sm + T5_TA));
      const uint64_t dk0 = t5_desc_mn(smem_addr_u32(sm + T5_TK));
      for (int n = 0; n < NT; ++n) {
        const uint32_t ph = (uint32_t)n & 1, sph = (uint32_t)(n >> 1) & 1;
        const int st = n & 1;
        const uint64_t dw = dw0 + (uint64_t)(st * 65536 >> 4);
        const uint32_t tD = tDD + 128u * ph;                 // [D1w | D1q] of this chunk; vt^T images over D1w
        if (!mbarrier_wait_bounded(w_full + st, sph, 44, T5_SPIN, a.status)) break;
        // [D1w | D1q] = S^T [w; qg]^T (D1w alone without an output), a 64-channel panel at a time: terms (S hi, x hi),
        // (S lo, x hi), (S hi, x lo)
        bool ok = true;
#pragma unroll
        for (int pan = 0; pan < 2; ++pan) {
          if (!mbarrier_wait_bounded(pan ? sa_ready1 : sa_ready0, ph, 43, T5_SPIN, a.status)) { ok = false; break; }
          t5_fence_after();
#pragma unroll
          for (int term = 0; term < 3; ++term)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              t5_mma_ts(tD, tSA + (term == 1 ? 64u : 0u) + 32u * pan + 8u * ks, dw + ((term == 2 ? 32768u : 0u) + pan * 16384u >> 4) + 2 * ks,
                        with_o ? id128 : id64, (pan | term | ks) ? 1u : 0u);
        }
        if (!ok) break;
        t5_commit(d1_full);
        t5_commit(w_empty + st);
        if (!mbarrier_wait_bounded(k_full, ph, 46, T5_SPIN, a.status)) break;
        // S^T += vt^T kg   (N = 128 channels, kg read in place as an MN-major operand; K = 64 tokens, the 16-token
        // steps {0, 2} first, {1, 3} second, as the vector warps finish them)
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          if (!mbarrier_wait_bounded(part ? va_ready1 : va_ready0, ph, 45, T5_SPIN, a.status)) { ok = false; break; }
          t5_fence_after();
#pragma unroll
          for (int term = 0; term < 3; ++term)
#pragma unroll
            for (int k2 = 0; k2 < 2; ++k2) {
              const int ks = 2 * k2 + part;
              t5_mma_ts(tS, tD + (term == 1 ? 16u : 0u) + 32u * (ks >> 1) + 8u * (ks & 1), dk0 + ((term == 2 ? 16384u : 0u) + ks * 2048u >> 4), id128mn, 1u);
            }
        }
        if (!ok) break;
        t5_commit(s_full);
        if (with_o) {
          // D1q += vt^T Aqk^T
#pragma unroll
          for (int term = 0; term < 3; ++term)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              t5_mma_ts(tD + 64, tD + (term == 1 ? 16u : 0u) + 32u * (ks >> 1) + 8u * (ks & 1), da0 + ((term == 2 ? 8192u : 0u) >> 4) + 2 * ks, id64, 1u);
          if (n + 1 == NT) t5_commit(o_full);
        }
        t5_commit(k_empty);
      }
    }
  } else {
    // ------------------------------ vector warps ------------------------------
    const int quarter = warp & 3, sub = (warp - 2) >> 2;
    const int v = quarter * 32 + lane;                         // this thread's row of S^T, D1w, D1q
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    uint32_t r[32], r2[32], ro[32];
    // initial state into tensor memory: this warp owns channels 32*sub .. +31 of each 64-channel panel of row v
#pragma unroll
    for (int pan = 0; pan < 2; ++pan) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int kc = 64 * pan + 32 * sub + j;
        r[j] = S0 ? __float_as_uint(S0[(int64_t)kc * 128 + v]) : (!with_u && kc == v ? __float_as_uint(1.f) : 0u);
      }
      t5_st32(tS + lane_base + 64 * pan + 32 * sub, r);
    }
    t5_wait_st();
    // o^T rows (this thread: value column v, 32 tokens in `ro`) -> o[token][v].  A 4 x 4 transpose inside each group of four
    // lanes turns 32 stores of 2 bytes per thread into 8 of 8 bytes (64 contiguous bytes per warp and token either way):
    // with the former the phase took 1860 cycles of a chunk's 5250.
    auto store_o = [&](int tok0) {
      uint32_t p[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t own = pack2_bf16(__uint_as_float(ro[2 * i]), __uint_as_float(ro[2 * i + 1]));     // tokens 2i, 2i + 1
        const uint32_t oth = __shfl_xor_sync(0xffffffffu, own, 1);
        p[i] = (lane & 1) ? __byte_perm(oth, own, 0x7632) : __byte_perm(own, oth, 0x5410);               // columns v & ~1, + 1 of token 2i + (lane & 1)
      }
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, (lane & 2) ? p[2 * m] : p[2 * m + 1], 2);
        const uint2 o4 = (lane & 2) ? make_uint2(got, p[2 * m + 1]) : make_uint2(p[2 * m], got);
        const int t = tok0 + 32 * sub + 4 * m + (lane & 3);
        bf16* dst = a.o + (((int64_t)b * a.Tb + n0 * 64 + t) * a.HV + hv) * 128 + (v & ~3);
        if (t < T_left && a.o_vec) *reinterpret_cast<uint2*>(dst) = o4;
        else if (t < T_left) {
          const uint32_t w2[2] = {o4.x, o4.y};
          for (int c = 0; c < 4; ++c) reinterpret_cast<uint16_t*>(dst)[c] = (uint16_t)(w2[c >> 1] >> (16 * (c & 1)));
        }
      }
    };
    bool ok = true;
    const float* dl = reinterpret_cast<const float*>(sm + T5_TU + 32768);
    const float4* up = reinterpret_cast<const float4*>(sm + T5_TU) + sub * 8 * 128 + v;       // [sub][j][v] float4
    for (int n = 0; n < NT && ok; ++n) {
      const uint32_t ph = (uint32_t)n & 1;
      if (n > 0 && !mbarrier_wait_bounded(s_full, ph ^ 1, 47, T5_SPIN, a.status)) { ok = false; break; }
      t5_fence_after();
      // ---- S^T -> bf16 hi / lo images, panel 0 then panel 1; then S^T diag(dl) back to tensor memory -------------------
      t5_ld32(tS + lane_base + 32 * sub, r);
      t5_ld32(tS + lane_base + 64 + 32 * sub, r2);
      t5_wait_ld();
#pragma unroll
      for (int pan = 0; pan < 2; ++pan) {
        uint32_t (&rr)[32] = pan ? r2 : r;
        uint32_t h[16], l[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) split2_bf16(__uint_as_float(rr[2 * e]), __uint_as_float(rr[2 * e + 1]), h[e], l[e]);
        t5_stn<16>(tSA + lane_base + 32 * pan + 16 * sub, h);
        t5_stn<16>(tSA + lane_base + 64 + 32 * pan + 16 * sub, l);
        t5_wait_st();
        t5_fence_before();
        __syncwarp();
        if (lane == 0) mbarrier_arrive(pan ? sa_ready1 : sa_ready0);
      }
      if (!mbarrier_wait_bounded(u_full, ph, 48, T5_SPIN, a.status)) { ok = false; break; }      // u^T and dl have landed
#pragma unroll
      for (int pan = 0; pan < 2; ++pan) {
        uint32_t (&rr)[32] = pan ? r2 : r;
        const int kc0 = 64 * pan + 32 * sub;                   // first channel of these 32 columns
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 d4 = *reinterpret_cast<const float4*>(dl + kc0 + j);
          rr[j] = __float_as_uint(__uint_as_float(rr[j]) * d4.x);
          rr[j + 1] = __float_as_uint(__uint_as_float(rr[j + 1]) * d4.y);
          rr[j + 2] = __float_as_uint(__uint_as_float(rr[j + 2]) * d4.z);
          rr[j + 3] = __float_as_uint(__uint_as_float(rr[j + 3]) * d4.w);
        }
        t5_st32(tS + lane_base + kc0, rr);
      }
      // ---- vt^T = u^T - D1w -> images, 16 tokens at a time -------------------------------------------------------
      t5_wait_st();                                             // the decayed S^T is in place before the update may start
      if (!mbarrier_wait_bounded(d1_full, ph, 49, T5_SPIN, a.status)) { ok = false; break; }
      t5_fence_after();
      t5_ld32(tDD + 128u * ph + lane_base + 32 * sub, r);
      float u[32];
#pragma unroll
      for (int j = 0; j < 8; ++j) { const float4 x = with_u ? up[j * 128] : make_float4(0.f, 0.f, 0.f, 0.f); u[4 * j] = x.x; u[4 * j + 1] = x.y; u[4 * j + 2] = x.z; u[4 * j + 3] = x.w; }
      t5_wait_ld();
#pragma unroll
      for (int q = 0; q < 2; ++q) {                             // 16 tokens: 8 columns of each image
        uint32_t h[8], l[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
          split2_bf16(u[16 * q + 2 * e] - __uint_as_float(r[16 * q + 2 * e]), u[16 * q + 2 * e + 1] - __uint_as_float(r[16 * q + 2 * e + 1]),
                      h[e], l[e]);
        t5_stn<8>(tDD + 128u * ph + lane_base + 32 * sub + 8 * q, h);
        t5_stn<8>(tDD + 128u * ph + lane_base + 32 * sub + 16 + 8 * q, l);
        t5_wait_st();
        t5_fence_before();
        __syncwarp();
        if (lane == 0) mbarrier_arrive(q ? va_ready1 : va_ready0);
      }
      if (lane == 0) mbarrier_arrive(u_empty);
      // ---- o^T of the previous chunk -> global, while the products of this one run (its D1q is the other buffer) --------
      // Its products lie before D1 of this chunk in the MMA thread's order, so the wait for d1_full above covers them.  A barrier
      // of their own could not be waited for here: the MMA thread has what it needs for the products of this chunk, and a warp
      // that it overtook by one phase would wait for a phase that nothing completes.
      if (n > 0 && with_o) {
        t5_ld32(tDD + 128u * (ph ^ 1) + 64 + lane_base + 32 * sub, ro);
        t5_wait_ld();
        store_o((n - 1) * 64);
      }
    }
    // the last products must have finished before o^T and the state are read and tensor memory is released
    if (ok && NT > 0 && !mbarrier_wait_bounded(s_full, (uint32_t)(NT - 1) & 1, 51, T5_SPIN, a.status)) ok = false;
    if (ok && NT > 0 && with_o && !mbarrier_wait_bounded(o_full, 0, 53, T5_SPIN, a.status)) ok = false;
    if (ok && NT > 0) {
      t5_fence_after();
      if (with_o) {
        t5_ld32(tDD + 128u * ((uint32_t)(NT - 1) & 1) + 64 + lane_base + 32 * sub, ro);
        t5_wait_ld();
        store_o((NT - 1) * 64);
      }
      if (S_out) {
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 32) {
          t5_ld32(tS + lane_base + 64 * sub + c0, r);
          t5_wait_ld();
          if (with_u) {
#pragma unroll
            for (int j = 0; j < 32; ++j) S_out[(int64_t)(64 * sub + c0 + j) * 128 + v] = __uint_as_float(r[j]);
          } else {                                               // a transition, transposed: the rows that the join reads side by side
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              *reinterpret_cast<uint4*>(S_out + (int64_t)v * 128 + 64 * sub + c0 + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
          }
        }
      }
    }
  }
  t5_fence_before();
  __syncthreads();
  if (warp == 1) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// ---- host ----------------------------------------------------------------------------------------------------
bool kch_kda_scan_tc5_enabled() {
  // default; KCH_KDA_SCAN=m selects the mma.sync scan (kda_scan_mma_kernel) for comparison
  static const bool on = [] { const char* e = getenv("KCH_KDA_SCAN"); return !(e && e[0] == 'm'); }();
  return on;
}

// ---- segments of a sequence side by side -----------------------------------------------------------------------------
// The update of a chunk is linear in the state, so a segment of chunks maps its start state to S -> M S + b.  Pass 1 finds b
// (the scan from a zero state) and M (the scan of the identity's rows, without values) of every segment but the first, which
// is scanned as it is, and the last, whose end nobody needs; the join walks the segments' start states; pass 2 scans all but
// the first segment from their start states.  Chain: 2 / nseg of the sequence's chunks instead of all of them, on
// (1 + 2 (nseg - 2)) CTAs a head instead of one.  All of it in the arithmetic of the plain scan, the join in fp32.
// A transition that expands (an entry beyond 4, or not finite: a gate that grows, keys far from unit length) could lose in M
// what the plain scan keeps; the segments of such a head run as one chain in pass 2.
// 1 x 8192 tokens, 16 heads, 6 segments: the scan alone 290 us as one chain; two passes of ~60 us and 19 of the join.
// km_split (kda_mma.cu) holds the rule.
// A CTA of the join walks the segments for 16 columns of a head's state; the transitions (64 KB each) are copied two steps ahead.
#define KJ_COLS 16
#define KJ_SMEM (2 * 128 * 128 * 4 + 128 * KJ_COLS * 4)
__global__ void __launch_bounds__(256) kda_join_kernel(float* starts, const float* trans, uint32_t* serial, int nseg) {
  extern __shared__ __align__(16) float kj_smem[];
  float4* sS = reinterpret_cast<float4*>(kj_smem + 2 * 128 * 128);      // [128][KJ_COLS / 4]
  const int64_t slot = (int64_t)gridDim.y * gridDim.z, bh = (int64_t)blockIdx.z * gridDim.y + blockIdx.y;
  const int tid = threadIdx.x, k = tid & 127, half = tid >> 7, c0 = blockIdx.x * KJ_COLS + 8 * half;
  const uint32_t sm32 = smem_addr_u32(kj_smem);
  chain_wait();
  auto fetch = [&](int s) {
    if (s + 1 < nseg) {
      const float* src = trans + ((int64_t)s * slot + bh) * (128 * 128);
      const uint32_t dst = sm32 + (uint32_t)(s & 1) * 65536u;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (tid + 256 * i) * 16u), "l"(src + (tid + 256 * i) * 4) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(1);
  fetch(2);
  {
    const float4* p = reinterpret_cast<const float4*>(starts + (slot + bh) * (128 * 128) + (int64_t)k * 128 + c0);
    sS[k * (KJ_COLS / 4) + 2 * half] = p[0];
    sS[k * (KJ_COLS / 4) + 2 * half + 1] = p[1];
  }
  bool expands = false;
  for (int s = 1; s + 1 < nseg; ++s) {
    float4* out = reinterpret_cast<float4*>(starts + ((int64_t)(s + 1) * slot + bh) * (128 * 128) + (int64_t)k * 128 + c0);
    const float4 b0 = out[0], b1 = out[1];
    float acc[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float* mt = kj_smem + (s & 1) * (128 * 128) + k;
    float big = 0.f;
#pragma unroll 16
    for (int j = 0; j < 128; ++j) {
      const float m = mt[j * 128];
      big = fmaxf(big, fabsf(m));
      expands |= m != m;
      const float4 x = sS[j * (KJ_COLS / 4) + 2 * half], y = sS[j * (KJ_COLS / 4) + 2 * half + 1];
      acc[0] = fmaf(m, x.x, acc[0]); acc[1] = fmaf(m, x.y, acc[1]); acc[2] = fmaf(m, x.z, acc[2]); acc[3] = fmaf(m, x.w, acc[3]);
      acc[4] = fmaf(m, y.x, acc[4]); acc[5] = fmaf(m, y.y, acc[5]); acc[6] = fmaf(m, y.z, acc[6]); acc[7] = fmaf(m, y.w, acc[7]);
    }
    expands |= big > 4.f;
    __syncthreads();
    fetch(s + 2);
    const float4 n0 = make_float4(acc[0], acc[1], acc[2], acc[3]), n1 = make_float4(acc[4], acc[5], acc[6], acc[7]);
    out[0] = sS[k * (KJ_COLS / 4) + 2 * half] = n0;
    out[1] = sS[k * (KJ_COLS / 4) + 2 * half + 1] = n1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  expands = __syncthreads_or(expands);             // every CTA of a head has read all of its transitions: they agree
  if (blockIdx.x == 0 && tid == 0) serial[bh] = expands ? 1u : 0u;
}

// Segments for the scan of NT chunks of BH heads (0: none fit): both passes (1.75 and 2.25 us a chunk; pass 1 computes no output)
// and ~2 us a segment in the join take the least.  Pass 1 stays within one wave of CTAs.
int kch_kda_scan_segments(int BH, int NT) {
  int best = 0;
  float best_us = 0.f;
  for (int P = 3; BH > 0 && (int64_t)BH * (1 + 2 * (P - 2)) <= KCH_SMS && P <= NT; ++P) {
    const int per = (NT + P - 1) / P;
    if ((NT + per - 1) / per != P) continue;         // the last segment would be empty
    const float us = (1.75f + 2.25f) * per + 2.f * P;
    if (!best || us < best_us) { best = P; best_us = us; }
  }
  return best;
}
// start states and transitions of the segments, then a flag per head
int64_t kch_kda_scan_split_bytes(int BH, int nseg) {
  return nseg ? (int64_t)2 * nseg * BH * 128 * 128 * 4 + (((int64_t)BH * 4 + 15) & ~(int64_t)15) : 0;
}

static int scan_launch(const T5Args& a, dim3 grid, cudaStream_t s) {
  const int smem = T5_TOTAL + 1024;
  auto kernel = a.nseg ? kda_scan_tc5_kernel<true> : kda_scan_tc5_kernel<false>;
  KCH_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  kernel<<<grid, T5_THREADS, smem, s>>>(a);
  KCH_LAUNCH_OK();
  return KCH_OK;
}

int kch_kda_scan_tc5_split(const void* workspace, void* split, int nseg, const float* initial_state, void* o, float* final_state,
                           int B, int T, int HV, int NT, unsigned int* status, cudaStream_t s) {
  T5Args a = {};
  a.ws = (const uint8_t*)workspace; a.S0 = initial_state; a.o = (bf16*)o; a.S_out = final_state; a.status = status;
  a.T = T; a.Tb = T; a.HV = HV; a.NT = NT;
  a.o_vec = ((uintptr_t)o & 7) == 0;
  const int64_t states = (int64_t)nseg * B * HV * 128 * 128;
  a.nseg = nseg; a.per = (NT + nseg - 1) / nseg; a.starts = (float*)split; a.trans = a.starts + states;
  uint32_t* serial = reinterpret_cast<uint32_t*>(a.trans + states);
  a.serial = serial;
  a.pass = 1;
  int rc = scan_launch(a, dim3(HV, B, 1 + 2 * (nseg - 2)), s);
  if (rc != KCH_OK) return rc;
  KCH_CUDA_OK(cudaFuncSetAttribute(kda_join_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KJ_SMEM));
  KCH_CUDA_OK(kch_launch_chained(kda_join_kernel, dim3(128 / KJ_COLS, HV, B), dim3(256), KJ_SMEM, s, 1, a.starts, (const float*)a.trans, serial, nseg));
  KCH_LAUNCH_OK();
  a.pass = 2;
  return scan_launch(a, dim3(HV, B, nseg - 1), s);
}

int kch_kda_scan_tc5(const void* workspace, const float* initial_state, void* o, float* final_state, int B, int T,
                     int Tb, int HV, int NT, unsigned int* status, cudaStream_t s) {
  T5Args a = {};
  a.ws = (const uint8_t*)workspace; a.S0 = initial_state; a.o = (bf16*)o; a.S_out = final_state; a.status = status;
  a.T = T; a.Tb = Tb; a.HV = HV; a.NT = NT;
  a.o_vec = ((uintptr_t)o & 7) == 0;
  return scan_launch(a, dim3(HV, B), s);
}
