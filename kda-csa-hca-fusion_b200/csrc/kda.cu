// KDA: gated delta rule with per-channel log-decay.
//   token recurrence : naive_recurrent_kda (ops_kda.py:222-258)
//   chunked WY form  : naive_chunk_kda     (ops_kda.py:375-424 prepare, 509-535 chain)
// All arithmetic is fp32; inputs are fp32 or bf16; the carried state is fp32 [B,HV,K,V].
#include <math.h>
#include <stdlib.h>

#include <type_traits>

#include "kch_common.cuh"
#include "mma_utils.cuh"

// =====================================================================================
// Token recurrence.  One CTA owns 32 value columns of one (batch, value head); its 4 warps
// split the K rows of the state, which lives in registers for the whole sequence.
// Per token: S <- diag(exp g) S ; S <- S + beta k (v - k^T S)^T ; o = (scale q)^T S.
// Decode (T=1) reads and writes the state exactly once: 2*K*V*4 bytes per (b, hv).
// S0 and S_out may be the same memory: every thread loads its own state elements before the token loop and
// stores the same elements after it.
// =====================================================================================
template <typename T, int KPT>
__global__ void __launch_bounds__(128)
kda_recurrent_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                     const T* __restrict__ g, const T* __restrict__ beta,
                     const float* S0, T* __restrict__ o, float* S_out,
                     int T_, int H, int HV, int K, int V, float scale, float g_min, int64_t ld_qk,
                     int64_t ld_v, int64_t ld_g, int64_t ld_b) {
  const int vb = blockIdx.x, hv = blockIdx.y, b = blockIdx.z;
  const int G = HV / H, h = hv / G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vcol = vb * 32 + lane;
  const bool vok = vcol < V;
  const int k0 = warp * KPT;
  __shared__ float sk[2][4 * KPT], sq[2][4 * KPT], sg[2][4 * KPT];
  __shared__ float red[4][32], red2[4][32];
  float s[KPT];
  const int64_t sbase = ((int64_t)b * HV + hv) * K * V;
#pragma unroll
  for (int i = 0; i < KPT; ++i) {
    int kk = k0 + i;
    s[i] = (S0 && vok && kk < K) ? S0[sbase + (int64_t)kk * V + vcol] : 0.f;
  }
  auto load_tok = [&](int t, int buf) {
    const int64_t qoff = ((int64_t)b * T_ + t) * ld_qk + (int64_t)h * K;
    const int64_t goff = ((int64_t)b * T_ + t) * ld_g + (int64_t)hv * K;
    for (int i = threadIdx.x; i < 4 * KPT; i += 128) {
      bool ok = i < K;
      sk[buf][i] = ok ? ldf(k + qoff + i) : 0.f;
      sq[buf][i] = ok ? ldf(q + qoff + i) * scale : 0.f;
      sg[buf][i] = ok ? expf(fmaxf(ldf(g + goff + i), g_min)) : 1.f;
    }
  };
  if (T_ > 0) load_tok(0, 0);
  __syncthreads();
  for (int t = 0; t < T_; ++t) {
    const int buf = t & 1;
    const int64_t voff = (((int64_t)b * T_ + t) * HV + hv);
    float part = 0.f;
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      s[i] *= sg[buf][k0 + i];
      part = fmaf(sk[buf][k0 + i], s[i], part);
    }
    red[warp][lane] = part;
    if (t + 1 < T_) load_tok(t + 1, buf ^ 1);
    __syncthreads();
    float pred = red[0][lane] + red[1][lane] + red[2][lane] + red[3][lane];
    float vv = vok ? ldf(v + ((int64_t)b * T_ + t) * ld_v + (int64_t)hv * V + vcol) : 0.f;
    float delta = ldf(beta + ((int64_t)b * T_ + t) * ld_b + hv) * (vv - pred);
    float op = 0.f;
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      s[i] = fmaf(sk[buf][k0 + i], delta, s[i]);
      op = fmaf(sq[buf][k0 + i], s[i], op);
    }
    red2[warp][lane] = op;
    __syncthreads();
    if (warp == 0 && vok)
      stf(o + voff * V + vcol, red2[0][lane] + red2[1][lane] + red2[2][lane] + red2[3][lane]);
  }
  if (S_out && vok) {
#pragma unroll
    for (int i = 0; i < KPT; ++i) {
      int kk = k0 + i;
      if (kk < K) S_out[sbase + (int64_t)kk * V + vcol] = s[i];
    }
  }
}

// One-token step (T = 1, K = V = 128), the form a decode step takes.  The 64 KB state of one (batch, value head) is
// contiguous: one bulk copy brings it into shared memory (no registers, no per-thread loads: three CTAs per SM keep
// 192 KB of requests in flight) and one bulk copy writes it back.  A thread takes RPT of a
// value column's four runs of 32 K rows; decay, key and scaled query of a K row travel as one float4 broadcast.  Both contractions over K (k^T S and
// q^T S) are four private runs added left to right, the order of kda_recurrent_kernel, so both return the same bits.
// Bound: HBM (128 KB per head) at large batches, where one thread per column (RPT = 4, three CTAs per SM) is enough and
// more threads only cost residency (25 us against 28 for 1024 heads); with at most two CTAs per SM in all, the chain
// copy -> two passes over the rows -> copy, whose middle four threads per column (RPT = 1) take from 2.2 to 0.7 us:
// 128 heads, within a step: 9.7 -> 9.1 us.
// The wait for the copy is bounded (status word, see kch_device_status).
#define KDS_STATE_BYTES (128 * 128 * 4)
#define KDS_SMEM (KDS_STATE_BYTES + 128 * 16 + 2 * 4 * 128 * 4 + 16)
struct KdsGate {                         // the gate's up-projection and activation, for a step that brings their input
  const bf16 *x, *W;                     // [B, 128] rows ld_x apart; [HV * 128, 128] rows ld_w apart
  int64_t ld_x, ld_w;
  float scale;                           // g = round(-round(softplus(round(W x))) * scale), the rounding points of the layer
  int settled;                           // the launch before does not write W
};
template <typename T, int RPT, bool GATE>
__global__ void __launch_bounds__(512 / RPT, RPT == 4 ? 3 : 2)
kda_decode_step_kernel(const T* q, const T* k, const T* v, const T* g, const T* beta, const float* S0, T* o, float* S_out, int H,
                       int HV, float scale, float g_min, int64_t ld_qk, int64_t ld_v, int64_t ld_g, int64_t ld_b,
                       const KdsGate gate, unsigned int* status) {
  constexpr int K = 128, V = 128;
  extern __shared__ __align__(128) uint8_t kds_raw[];
  float* st = reinterpret_cast<float*>(kds_raw);                                   // [K][V]
  float4* sgkq = reinterpret_cast<float4*>(kds_raw + KDS_STATE_BYTES);             // {exp(g), k, scale * q, -} of K row i
  float* sp = reinterpret_cast<float*>(kds_raw + KDS_STATE_BYTES + 128 * 16);      // [2][4][V] sums of the runs
  uint64_t* bar = reinterpret_cast<uint64_t*>(kds_raw + KDS_STATE_BYTES + 128 * 16 + 2 * 4 * V * 4);
  const int hv = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int h = hv / (HV / H);
  const int64_t sbase = ((int64_t)b * HV + hv) * K * V;
  if (tid == 0) {
    mbarrier_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the head's 128 x 128 gate weights: four threads a row, 64 bytes each
  static_assert(!GATE || RPT == 1, "one row of the gate's weights per four threads");
  uint4 wraw[4];
  auto load_gate_weights = [&]() {
    const uint4* p = reinterpret_cast<const uint4*>(gate.W + ((int64_t)hv * K + (tid >> 2)) * gate.ld_w + 32 * (tid & 3));
#pragma unroll
    for (int i = 0; i < 4; ++i) wraw[i] = p[i];
  };
  if (GATE && gate.settled) load_gate_weights();
  chain_wait();
  chain_trigger();
  if (tid == 0 && S0) {
    mbarrier_expect_tx(bar, KDS_STATE_BYTES);
    bulk_copy_g2s(st, S0 + sbase, KDS_STATE_BYTES, bar);
  }
  if (GATE && !gate.settled) load_gate_weights();
  const int c = tid & 127, run0 = (tid >> 7) * RPT;    // value column, first of this thread's runs of 32 K rows
  const float bt = ldf(beta + (int64_t)b * ld_b + hv);
  const float vv = ldf(v + (int64_t)b * ld_v + (int64_t)hv * V + c);
  if constexpr (GATE) {
    uint4 xraw[4];
    const uint4* xp = reinterpret_cast<const uint4*>(gate.x + (int64_t)b * gate.ld_x + 32 * (tid & 3));
#pragma unroll
    for (int i = 0; i < 4; ++i) xraw[i] = xp[i];
    if (tid < K) {
      const int64_t qoff = (int64_t)b * ld_qk + (int64_t)h * K;
      reinterpret_cast<float*>(sgkq + tid)[1] = ldf(k + qoff + tid);
      reinterpret_cast<float*>(sgkq + tid)[2] = ldf(q + qoff + tid) * scale;
    }
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t w4[4] = {wraw[i].x, wraw[i].y, wraw[i].z, wraw[i].w};
      const uint32_t x4[4] = {xraw[i].x, xraw[i].y, xraw[i].z, xraw[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        dot = fmaf(__uint_as_float(w4[e] << 16), __uint_as_float(x4[e] << 16), dot);
        dot = fmaf(__uint_as_float(w4[e] & 0xFFFF0000u), __uint_as_float(x4[e] & 0xFFFF0000u), dot);
      }
    }
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
    if ((tid & 3) == 0) {
      // the activation as the projection's epilogue applies it (gemm_decode.cu)
      const float t = round_to<bf16>(dot);
      const float gv = round_to<bf16>(-round_to<bf16>(t > 20.f ? t : __logf(1.0f + __expf(t))) * gate.scale);
      reinterpret_cast<float*>(sgkq + (tid >> 2))[0] = expf(fmaxf(gv, g_min));
    }
  } else if (tid < K) {
    const int64_t qoff = (int64_t)b * ld_qk + (int64_t)h * K, goff = (int64_t)b * ld_g + (int64_t)hv * K;
    sgkq[tid] = make_float4(expf(fmaxf(ldf(g + goff + tid), g_min)), ldf(k + qoff + tid), ldf(q + qoff + tid) * scale, 0.f);
  }
  if (!S0) {
    for (int i = 32 * run0; i < 32 * (run0 + RPT); ++i) st[i * V + c] = 0.f;
  }
  __syncthreads();
  bool ok = true;
  if (S0) ok = mbarrier_wait_bounded(bar, 0, KCH_STATUS_KDA_STEP, 1u << 24, status);
#pragma unroll
  for (int r = run0; r < run0 + RPT; ++r) {
    const float* col = st + 32 * r * V + c;
    const float4* row = sgkq + 32 * r;
    float acc = 0.f;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const float4 x = row[i];
      acc = fmaf(x.y, col[i * V] * x.x, acc);
    }
    sp[r * V + c] = acc;
  }
  __syncthreads();
  const float delta = bt * (vv - (sp[c] + sp[V + c] + sp[2 * V + c] + sp[3 * V + c]));
#pragma unroll
  for (int r = run0; r < run0 + RPT; ++r) {
    float* col = st + 32 * r * V + c;
    const float4* row = sgkq + 32 * r;
    float acc = 0.f;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const float4 x = row[i];
      const float sv = fmaf(x.y, delta, col[i * V] * x.x);
      col[i * V] = sv;
      acc = fmaf(x.z, sv, acc);
    }
    sp[(4 + r) * V + c] = acc;
  }
  if (S_out) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");          // the bulk store reads what the threads wrote
  __syncthreads();
  if (S_out && tid == 0 && ok) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(S_out + sbase), "r"(smem_addr_u32(st)), "r"((uint32_t)KDS_STATE_BYTES) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
  if (run0 == 0 && ok)
    stf(o + ((int64_t)b * HV + hv) * V + c, sp[4 * V + c] + sp[5 * V + c] + sp[6 * V + c] + sp[7 * V + c]);
  if (S_out && tid == 0 && ok) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // shared memory must outlive the copy
}

// Steps of up to two heads an SM: one row a thread, and the form that projects the gate itself.  Beyond that the 32 KB of weights
// that every CTA reads cost as much as the launch that they save (64 sequences, 16 heads, whole step: 356 us with the launch, 360
// without; 8 sequences: 199 and 185).
static bool kds_few(int B, int HV) { return (int64_t)HV * B <= 2 * KCH_SMS; }

template <typename T, bool GATE>
static int launch_kda_step(const T* q, const T* k, const T* v, const T* g, const T* beta, const float* S0, T* o, float* S_out, int B, int H,
                           int HV, float scale, float g_min, int64_t ld_qk, int64_t ld_v, int64_t ld_g, int64_t ld_b, const KdsGate& gate,
                           cudaStream_t s) {
  unsigned int* status = kch_status_device_ptr();
  KCH_REQUIRE(status != nullptr, "kch_kda_recurrent: cannot resolve the device status word");
#define KDS_GO(RPT_)                                                                                                               \
  do {                                                                                                                             \
    KCH_CUDA_OK(cudaFuncSetAttribute(kda_decode_step_kernel<T, RPT_, GATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, KDS_SMEM)); \
    KCH_CUDA_OK(kch_launch_chained(kda_decode_step_kernel<T, RPT_, GATE>, dim3(HV, B), dim3(512 / RPT_), KDS_SMEM, s, 1, q, k, v, g,  \
                                   beta, S0, o, S_out, H, HV, scale, g_min, ld_qk, ld_v, ld_g, ld_b, gate, status));               \
  } while (0)
  if constexpr (GATE) {
    KDS_GO(1);
  } else {
    if (kds_few(B, HV)) KDS_GO(1);
    else KDS_GO(4);
  }
#undef KDS_GO
  KCH_LAUNCH_OK();
  return KCH_OK;
}

// KCH_KDA_DECODE=o keeps the general kernel for the one-token step, behind a gate projected by a launch of its own, for comparison
static bool kds_general() {
  static const bool on = [] { const char* e = getenv("KCH_KDA_DECODE"); return e && e[0] == 'o'; }();
  return on;
}

extern "C" int kch_kda_step_gate_supported(int B, int HV, int K, int V, int dtype) {
  return dtype == KCH_BF16 && K == 128 && V == 128 && B >= 1 && HV >= 1 && kds_few(B, HV) && !kds_general();
}

// The one-token step of a layer whose gate has not been projected up yet (see KdsGate).  As a launch of its own the up-projection
// (0.5 MB of weights) took 4.5 us of a step between the two it depends on; here its weights are under way before the launch
// before has finished, and its 16 K products a head hide behind the copy of the state.
extern "C" int kch_kda_step_gate(const void* q, const void* k, const void* v, const void* gate_x, const void* W_gup, const void* beta,
                                 const float* initial_state, void* o, float* final_state, int B, int H, int HV, int K, int V, float scale,
                                 float g_clamp_min, float gate_scale, int dtype, int64_t ld_qk, int64_t ld_v, int64_t ld_gate, int64_t ld_wg,
                                 int64_t ld_beta, int w_settled, void* stream) {
  KCH_REQUIRE(kch_kda_step_gate_supported(B, HV, K, V, dtype),
              "kch_kda_step_gate: bf16 with K = V = 128 and B * HV from 1 to 296 only (dtype tag %d, K=%d, V=%d, B=%d, HV=%d)", dtype, K, V, B, HV);
  KCH_REQUIRE(H >= 1 && HV % H == 0, "kch_kda_step_gate: H=%d HV=%d", H, HV);
  KCH_REQUIRE(q && k && v && gate_x && W_gup && beta && o, "kch_kda_step_gate: an operand is missing");
  KCH_REQUIRE(((((uintptr_t)gate_x | (uintptr_t)W_gup | (uintptr_t)initial_state | (uintptr_t)final_state) & 15) == 0) && (ld_gate % 8) == 0 && (ld_wg % 8) == 0,
              "kch_kda_step_gate: gate input, weights and states must be 16-byte aligned with strides that are multiples of 8 elements");
  const KdsGate gate = {(const bf16*)gate_x, (const bf16*)W_gup, ld_gate, ld_wg, gate_scale, w_settled};
  return launch_kda_step<bf16, true>((const bf16*)q, (const bf16*)k, (const bf16*)v, nullptr, (const bf16*)beta, initial_state, (bf16*)o,
                                     final_state, B, H, HV, scale, g_clamp_min, ld_qk, ld_v, 0, ld_beta, gate, kch_stream(stream));
}

extern "C" int kch_kda_recurrent(const void* q, const void* k, const void* v, const void* g,
                                 const void* beta, const float* initial_state, void* o,
                                 float* final_state, int B, int T, int H, int HV, int K, int V,
                                 float scale, float g_clamp_min, int dtype, int64_t ld_qk, int64_t ld_v,
                                 int64_t ld_g, int64_t ld_beta, void* stream) {
  if (ld_qk <= 0) ld_qk = (int64_t)H * K;
  if (ld_v <= 0) ld_v = (int64_t)HV * V;
  if (ld_g <= 0) ld_g = (int64_t)HV * K;
  if (ld_beta <= 0) ld_beta = HV;
  KCH_REQUIRE(H >= 1, "H=%d must be >= 1", H);
  KCH_REQUIRE(K >= 1, "K=%d must be >= 1", K);
  KCH_REQUIRE(V >= 1, "V=%d must be >= 1", V);
  KCH_REQUIRE(HV >= 1 && HV % H == 0, "HV=%d must be divisible by H=%d (GVA factor)", HV, H);
  KCH_REQUIRE(K <= 256, "K=%d exceeds the supported maximum of 256", K);
  KCH_REQUIRE(B >= 0 && T >= 0, "B=%d T=%d", B, T);
  if (B == 0) return KCH_OK;
  if (T == 0 && !final_state) return KCH_OK;
  dim3 grid((V + 31) / 32, HV, B), block(128);
  cudaStream_t s = kch_stream(stream);
  if (T == 1 && K == 128 && V == 128 && !kds_general() && (((uintptr_t)initial_state | (uintptr_t)final_state) & 15) == 0) {
    const KdsGate none = {};
    KCH_DISPATCH_FLOAT(dtype, T_, return (launch_kda_step<T_, false>((const T_*)q, (const T_*)k, (const T_*)v, (const T_*)g, (const T_*)beta,
                                                                     initial_state, (T_*)o, final_state, B, H, HV, scale, g_clamp_min, ld_qk,
                                                                     ld_v, ld_g, ld_beta, none, s)));
  }
  int kpt = (K + 3) / 4;
#define GO(T_, KPT)                                                                              \
  kda_recurrent_kernel<T_, KPT><<<grid, block, 0, s>>>((const T_*)q, (const T_*)k, (const T_*)v, \
      (const T_*)g, (const T_*)beta, initial_state, (T_*)o, final_state, T, H, HV, K, V, scale,  \
      g_clamp_min, ld_qk, ld_v, ld_g, ld_beta)
#define GOK(T_)                      \
  do {                               \
    if (kpt <= 4) GO(T_, 4);         \
    else if (kpt <= 8) GO(T_, 8);    \
    else if (kpt <= 16) GO(T_, 16);  \
    else if (kpt <= 32) GO(T_, 32);  \
    else GO(T_, 64);                 \
  } while (0)
  KCH_DISPATCH_FLOAT(dtype, T_, GOK(T_));
#undef GOK
#undef GO
  KCH_LAUNCH_OK();
  return KCH_OK;
}

// =====================================================================================
// Chunked form in fp32 on CUDA cores, for every geometry the tensor-core kernels do not take (fp32 inputs, K or V other
// than 128).  A record holds L tokens: as many whole chunks of C = min(chunk_size, 64, K) as fit into 64 (zero rows pad it
// to 64 rows), because a longer record means fewer dependent steps in stage 2 and the mathematics does not depend on the
// length -- but for a gate that grows: the exponent of a pair is clamped at 50 within a chunk of C tokens and exact between
// chunks, where the state carries it.  K is padded to KT = 64 or 128 channels.
//
// Stage 1, one CTA of 4*KT threads per (b, hv, chunk), all chunks in parallel:
//   gamma = cumsum(g), A (strictly lower), Tm = (I+A)^-1 diag(beta),
//   w = Tm (exp(gamma) k), u = Tm v, Aqk (lower incl. diagonal),
//   qg = scale q exp(gamma), kg = k exp(gamma_last - gamma), dl = exp(gamma_last)
// into one record per chunk that stage 2 streams.  Bound: instruction issue.  What made it long was one exponential
// per (i, j, channel): 262 K of them per chunk and a 64-deep serial substitution.  Now the exponent difference is
// factored around a row between the two halves of a block (both factors <= 1 for a decay, so nothing overflows, and
// what underflows is smaller still), halving the blocks from 32 to 4 rows: 8 K exponentials a level and plain products;
// only the 4 x 4 diagonal blocks take the difference pair by pair.  The inverse is built from 8 x 8 blocks upwards.
// Of the 78 K cycles that a chunk then took, 14 K were the diagonal blocks (a warp a pair, two reductions each), 9 K the loads
// (scalar, a few in flight), 8 K the element-wise outputs, 7 K the loads of v, 10 K the products of the two widest levels (2 x 2
// tiles: the return path of shared memory): 16-byte loads all under way at once, a warp a diagonal block, 4 x 4 tiles.
// 1024 tokens, 4 heads, K = V = 128, fp32: 202 -> 42 -> 29 us.  What holds zero rows only is skipped (8 tokens: 41 -> 23 us,
// both stages).
// A record whose gate is positive or not finite somewhere takes every pair directly.
// =====================================================================================
#define KC_C 64
#define KC_AS 68                       // row stride of the 64 x 64 tiles (16-byte rows, 8 rows on 32 banks)

// one chunk record, in floats: w, qg, kg [64][KT+4]; Aqk [64][68]; dl [KT]; u [V/8][64][8]
__host__ __device__ inline int64_t kc_record_floats(int KT, int V) {
  return 3ll * KC_C * (KT + 4) + KC_C * KC_AS + KT + (int64_t)((V + 7) / 8) * 8 * KC_C;
}

// four consecutive elements as fp32, from a 16-byte (fp32) or 8-byte (bf16) boundary
__device__ __forceinline__ float4 kc_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 kc_load4(const bf16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xFFFF0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xFFFF0000u));
}
// sum of each of N values (a power of two) over groups of G lanes; lane l of a group is left with the N / G sums from l * N / G on
template <int N, int G>
__device__ __forceinline__ void kc_reduce(float (&v)[N], int lane) {
  static_assert(N >= G, "a value per lane at least");
  int n = N;
#pragma unroll
  for (int off = G >> 1; off > 0; off >>= 1) {
    n >>= 1;
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i < n) {
        const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
  }
}

template <typename T, int KT>
__global__ void __launch_bounds__(4 * KT)
kda_chunk_prepare_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                         const T* __restrict__ g, const T* __restrict__ beta, float* __restrict__ ws, int T_,
                         int H, int HV, int K, int V, int NT, int L, int C, float scale, float g_min,
                         int64_t ld_qk, int64_t ld_v, int64_t ld_g, int64_t ld_b, int vec) {
  constexpr int NTH = 4 * KT, KS = KT + 4, NW = NTH / 32;
  extern __shared__ __align__(16) float smem[];
  float* sk = smem;                    // [64][KS] k
  float* sq = sk + KC_C * KS;          // [64][KS] scale * q
  float* sgam = sq + KC_C * KS;        // [64][KS] running sum of g from the start of the row's segment of 16
  float* sx = sgam + KC_C * KS;        // [64][KS] k with one side of the factored exponent; later exp(gamma) k, then v
  float* sy = sx + KC_C * KS;          // [32][KS] the same for q (rows on the i side)
  float* sT = sy;                      // [64][68] (I + A)^-1, then Tm, once the factors are done with
  float* sA = sy + (32 * KS > KC_C * KC_AS ? 32 * KS : KC_C * KC_AS);      // [64][68] A
  float* sbeta = sA + KC_C * KC_AS;    // [64]
  float* stot = sbeta + KC_C;          // [4][KT] sums over the segments
  const int n = blockIdx.x, hv = blockIdx.y, b = blockIdx.z;
  const int h = hv / (HV / H);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = n * L, t_end = min(t0 + L, T_), rows = t_end - t0;      // this record's tokens; rows behind them are zero
  float* rec = ws + (((int64_t)b * HV + hv) * NT + n) * kc_record_floats(KT, V);
  float* o_w = rec;
  float* o_qg = o_w + KC_C * KS;
  float* o_kg = o_qg + KC_C * KS;
  float* o_aqk = o_kg + KC_C * KS;
  float* o_dl = o_aqk + KC_C * KC_AS;
  float* o_u = o_dl + KT;

  bool odd_gate = false;
  if (vec & 1) {                                         // all twelve loads of a thread are under way before the first is used
    float4 kv[4], qv[4], gv[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int idx = tid + r * NTH, i = idx / (KT / 4), kk = 4 * (idx % (KT / 4)), t = t0 + i;
      kv[r] = qv[r] = gv[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < t_end && kk < K) {
        const int64_t qoff = ((int64_t)b * T_ + t) * ld_qk + (int64_t)h * K + kk;
        kv[r] = kc_load4(k + qoff);
        qv[r] = kc_load4(q + qoff);
        gv[r] = kc_load4(g + ((int64_t)b * T_ + t) * ld_g + (int64_t)hv * K + kk);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int idx = tid + r * NTH, i = idx / (KT / 4), kk = 4 * (idx % (KT / 4));
      if (t0 + i < t_end && kk < K) {
        float* gp = &gv[r].x;
        float* qp = &qv[r].x;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          gp[e] = fmaxf(gp[e], g_min);
          odd_gate |= !(gp[e] <= 0.f && gp[e] > -1e30f);
          qp[e] *= scale;
        }
      }
      *reinterpret_cast<float4*>(sk + i * KS + kk) = kv[r];
      *reinterpret_cast<float4*>(sq + i * KS + kk) = qv[r];
      *reinterpret_cast<float4*>(sgam + i * KS + kk) = gv[r];
    }
  } else {
#pragma unroll 4
    for (int idx = tid; idx < KC_C * KT; idx += NTH) {
      const int i = idx / KT, kk = idx % KT, t = t0 + i;
      float kv = 0.f, qv = 0.f, gv = 0.f;
      if (t < t_end && kk < K) {
        const int64_t qoff = ((int64_t)b * T_ + t) * ld_qk + (int64_t)h * K + kk;
        kv = ldf(k + qoff);
        qv = ldf(q + qoff) * scale;
        gv = fmaxf(ldf(g + ((int64_t)b * T_ + t) * ld_g + (int64_t)hv * K + kk), g_min);
        odd_gate |= !(gv <= 0.f && gv > -1e30f);
      }
      sk[i * KS + kk] = kv;
      sq[i * KS + kk] = qv;
      sgam[i * KS + kk] = gv;
    }
  }
  if (tid < KC_C) sbeta[tid] = t0 + tid < t_end ? ldf(beta + ((int64_t)b * T_ + t0 + tid) * ld_b + hv) : 0.f;
  for (int idx = tid; idx < KC_C * KC_AS; idx += NTH) {
    sA[idx] = 0.f;
    if (idx % KC_AS > idx / KC_AS) o_aqk[idx] = 0.f;
  }
  const bool direct = __syncthreads_or(odd_gate);
  // running sums: four threads per channel, 16 rows each.  They stay relative to their segment: a difference of two
  // rows is then put together from short sums (gamma itself grows to tens, and its rounding with it)
  {
    const int kk = tid % KT, seg = tid / KT;
    float r[16], acc = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = sgam[(16 * seg + i) * KS + kk];
#pragma unroll
    for (int i = 0; i < 16; ++i) { acc += r[i]; r[i] = acc; }
    stot[seg * KT + kk] = acc;
#pragma unroll
    for (int i = 0; i < 16; ++i) sgam[(16 * seg + i) * KS + kk] = r[i];
  }
  __syncthreads();
  // A and Aqk below the diagonal blocks, half block size 32, 16, 8, 4
  if (!direct) {
#pragma unroll
    for (int s = 32; s >= 4; s >>= 1) {
      if (s >= rows) continue;                            // blocks of zero rows only
#pragma unroll 4
      for (int idx = tid; idx < KC_C * KT; idx += NTH) {
        const int i = idx / KT, kk = idx % KT;
        const float rl = sgam[i * KS + kk];
        const int seg = i >> 4;
        if (i & s) {                                      // gamma_i - gamma_ref, ref = the last row of the other half
          const float d = s == 32 ? (seg == 3 ? rl + stot[2 * KT + kk] : rl)
                        : s == 16 ? rl : rl - sgam[((i & ~(2 * s - 1)) + s - 1) * KS + kk];
          const float e = expf(d);
          sx[i * KS + kk] = sk[i * KS + kk] * e;
          sy[((i / (2 * s)) * s + (i & (s - 1))) * KS + kk] = sq[i * KS + kk] * e;
        } else {
          float d;                                        // gamma_ref - gamma_i
          if (s >= 16) {
            d = stot[seg * KT + kk] - rl;
            if (s == 32 && seg == 0) d += stot[KT + kk];
          } else {
            d = sgam[((i & ~(2 * s - 1)) + s - 1) * KS + kk] - rl;
          }
          sx[i * KS + kk] = sk[i * KS + kk] * expf(d);
        }
      }
      __syncthreads();
      if (s >= 16) {
        // 4 x 4 outputs of A and of Aqk per thread group, the channels dealt out to SPL neighbouring lanes (a 16-byte read is
        // four cycles of the return path however many lanes share it: 12 reads feed 128 multiply-adds, 6 fed 32)
        constexpr int SP32 = NTH / 64;
        auto tile4 = [&](auto spl_tag) {
          constexpr int SPL = decltype(spl_tag)::value;
          const int tile = tid / SPL, ks = tid % SPL, per = (s / 4) * (s / 4), blk = tile / per, tb = tile % per;
          const int ti = tb / (s / 4), tj = tb % (s / 4);
          const int i0 = blk * 2 * s + s + 4 * ti, j0 = blk * 2 * s + 4 * tj, y0 = blk * s + 4 * ti;
          float acc[32] = {};
          for (int f = ks; f < KT / 4; f += SPL) {
            float4 xi[4], yi[4], xj[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              xi[e] = *reinterpret_cast<const float4*>(sx + (i0 + e) * KS + 4 * f);
              yi[e] = *reinterpret_cast<const float4*>(sy + (y0 + e) * KS + 4 * f);
              xj[e] = *reinterpret_cast<const float4*>(sx + (j0 + e) * KS + 4 * f);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                float& a = acc[4 * e + c];
                float& aq = acc[16 + 4 * e + c];
                a = fmaf(xi[e].x, xj[c].x, a); a = fmaf(xi[e].y, xj[c].y, a); a = fmaf(xi[e].z, xj[c].z, a); a = fmaf(xi[e].w, xj[c].w, a);
                aq = fmaf(yi[e].x, xj[c].x, aq); aq = fmaf(yi[e].y, xj[c].y, aq); aq = fmaf(yi[e].z, xj[c].z, aq); aq = fmaf(yi[e].w, xj[c].w, aq);
              }
          }
          kc_reduce<32, SPL>(acc, lane);
#pragma unroll
          for (int u = 0; u < 32 / SPL; ++u) {
            const int v = ks * (32 / SPL) + u, e = (v & 15) >> 2, c = v & 3;
            if (v < 16) sA[(i0 + e) * KC_AS + j0 + c] = acc[u] * sbeta[i0 + e];
            else o_aqk[(i0 + e) * KC_AS + j0 + c] = acc[u];
          }
        };
        if (s == 32) tile4(std::integral_constant<int, SP32>{});
        else tile4(std::integral_constant<int, 2 * SP32>{});
        __syncthreads();
        continue;
      }
      // narrower blocks: 2 x 2 outputs per thread group, the channels of a group dealt out to `split` neighbouring lanes
      const int split = NTH / (8 * s);
      const int tile = tid / split, ks = tid % split;
      const int per = (s / 2) * (s / 2);                  // tiles of one block
      const int blk = tile / per, tb = tile % per;
      int ti, tj;
      if (s >= 8) {                                       // 4 x 4 tiles per 16: four rows each side per warp
        const int t16 = tb % 16, hi = tb / 16, side = s / 8;
        ti = 4 * (hi / side) + t16 / 4;
        tj = 4 * (hi % side) + t16 % 4;
      } else {
        ti = tb / 2;
        tj = tb % 2;
      }
      const int i0 = blk * 2 * s + s + 2 * ti, j0 = blk * 2 * s + 2 * tj, y0 = blk * s + 2 * ti;
      float a[2][2] = {}, aq[2][2] = {};
      for (int f = ks; f < KT / 4; f += split) {
        float4 xi[2], yi[2], xj[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          xi[e] = *reinterpret_cast<const float4*>(sx + (i0 + e) * KS + 4 * f);
          yi[e] = *reinterpret_cast<const float4*>(sy + (y0 + e) * KS + 4 * f);
          xj[e] = *reinterpret_cast<const float4*>(sx + (j0 + e) * KS + 4 * f);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            a[e][c] = fmaf(xi[e].x, xj[c].x, a[e][c]); a[e][c] = fmaf(xi[e].y, xj[c].y, a[e][c]);
            a[e][c] = fmaf(xi[e].z, xj[c].z, a[e][c]); a[e][c] = fmaf(xi[e].w, xj[c].w, a[e][c]);
            aq[e][c] = fmaf(yi[e].x, xj[c].x, aq[e][c]); aq[e][c] = fmaf(yi[e].y, xj[c].y, aq[e][c]);
            aq[e][c] = fmaf(yi[e].z, xj[c].z, aq[e][c]); aq[e][c] = fmaf(yi[e].w, xj[c].w, aq[e][c]);
          }
      }
      for (int o = split >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            a[e][c] += __shfl_xor_sync(0xffffffffu, a[e][c], o);
            aq[e][c] += __shfl_xor_sync(0xffffffffu, aq[e][c], o);
          }
      if (ks == 0) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            sA[(i0 + e) * KC_AS + j0 + c] = a[e][c] * sbeta[i0 + e];
            o_aqk[(i0 + e) * KC_AS + j0 + c] = aq[e][c];
          }
      }
      __syncthreads();
    }
  }
  for (int idx = tid; idx < KC_C * KC_AS; idx += NTH) sT[idx] = 0.f;
  // V of the first tile of columns: under way while the triangle is finished and inverted
  float4 vraw[4];
  if (vec & 2) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int idx = tid + r * NTH, i = idx / (KT / 4), c = 4 * (idx % (KT / 4)), t = t0 + i;
      vraw[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t < t_end && c < V) vraw[r] = kc_load4(v + ((int64_t)b * T_ + t) * ld_v + (int64_t)hv * V + c);
    }
  }
  if (!direct) {
    // the 4 x 4 diagonal blocks: a warp per block, its lanes over the channels, the 6 + 10 sums of a block reduced together
    // (a warp per pair, two reductions each, took a fifth of the stage)
    for (int blk = warp; blk < (rows + 3) / 4; blk += NW) {
      const int r0 = 4 * blk;
      float acc[16] = {};                                 // A (1,0) (2,0) (2,1) (3,0) (3,1) (3,2), then Aqk with the diagonal
#pragma unroll
      for (int c = 0; c < KT / 32; ++c) {
        const int kk = lane + 32 * c;
        float kr[4], qr[4], gr[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          kr[e] = sk[(r0 + e) * KS + kk];
          qr[e] = sq[(r0 + e) * KS + kk];
          gr[e] = sgam[(r0 + e) * KS + kk];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j <= i; ++j) {
            const float e = i == j ? kr[j] : expf(gr[i] - gr[j]) * kr[j];
            if (j < i) acc[i * (i - 1) / 2 + j] = fmaf(kr[i], e, acc[i * (i - 1) / 2 + j]);
            acc[6 + i * (i + 1) / 2 + j] = fmaf(qr[i], e, acc[6 + i * (i + 1) / 2 + j]);
          }
      }
#pragma unroll
      for (int v = 0; v < 16; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], 16);
      kc_reduce<16, 16>(acc, lane);
      const int v = lane & 15, w = v < 6 ? v : v - 6;
      if (lane < 16) {
        if (v < 6) {
          const int i = 1 + (w >= 1) + (w >= 3), j = w - i * (i - 1) / 2;
          sA[(r0 + i) * KC_AS + r0 + j] = acc[0] * sbeta[r0 + i];
        } else {
          const int i = (w >= 1) + (w >= 3) + (w >= 6), j = w - i * (i + 1) / 2;
          o_aqk[(r0 + i) * KC_AS + r0 + j] = acc[0];
        }
      }
    }
  } else {
    // every pair of the triangle: a warp per pair, its lanes over the channels
    for (int p = warp; p < KC_C * (KC_C + 1) / 2; p += NW) {
      int i = (int)((sqrtf(8.f * p + 1.f) - 1.f) * 0.5f);
      if ((i + 1) * (i + 2) / 2 <= p) ++i;
      if (i * (i + 1) / 2 > p) --i;
      const int j = p - i * (i + 1) / 2;
      if (i >= rows) break;
      float a = 0.f, aq = 0.f;
#pragma unroll
      for (int c = 0; c < KT / 32; ++c) {
        const int kk = lane + 32 * c;
        float d = sgam[i * KS + kk] - sgam[j * KS + kk];
        for (int s = j >> 4; s < i >> 4; ++s) d += stot[s * KT + kk];
        if (i / C == j / C) d = fminf(d, 50.f);
        const float e = expf(d) * sk[j * KS + kk];
        a = fmaf(sk[i * KS + kk], e, a);
        aq = fmaf(sq[i * KS + kk], e, aq);
      }
      a = warp_sum(a);
      aq = warp_sum(aq);
      if (lane == 0) {
        if (j < i) sA[i * KC_AS + j] = a * sbeta[i];
        o_aqk[i * KC_AS + j] = aq;
      }
    }
  }
  __syncthreads();
  // (I + A)^-1: the 8 x 8 diagonal blocks by substitution (a thread per column) ...
  if (tid < KC_C) {
    const int c = tid & 7, b0 = tid & ~7;
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float acc = i == c ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) acc = fmaf(-sA[(b0 + i) * KC_AS + b0 + j], x[j], acc);
      x[i] = i < c ? 0.f : acc;
      sT[(b0 + i) * KC_AS + b0 + c] = x[i];
    }
  }
  // ... meanwhile the element-wise outputs, and exp(gamma) k as the operand of w
  {
    const int kk = tid % KT, seg = tid / KT;
    float before = 0.f, after = stot[seg * KT + kk];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float x = stot[s * KT + kk];
      before += s < seg ? x : 0.f;
      after += s > seg ? x : 0.f;
    }
#pragma unroll 4
    for (int i = 16 * seg; i < 16 * seg + 16; ++i) {
      const float gl = sgam[i * KS + kk], kv = sk[i * KS + kk], eg = expf(gl + before);        // gamma; then gamma_last - gamma
      sx[i * KS + kk] = eg * kv;
      o_qg[i * KS + kk] = sq[i * KS + kk] * eg;
      o_kg[i * KS + kk] = kv * expf(after - gl);
      if (i == KC_C - 1) o_dl[kk] = eg;
    }
  }
  __syncthreads();
  // ... then [[T00, 0], [-T11 A10 T00, T11]] for blocks of 8, 16 and 32
#pragma unroll
  for (int s = 8; s <= 32; s <<= 1) {
    if (s >= rows) continue;
    for (int idx = tid; idx < 32 * s; idx += NTH) {
      const int blk = idx / (s * s), i = (idx / s) % s, c = idx % s, r0 = blk * 2 * s;
      float acc = 0.f;
#pragma unroll 8
      for (int j = 0; j < s; ++j) acc = fmaf(sA[(r0 + s + i) * KC_AS + r0 + j], sT[(r0 + j) * KC_AS + r0 + c], acc);
      sgam[blk * s * s + i * s + c] = acc;
    }
    __syncthreads();
    for (int idx = tid; idx < 32 * s; idx += NTH) {
      const int blk = idx / (s * s), i = (idx / s) % s, c = idx % s, r0 = blk * 2 * s;
      float acc = 0.f;
#pragma unroll 8
      for (int j = 0; j < s; ++j) acc = fmaf(sT[(r0 + s + i) * KC_AS + r0 + s + j], sgam[blk * s * s + j * s + c], acc);
      sT[(r0 + s + i) * KC_AS + r0 + c] = -acc;
    }
    __syncthreads();
  }
  for (int idx = tid; idx < KC_C * KC_C; idx += NTH) sT[(idx / KC_C) * KC_AS + idx % KC_C] *= sbeta[idx % KC_C];
  __syncthreads();
  // w = Tm (exp(gamma) k), then u = Tm v in tiles of KT columns: 4 rows x 4 columns per thread
  const int ti = tid / (KT / 4), tc = 4 * (tid % (KT / 4));
  auto product = [&](float (&acc)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
    for (int j = 0; j < 4 * ti + 4; j += 4) {
      float4 tr[4], xv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        tr[r] = *reinterpret_cast<const float4*>(sT + (4 * ti + r) * KC_AS + j);
        xv[r] = *reinterpret_cast<const float4*>(sx + (j + r) * KS + tc);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float tj[4] = {tr[r].x, tr[r].y, tr[r].z, tr[r].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[r][0] = fmaf(tj[e], xv[e].x, acc[r][0]); acc[r][1] = fmaf(tj[e], xv[e].y, acc[r][1]);
          acc[r][2] = fmaf(tj[e], xv[e].z, acc[r][2]); acc[r][3] = fmaf(tj[e], xv[e].w, acc[r][3]);
        }
      }
    }
  };
  float acc[4][4];
  product(acc);
#pragma unroll
  for (int r = 0; r < 4; ++r)
    *reinterpret_cast<float4*>(o_w + (4 * ti + r) * KS + tc) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
  for (int v0 = 0; v0 < V; v0 += KT) {
    __syncthreads();
    if (v0 == 0 && (vec & 2)) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int idx = tid + r * NTH;
        *reinterpret_cast<float4*>(sx + (idx / (KT / 4)) * KS + 4 * (idx % (KT / 4))) = vraw[r];
      }
    } else {
#pragma unroll 4
      for (int idx = tid; idx < KC_C * KT; idx += NTH) {
        const int i = idx / KT, c = idx % KT, t = t0 + i;
        sx[i * KS + c] = t < t_end && v0 + c < V ? ldf(v + ((int64_t)b * T_ + t) * ld_v + (int64_t)hv * V + v0 + c) : 0.f;
      }
    }
    __syncthreads();
    product(acc);
    if (v0 + tc < V) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4*>(o_u + ((int64_t)((v0 + tc) / 8) * KC_C + 4 * ti + r) * 8 + (tc & 7)) =
            make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    }
  }
}

// =====================================================================================
// Stage 2 (sequential over chunks): one CTA owns VS = 8 or 4 value columns of one (batch, value head) and keeps that slice of
// the state in shared memory.
//   vt = u - w S ; o = qg S + Aqk vt ; S <- diag(dl) S + kg^T vt
// Bound: shared-memory wavefronts (each operand row is read once per VS columns) and the four barriers of a chunk.
// Few columns instead of 32: a chunk's step is shortened, not the chain of chunks, by spreading a head over
// V / VS CTAs (a single sequence of a few heads leaves the chip idle otherwise); the next chunk's operands are
// bulk-copied into the buffers as each product releases them, so no step waits for memory.
// 1024 tokens, 4 heads, K = V = 128, fp32: 257 -> 52 us with 8 columns -> 37 with 4 (16 dependent chunks); 2 x 2011 tokens, 4
// heads of 64: 76 -> 48.
// =====================================================================================
template <typename T, int KT, int VS>
__global__ void __launch_bounds__(256)
kda_chunk_scan_kernel(const float* __restrict__ ws, const float* __restrict__ S0, T* __restrict__ o,
                      float* __restrict__ S_out, int T_, int HV, int K, int V, int NT, int L, unsigned int* status) {
  constexpr int KS = KT + 4, IG = 256 / KT, IR = KC_C / IG, N4 = VS / 4;
  extern __shared__ __align__(16) float smem[];
  float* sw = smem;                          // [64][KS], then qg [64][KS]
  float* sqg = sw + KC_C * KS;
  float* skg = sqg + KC_C * KS;              // [64][KS]
  float* saqk = skg + KC_C * KS;             // [64][68], dl [KT] behind it as in the record
  float* sdl = saqk + KC_C * KC_AS;
  float* su = sdl + KT;                      // [64][8]: the record keeps u in groups of 8 columns
  float* sS = su + KC_C * 8;                 // [KT][VS]
  float* svt = sS + KT * VS;                 // [64][VS]
  float4* red = reinterpret_cast<float4*>(svt + KC_C * VS);          // [4][N4][64]: partial sums of w S, then of o
  float4* red3 = red + 4 * N4 * KC_C;                                // [IG][N4][KT]: partial sums of kg^T vt
  uint64_t* bars = reinterpret_cast<uint64_t*>(red3 + IG * N4 * KT); // w + qg + u | Aqk + dl | kg
  const int vb = blockIdx.x, hv = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x;
  const int v0 = vb * VS, u4 = (v0 & 7) / 4;            // first of its columns; its first float4 of a group of 8
  const int64_t bh = (int64_t)b * HV + hv, rf = kc_record_floats(KT, V), sbase = bh * K * V;
  const float* rec = ws + bh * NT * rf;
  auto load_w = [&](int n) {
    mbarrier_expect_tx(&bars[0], (2 * KC_C * KS + KC_C * 8) * 4);
    bulk_copy_g2s(sw, rec + n * rf, 2 * KC_C * KS * 4, &bars[0]);
    bulk_copy_g2s(su, rec + n * rf + 3 * KC_C * KS + KC_C * KC_AS + KT + (int64_t)(v0 / 8) * KC_C * 8, KC_C * 8 * 4, &bars[0]);
  };
  auto load_a = [&](int n) {
    mbarrier_expect_tx(&bars[1], (KC_C * KC_AS + KT) * 4);
    bulk_copy_g2s(saqk, rec + n * rf + 3 * KC_C * KS, (KC_C * KC_AS + KT) * 4, &bars[1]);
  };
  auto load_k = [&](int n) {
    mbarrier_expect_tx(&bars[2], KC_C * KS * 4);
    bulk_copy_g2s(skg, rec + n * rf + 2 * KC_C * KS, KC_C * KS * 4, &bars[2]);
  };
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbarrier_init(&bars[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    load_w(0);
    load_a(0);
    load_k(0);
  }
  for (int idx = tid; idx < KT * VS; idx += 256) {
    const int kk = idx / VS, c = idx % VS;
    sS[idx] = (S0 && kk < K && v0 + c < V) ? S0[sbase + (int64_t)kk * V + v0 + c] : 0.f;
  }
  __syncthreads();
  const int r = tid & 63, ks = tid >> 6;
  bool ok = true;
  auto add4 = [](float4& a, float x, const float4& y) {
    a.x = fmaf(x, y.x, a.x); a.y = fmaf(x, y.y, a.y); a.z = fmaf(x, y.z, a.z); a.w = fmaf(x, y.w, a.w);
  };
  const float4* S4 = reinterpret_cast<const float4*>(sS);
  const float4* vt4 = reinterpret_cast<const float4*>(svt);
  for (int n = 0; n < NT; ++n) {
    ok = ok && mbarrier_wait_bounded(&bars[0], n & 1, KCH_STATUS_KDA_CHUNK, 1u << 24, status);
    // partial sums of w S and qg S: row r, a quarter of the channels
    float4 aw[N4] = {}, aq[N4] = {};
#pragma unroll 4
    for (int kk = ks * (KT / 4); kk < (ks + 1) * (KT / 4); kk += 4) {
      const float4 w4 = *reinterpret_cast<const float4*>(sw + r * KS + kk);
      const float4 q4 = *reinterpret_cast<const float4*>(sqg + r * KS + kk);
      const float wv[4] = {w4.x, w4.y, w4.z, w4.w}, qv[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int c = 0; c < N4; ++c) {
          const float4 s = S4[N4 * (kk + e) + c];
          add4(aw[c], wv[e], s);
          add4(aq[c], qv[e], s);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < N4; ++c) red[(ks * N4 + c) * KC_C + r] = aw[c];
    __syncthreads();
    if (tid < N4 * KC_C) {
      const int c4 = tid >> 6;
      float4 x = reinterpret_cast<const float4*>(su)[2 * r + u4 + c4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float4 y = red[(p * N4 + c4) * KC_C + r];
        x.x -= y.x; x.y -= y.y; x.z -= y.z; x.w -= y.w;
      }
      reinterpret_cast<float4*>(svt)[N4 * r + c4] = x;
    }
    __syncthreads();
    if (tid == 0 && ok && n + 1 < NT) load_w(n + 1);
    ok = ok && mbarrier_wait_bounded(&bars[1], n & 1, KCH_STATUS_KDA_CHUNK, 1u << 24, status);
#pragma unroll
    for (int j = ks * 16; j < ks * 16 + 16; j += 4) {
      const float4 a4 = *reinterpret_cast<const float4*>(saqk + r * KC_AS + j);
      const float av[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int c = 0; c < N4; ++c) add4(aq[c], av[e], vt4[N4 * (j + e) + c]);
      }
    }
#pragma unroll
    for (int c = 0; c < N4; ++c) red[(ks * N4 + c) * KC_C + r] = aq[c];
    ok = ok && mbarrier_wait_bounded(&bars[2], n & 1, KCH_STATUS_KDA_CHUNK, 1u << 24, status);
    {
      const int kk = tid % KT, ig = tid / KT;
      float4 as[N4] = {};
#pragma unroll 8
      for (int i = ig * IR; i < (ig + 1) * IR; ++i) {
        const float kv = skg[i * KS + kk];
#pragma unroll
        for (int c = 0; c < N4; ++c) add4(as[c], kv, vt4[N4 * i + c]);
      }
#pragma unroll
      for (int c = 0; c < N4; ++c) red3[(ig * N4 + c) * KT + kk] = as[c];
    }
    __syncthreads();
    if (tid == 0 && ok && n + 1 < NT) load_k(n + 1);
    for (int idx = tid; idx < N4 * KT; idx += 256) {
      const int kk = idx % KT, c4 = idx / KT;
      float4 x = reinterpret_cast<float4*>(sS)[N4 * kk + c4];
      const float d = sdl[kk];
      x.x *= d; x.y *= d; x.z *= d; x.w *= d;
#pragma unroll
      for (int p = 0; p < IG; ++p) {
        const float4 y = red3[(p * N4 + c4) * KT + kk];
        x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
      }
      reinterpret_cast<float4*>(sS)[N4 * kk + c4] = x;
    }
    if (tid >= 256 - N4 * KC_C) {          // (with four columns: warps that had no share of the state)
      const int c4 = N4 == 1 ? 0 : (tid - 128) >> 6, t = n * L + r;
      float4 x = red[c4 * KC_C + r];
#pragma unroll
      for (int p = 1; p < 4; ++p) {
        const float4 y = red[(p * N4 + c4) * KC_C + r];
        x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
      }
      if (r < L && t < T_ && ok) {
        T* orow = o + (((int64_t)b * T_ + t) * HV + hv) * V + v0 + 4 * c4;
        const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (v0 + 4 * c4 + c < V) stf(orow + c, xv[c]);
      }
    }
    __syncthreads();
    if (tid == 0 && ok && n + 1 < NT) load_a(n + 1);
  }
  if (!ok) {            // give copies still in flight time to land before the shared memory goes
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    return;
  }
  if (S_out)
    for (int idx = tid; idx < KT * VS; idx += 256) {
      const int kk = idx / VS, c = idx % VS;
      if (kk < K && v0 + c < V) S_out[sbase + (int64_t)kk * V + v0 + c] = sS[idx];
    }
}

static size_t kc_prepare_smem(int KT) {
  const int KS = KT + 4;
  return ((size_t)4 * KC_C * KS + (32 * KS > KC_C * KC_AS ? 32 * KS : KC_C * KC_AS) + KC_C * KC_AS + KC_C + 4 * KT) * sizeof(float);
}
static size_t kc_scan_smem(int KT, int VS) {
  return ((size_t)3 * KC_C * (KT + 4) + KC_C * KC_AS + KT + KC_C * 8 + KC_C * VS + KT * VS + 4 * VS * KC_C +
          (256 / KT) * VS * KT) * sizeof(float) + 3 * sizeof(uint64_t);
}
static int kc_padded_k(int K) { return K <= 64 ? 64 : 128; }
// tokens of a chunk (what the clamp of a growing gate's exponents counts by), and of a record
static int kc_chunk(int K, int chunk_size) {
  const int C = chunk_size < KC_C ? chunk_size : KC_C;
  return C < K ? C : K;
}
static int kc_record_tokens(int C) { return KC_C / C * C; }
static int64_t kc_records(int T, int K, int chunk_size) {
  const int L = kc_record_tokens(kc_chunk(K, chunk_size));
  return ((int64_t)T + L - 1) / L;
}
static int64_t kc_workspace_bytes(int B, int T, int HV, int K, int V, int chunk_size) {
  return (int64_t)B * HV * kc_records(T, K, chunk_size) * kc_record_floats(kc_padded_k(K), V) * 4 + 16;   // + alignment of the base
}

// tensor-core path (kda_mma.cu)
bool kch_kda_mma_supported(int K, int V, int chunk_size, float g_clamp_min, int dtype);
int64_t kch_kda_mma_workspace_bytes(int B, int T, int HV);
int kch_kda_chunk_mma(const void* q, const void* k, const void* v, const void* g, const void* beta,
                      const float* initial_state, void* o, float* final_state, int B, int T, int H, int HV,
                      float scale, float g_clamp_min, int64_t ld_qk, int64_t ld_v, int64_t ld_g, int64_t ld_beta,
                      void* workspace, int64_t workspace_bytes, void* stream, float gate_scale);

extern "C" int64_t kch_kda_chunk_workspace_bytes(int B, int T, int HV, int K, int V, int chunk_size) {
  if (B <= 0 || T <= 0 || HV <= 0 || K <= 0 || V <= 0 || chunk_size < 1) return 0;
  if (K > 128) return 0;                       // runs as the token recurrence
  int64_t need = kc_workspace_bytes(B, T, HV, K, V, chunk_size);
  // the dtype is not known here: size for whichever path may run
  if (kch_kda_mma_supported(K, V, chunk_size, 0.f, KCH_BF16)) {
    int64_t m = kch_kda_mma_workspace_bytes(B, T, HV);
    if (m > need) need = m;
  }
  return need;
}

static int kda_chunk_impl(const void* q, const void* k, const void* v, const void* g,
                          const void* beta, const float* initial_state, void* o,
                          float* final_state, int B, int T, int H, int HV, int K, int V,
                          int chunk_size, float scale, float g_clamp_min, int dtype, int64_t ld_qk,
                          int64_t ld_v, int64_t ld_g, int64_t ld_beta, void* workspace,
                          int64_t workspace_bytes, void* stream, float gate_scale) {
  if (ld_qk <= 0) ld_qk = (int64_t)H * K;
  if (ld_v <= 0) ld_v = (int64_t)HV * V;
  if (ld_g <= 0) ld_g = (int64_t)HV * K;
  if (ld_beta <= 0) ld_beta = HV;
  KCH_REQUIRE(H >= 1, "H=%d must be >= 1", H);
  KCH_REQUIRE(K >= 1, "K=%d must be >= 1", K);
  KCH_REQUIRE(V >= 1, "V=%d must be >= 1", V);
  KCH_REQUIRE(chunk_size >= 1, "chunk_size=%d must be >= 1", chunk_size);
  KCH_REQUIRE(HV >= 1 && HV % H == 0, "HV=%d must be divisible by H=%d (GVA factor)", HV, H);
  KCH_REQUIRE(B >= 0 && T >= 0, "B=%d T=%d", B, T);
  if (gate_scale != 0.f)
    KCH_REQUIRE(T > 0 && K <= 128 && kch_kda_mma_supported(K, V, chunk_size, g_clamp_min, dtype),
                "kch_kda_chunk_gate: the fused gate activation needs bf16, K = V = 128, chunk_size = 64 (K=%d V=%d chunk=%d)",
                K, V, chunk_size);
  if (K > 128)  // state slice + staging tiles exceed shared memory: same maths, token form
    return kch_kda_recurrent(q, k, v, g, beta, initial_state, o, final_state, B, T, H, HV, K, V, scale,
                             g_clamp_min, dtype, ld_qk, ld_v, ld_g, ld_beta, stream);
  if (B == 0) return KCH_OK;
  if (T > 0 && kch_kda_mma_supported(K, V, chunk_size, g_clamp_min, dtype))
    return kch_kda_chunk_mma(q, k, v, g, beta, initial_state, o, final_state, B, T, H, HV, scale, g_clamp_min,
                             ld_qk, ld_v, ld_g, ld_beta, workspace, workspace_bytes, stream, gate_scale);
  if (T == 0) {
    if (final_state) {
      size_t nb = (size_t)B * HV * K * V * sizeof(float);
      if (initial_state) KCH_CUDA_OK(cudaMemcpyAsync(final_state, initial_state, nb, cudaMemcpyDeviceToDevice, kch_stream(stream)));
      else KCH_CUDA_OK(cudaMemsetAsync(final_state, 0, nb, kch_stream(stream)));
    }
    return KCH_OK;
  }
  const int C = kc_chunk(K, chunk_size), L = kc_record_tokens(C), NT = (int)kc_records(T, K, chunk_size), KT = kc_padded_k(K);
  const int64_t need = kc_workspace_bytes(B, T, HV, K, V, chunk_size);
  KCH_REQUIRE(workspace && workspace_bytes >= need, "kch_kda_chunk: workspace %lld < %lld bytes",
              (long long)workspace_bytes, (long long)need);
  float* ws = (float*)(((uintptr_t)workspace + 15) & ~(uintptr_t)15);
  unsigned int* status = kch_status_device_ptr();
  KCH_REQUIRE(status != nullptr, "kch_kda_chunk: cannot resolve the device status word");
  cudaStream_t s = kch_stream(stream);
  // value columns of a CTA of the scan: 8, or 4 where twice the CTAs still get an SM each (beyond that two of them would share
  // one and read every operand row twice as often)
  const int VS = (int64_t)((V + 3) / 4) * HV * B <= KCH_SMS ? 4 : 8;
  // four elements a load: q, k, g (1), v (2)
  const int es = dtype == KCH_BF16 ? 2 : 4;
  const int vec = ((K % 4) == 0 && (ld_qk % 4) == 0 && (ld_g % 4) == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)g) % (4 * es)) == 0 ? 1 : 0) |
                  ((V % 4) == 0 && (ld_v % 4) == 0 && ((uintptr_t)v % (4 * es)) == 0 ? 2 : 0);
  const size_t smem1 = kc_prepare_smem(KT), smem2 = kc_scan_smem(KT, VS);
  const dim3 g1(NT, HV, B), g2((V + VS - 1) / VS, HV, B);
#define GO(T_, KT_, VS_)                                                                                       \
  do {                                                                                                    \
    KCH_CUDA_OK(cudaFuncSetAttribute(kda_chunk_prepare_kernel<T_, KT_>,                                   \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1));           \
    KCH_CUDA_OK(cudaFuncSetAttribute(kda_chunk_scan_kernel<T_, KT_, VS_>,                                      \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2));           \
    kda_chunk_prepare_kernel<T_, KT_><<<g1, 4 * KT_, smem1, s>>>((const T_*)q, (const T_*)k,              \
        (const T_*)v, (const T_*)g, (const T_*)beta, ws, T, H, HV, K, V, NT, L, C, scale, g_clamp_min,    \
        ld_qk, ld_v, ld_g, ld_beta, vec);                                                                        \
    kda_chunk_scan_kernel<T_, KT_, VS_><<<g2, 256, smem2, s>>>(ws, initial_state, (T_*)o, final_state, T, HV,  \
        K, V, NT, L, status);                                                                             \
  } while (0)
  KCH_DISPATCH_FLOAT(dtype, T_, {
    if (KT == 64) { if (VS == 4) GO(T_, 64, 4); else GO(T_, 64, 8); }
    else if (VS == 4) GO(T_, 128, 4);
    else GO(T_, 128, 8);
  });
#undef GO
  kch_note_launch(1);  // two kernels per call
  KCH_LAUNCH_OK();
  return KCH_OK;
}

extern "C" int kch_kda_chunk(const void* q, const void* k, const void* v, const void* g,
                             const void* beta, const float* initial_state, void* o,
                             float* final_state, int B, int T, int H, int HV, int K, int V,
                             int chunk_size, float scale, float g_clamp_min, int dtype, int64_t ld_qk,
                             int64_t ld_v, int64_t ld_g, int64_t ld_beta, void* workspace,
                             int64_t workspace_bytes, void* stream) {
  return kda_chunk_impl(q, k, v, g, beta, initial_state, o, final_state, B, T, H, HV, K, V, chunk_size, scale,
                        g_clamp_min, dtype, ld_qk, ld_v, ld_g, ld_beta, workspace, workspace_bytes, stream, 0.f);
}

extern "C" int kch_kda_chunk_gate_supported(int K, int V, int chunk_size, float g_clamp_min, int dtype) {
  return K <= 128 && kch_kda_mma_supported(K, V, chunk_size, g_clamp_min, dtype) ? 1 : 0;
}

extern "C" int kch_kda_chunk_gate(const void* q, const void* k, const void* v, const void* g_pre,
                                  const void* beta, const float* initial_state, void* o,
                                  float* final_state, int B, int T, int H, int HV, int K, int V,
                                  int chunk_size, float scale, float g_clamp_min, float gate_scale, int dtype,
                                  int64_t ld_qk, int64_t ld_v, int64_t ld_g, int64_t ld_beta, void* workspace,
                                  int64_t workspace_bytes, void* stream) {
  KCH_REQUIRE(gate_scale > 0.f, "kch_kda_chunk_gate: gate_scale=%g must be > 0", (double)gate_scale);
  return kda_chunk_impl(q, k, v, g_pre, beta, initial_state, o, final_state, B, T, H, HV, K, V, chunk_size, scale,
                        g_clamp_min, dtype, ld_qk, ld_v, ld_g, ld_beta, workspace, workspace_bytes, stream, gate_scale);
}
