// Linear layer  C[M,N] = A[M,K] . W[N,K]^T  (nn.Linear weight layout), fp32 accumulation,
// result rounded once to the storage type, optional residual add (in fp32, rounded once more, which
// is what `residual + o_proj(o)` does on stored tensors).
//
// This file holds the CUDA-core versions: gemm_f32_kernel for fp32 operands that 16-byte copies can read, and
// gemm_simt_kernel for any shape, any leading dimensions, fp32 or bf16: what neither the former nor the tensor-core
// kernel takes (see gemm_tcgen05.cu).
#include "kch_common.cuh"

#define SG_BM 64
#define SG_BN 64
#define SG_BK 16

template <typename T>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T* __restrict__ A, const T* __restrict__ W, T* __restrict__ C,
                 const T* __restrict__ R, int64_t M, int N, int K, int64_t lda, int64_t ldw,
                 int64_t ldc, int64_t ldr) {
  __shared__ float sa[SG_BK][SG_BM + 1];
  __shared__ float sw[SG_BK][SG_BN + 1];
  const int64_t m0 = (int64_t)blockIdx.x * SG_BM;
  const int n0 = blockIdx.y * SG_BN;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += SG_BK) {
    for (int idx = threadIdx.x; idx < SG_BM * SG_BK; idx += 256) {
      int r = idx / SG_BK, kk = idx % SG_BK;
      int64_t mm = m0 + r;
      sa[kk][r] = (mm < M && k0 + kk < K) ? ldf(A + mm * lda + k0 + kk) : 0.f;
    }
    for (int idx = threadIdx.x; idx < SG_BN * SG_BK; idx += 256) {
      int r = idx / SG_BK, kk = idx % SG_BK;
      int nn = n0 + r;
      sw[kk][r] = (nn < N && k0 + kk < K) ? ldf(W + (int64_t)nn * ldw + k0 + kk) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < SG_BK; ++kk) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = sa[kk][ty * 4 + i]; w[i] = sw[kk][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int64_t mm = m0 + ty * 4 + i;
    if (mm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int nn = n0 + tx * 4 + j;
      if (nn >= N) continue;
      float v = round_to<T>(acc[i][j]);
      if (R) v += ldf(R + mm * ldr + nn);
      stf(C + mm * ldc + nn, v);
    }
  }
}

// ---- fp32, 16-byte aligned operands -----------------------------------------------------------------------------------
// The kernel above loads scalars and has one buffer: every 16-wide step of K waits for global memory, 45 us for
// 662 x 840 x 256 (6 TFLOP/s) whatever the tile count.  Here 16-byte cp.async copies run GF_STAGES - 1 steps of 32 ahead, the
// operands stay in their row-major layout in shared memory (36-float rows: the 8 rows of a quarter warp's 16-byte reads fall
// into distinct banks) and a thread multiplies four consecutive k of a 4 x 4 block per 8 such reads.  Tiles of 32 x 64: the
// small models' 500 to 2000 rows give 80 to 900 CTAs.  Two thread groups take the two halves of each step of K and add up at
// the end: a warp per scheduler issues an instruction every ~2.5 cycles only (the 15 products of the default stack, 662 rows:
// 528 us scalar, 175 with one group, 151 with two).  Bound: the shared-memory return path, 32 cycles per 4 x 4 x 4 block of a
// warp against 16 of the FMA pipe, then the latency of the copies.
// Activation segments are applied to the sums (same functions and rounding as kch_activation).
#define GF_BM 32
#define GF_BN 64
#define GF_BK 32
#define GF_LD 36
#define GF_STAGES 4
#define GF_KG 2
#define GF_STAGE_FLOATS ((GF_BM + GF_BN) * GF_LD)

struct GfEpilogue {
  int nseg;
  int end[8], act[8];
  float param[8];
  int group;                             // silu + L2 norm: divides 64, segments start and end on multiples of 64
};

__global__ void __launch_bounds__(128 * GF_KG)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                const float* __restrict__ R, int64_t M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, int64_t ldr,
                const __grid_constant__ GfEpilogue ep) {
  extern __shared__ __align__(16) float gf_smem[];
  const int64_t m0 = (int64_t)blockIdx.x * GF_BM;
  const int n0 = blockIdx.y * GF_BN;
  const int tid = threadIdx.x, tx = tid & 15, ty = (tid >> 4) & 7, kg = tid >> 7;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(gf_smem);
  const int KT = (K + GF_BK - 1) / GF_BK;
  auto copy16 = [](uint32_t dst, const float* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
  };
  const int lr = tid >> 3, lk = (tid & 7) * 4;       // 32 rows x 8 granules of 4 floats per pass
  auto issue = [&](int kt) {
    if (kt < KT) {
      const uint32_t st = sbase + (uint32_t)(kt % GF_STAGES) * (GF_STAGE_FLOATS * 4);
      const int k = kt * GF_BK + lk;
      const bool kok = k < K;
#pragma unroll
      for (int p = 0; p < GF_BM / 32; ++p) {
        const int r = lr + 32 * p;
        const bool on = kok && m0 + r < M;
        copy16(st + (uint32_t)(r * GF_LD + lk) * 4, on ? A + (m0 + r) * lda + k : A, on);
      }
#pragma unroll
      for (int p = 0; p < GF_BN / 32; ++p) {
        const int r = lr + 32 * p;
        const bool on = kok && n0 + r < N;
        copy16(st + (uint32_t)((GF_BM + r) * GF_LD + lk) * 4, on ? W + (int64_t)(n0 + r) * ldw + k : W, on);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < GF_STAGES - 1; ++s) issue(s);
  float acc[4][4] = {};                              // rows ty + 8 i, columns tx + 16 j
  for (int kt = 0; kt < KT; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GF_STAGES - 2) : "memory");
    __syncthreads();                                 // step kt has landed for all; the stage refilled below was read in step kt - 1
    issue(kt + GF_STAGES - 1);
    const float* sa = gf_smem + (kt % GF_STAGES) * GF_STAGE_FLOATS + ty * GF_LD;
    const float* sw = gf_smem + (kt % GF_STAGES) * GF_STAGE_FLOATS + (GF_BM + tx) * GF_LD;
#pragma unroll
    for (int kk = 0; kk < GF_BK / GF_KG; kk += 4) {
      const int k4 = kg * (GF_BK / GF_KG) + kk;
      float4 a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const float4*>(sa + 8 * i * GF_LD + k4);
        w[i] = *reinterpret_cast<const float4*>(sw + 16 * i * GF_LD + k4);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    }
  }
  // the two halves of each step of K: thread group kg finishes rows 2 kg and 2 kg + 1 of the four.  (Columns past K were
  // zero-filled in both operands; rows past M / N are not stored.)
  float4* xch = reinterpret_cast<float4*>(gf_smem);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    xch[(i * GF_KG + kg) * 128 + (tid & 127)] = kg ? make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3])
                                                   : make_float4(acc[2 + i][0], acc[2 + i][1], acc[2 + i][2], acc[2 + i][3]);
  }
  __syncthreads();
  float c[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 o = xch[(i * GF_KG + 1 - kg) * 128 + (tid & 127)];
    c[i][0] = (kg ? acc[2 + i][0] : acc[i][0]) + o.x; c[i][1] = (kg ? acc[2 + i][1] : acc[i][1]) + o.y;
    c[i][2] = (kg ? acc[2 + i][2] : acc[i][2]) + o.z; c[i][3] = (kg ? acc[2 + i][3] : acc[i][3]) + o.w;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int nn = n0 + tx + 16 * j;
    int act = 0;
    float param = 0.f;
    for (int s = ep.nseg - 1; s >= 0; --s)
      if (nn < ep.end[s]) { act = ep.act[s]; param = ep.param[s]; }
    if (act == KCH_ACT_SILU || act == KCH_ACT_SILU_L2NORM) {
#pragma unroll
      for (int i = 0; i < 2; ++i) c[i][j] = silu_f(c[i][j]);
    } else if (act == KCH_ACT_SIGMOID) {
#pragma unroll
      for (int i = 0; i < 2; ++i) c[i][j] = sigmoid_f(c[i][j]);
    } else if (act == KCH_ACT_NEG_SOFTPLUS) {
#pragma unroll
      for (int i = 0; i < 2; ++i) c[i][j] = -softplus_f(c[i][j]) * param;
    }
  }
  {
    // silu + L2 norm: the segments cover whole 64-column tiles, so this holds for all columns of the CTA or for none
    int act = 0;
    for (int s = ep.nseg - 1; s >= 0; --s)
      if (n0 < ep.end[s]) act = ep.act[s];
    if (act == KCH_ACT_SILU_L2NORM) {
      // a group of 64: the 16 lanes of a row and their four columns; of 32: column pairs {0, 1}, {2, 3}; of 16: one column;
      // narrower: `group` neighbouring lanes
      const int group = ep.group, span = group < 16 ? group : 16, cols = group > 16 ? group / 16 : 1;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float ss[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) ss[j] = c[i][j] * c[i][j];
        if (cols >= 2) { ss[0] += ss[1]; ss[1] = ss[0]; ss[2] += ss[3]; ss[3] = ss[2]; }
        if (cols == 4) { ss[0] += ss[2]; ss[1] = ss[2] = ss[3] = ss[0]; }
        for (int o = span >> 1; o > 0; o >>= 1)
#pragma unroll
          for (int j = 0; j < 4; ++j) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], o);
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] /= fmaxf(sqrtf(ss[j]), 1e-12f);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int64_t mm = m0 + ty + 8 * (2 * kg + i);
    if (mm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int nn = n0 + tx + 16 * j;
      if (nn >= N) continue;
      float v = c[i][j];
      if (R) v += R[mm * ldr + nn];
      C[mm * ldc + nn] = v;
    }
  }
}

// Row counts up to 2^31 tiles; K and the strides keep every 16-byte copy aligned.
static bool gemm_f32_ok(const void* A, const void* W, int64_t M, int N, int K, int64_t lda, int64_t ldw, int dtype) {
  return dtype == KCH_F32 && (K % 4) == 0 && (lda % 4) == 0 && (ldw % 4) == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 &&
         (N + GF_BN - 1) / GF_BN <= 65535 && ceil_div64(M, GF_BM) <= 0x7FFFFFFF;
}

// Can the segments of `e` be applied by gemm_f32_kernel?  A silu + L2-norm segment has to consist of whole 64-column tiles
// and its groups have to divide them.
bool kch_linear_f32_epilogue_ok(const kch_epilogue* e, const void* A, const void* W, int64_t M, int N, int K, int64_t lda,
                                int64_t ldw, int dtype) {
  if (!gemm_f32_ok(A, W, M, N, K, lda, ldw, dtype)) return false;
  int start = 0;
  for (int i = 0; i < e->n_segments; ++i) {
    const int end = e->seg_end[i], act = e->seg_act[i];
    if (end <= start || end > N) return false;                    // named by the general path
    if (act < 0 || act > KCH_ACT_SILU_L2NORM) return false;
    if (act == KCH_ACT_SILU_L2NORM && (start % 64 || end % 64 || e->group < 1 || e->group > 64 || 64 % e->group)) return false;
    start = end;
  }
  return true;
}

int kch_linear_f32(const void* A, const void* W, void* C, const void* residual, int64_t M, int N, int K, int64_t lda,
                   int64_t ldw, int64_t ldc, int64_t ldr, const kch_epilogue* e, void* stream) {
  GfEpilogue ep = {};
  if (e) {
    ep.nseg = e->n_segments;
    ep.group = e->group;
    for (int i = 0; i < e->n_segments; ++i) { ep.end[i] = e->seg_end[i]; ep.act[i] = e->seg_act[i]; ep.param[i] = e->seg_param[i]; }
  }
  const int smem = GF_STAGES * GF_STAGE_FLOATS * 4;
  KCH_CUDA_OK(cudaFuncSetAttribute(gemm_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  dim3 grid((unsigned)ceil_div64(M, GF_BM), (N + GF_BN - 1) / GF_BN);
  gemm_f32_kernel<<<grid, 128 * GF_KG, smem, kch_stream(stream)>>>((const float*)A, (const float*)W, (float*)C, (const float*)residual,
                                                          M, N, K, lda, ldw, ldc, ldr, ep);
  KCH_LAUNCH_OK();
  return KCH_OK;
}

int kch_linear_simt(const void* A, const void* W, void* C, const void* residual, int64_t M, int N, int K,
                    int64_t lda, int64_t ldw, int64_t ldc, int64_t ldr, int dtype, void* stream) {
  if (M == 0 || N == 0) return KCH_OK;
  if (gemm_f32_ok(A, W, M, N, K, lda, ldw, dtype)) return kch_linear_f32(A, W, C, residual, M, N, K, lda, ldw, ldc, ldr, nullptr, stream);
  dim3 grid((unsigned)ceil_div64(M, SG_BM), (N + SG_BN - 1) / SG_BN), block(256);
  KCH_DISPATCH_FLOAT(dtype, T, (gemm_simt_kernel<T><<<grid, block, 0, kch_stream(stream)>>>(
      (const T*)A, (const T*)W, (T*)C, (const T*)residual, M, N, K, lda, ldw, ldc, ldr)));
  KCH_LAUNCH_OK();
  return KCH_OK;
}
