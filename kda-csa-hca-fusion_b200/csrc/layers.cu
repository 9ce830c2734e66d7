// Whole layers in one call: the launches of a KDA, CSA or HCA layer over several tokens, issued from here one after the
// other.  Every launch is one of the library's own entry points with the arguments that the Python wrappers give it; what
// goes away is the host work between them (tensor objects, views, allocations and a ctypes call each: 15 to 20 us a launch,
// which is more than most of these kernels take below ~4000 tokens).  Intermediate results lie in one caller workspace, over one
// another where one is dead before the next is written.
#include <math.h>
#include <string.h>

#include "kch_common.cuh"

int kch_rownorm_groups(const void* x, int64_t ld, int groups, void* y, float* norms, int64_t rows, int c, int dtype,
                       int out_dtype, void* stream);      // elementwise.cu

namespace {
// 256-byte aligned pieces of a workspace; with a null base it only counts.  The pieces behind `again(mark)` lie where those
// behind `mark` did, which are not read any more when they are written (one stream, launch after launch).
struct Carve {
  uint8_t* base;
  int64_t used = 0, most = 0;
  explicit Carve(void* p) : base((uint8_t*)p) {}
  void* take(int64_t bytes) {
    void* p = base ? base + used : nullptr;
    used += (bytes + 255) & ~(int64_t)255;
    if (used > most) most = used;
    return p;
  }
  void again(int64_t mark) { used = mark; }
};
inline int64_t esize(int dtype) { return dtype == KCH_BF16 ? 2 : 4; }
inline const void* at(const void* p, int64_t elems, int dtype) { return (const uint8_t*)p + elems * esize(dtype); }
}  // namespace
#define LY_GO(expr)                 \
  do {                              \
    const int rc_ = (expr);         \
    if (rc_ != KCH_OK) return rc_;  \
  } while (0)

// ---- small helpers on the device -----------------------------------------------------------------------------------
// Rows of up to 9 matrices one after the other, then zero rows up to n: the fused weight of a call that brings its weights
// one by one.  One 16-byte chunk a thread (row bytes are a multiple of 16).
#define LY_MAX_PARTS 9
struct ConcatArgs {
  const uint8_t* src[LY_MAX_PARTS];
  int64_t ld[LY_MAX_PARTS];               // bytes between rows
  int end[LY_MAX_PARTS];
  int parts;
};
__global__ void concat_rows_kernel(ConcatArgs a, uint8_t* dst, int64_t row_bytes, int n) {
  const int64_t chunks = row_bytes / 16, i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= chunks * n) return;
  const int r = (int)(i / chunks);
  const int64_t o = (i % chunks) * 16;
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  int start = 0;
  for (int p = 0; p < a.parts; ++p) {
    if (r < a.end[p]) { v = *reinterpret_cast<const uint4*>(a.src[p] + (int64_t)(r - start) * a.ld[p] + o); break; }
    start = a.end[p];
  }
  *reinterpret_cast<uint4*>(dst + (int64_t)r * row_bytes + o) = v;
}

// rows of `width` elements, ld apart, as dense fp32
template <typename T>
__global__ void widen_rows_kernel(const T* __restrict__ x, int64_t ld, float* __restrict__ y, int64_t rows, int width) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows * width) y[i] = ldf(x + (i / width) * ld + i % width);
}

static int concat_rows(const kch_weight_part* parts, int count, void* dst, int K, int n, int dtype, cudaStream_t s) {
  ConcatArgs a = {};
  KCH_REQUIRE(count >= 1 && count <= LY_MAX_PARTS, "kch layer: %d weight parts", count);
  const int64_t row_bytes = K * esize(dtype);
  a.parts = count;
  int end = 0;
  for (int i = 0; i < count; ++i) {
    a.src[i] = (const uint8_t*)parts[i].w;
    a.ld[i] = parts[i].ld * esize(dtype);
    a.end[i] = end += parts[i].rows;
    KCH_REQUIRE(((row_bytes | a.ld[i] | (int64_t)(uintptr_t)parts[i].w) & 15) == 0, "kch layer: weight part %d is not 16-byte aligned", i);
  }
  KCH_REQUIRE(end <= n, "kch layer: %d weight rows, room for %d", end, n);
  const int64_t total = row_bytes / 16 * n;
  concat_rows_kernel<<<(unsigned)ceil_div64(total, 256), 256, 0, s>>>(a, (uint8_t*)dst, row_bytes, n);
  KCH_LAUNCH_OK();
  return KCH_OK;
}

// LayerNorm of the layer's input into the workspace, where there is one
static int layer_norm(const kch_layer_common* l, const void** x, int64_t* ld, void* xn, void* stream) {
  *x = l->x;
  *ld = l->ld_x;
  if (!l->norm_w) return KCH_OK;
  KCH_REQUIRE(l->ld_x == l->d, "kch layer: a normalised input has dense rows (ld %lld, d %d)", (long long)l->ld_x, l->d);
  LY_GO(kch_layernorm(l->x, l->norm_w, l->norm_b, xn, (int64_t)l->B * l->T, l->d, l->eps, l->dtype, l->norm_dtype, stream));
  *x = xn;
  *ld = l->d;
  return KCH_OK;
}
static int layer_checks(const kch_layer_common* l, const char* fn) {
  KCH_REQUIRE(l->B >= 1 && l->T >= 1 && l->d >= 1 && l->x, "%s: B=%d T=%d d=%d", fn, l->B, l->T, l->d);
  KCH_REQUIRE(l->dtype == KCH_F32 || l->dtype == KCH_BF16, "%s: dtype tag %d", fn, l->dtype);
  KCH_REQUIRE((l->norm_w == nullptr) == (l->norm_b == nullptr), "%s: LayerNorm weight and bias come together", fn);
  KCH_REQUIRE(!l->W_o || l->out, "%s: an output projection needs `out`", fn);
  return KCH_OK;
}
// o_proj (+ residual) of the heads' outputs, where the call asks for it
static int layer_out(const kch_layer_common* l, const void* o, int width, void* stream) {
  if (!l->W_o) return KCH_OK;
  return kch_linear(o, l->W_o, l->out, l->residual, (int64_t)l->B * l->T, l->d_out, width, width, l->ld_wo, l->d_out, l->ld_res,
                    l->dtype, stream);
}

// ---- CSA ----------------------------------------------------------------------------------------------------------------
struct CsaWs { void *xn, *w, *wq, *proj, *qq, *idx, *qn, *kn, *wf, *topk, *comp_n, *local, *core; float *comp, *kcomp; int64_t topk_bytes; };
static bool csa_raw_q(const kch_csa_layer_args* a) {
  return a->l.dtype == KCH_BF16 && a->c_I == 64 && a->T_blocks > 0 && a->n_q % 8 == 0 && ((int64_t)a->nh * a->c) % 8 == 0;
}
static int attend_key_dtype(int dtype, int c, int nh, float scale) {     // unit keys in bf16 for the tensor-core attention kernels
  return dtype == KCH_BF16 && c == 128 && nh <= 16 && fabsf(scale) <= 16.f ? KCH_BF16 : KCH_F32;
}
static int64_t csa_carve(const kch_csa_layer_args* a, void* base, CsaWs* w) {
  const kch_layer_common* l = &a->l;
  const int64_t rows = (int64_t)l->B * l->T, es = esize(l->dtype), nb = (int64_t)l->B * a->T_blocks;
  const int64_t ks = esize(attend_key_dtype(l->dtype, a->c, a->nh, a->scale));
  Carve c(base);
  w->w = a->W ? nullptr : c.take((int64_t)a->n_w * l->d * es);
  w->wq = a->Wq ? nullptr : c.take((int64_t)a->n_q * a->dc * es);
  w->proj = a->proj ? a->proj : c.take(rows * a->n_w * es);
  w->qq = c.take(rows * a->n_q * es);
  w->comp = a->comp ? a->comp : (float*)c.take(nb * a->c * 4);
  w->kcomp = a->kcomp ? a->kcomp : (float*)c.take(nb * a->c_I * 4);
  w->idx = a->topk > 0 ? c.take(rows * a->topk * 4) : nullptr;
  // the input projection's operand, then what the selection needs, then what the attention does
  const int64_t mark = c.used;
  w->xn = l->norm_w ? c.take(rows * l->d * es) : nullptr;
  c.again(mark);
  w->qn = w->kn = w->wf = w->topk = nullptr;
  w->topk_bytes = 0;
  if (a->topk > 0) {
    w->kn = c.take(nb * a->c_I * 4);
    w->wf = c.take(rows * a->nIh * 4);
    if (csa_raw_q(a)) {
      w->topk_bytes = kch_indexer_workspace_bytes_ex(l->B, l->T, a->T_blocks, KCH_BF16);
    } else {
      w->qn = c.take(rows * a->nIh * a->c_I * 4);
      w->topk_bytes = kch_indexer_workspace_bytes(l->B, l->T, a->T_blocks, a->nIh, a->c_I);
    }
    w->topk = c.take(w->topk_bytes);
  }
  c.again(mark);
  w->comp_n = c.take(nb * a->c * ks);
  w->local = a->sliding_window > 0 ? c.take(rows * a->c * ks) : nullptr;
  w->core = a->l.W_o ? c.take(rows * a->nh * a->c * es) : nullptr;
  return c.most;
}
static int csa_checks(const kch_csa_layer_args* a) {
  LY_GO(layer_checks(&a->l, "kch_csa_layer"));
  KCH_REQUIRE(a->m >= 1 && a->c >= 1 && a->c_I >= 1 && a->dc >= 1 && a->nh >= 1 && a->nIh >= 1 && a->topk >= 0 && a->sliding_window >= 0,
              "kch_csa_layer: m=%d c=%d c_I=%d dc=%d nh=%d nIh=%d topk=%d window=%d", a->m, a->c, a->c_I, a->dc, a->nh, a->nIh,
              a->topk, a->sliding_window);
  KCH_REQUIRE(a->T_blocks == a->l.T / a->m && a->T_blocks >= 1, "kch_csa_layer: %d tokens hold %d blocks of %d, T_blocks=%d",
              a->l.T, a->l.T / a->m, a->m, a->T_blocks);
  KCH_REQUIRE(a->n_w >= 4 * a->c + 2 * a->c_I + a->dc + a->nIh && a->n_q >= a->nh * a->c + a->nIh * a->c_I,
              "kch_csa_layer: fused widths %d, %d", a->n_w, a->n_q);
  KCH_REQUIRE(a->Ba && a->Bb && a->B_idx, "kch_csa_layer: the biases are missing");
  return KCH_OK;
}
extern "C" int64_t kch_csa_layer_workspace_bytes(const kch_csa_layer_args* a) {
  CsaWs w;
  return csa_carve(a, nullptr, &w);
}
extern "C" int kch_csa_layer(const kch_csa_layer_args* a, void* stream) {
  LY_GO(csa_checks(a));
  const kch_layer_common* l = &a->l;
  CsaWs w;
  KCH_REQUIRE(l->workspace && ((uintptr_t)l->workspace & 255) == 0 && csa_carve(a, l->workspace, &w) <= l->workspace_bytes,
              "kch_csa_layer: workspace of %lld bytes", (long long)l->workspace_bytes);
  cudaStream_t s = kch_stream(stream);
  const int dt = l->dtype, B = l->B, T = l->T, n = a->T_blocks, c = a->c, cI = a->c_I;
  const int64_t rows = (int64_t)B * T, Tc = (int64_t)n * a->m, nw = a->n_w;
  const void *x, *W = a->W, *Wq = a->Wq;
  int64_t ld_x, ldw = a->ld_w, ldwq = a->ld_wq;
  LY_GO(layer_norm(l, &x, &ld_x, w.xn, stream));
  if (!W) { LY_GO(concat_rows(a->parts, 8, w.w, l->d, a->n_w, dt, s)); W = w.w; ldw = l->d; }
  if (!Wq) { LY_GO(concat_rows(a->parts + 8, 2, w.wq, a->dc, a->n_q, dt, s)); Wq = w.wq; ldwq = a->dc; }
  LY_GO(kch_linear(x, W, w.proj, nullptr, rows, a->n_w, l->d, ld_x, ldw, nw, 0, dt, stream));
  const void *Ca = w.proj, *Cb = at(Ca, c, dt), *Za = at(Ca, 2 * c, dt), *Zb = at(Ca, 3 * c, dt), *Ki = at(Ca, 4 * c, dt),
             *Zi = at(Ca, 4 * c + cI, dt), *cQ = at(Ca, 4 * c + 2 * cI, dt), *wi = at(Ca, 4 * c + 2 * cI + a->dc, dt);
  LY_GO(kch_compress_kv_overlapped(Ca, Cb, Za, Zb, a->Ba, a->Bb, nullptr, nullptr, c, w.comp, B, Tc, c, a->m, nw, T, (int64_t)n * c,
                                   dt, a->bias_dtype, stream));
  LY_GO(kch_compress_kv(Ki, Zi, a->B_idx, w.kcomp, B, Tc, cI, a->m, nw, T, (int64_t)n * cI, dt, a->bias_dtype, stream));
  LY_GO(kch_linear(cQ, Wq, w.qq, nullptr, rows, a->n_q, a->dc, nw, ldwq, a->n_q, 0, dt, stream));
  if (a->topk > 0) {
    const void* qi = at(w.qq, (int64_t)a->nh * c, dt);
    LY_GO(kch_rownorm(w.kcomp, cI, w.kn, nullptr, (int64_t)B * n, cI, KCH_F32, KCH_F32, stream));
    const unsigned gw = (unsigned)ceil_div64(rows * a->nIh, 256);
    KCH_DISPATCH_FLOAT(dt, T_, (widen_rows_kernel<T_><<<gw, 256, 0, s>>>((const T_*)wi, nw, (float*)w.wf, rows, a->nIh)));
    KCH_LAUNCH_OK();
    if (csa_raw_q(a)) {
      LY_GO(kch_indexer_topk_ex(qi, KCH_BF16, a->n_q, 1, (const float*)w.kn, (const float*)w.wf, (int32_t*)w.idx, B, T, n, a->nIh, cI,
                                a->topk, 1.f, a->m, 0, -1, 0, 0, w.topk, w.topk_bytes, stream));
    } else {
      LY_GO(kch_rownorm_groups(qi, a->n_q, a->nIh, w.qn, nullptr, rows * a->nIh, cI, dt, KCH_F32, stream));
      LY_GO(kch_indexer_topk((const float*)w.qn, (const float*)w.kn, (const float*)w.wf, (int32_t*)w.idx, B, T, n, a->nIh, cI, a->topk,
                             1.f, a->m, 0, -1, 0, 0, w.topk, w.topk_bytes, stream));
    }
  }
  const int kdt = attend_key_dtype(dt, c, a->nh, a->scale);
  kch_attend_args t = {};
  t.q = w.qq; t.q_dtype = dt; t.q_ld = a->n_q; t.q_normalize = 1;
  t.B = B; t.T = T; t.nh = a->nh; t.c = c;
  if (a->topk > 0) {
    LY_GO(kch_rownorm(w.comp, c, w.comp_n, nullptr, (int64_t)B * n, c, KCH_F32, kdt, stream));
    t.comp = w.comp_n; t.comp_dtype = kdt; t.comp_ld = c; t.comp_batch_rows = n; t.n_comp = n;
    t.sel_indices = (const int32_t*)w.idx; t.topk = a->topk;
  }
  t.m = a->m; t.n_visible = -1;
  if (a->sliding_window > 0) {
    LY_GO(kch_rownorm(Ca, nw, w.local, nullptr, rows, c, dt, kdt, stream));
    t.win = w.local; t.win_dtype = kdt; t.win_ld = c; t.win_batch_rows = T; t.sliding_window = a->sliding_window;
  }
  t.sink = a->sink; t.sink_dtype = a->sink_dtype; t.scale = a->scale;
  t.out = l->W_o ? w.core : l->out; t.out_dtype = dt;
  LY_GO(kch_attend_distinct(&t, stream));
  return layer_out(l, t.out, a->nh * c, stream);
}

// ---- HCA ----------------------------------------------------------------------------------------------------------------
struct HcaWs { void *xn, *w, *proj, *q, *comp_n, *local, *core; float* comp; };
static int64_t hca_carve(const kch_hca_layer_args* a, void* base, HcaWs* w) {
  const kch_layer_common* l = &a->l;
  const int64_t rows = (int64_t)l->B * l->T, es = esize(l->dtype), nb = (int64_t)l->B * a->T_blocks;
  const int64_t ks = esize(attend_key_dtype(l->dtype, a->c, a->nh, a->scale));
  Carve c(base);
  w->w = a->W ? nullptr : c.take((int64_t)a->n_w * l->d * es);
  w->proj = a->proj ? a->proj : c.take(rows * a->n_w * es);
  w->q = c.take(rows * a->nh * a->c * es);
  w->comp = a->comp ? a->comp : (float*)c.take(nb * a->c * 4);
  const int64_t mark = c.used;            // the input projection's operand, then what the attention needs
  w->xn = l->norm_w ? c.take(rows * l->d * es) : nullptr;
  c.again(mark);
  w->comp_n = c.take(nb * a->c * ks);
  w->local = a->sliding_window > 0 ? c.take(rows * a->c * ks) : nullptr;
  w->core = l->W_o ? c.take(rows * a->nh * a->c * es) : nullptr;
  return c.most;
}
extern "C" int64_t kch_hca_layer_workspace_bytes(const kch_hca_layer_args* a) {
  HcaWs w;
  return hca_carve(a, nullptr, &w);
}
extern "C" int kch_hca_layer(const kch_hca_layer_args* a, void* stream) {
  const kch_layer_common* l = &a->l;
  LY_GO(layer_checks(l, "kch_hca_layer"));
  KCH_REQUIRE(a->m2 >= 1 && a->c >= 1 && a->dc >= 1 && a->nh >= 1 && a->sliding_window >= 0, "kch_hca_layer: m2=%d c=%d dc=%d nh=%d window=%d",
              a->m2, a->c, a->dc, a->nh, a->sliding_window);
  KCH_REQUIRE(a->T_blocks == l->T / a->m2 && a->T_blocks >= 1, "kch_hca_layer: %d tokens hold %d blocks of %d, T_blocks=%d", l->T,
              l->T / a->m2, a->m2, a->T_blocks);
  KCH_REQUIRE(a->n_w >= 2 * a->c + a->dc && a->Wq && a->B_pos, "kch_hca_layer: fused width %d", a->n_w);
  HcaWs w;
  KCH_REQUIRE(l->workspace && ((uintptr_t)l->workspace & 255) == 0 && hca_carve(a, l->workspace, &w) <= l->workspace_bytes,
              "kch_hca_layer: workspace of %lld bytes", (long long)l->workspace_bytes);
  cudaStream_t s = kch_stream(stream);
  const int dt = l->dtype, B = l->B, T = l->T, n = a->T_blocks, c = a->c;
  const int64_t rows = (int64_t)B * T, nw = a->n_w;
  const void *x, *W = a->W;
  int64_t ld_x, ldw = a->ld_w;
  LY_GO(layer_norm(l, &x, &ld_x, w.xn, stream));
  if (!W) { LY_GO(concat_rows(a->parts, 3, w.w, l->d, a->n_w, dt, s)); W = w.w; ldw = l->d; }
  LY_GO(kch_linear(x, W, w.proj, nullptr, rows, a->n_w, l->d, ld_x, ldw, nw, 0, dt, stream));
  LY_GO(kch_compress_kv(w.proj, at(w.proj, c, dt), a->B_pos, w.comp, B, (int64_t)n * a->m2, c, a->m2, nw, T, (int64_t)n * c, dt,
                        a->bias_dtype, stream));
  const int kdt = attend_key_dtype(dt, c, a->nh, a->scale);
  LY_GO(kch_rownorm(w.comp, c, w.comp_n, nullptr, (int64_t)B * n, c, KCH_F32, kdt, stream));
  LY_GO(kch_linear(at(w.proj, 2 * c, dt), a->Wq, w.q, nullptr, rows, a->nh * c, a->dc, nw, a->ld_wq, (int64_t)a->nh * c, 0, dt, stream));
  kch_attend_args t = {};
  t.q = w.q; t.q_dtype = dt; t.q_ld = (int64_t)a->nh * c; t.q_normalize = 1;
  t.B = B; t.T = T; t.nh = a->nh; t.c = c;
  t.comp = w.comp_n; t.comp_dtype = kdt; t.comp_ld = c; t.comp_batch_rows = n; t.n_comp = n;
  t.m = a->m2; t.n_visible = -1;
  if (a->sliding_window > 0) {
    LY_GO(kch_rownorm(w.proj, nw, w.local, nullptr, rows, c, dt, kdt, stream));
    t.win = w.local; t.win_dtype = kdt; t.win_ld = c; t.win_batch_rows = T; t.sliding_window = a->sliding_window;
  }
  t.sink = a->sink; t.sink_dtype = a->sink_dtype; t.scale = a->scale;
  t.out = l->W_o ? w.core : l->out; t.out_dtype = dt;
  LY_GO(kch_attend(&t, stream));
  return layer_out(l, t.out, a->nh * c, stream);
}

// ---- KDA ----------------------------------------------------------------------------------------------------------------
struct KdaWs { void *xn, *xc, *proj, *g, *o, *chunk; int64_t chunk_bytes; };
static bool kda_fused_norm(const kch_kda_layer_args* a) {
  const kch_layer_common* l = &a->l;
  return l->norm_w && l->dtype == KCH_BF16 && l->T >= 2 && l->d % 256 == 0 && l->d <= 2048;
}
static bool kda_chunked(const kch_kda_layer_args* a) { return a->chunk_size >= 1 && a->l.T >= a->chunk_size; }
static bool kda_raw_gate(const kch_kda_layer_args* a) {
  return kda_chunked(a) && a->decay_scale > 0.f && kch_kda_chunk_gate_supported(a->K, a->V, a->chunk_size, a->g_clamp_min, a->l.dtype);
}
static int64_t kda_carve(const kch_kda_layer_args* a, void* base, KdaWs* w) {
  const kch_layer_common* l = &a->l;
  const int64_t rows = (int64_t)l->B * l->T, es = esize(l->dtype);
  Carve c(base);
  w->proj = c.take(rows * a->n_w * es);
  w->g = c.take(rows * a->HV * a->K * es);
  w->o = c.take(rows * a->HV * a->V * es);
  const int64_t mark = c.used;            // the input projection's operand, then the chunk records
  w->xn = l->norm_w && !kda_fused_norm(a) ? c.take(rows * l->d * es) : nullptr;
  w->xc = c.take(rows * l->d * es);
  c.again(mark);
  w->chunk_bytes = kda_chunked(a) ? kch_kda_chunk_workspace_bytes(l->B, l->T, a->HV, a->K, a->V, a->chunk_size) : 0;
  w->chunk = c.take(w->chunk_bytes);
  return c.most;
}
extern "C" int64_t kch_kda_layer_workspace_bytes(const kch_kda_layer_args* a) {
  KdaWs w;
  return kda_carve(a, nullptr, &w);
}
extern "C" int kch_kda_layer(const kch_kda_layer_args* a, void* stream) {
  const kch_layer_common* l = &a->l;
  LY_GO(layer_checks(l, "kch_kda_layer"));
  KCH_REQUIRE(l->T >= 2 && l->ld_x == l->d && l->W_o, "kch_kda_layer: T=%d ld_x=%lld", l->T, (long long)l->ld_x);
  KCH_REQUIRE(a->H >= 1 && a->HV >= 1 && a->HV % a->H == 0 && a->K >= 1 && a->V >= 1, "kch_kda_layer: H=%d HV=%d K=%d V=%d", a->H, a->HV, a->K, a->V);
  const int nq = a->H * a->K, nv = a->HV * a->V, used = 2 * nq + nv + a->K + a->HV;
  KCH_REQUIRE(a->n_w >= used && a->W && a->W_gup && a->conv_w && a->conv_b && a->lookback_out, "kch_kda_layer: fused width %d of %d", a->n_w, used);
  KdaWs w;
  KCH_REQUIRE(l->workspace && ((uintptr_t)l->workspace & 255) == 0 && kda_carve(a, l->workspace, &w) <= l->workspace_bytes,
              "kch_kda_layer: workspace of %lld bytes", (long long)l->workspace_bytes);
  const int dt = l->dtype, B = l->B, T = l->T;
  const int64_t rows = (int64_t)B * T, es = esize(dt), nw = a->n_w;
  if (kda_fused_norm(a)) {
    LY_GO(kch_layernorm_short_conv(l->x, l->norm_w, l->norm_b, l->eps, a->lookback, a->conv_w, a->conv_b, w.xc, a->lookback_out, B, T, l->d,
                                   dt, l->norm_dtype, stream));
  } else {
    const void* x;
    int64_t ld_x;
    LY_GO(layer_norm(l, &x, &ld_x, w.xn, stream));
    LY_GO(kch_short_conv(x, a->lookback, a->conv_w, a->conv_b, w.xc, B, T, l->d, dt, stream));
    // the last two rows of every sequence
    const size_t two = (size_t)2 * l->d * es;
    KCH_CUDA_OK(cudaMemcpy2DAsync(a->lookback_out, two, at(x, (int64_t)(T - 2) * l->d, dt), (size_t)T * l->d * es, two, B,
                                  cudaMemcpyDeviceToDevice, kch_stream(stream)));
  }
  const bool raw = kda_raw_gate(a);
  kch_epilogue ep = {};
  const int ends[5] = {nq, 2 * nq, 2 * nq + nv, 2 * nq + nv + a->K, a->n_w};
  const int acts[5] = {KCH_ACT_SILU_L2NORM, KCH_ACT_SILU_L2NORM, KCH_ACT_SILU, 0, KCH_ACT_SIGMOID};
  ep.n_segments = 5;
  ep.group = a->K;
  memcpy(ep.seg_end, ends, sizeof(ends));
  memcpy(ep.seg_act, acts, sizeof(acts));
  LY_GO(kch_linear_ex(w.xc, a->W, w.proj, nullptr, rows, a->n_w, l->d, l->d, a->ld_w, nw, 0, dt, &ep, stream));
  kch_epilogue eg = {};
  eg.n_segments = 1;
  eg.group = 1;
  eg.seg_end[0] = a->HV * a->K;
  eg.seg_act[0] = KCH_ACT_NEG_SOFTPLUS;
  eg.seg_param[0] = a->decay_scale;
  LY_GO(kch_linear_ex(at(w.proj, 2 * nq + nv, dt), a->W_gup, w.g, nullptr, rows, a->HV * a->K, a->K, nw, a->ld_wg, (int64_t)a->HV * a->K, 0,
                      dt, raw ? nullptr : &eg, stream));
  // q, k, v and beta are column slices of the fused projection; what the operator cannot read in place is refused by it
  const void *q = w.proj, *k = at(q, nq, dt), *v = at(q, 2 * nq, dt), *beta = at(q, 2 * nq + nv + a->K, dt);
  const int64_t ldg = (int64_t)a->HV * a->K;
  if (!kda_chunked(a)) {
    LY_GO(kch_kda_recurrent(q, k, v, w.g, beta, a->state, w.o, a->state_out, B, T, a->H, a->HV, a->K, a->V, a->scale, a->g_clamp_min, dt, nw, nw,
                            ldg, nw, stream));
  } else if (raw) {
    LY_GO(kch_kda_chunk_gate(q, k, v, w.g, beta, a->state, w.o, a->state_out, B, T, a->H, a->HV, a->K, a->V, a->chunk_size, a->scale,
                             a->g_clamp_min, a->decay_scale, dt, nw, nw, ldg, nw, w.chunk, w.chunk_bytes, stream));
  } else {
    LY_GO(kch_kda_chunk(q, k, v, w.g, beta, a->state, w.o, a->state_out, B, T, a->H, a->HV, a->K, a->V, a->chunk_size, a->scale, a->g_clamp_min,
                        dt, nw, nw, ldg, nw, w.chunk, w.chunk_bytes, stream));
  }
  return layer_out(l, w.o, a->HV * a->V, stream);
}

// ---- a prompt into an empty or block-aligned cache --------------------------------------------------------------------
extern "C" int64_t kch_cache_append_prompt_workspace_bytes(const kch_cache_append_args* a, int64_t T) {
  if (!a || a->m < 1 || T < 0) return 0;
  Carve c(nullptr);
  c.take(a->B * (T / a->m) * (int64_t)a->c * 4);
  c.take(a->B * (T / a->m) * (int64_t)a->c_I * 4);
  return c.used;
}
extern "C" int kch_cache_append_prompt(const kch_cache_append_args* a, int64_t T, int64_t bs_c, int64_t bs_i, int64_t ring_n,
                                       int64_t tokens_seen, const float* rows, const float* key_rows, void* workspace,
                                       int64_t workspace_bytes, void* stream) {
  KCH_REQUIRE(a && a->B >= 1 && a->c >= 1 && a->m >= 1 && T >= 1, "kch_cache_append_prompt: incomplete arguments");
  KCH_REQUIRE(a->acc_len == 0 && a->comp_kind == a->dtype, "kch_cache_append_prompt: an open block (%d tokens) or 8-bit rows (kind %d)",
              a->acc_len, a->comp_kind);
  const int64_t n = T / a->m;
  const bool csa = a->Cb != nullptr;
  if (n > 0) {
    KCH_REQUIRE(a->comp && a->comp_norms && a->Ba && a->n_blocks >= 0 && a->n_blocks + n <= a->capacity && (!csa || (a->kcomp && a->kcomp_norms && a->Bb && a->B_idx)),
                "kch_cache_append_prompt: no room for %lld rows behind %d of %lld", (long long)n, a->n_blocks, (long long)a->capacity);
    KCH_REQUIRE(a->ld_c >= a->c && (a->B == 1 || bs_c % a->ld_c == 0) && (!csa || (a->ld_i >= a->c_I && (a->B == 1 || bs_i % a->ld_i == 0))),
                "kch_cache_append_prompt: sequences %lld / %lld elements apart, tokens %lld / %lld", (long long)bs_c, (long long)bs_i,
                (long long)a->ld_c, (long long)a->ld_i);
    Carve w(workspace);
    float* r = (float*)w.take(a->B * n * a->c * 4);
    float* k = (float*)w.take(a->B * n * a->c_I * 4);
    KCH_REQUIRE((rows && (!csa || key_rows)) || (workspace && w.used <= workspace_bytes), "kch_cache_append_prompt: workspace of %lld bytes",
                (long long)workspace_bytes);
    const int64_t br = a->B > 1 ? bs_c / a->ld_c : T;
    if (!rows) {
      if (csa)
        LY_GO(kch_compress_kv_overlapped(a->Ca, a->Cb, a->Za, a->Zb, a->Ba, a->Bb, a->has_prev ? a->prev_Cb : nullptr,
                                         a->has_prev ? a->prev_Zb : nullptr, a->c, r, a->B, n * a->m, a->c, a->m, a->ld_c, br, n * a->c,
                                         a->dtype, a->dtype, stream));
      else
        LY_GO(kch_compress_kv(a->Ca, a->Za, a->Ba, r, a->B, n * a->m, a->c, a->m, a->ld_c, br, n * a->c, a->dtype, a->dtype, stream));
      rows = r;
    }
    LY_GO(kch_cache_store_rows(rows, n, a->c, a->B, a->comp, a->comp_norms, a->capacity, a->n_blocks, a->dtype, stream));
    if (csa) {
      if (!key_rows) {
        LY_GO(kch_compress_kv(a->K_idx, a->Z_idx, a->B_idx, k, a->B, n * a->m, a->c_I, a->m, a->ld_i, a->B > 1 ? bs_i / a->ld_i : T,
                              n * a->c_I, a->dtype, a->dtype, stream));
        key_rows = k;
      }
      LY_GO(kch_cache_store_rows(key_rows, n, a->c_I, a->B, a->kcomp, a->kcomp_norms, a->capacity, a->n_blocks, a->dtype, stream));
    }
  }
  return kch_cache_append_rows(a, T, bs_c, bs_i, ring_n, tokens_seen, stream);
}
