// Chains of launches enqueued by one call: the sparse MoE block's inference forward after its router GEMM, and the
// forward and backward of the expert MLP with LoRA.  At small sizes the kernels of a chain take less time than a host
// that goes back to Python between them (a decode step: 45 us of kernels, 190 us of host); nothing here touches device
// memory or changes what is launched.
#include <cmath>

#include "common.cuh"

using namespace moe;

namespace {

struct Carve {  // consecutive 256-byte aligned pieces of one scratch buffer
  uint8_t* base;
  size_t used = 0;
  void* take(size_t bytes) {
    void* p = base ? base + used : nullptr;
    used += (bytes + 255) & ~(size_t)255;
    return p;
  }
};

struct BlockScratch {
  void *weights, *experts, *counts, *sorted_of, *source_of, *sort_ws, *gemm_ws, *xs, *h, *y;
  size_t sort_bytes, gemm_bytes, total;
};

BlockScratch carve(void* base, int64_t T, int H, int I, int E, int k, int dtype) {
  Carve c{(uint8_t*)base};
  BlockScratch b;
  const int64_t M = T * k;
  const size_t esz = dtype_size(dtype);
  b.sort_bytes = moe_sort_workspace_bytes(M, E);
  b.gemm_bytes = moe_grouped_gemm_workspace_bytes(0, M, I, H, E);
  b.weights = c.take((size_t)M * esz);
  b.experts = c.take((size_t)M * sizeof(int64_t));
  b.counts = c.take((size_t)E * sizeof(int32_t));
  b.sorted_of = c.take((size_t)M * sizeof(int32_t));
  b.source_of = c.take((size_t)M * sizeof(int32_t));
  b.sort_ws = c.take(b.sort_bytes);
  b.gemm_ws = c.take(b.gemm_bytes);
  b.h = c.take((size_t)M * I * esz);
  b.xs = c.take((size_t)M * H * esz);
  b.y = b.xs;  // the expanded tokens have been read when the down projection writes
  b.total = c.used;
  return b;
}

bool block_shape_ok(int64_t T, int H, int I, int E, int k, int dtype) {
  return T > 0 && H > 0 && I > 0 && E > 0 && E <= 1024 && k > 0 && k <= 32 && k <= E && T <= 0x7fffffffLL &&
         T * k <= 0x7fffffffLL - 1024 && is_float_dtype(dtype);
}

// The factor s of a LoRA product as thin * 2^log2.  `thin` goes onto the fp32 accumulator of the thin factor (t = s x A^T,
// d = s dy B), which is then rounded to 16 bits; 2^log2 onto the accumulators of the products with the thin factor.
// bf16 has fp32's range: all of s in one go.  In fp16 it would cost thin factors small ones their low bits or large ones
// their range: 1 <= |thin| < 2, and +-1 for powers of two, so that the thin factors are held as they are.
struct Factor {
  float thin = 1.f;
  int log2 = 0;
  Factor(float s, int dtype) : thin(s) {
    if (dtype != MOE_F16 || s == 0.f || !std::isfinite(s)) return;
    thin = 2.f * std::frexp(s, &log2);
    --log2;
  }
  float pow2() const { return std::ldexp(1.f, log2); }
};

// Whether the accumulators can be rescaled by the factors (by at most 2^15 between two products).
bool factors_ok(const Factor* f) {
  for (int i = 0; i < 3; ++i)
    if (f[i].log2 < -7 || f[i].log2 > 7) return false;
  return true;
}

}  // namespace

MOE_API size_t moe_block_fwd_scratch_bytes(int64_t T, int H, int I, int E, int k, int dtype) {
  return block_shape_ok(T, H, I, E, k, dtype) ? carve(nullptr, T, H, I, E, k, dtype).total : 0;
}

MOE_API int moe_block_fwd(const void* x, const void* logits, const void* w_gate, const void* w_up, const void* w_down,
                          void* out, int64_t T, int H, int I, int E, int k, int norm_topk, int dtype, void* scratch,
                          size_t scratch_bytes, void* stream) {
  if (!is_float_dtype(dtype)) return MOE_ERR_DTYPE;
  if (!block_shape_ok(T, H, I, E, k, dtype)) return MOE_ERR_SHAPE;
  if (!x || !logits || !w_gate || !w_up || !w_down || !out || !scratch) return MOE_ERR_NULL;
  const BlockScratch b = carve(scratch, T, H, I, E, k, dtype);
  if (((uintptr_t)scratch & 255) || scratch_bytes < b.total) return MOE_ERR_WORKSPACE;
  // what the fused gate / up kernel refuses is refused here, before anything is enqueued
  if (dtype == MOE_F32 || H % 8 || I % 8 || moe_get_gemm_path() != MOE_PATH_AUTO || (((uintptr_t)w_gate | (uintptr_t)w_up) & 15))
    return MOE_ERR_UNSUPPORTED;
  const int64_t M = T * k;
  int st;
  if ((st = moe_router_softmax_topk(logits, dtype, T, E, k, norm_topk, b.weights, dtype, (int64_t*)b.experts, stream)) != MOE_OK) return st;
  if ((st = moe_sort_by_expert(b.experts, MOE_I64, M, E, (int32_t*)b.counts, (int32_t*)b.source_of, (int32_t*)b.sorted_of, b.sort_ws,
                               b.sort_bytes, stream)) != MOE_OK) return st;
  if ((st = moe_expand_rows(x, (const int32_t*)b.sorted_of, k, b.xs, T, H, dtype, stream)) != MOE_OK) return st;
  if ((st = moe_gate_up_silu_fwd(b.xs, w_gate, w_up, b.counts, MOE_I32, b.h, M, I, H, E, dtype, b.gemm_ws, b.gemm_bytes, stream)) != MOE_OK) return st;
  if ((st = moe_grouped_gemm_fwd(b.h, w_down, b.counts, MOE_I32, b.y, M, H, I, E, dtype, dtype, b.gemm_ws, b.gemm_bytes, stream)) != MOE_OK) return st;
  return moe_combine(b.y, (const int32_t*)b.sorted_of, b.weights, out, T, k, H, dtype, stream);
}

// The expert MLP with LoRA on dense 16-bit weights.  Refusals of the parts come back unchanged; the caller has
// checked that there are none (extents, alignment), so that a chain is not left half enqueued.
MOE_API int moe_lora_mlp_fwd(const moe_lora_weights* w, const void* x, const void* m_sizes, int msd, void* e, void* g, void* h,
                             void* t_gu, void* t_w, void* y, int64_t M, int H, int I, int E, int dtype, void* stream) {
  if (!w || !x || !e || !g || !h || !t_gu || !t_w || !y) return MOE_ERR_NULL;
  const int rg = w->rank[0], ru = w->rank[1], rw = w->rank[2];
  if (M <= 0 || H <= 0 || I <= 0 || rg <= 0 || ru <= 0 || rw <= 0) return MOE_ERR_SHAPE;
  const int64_t ld = rg + ru;
  uint8_t* t_u = (uint8_t*)t_gu + (size_t)rg * dtype_size(dtype);
  const Factor f[3] = {{w->scale[0], dtype}, {w->scale[1], dtype}, {w->scale[2], dtype}};
  if (!factors_ok(f)) return MOE_ERR_UNSUPPORTED;
  auto sum2 = [&](const void* x0, int i, int k0, const void* t, int64_t ldt, void* out, int N) {
    const void* xs[2] = {x0, t};
    const void* ws[2] = {w->base[i], w->b[i]};
    const int64_t lds[2] = {k0, ldt};
    const int ks[2] = {k0, w->rank[i]};
    const int log2_scale[2] = {0, f[i].log2};
    return grouped_gemm_sum_scaled(0, 2, xs, lds, ws, ks, log2_scale, m_sizes, msd, out, M, N, E, dtype, stream);
  };
  int st;
  // thin factors of the LoRA products: gate and up side by side (x is read once), down
  if ((st = moe_lora_project(0, x, w->a[0], rg, f[0].thin, w->a[1], ru, f[1].thin, m_sizes, msd, t_gu, ld, M, H, E, dtype, stream)) != MOE_OK) return st;
  if ((st = sum2(x, 0, H, t_gu, ld, e, I)) != MOE_OK) return st;
  if ((st = sum2(x, 1, H, t_u, ld, g, I)) != MOE_OK) return st;
  if ((st = moe_silu_mul_fwd(e, g, h, M * I, dtype, stream)) != MOE_OK) return st;
  if ((st = moe_lora_project(0, h, w->a[2], rw, f[2].thin, nullptr, 0, 1.f, m_sizes, msd, t_w, rw, M, I, E, dtype, stream)) != MOE_OK) return st;
  return sum2(h, 2, I, t_w, rw, y, H);
}

MOE_API int moe_lora_mlp_bwd(const moe_lora_weights* w, const moe_lora_grads* grads, const void* dy, const void* x,
                             const void* m_sizes, int msd, void* e, void* g, const void* t_gu, const void* t_w, void* dh,
                             void* d_gu, void* d_w, void* dx, int64_t M, int H, int I, int E, int dtype, void* ws,
                             size_t ws_bytes, void* stream) {
  if (!w || !grads || !dy || !x || !e || !g || !t_gu || !t_w || !dh || !d_gu || !d_w) return MOE_ERR_NULL;
  const int rg = w->rank[0], ru = w->rank[1], rw = w->rank[2];
  if (M <= 0 || H <= 0 || I <= 0 || rg <= 0 || ru <= 0 || rw <= 0) return MOE_ERR_SHAPE;
  const int64_t ld = rg + ru;
  const size_t off = (size_t)rg * dtype_size(dtype);
  const uint8_t* t_u = (const uint8_t*)t_gu + off;
  uint8_t* d_u = (uint8_t*)d_gu + off;
  const Factor f[3] = {{w->scale[0], dtype}, {w->scale[1], dtype}, {w->scale[2], dtype}};
  if (!factors_ok(f)) return MOE_ERR_UNSUPPORTED;
  auto dw = [&](int i, const void* x_, int64_t ldx, int K, const void* dy_, int64_t ldy, int N, void* out) {
    return grouped_gemm_dw_scaled(x_, ldx, dy_, ldy, m_sizes, msd, out, nullptr, 0, f[i].pow2(), 1.f, M, N, K, E, dtype, ws,
                                  ws_bytes, stream);
  };
  int st;
  if ((st = moe_lora_project(1, dy, w->b[2], rw, f[2].thin, nullptr, 0, 1.f, m_sizes, msd, d_w, rw, M, H, E, dtype, stream)) != MOE_OK) return st;
  {
    const void* xs[2] = {dy, d_w};
    const void* wt[2] = {w->base[2], w->a[2]};
    const int64_t lds[2] = {H, rw};
    const int ks[2] = {H, rw};
    const int log2_scale[2] = {0, f[2].log2};
    if ((st = grouped_gemm_sum_scaled(1, 2, xs, lds, wt, ks, log2_scale, m_sizes, msd, dh, M, I, E, dtype, stream)) != MOE_OK) return st;
  }
  // dh, e, g become h, de, dg
  if ((st = moe_silu_mul_bwd_inplace(dh, e, g, M * I, dtype, stream)) != MOE_OK) return st;
  if ((st = dw(2, dh, I, I, d_w, rw, rw, grads->da[2])) != MOE_OK) return st;
  if ((st = dw(2, t_w, rw, rw, dy, H, H, grads->db[2])) != MOE_OK) return st;
  if ((st = moe_lora_project(1, e, w->b[0], rg, f[0].thin, nullptr, 0, 1.f, m_sizes, msd, d_gu, ld, M, I, E, dtype, stream)) != MOE_OK) return st;
  if ((st = moe_lora_project(1, g, w->b[1], ru, f[1].thin, nullptr, 0, 1.f, m_sizes, msd, d_u, ld, M, I, E, dtype, stream)) != MOE_OK) return st;
  if (rg + ru <= 128) {  // both gradients of a from one read of x
    if ((st = grouped_gemm_dw_scaled(x, H, d_gu, ld, m_sizes, msd, grads->da[0], grads->da[1], rg, f[0].pow2(), f[1].pow2(), M,
                                     rg + ru, H, E, dtype, ws, ws_bytes, stream)) != MOE_OK) return st;
  } else {
    if ((st = dw(0, x, H, H, d_gu, ld, rg, grads->da[0])) != MOE_OK) return st;
    if ((st = dw(1, x, H, H, d_u, ld, ru, grads->da[1])) != MOE_OK) return st;
  }
  if ((st = dw(0, t_gu, ld, rg, e, I, I, grads->db[0])) != MOE_OK) return st;
  if ((st = dw(1, t_u, ld, ru, g, I, I, grads->db[1])) != MOE_OK) return st;
  if (!dx) return MOE_OK;
  const void* xs[4] = {e, d_gu, g, d_u};
  const void* wt[4] = {w->base[0], w->a[0], w->base[1], w->a[1]};
  const int64_t lds[4] = {I, ld, I, ld};
  const int ks[4] = {I, rg, I, ru};
  const int log2_scale[4] = {0, f[0].log2, 0, f[1].log2};
  return grouped_gemm_sum_scaled(1, 4, xs, lds, wt, ks, log2_scale, m_sizes, msd, dx, M, H, E, dtype, stream);
}
