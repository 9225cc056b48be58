// The layer loop of a plain dense decoder over a ragged batch of prompt tokens, walked here instead of in Python: the same kernels in the
// same order with the same choices (models/llm/transformer.py, DecoderModel.forward_hidden), nine launches a layer.
//
// Why: a launch through the Python ops costs 15 us of host time (argument objects, output tensors, checks), so a short prompt
// through 24 layers of a small model took 3.4 ms of which the device was busy for one; from here a launch costs 3 us. What
// lies between the kernels is scratch that the caller allocates once for the whole stack.
#include "common.cuh"

extern "C" {
int b200_norm(const void*, const void*, void*, const void*, const void*, const void*, const void*, void*, void*, float*, int, int, int, int,
              float, int, int, int, const float*, int, int, cudaStream_t);
int b200_gemm(const void*, const void*, void*, int, int, int, long long, long long, long long, int, const float*, const float*, const void*,
              const void*, const void*, int, int, void*, long long, void*, cudaStream_t);
int b200_gemm_deferred_plan(int, int, int, int, long long);
int b200_gemm_deferred(const void*, const void*, int, int, int, long long, long long, int, const float*, const float*, void*, long long, float*,
                       void*, cudaStream_t);
int b200_rope_kv(const void*, void*, void*, void*, void*, void*, const int*, const long long*, const void*, const void*, const float*, int, int,
                 int, int, int, int, int, float, float, const float*, int, int, const void*, cudaStream_t);
int b200_attn_prefill_tc(const void*, const void*, const void*, void*, const int*, const int*, const int*, int, int, int, int, int, int, int,
                         long long, int, float, void*, cudaStream_t);
int b200_attn_prefill(const void*, const void*, const void*, void*, const int*, const int*, const int*, const int*, int, int, int, int, int, int,
                      int, int, int, int, int, int, float, float, cudaStream_t);
int b200_glu(const void*, void*, void*, float*, int, int, int, int, const float*, int, int, cudaStream_t);
int b200_glu_form(int, int, int, int);
int b200_gemm_glu(const void*, const void*, void*, void*, void*, int, int, int, long long, long long, long long, int, const float*, const float*,
                  int, int, void*, cudaStream_t);
int b200_gemv_glu(const void*, const void*, void*, int, int, int, long long, long long, long long, int, cudaStream_t);
}

namespace b200 {

struct DenseSizes {
  int tokens, hidden, hq, hkv, d, ffn;
  int qkv() const { return (hq + 2 * hkv) * d; }
  int att() const { return hq * d; }
};

static long long padded(long long bytes) { return (bytes + 255) / 256 * 256; }

// What the policy leaves unsummed of a layer's four products (see b200_gemm_deferred_plan), and the bytes of the ranges. The policy follows
// switches that another thread can turn between the call that asks for the scratch's size and the launch, so a launch asks once, for all
// layers, and compares with the size that it was given.
struct DensePlan {
  int qkv, o, gate_up, down;
  long long part;
};

static DensePlan dense_plan(const DenseSizes& z, long long ws_bytes) {
  DensePlan p{};
  auto one = [&](int n, int k) {
    const int plan = z.tokens <= 128 ? b200_gemm_deferred_plan(z.tokens, n, k, 0, ws_bytes) : 0;
    const long long bytes = padded(static_cast<long long>((n + 127) / 128) * (plan & 0xffff) * (plan >> 16) * 128 * 4);
    if (bytes > p.part) p.part = bytes;
    return plan;
  };
  p.qkv = one(z.qkv(), z.hidden);
  p.o = one(z.hidden, z.att());
  p.gate_up = one(2 * z.ffn, z.hidden);
  p.down = one(z.hidden, z.ffn);
  return p;
}

static long long dense_scratch(const DenseSizes& z, const DensePlan& plan) {
  const long long t = z.tokens;
  return 4 * padded(t * z.hidden * 2) + padded(t * z.qkv() * 2) + 2 * padded(t * z.att() * 2) + padded(t * 2 * z.ffn * 2) + padded(t * z.ffn * 2) +
         plan.part;
}

// A product, or its unsummed ranges where the policy leaves them to the kernel behind it
struct Product {
  const __nv_bfloat16* y = nullptr;
  const float* part = nullptr;
  int splits = 0, bn = 0;
};

}  // namespace b200

using namespace b200;

B200_API long long b200_dense_layers_scratch(int tokens, int hidden, int hq, int hkv, int d, int ffn, long long gemm_ws_bytes) {
  const DenseSizes z{tokens, hidden, hq, hkv, d, ffn};
  return dense_scratch(z, dense_plan(z, gemm_ws_bytes));
}

// x [tokens][hidden] bf16 -> out = norm(stream) behind all layers. layer_ptrs: seven pointers a layer (in_norm, qkv, qkv bias or null, o,
// post_norm, gate_up, down), rows of weights dense. kv: pools [layers][2][pages][hkv][page][d]. cu_q, kv_lens, block_table as in
// b200_attn_prefill. scratch: b200_dense_layers_scratch bytes on a 256-byte boundary. Returns the number of ops launched, or the
// negative code of the one that failed; -14, and nothing is launched: the scratch is too small for the policy as it is now.
B200_API int b200_dense_layers(const void* x, void* out, const void* const* layer_ptrs, const void* final_norm, void* kv, long long layer_stride,
                               long long v_offset, const int* block_table, const int* kv_lens, const int* cu_q, const int* positions,
                               const long long* slots, const float* inv_freq, int tokens, int seqs, int max_q_len, int max_kv_len, int layers,
                               int hidden, int hq, int hkv, int d, int ffn, int rot, int style, int page, int max_pages, long long pages, int act,
                               int plus_one, float eps, float theta, float scale, void* gemm_ws, long long gemm_ws_bytes, void* scratch,
                               long long scratch_bytes, void* status, cudaStream_t stream) {
  const DenseSizes z{tokens, hidden, hq, hkv, d, ffn};
  const DensePlan plans = dense_plan(z, gemm_ws_bytes);
  if (dense_scratch(z, plans) > scratch_bytes) return -14;
  const long long t = tokens;
  uint8_t* at = static_cast<uint8_t*>(scratch);
  auto take = [&](long long bytes) {
    uint8_t* r = at;
    at += padded(bytes);
    return reinterpret_cast<__nv_bfloat16*>(r);
  };
  __nv_bfloat16 *h = take(t * hidden * 2), *y = take(t * hidden * 2), *res[2] = {take(t * hidden * 2), take(t * hidden * 2)};
  __nv_bfloat16 *qkv = take(t * z.qkv() * 2), *q = take(t * z.att() * 2), *att = take(t * z.att() * 2), *gu = take(t * 2 * ffn * 2), *a = take(t * ffn * 2);
  float* part = reinterpret_cast<float*>(at);
  int launches = 0, rc = 0;
  auto ok = [&](int code) {
    rc = code;
    ++launches;
    return code == 0;
  };
  // dst [tokens][n] = in w^T (+ bias), or the K ranges of `plan`, which the kernel behind it adds (and the bias)
  auto product = [&](const void* in, const void* w, const void* bias, __nv_bfloat16* dst, int n, int k, int plan, Product& p) {
    p = Product{};
    if (plan) {
      p.part = part;
      p.splits = plan & 0xffff;
      p.bn = plan >> 16;
      const int c = b200_gemm_deferred(in, w, tokens, n, k, k, k, 0, nullptr, nullptr, gemm_ws, gemm_ws_bytes, part, status, stream);
      if (c != -13) return ok(c);                      // -13: the reduce form was switched meanwhile
      p = Product{};
    }
    p.y = dst;
    return ok(b200_gemm(in, w, dst, tokens, n, k, k, k, n, 0, nullptr, nullptr, bias, nullptr, nullptr, 0, 0, gemm_ws, gemm_ws_bytes, status, stream));
  };
  auto norm = [&](const Product& p, const void* residual, void* sum, const void* w, void* dst) {
    return ok(b200_norm(p.y, residual, sum, w, nullptr, nullptr, nullptr, dst, nullptr, nullptr, tokens, hidden, 0, 0, eps, 0, plus_one, 0, p.part,
                        p.splits, p.bn, stream));
  };
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  Product cur, p;
  cur.y = static_cast<const __nv_bfloat16*>(x);
  const void* stream_in = nullptr;
  for (int li = 0; li < layers; ++li) {
    const void* const* w = layer_ptrs + 7 * li;
    __nv_bfloat16* kc = static_cast<__nv_bfloat16*>(kv) + li * layer_stride;
    __nv_bfloat16* vc = kc + v_offset;
    if (!norm(cur, stream_in, stream_in ? res[0] : nullptr, w[0], h)) return rc;
    if (stream_in == nullptr) stream_in = x; else stream_in = res[0];
    if (!product(h, w[1], w[2], qkv, z.qkv(), hidden, plans.qkv, p)) return rc;
    if (!ok(b200_rope_kv(p.y, q, kc, vc, nullptr, nullptr, positions, slots, nullptr, nullptr, inv_freq, tokens, hq, hkv, d, rot, style, page, theta, eps,
                         p.part, p.splits, p.bn, p.part ? w[2] : nullptr, stream)))
      return rc;
    int code = 1;                                      // 1: short prompts, for which the other kernel is faster
    if (d == 128 && scale > 0.f && (page == 8 || page == 16 || page == 32 || page == 64) && aligned(kc) && aligned(vc))
      code = b200_attn_prefill_tc(q, kc, vc, att, block_table, kv_lens, cu_q, seqs, tokens, max_q_len, hq, hkv, page, max_pages, pages, max_kv_len,
                                  scale, status, stream);
    if (code == 1)
      code = b200_attn_prefill(q, kc, vc, att, block_table, kv_lens, cu_q, nullptr, seqs, max_q_len, 0, 0, hq, hkv, d, page, max_pages, 1, 1, 0, scale, 0.f,
                               stream);
    if (!ok(code)) return rc;
    if (!product(att, w[3], nullptr, y, hidden, z.att(), plans.o, p)) return rc;
    if (!norm(p, stream_in, res[1], w[4], h)) return rc;
    // as ops.linear_glu: one kernel for a handful of tokens and for many, otherwise the product and the activation
    const int form = b200_glu_form(tokens, ffn, hidden, 0);
    code = -12;
    if (form == 1 && aligned(w[5])) code = b200_gemv_glu(h, w[5], a, tokens, ffn, hidden, hidden, hidden, ffn, act, stream);
    else if (form == 2) code = b200_gemm_glu(h, w[5], a, nullptr, nullptr, tokens, ffn, hidden, hidden, hidden, ffn, 0, nullptr, nullptr, act, 128, status, stream);
    if (code != -12) {
      if (!ok(code)) return rc;
    } else {
      if (!product(h, w[5], nullptr, gu, 2 * ffn, hidden, plans.gate_up, p)) return rc;
      if (!ok(b200_glu(p.y, a, nullptr, nullptr, tokens, ffn, act, 0, p.part, p.splits, p.bn, stream))) return rc;
    }
    if (!product(a, w[6], nullptr, y, hidden, ffn, plans.down, cur)) return rc;
    stream_in = res[1];
  }
  if (!norm(cur, stream_in, res[0], final_norm, out)) return rc;
  return launches;
}
