// The layer loop of a plain dense decoder over a ragged batch of prompt tokens, walked here instead of in Python: the same kernels in the
// same order with the same choices (models/llm/transformer.py, DecoderModel.forward_hidden), nine launches a layer.
//
// Why: a launch through the Python ops costs 15 us of host time (argument objects, output tensors, checks), so a short prompt
// through 24 layers of a small model took 3.4 ms of which the device was busy for one; from here a launch costs 3 us. What
// lies between the kernels is scratch that the caller allocates once for the whole stack.
#include "layer_ops.cuh"

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
  int form;                                            // of the gated product, see b200_glu_form
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
  p.form = b200_glu_form(z.tokens, z.ffn, z.hidden, 0);
  return p;
}

// Where a layer's intermediates lie in the scratch, in bytes. The halves of a layer take turns in one region: q, k and v are dead when
// attention has run, whose output takes the place of the packed projection and is dead when the product behind it has; the gate and up rows
// exist only where the gated product does not form the activation itself. 8192 tokens of 4096 features with 32 + 16 heads of 128 and a
// feed-forward of 14336: 1.2 GB with a place for each -> 0.5 GB.
struct DenseLayout {
  long long h, y, res[2], qkv, q, att, gu, a, part, total;
};

static DenseLayout dense_layout(const DenseSizes& z, const DensePlan& plan) {
  const long long t = z.tokens, row = padded(t * z.hidden * 2), qkv = padded(t * z.qkv() * 2), att = padded(t * z.att() * 2), a = padded(t * z.ffn * 2);
  const long long gu = plan.form == 0 ? padded(t * 2 * z.ffn * 2) : 0;
  DenseLayout l{};
  l.y = row;
  l.res[0] = 2 * row;
  l.res[1] = 3 * row;
  l.qkv = l.att = l.a = 4 * row;
  l.q = l.qkv + qkv;
  l.gu = l.a + a;
  l.part = 4 * row + (qkv + att > gu + a ? qkv + att : gu + a);
  l.total = l.part + plan.part;
  return l;
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
  return dense_layout(z, dense_plan(z, gemm_ws_bytes)).total;
}

// x [tokens][hidden] bf16 -> out = norm(stream) behind all layers. layer_ptrs: seven pointers a layer (in_norm, qkv, qkv bias or null, o,
// post_norm, gate_up, down), rows of weights dense, on 16-byte boundaries and multiples of 8 values long. kv: pools
// [layers][2][pages][hkv][page][d]. cu_q, kv_lens, block_table as in b200_attn_prefill. scratch: b200_dense_layers_scratch bytes on a 256-byte boundary. Returns the number of ops launched, or the
// negative code of the one that failed; -14, and nothing is launched: the scratch is too small for the policy as it is now.
B200_API int b200_dense_layers(const void* x, void* out, const void* const* layer_ptrs, const void* final_norm, void* kv, long long layer_stride,
                               long long v_offset, const int* block_table, const int* kv_lens, const int* cu_q, const int* positions,
                               const long long* slots, const float* inv_freq, int tokens, int seqs, int max_q_len, int max_kv_len, int layers,
                               int hidden, int hq, int hkv, int d, int ffn, int rot, int style, int page, int max_pages, long long pages, int act,
                               int plus_one, float eps, float theta, float scale, void* gemm_ws, long long gemm_ws_bytes, void* scratch,
                               long long scratch_bytes, void* status, cudaStream_t stream) {
  const DenseSizes z{tokens, hidden, hq, hkv, d, ffn};
  const DensePlan plans = dense_plan(z, gemm_ws_bytes);
  const DenseLayout at = dense_layout(z, plans);
  if (at.total > scratch_bytes) return -14;
  auto place = [&](long long offset) { return reinterpret_cast<__nv_bfloat16*>(static_cast<uint8_t*>(scratch) + offset); };
  __nv_bfloat16 *const h = place(at.h), *const y = place(at.y), *const res[2] = {place(at.res[0]), place(at.res[1])};
  __nv_bfloat16 *const qkv = place(at.qkv), *const q = place(at.q), *const att = place(at.att), *const gu = place(at.gu), *const a = place(at.a);
  float* const part = reinterpret_cast<float*>(place(at.part));
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
    if (plans.form == 1) code = b200_gemv_glu(h, w[5], a, tokens, ffn, hidden, hidden, hidden, ffn, act, stream);
    else if (plans.form == 2) code = b200_gemm_glu(h, w[5], a, nullptr, nullptr, tokens, ffn, hidden, hidden, hidden, ffn, 0, nullptr, nullptr, act, 128, status, stream);
    if (plans.form != 0) {
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
