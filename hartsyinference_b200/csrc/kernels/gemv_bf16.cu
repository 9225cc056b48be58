// Linear layers of one to four tokens with bf16 weights: out[t][n] = epilogue(sum over k of x[t][k] w[n][k]).
//
// With so few tokens a product is one pass over the weights and a chain of latencies: the tcgen05 form stages
// 128-row tiles, cuts small ones along K and leaves the sums to another kernel. Here a warp holds kRows rows of
// weights in flight (16 bytes a lane, four or more loads before the first use, the first ones requested before the
// wait for the kernel in front, which only produces x); products and sums are fp32 FMAs. Where the rows are too
// few for the machine, up to eight warps share a row and meet in shared memory: one launch, no scratch.
//
// Bound by HBM from about 10 MB of weights on (128256 x 4096, one token: 153 us, 6.85 TB/s), by latency below
// (1152 x 896 6.3 -> 2.3 us, 896 x 4864 7.5 -> 3.9 us, 4096 x 4096 9.6 -> 5.4 us against the tcgen05 form with its
// reduce). Every further token adds reads of x and FMAs per weight, so it wins for one token everywhere, for three
// and four with small matrices only: the line is drawn where it is called.
//
// The norm in front (kNorm) and the rotation behind (kRope) can be taken along, and weights further on brought to L2 meanwhile: one
// token through 24 layers of 896 features 630 us with eight launches a layer, 534 with five, 488 with the weights ahead.
#include <type_traits>

#include "layer_ops.cuh"

namespace b200 {

struct GemvBf16Params {
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;
  __nv_bfloat16* out;
  int n, k;
  long long ldx, ldw, ldc;
  const __nv_bfloat16* bias;      // per output feature, may be null (as all three)
  const __nv_bfloat16* gate;
  const __nv_bfloat16* residual;
  int act, act_col;
  int share;                      // warps that share a row: 1, 2, 4 or 8
  int glu_act;                    // kGlu: 0 = SiLU, 1 = GELU-tanh
};
// What the forms with a norm take besides. (A struct of its own: in the other kernels' parameters these fields alone made the compiler keep fewer
// loads in flight, two tokens of 2304 x 4096 6.7 -> 7.8 us.)
struct GemvNormParams : GemvBf16Params {
  // kNorm: x is the residual stream and the product reads its RMS norm
  const __nv_bfloat16* norm_w;    // [k]
  float eps;
  int plus_one;                   // the norm multiplies by 1 + w
  // kRope: w holds q, k and v heads of d rows each (n = pairs of all heads)
  __nv_bfloat16 *q_out, *k_cache, *v_cache;     // [tokens][hq][d]; pages [pages][hkv][page][d]
  const int* positions;
  const long long* slots;         // < 0: k and v are not stored
  const float* inv_freq;          // [rot / 2]
  int hq, hkv, d, rot, style, page;
  int early;                      // the kernel behind may be launched from the start on
  // kNorm: weights of products further on that are brought to L2 meanwhile
  const uint8_t* ahead[2];
  long long ahead_bytes[2];
};
constexpr long long kAheadMost = 24ll << 20;      // of one weight: what waits in L2 shall not push itself out
constexpr int kAheadPiece = 8192;

constexpr int kGemvDepth = 4;     // 16-byte loads of a row in flight per lane

enum GemvForm { kPlain, kGlu, kRope };

// Elements e0, e1 of a head that pair i turns into each other; behind the rotated part two neighbours.
__device__ __forceinline__ void gemv_pair(const GemvNormParams& p, int i, int& e0, int& e1) {
  const int half = p.rot >> 1;
  if (i >= half || p.style != 0) {
    e0 = i >= half ? p.rot + 2 * (i - half) : 2 * i;
    e1 = e0 + 1;
  } else {
    e0 = i;
    e1 = i + half;
  }
}

// kGlu: w holds the gate rows and, n rows on, the up rows; a warp takes kOut of both and writes act(gate) * up.
// kRope: a unit is a pair of rows of one head, which leaves rotated, q to q_out and k and v into their pages.
// kNorm: every block norms the rows of x on its own, into shared memory, while its first weights are on their way; a launch for
// the norm and what it writes and reads again are saved (896 features: norm 1.5 us and product 2.3 against 3.4, gated 1.5 and 5.5
// against 6.4).
template <int kTokens, int kOut, int kForm = kPlain, bool kNorm = false>
__global__ void __launch_bounds__(256) gemv_bf16_kernel(const std::conditional_t<kNorm, GemvNormParams, GemvBf16Params> p) {
  static_assert(kForm != kRope || kNorm);
  constexpr int kRows = kForm != kPlain ? 2 * kOut : kOut;        // weight rows of a warp: the second rows of its units follow the first ones
  extern __shared__ __align__(16) uint8_t gemv_smem[];            // kNorm: the normed rows [tokens][k]
  __shared__ float part[8][kTokens * kRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / p.share, slice = warp - group * p.share;
  const int row0 = (blockIdx.x * (8 / p.share) + group) * kOut;
  const int nvec = p.k >> 3, step = 32 * p.share;
  const uint4* wr[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {    // rows past the end are not stored
    long long row = min(row0 + r % kOut, p.n - 1) + (r >= kOut ? p.n : 0);
    if constexpr (kForm == kRope) {
      const int unit = min(row0 + r % kOut, p.n - 1), h = unit / (p.d >> 1);
      int e0, e1;
      gemv_pair(p, unit - h * (p.d >> 1), e0, e1);
      row = static_cast<long long>(h) * p.d + (r >= kOut ? e1 : e0);
    }
    wr[r] = reinterpret_cast<const uint4*>(p.w + row * p.ldw);
  }
  float acc[kRows][kTokens];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int t = 0; t < kTokens; ++t) acc[r][t] = 0.f;
  uint4 wv[kRows][kGemvDepth];
  auto request = [&](int v0) {
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int u = 0; u < kGemvDepth; ++u) {
        const int v = v0 + u * step;
        wv[r][u] = make_uint4(0u, 0u, 0u, 0u);
        if (v < nvec) wv[r][u] = __ldg(wr[r] + v);
      }
  };
  int v0 = slice * 32 + lane;
  request(v0);
  __nv_bfloat16* const xs = reinterpret_cast<__nv_bfloat16*>(gemv_smem);
  const long long ldx = kNorm ? p.k : p.ldx;
  if constexpr (kNorm) {
    __shared__ float sums[8][kTokens];
    if (warp == 0) {
#pragma unroll
      for (int a = 0; a < 2; ++a)
        for (long long at = (static_cast<long long>(blockIdx.x) * 32 + lane) * kAheadPiece; at < p.ahead_bytes[a]; at += static_cast<long long>(gridDim.x) * 32 * kAheadPiece) {
          const uint32_t bytes = static_cast<uint32_t>(min(static_cast<long long>(kAheadPiece), p.ahead_bytes[a] - at));
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.ahead[a] + at), "r"(bytes) : "memory");
        }
    }
    pdl_wait();
    // With kRope attention follows, whose blocks share the keys: launched while the last blocks here still run they crowd the processors
    // that are free first, and the fullest one ends late (a layer of 4096 features and 9000 keys 117.4 us, without the trigger 110.1; of
    // 1536 and 4000 53.2 and 48.7, and 40 44.8 and 43.5). Only few blocks of little work gain by being there early: heads of 64 values and
    // at most 256 keys (896 features: 64 keys 20.5 us early, 20.9 late, 256 22.5 and 22.6, 512 23.6 and 23.5; heads of 128 42.4 and 42.6 for
    // 128 keys, 43.3 and 42.6 for 256).
    if (kForm != kRope || p.early) pdl_trigger();
    float ss[kTokens];
#pragma unroll
    for (int t = 0; t < kTokens; ++t) {
      ss[t] = 0.f;
      for (int v = threadIdx.x; v < nvec; v += 256) {
        const uint4 raw = *reinterpret_cast<const uint4*>(p.x + t * p.ldx + static_cast<long long>(v) * 8);
        *reinterpret_cast<uint4*>(xs + t * p.k + v * 8) = raw;
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float a = __uint_as_float(w[i] << 16), b = __uint_as_float(w[i] & 0xffff0000u);
          ss[t] += a * a + b * b;
        }
      }
      ss[t] = warp_sum(ss[t]);
      if (lane == 0) sums[warp][t] = ss[t];
    }
    __syncthreads();
    const float one = p.plus_one ? 1.f : 0.f;
    float rstd[kTokens];
#pragma unroll
    for (int t = 0; t < kTokens; ++t) {
      float q = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) q += sums[i][t];
      rstd[t] = rsqrtf(q / p.k + p.eps);
    }
    for (int v = threadIdx.x; v < nvec; v += 256) {
      const uint4 g4 = __ldg(reinterpret_cast<const uint4*>(p.norm_w) + v);
      const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int t = 0; t < kTokens; ++t) {
        const uint4 raw = *reinterpret_cast<const uint4*>(xs + t * p.k + v * 8);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        uint32_t y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          y[i] = pack_bf16x2(__uint_as_float(w[i] << 16) * rstd[t] * (one + __uint_as_float(g[i] << 16)),
                             __uint_as_float(w[i] & 0xffff0000u) * rstd[t] * (one + __uint_as_float(g[i] & 0xffff0000u)));
        *reinterpret_cast<uint4*>(xs + t * p.k + v * 8) = make_uint4(y[0], y[1], y[2], y[3]);
      }
    }
    __syncthreads();
  } else {
    pdl_wait();
    pdl_trigger();
  }
  const __nv_bfloat16* const x = kNorm ? xs : p.x;
  for (; v0 < nvec; v0 += kGemvDepth * step) {
#pragma unroll
    for (int u = 0; u < kGemvDepth; ++u) {
      const int v = v0 + u * step;
      const bool inside = v < nvec;                          // past the end both operands are zeros
#pragma unroll
      for (int t = 0; t < kTokens; ++t) {
        // plain loads: x may have been written by the kernel in front
        uint4 xr = make_uint4(0u, 0u, 0u, 0u);
        if (inside) xr = *reinterpret_cast<const uint4*>(x + t * ldx + static_cast<long long>(v) * 8);
        const uint32_t xw[4] = {xr.x, xr.y, xr.z, xr.w};
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const uint32_t ww[4] = {wv[r][u].x, wv[r][u].y, wv[r][u].z, wv[r][u].w};
          float a = acc[r][t];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // a bf16 is the upper half of its fp32
            a = fmaf(__uint_as_float(ww[i] << 16), __uint_as_float(xw[i] << 16), a);
            a = fmaf(__uint_as_float(ww[i] & 0xffff0000u), __uint_as_float(xw[i] & 0xffff0000u), a);
          }
          acc[r][t] = a;
        }
      }
    }
    if (v0 + kGemvDepth * step < nvec) request(v0 + kGemvDepth * step);
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int t = 0; t < kTokens; ++t) {
      const float s = warp_sum(acc[r][t]);
      if (lane == 0) part[warp][r * kTokens + t] = s;
    }
  if (p.share > 1) __syncthreads(); else __syncwarp();
  if (slice != 0 || lane >= kOut * kTokens) return;
  const int r = lane / kTokens, t = lane - r * kTokens, col = row0 + r;
  if (col >= p.n) return;
  float v = 0.f;
  for (int s = 0; s < p.share; ++s) v += part[warp + s][lane];
  if constexpr (kForm == kRope) {
    float u = 0.f;
    for (int s = 0; s < p.share; ++s) u += part[warp + s][kOut * kTokens + lane];
    const int h = col / (p.d >> 1), i = col - h * (p.d >> 1);
    int e0, e1;
    gemv_pair(p, i, e0, e1);
    if (p.bias) {
      v += __bfloat162float(p.bias[h * p.d + e0]);
      u += __bfloat162float(p.bias[h * p.d + e1]);
    }
    v = __bfloat162float(__float2bfloat16(v));         // as the projection would have stored them
    u = __bfloat162float(__float2bfloat16(u));
    if (h < p.hq + p.hkv && i < (p.rot >> 1)) {
      float sn, cs;
      sincosf(static_cast<float>(p.positions[t]) * p.inv_freq[i], &sn, &cs);
      const float a = v * cs - u * sn;
      u = u * cs + v * sn;
      v = a;
    }
    __nv_bfloat16* dst = p.q_out + (static_cast<long long>(t) * p.hq + h) * p.d;
    if (h >= p.hq) {
      const long long slot = p.slots[t];
      if (slot < 0) return;
      const bool key = h < p.hq + p.hkv;
      dst = (key ? p.k_cache : p.v_cache) + ((slot / p.page * p.hkv + (h - p.hq - (key ? 0 : p.hkv))) * p.page + slot % p.page) * p.d;
    }
    dst[e0] = __float2bfloat16(v);
    dst[e1] = __float2bfloat16(u);
    return;
  }
  if constexpr (kForm == kGlu) {
    float u = 0.f;
    for (int s = 0; s < p.share; ++s) u += part[warp + s][kOut * kTokens + lane];
    p.out[t * p.ldc + col] = __float2bfloat16((p.glu_act == 0 ? silu(v) : gelu_tanh(v)) * u);
    return;
  }
  if (p.bias) v += __bfloat162float(p.bias[col]);
  if (col >= p.act_col) {
    if (p.act == 1) v = gelu_tanh(v);
    else if (p.act == 2) v = silu(v);
    else if (p.act == 3) v = relu2(v);
    else if (p.act == 4) v = tanhf(v);
  }
  if (p.gate) v *= __bfloat162float(p.gate[col]);
  if (p.residual) v += __bfloat162float(p.residual[t * p.ldc + col]);
  p.out[t * p.ldc + col] = __float2bfloat16(v);
}

// x [m][k] and w [n][k] on 16-byte boundaries with rows a multiple of 16 bytes apart, k % 8 == 0, 1 <= m <= 4; the
// other arguments as in b200_gemm.
int gemv_bf16(const void* x, const void* w, void* out, int m, int n, int k, long long ldx, long long ldw, long long ldc,
              const void* bias, const void* gate, const void* residual, int act, cudaStream_t stream) {
  GemvBf16Params p{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(out),
                   n, k, ldx, ldw, ldc, static_cast<const __nv_bfloat16*>(bias), static_cast<const __nv_bfloat16*>(gate),
                   static_cast<const __nv_bfloat16*>(residual), act & 255, act >> 8, 1, 0};
  // Rows per warp: as many as leave the machine about two thousand warps, since rows of one warp share the reads of
  // x. Few rows: warps share them until there are that many, but keep a full round of loads each.
  const int rows = n >= 8192 ? 4 : n >= 4096 ? 2 : 1;
  while (p.share < 8 && (n + rows - 1) / rows * p.share < 2368 && k >= 2 * p.share * 32 * 8 * 2) p.share *= 2;
  const int per_block = 8 / p.share * rows;
  const dim3 grid((n + per_block - 1) / per_block);
  auto go = [&](auto* kernel) { return launch_pdl(kernel, grid, dim3(256), 0, stream, p); };
  cudaError_t e;
#define GEMV_ROWS(R) (m == 1 ? go(gemv_bf16_kernel<1, R>) : m == 2 ? go(gemv_bf16_kernel<2, R>) : m == 3 ? go(gemv_bf16_kernel<3, R>) : go(gemv_bf16_kernel<4, R>))
  e = rows == 4 ? GEMV_ROWS(4) : rows == 2 ? GEMV_ROWS(2) : GEMV_ROWS(1);
#undef GEMV_ROWS
  return e == cudaSuccess ? 0 : -300;
}

bool handful(int m, int n, int k, int dtype);          // see gemm_tcgen05.cu

}  // namespace b200

using namespace b200;

// out[m][f] = act(x w_gate^T) * (x w_up^T) for w [2f][k] (gate rows first), act 0 = SiLU, 1 = GELU-tanh: the gated
// feed-forward's first half in one launch, neither product rounded on the way. 1 <= m <= 4, k % 8 == 0, x and w on 16-byte
// boundaries with rows a multiple of 16 bytes apart; -2 otherwise.
B200_API int b200_gemv_glu(const void* x, const void* w, void* out, int m, int f, int k, long long ldx, long long ldw,
                           long long ldc, int act, cudaStream_t stream) {
  if (m < 1 || m > 4 || f < 1 || k < 8 || k % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) != 0)
    return -2;
  GemvBf16Params p{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(out),
                   f, k, ldx, ldw, ldc, nullptr, nullptr, nullptr, 0, 0, 1, act};
  const int rows = f >= 4096 ? 2 : 1;      // pairs of rows per warp, see gemv_bf16
  while (p.share < 8 && (f + rows - 1) / rows * p.share < 2368 && k >= 2 * p.share * 32 * 8 * 2) p.share *= 2;
  const int per_block = 8 / p.share * rows;
  const dim3 grid((f + per_block - 1) / per_block);
  auto go = [&](auto* kernel) { return launch_pdl(kernel, grid, dim3(256), 0, stream, p); };
  cudaError_t e;
#define GLU_ROWS(R) (m == 1 ? go(gemv_bf16_kernel<1, R, kGlu>) : m == 2 ? go(gemv_bf16_kernel<2, R, kGlu>) : m == 3 ? go(gemv_bf16_kernel<3, R, kGlu>) : go(gemv_bf16_kernel<4, R, kGlu>))
  e = rows == 2 ? GLU_ROWS(2) : GLU_ROWS(1);
#undef GLU_ROWS
  return e == cudaSuccess ? 0 : -300;
}

// Whether b200_gemv_norm_qkv and b200_gemv_norm_glu take m rows of depth k against n weight rows: where the product itself would
// leave the tensor core, and the normed rows fit the shared memory that needs no asking for.
B200_API int b200_gemv_norm_fits(int m, int n, int k) {
  return m >= 1 && m <= 4 && k >= 8 && n >= 1 && m * k * 2 <= 47 * 1024 && handful(m, n, k, 0) ? 1 : 0;
}

// What b200_gemv_norm_* bring to L2 for products further on: whole multiples of 16 bytes on 16-byte boundaries, not too much
static void set_ahead(GemvNormParams& p, const void* a, long long a_bytes, const void* b, long long b_bytes) {
  const void* ptr[2] = {a, b};
  const long long bytes[2] = {a_bytes, b_bytes};
  for (int i = 0; i < 2; ++i) {
    if (ptr[i] == nullptr || bytes[i] < 16 || bytes[i] > kAheadMost || (reinterpret_cast<uintptr_t>(ptr[i]) & 15)) continue;
    p.ahead[i] = static_cast<const uint8_t*>(ptr[i]);
    p.ahead_bytes[i] = bytes[i] & ~15ll;
  }
}

// b200_gemv_glu of norm(x): x [m][k] the residual stream, norm_w [k] (16-byte boundary). -2: see b200_gemv_norm_fits.
B200_API int b200_gemv_norm_glu(const void* x, const void* norm_w, const void* w, void* out, int m, int f, int k, long long ldx,
                                long long ldw, long long ldc, int act, float eps, int plus_one, const void* ahead_a, long long ahead_a_bytes,
                                const void* ahead_b, long long ahead_b_bytes, cudaStream_t stream) {
  if (f < 1 || f > (1 << 30) || !b200_gemv_norm_fits(m, 2 * f, k) || ldx % 8 != 0 || ldw % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(norm_w)) & 15) != 0)
    return -2;
  GemvNormParams p{{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(out),
                   f, k, ldx, ldw, ldc, nullptr, nullptr, nullptr, 0, 0, 1, act}};
  p.norm_w = static_cast<const __nv_bfloat16*>(norm_w);
  p.eps = eps;
  p.plus_one = plus_one;
  set_ahead(p, ahead_a, ahead_a_bytes, ahead_b, ahead_b_bytes);
  const int rows = f >= 4096 ? 2 : 1;
  while (p.share < 8 && (f + rows - 1) / rows * p.share < 2368 && k >= 2 * p.share * 32 * 8 * 2) p.share *= 2;
  const int per_block = 8 / p.share * rows;
  const dim3 grid((f + per_block - 1) / per_block);
  auto go = [&](auto* kernel) { return launch_pdl(kernel, grid, dim3(256), static_cast<size_t>(m) * k * 2, stream, p); };
  cudaError_t e;
#define GLU_ROWS(R) (m == 1 ? go(gemv_bf16_kernel<1, R, kGlu, true>) : m == 2 ? go(gemv_bf16_kernel<2, R, kGlu, true>) : m == 3 ? go(gemv_bf16_kernel<3, R, kGlu, true>) : go(gemv_bf16_kernel<4, R, kGlu, true>))
  e = rows == 2 ? GLU_ROWS(2) : GLU_ROWS(1);
#undef GLU_ROWS
  return e == cudaSuccess ? 0 : -300;
}

// q | k | v = norm(x) w^T + bias of m decoded tokens with the rotary embedding (b200_rope_kv without head norms) in the epilogue: q to
// q_out [m][hq][d], k and v into their pages. Three launches in one. early: the next kernel in the stream may be launched while this one runs. d even, rot even and at most d, inv_freq [rot / 2].
B200_API int b200_gemv_norm_qkv(const void* x, const void* norm_w, const void* w, const void* bias, void* q_out, void* k_cache, void* v_cache,
                                const int* positions, const long long* slots, const float* inv_freq, int m, int k, long long ldx, long long ldw,
                                int hq, int hkv, int d, int rot, int style, int page, float eps, int plus_one,
                                const void* ahead_a, long long ahead_a_bytes, const void* ahead_b, long long ahead_b_bytes, int early,
                                cudaStream_t stream) {
  const long long n = static_cast<long long>(hq + 2 * hkv) * d;
  if (hq < 1 || hkv < 1 || d < 2 || d % 2 != 0 || rot < 0 || rot % 2 != 0 || rot > d || page < 1 || n > (1 << 30) || (rot > 0 && inv_freq == nullptr) ||
      !b200_gemv_norm_fits(m, static_cast<int>(n), k) || ldx % 8 != 0 || ldw % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(norm_w)) & 15) != 0)
    return -2;
  GemvNormParams p{{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), nullptr,
                   static_cast<int>(n / 2), k, ldx, ldw, 0, static_cast<const __nv_bfloat16*>(bias), nullptr, nullptr, 0, 0, 1, 0}};
  p.norm_w = static_cast<const __nv_bfloat16*>(norm_w);
  p.eps = eps;
  p.plus_one = plus_one;
  set_ahead(p, ahead_a, ahead_a_bytes, ahead_b, ahead_b_bytes);
  p.q_out = static_cast<__nv_bfloat16*>(q_out);
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.positions = positions;
  p.slots = slots;
  p.inv_freq = inv_freq;
  p.hq = hq; p.hkv = hkv; p.d = d; p.rot = rot; p.style = style; p.page = page;
  p.early = early;
  while (p.share < 8 && p.n * p.share < 2368 && k >= p.share * 32 * 8 * 2) p.share *= 2;      // half a round of loads each is enough: the chain counts
  const int per_block = 8 / p.share;
  const dim3 grid((p.n + per_block - 1) / per_block);
  auto go = [&](auto* kernel) { return launch_pdl(kernel, grid, dim3(256), static_cast<size_t>(m) * k * 2, stream, p); };
  const cudaError_t e = m == 1 ? go(gemv_bf16_kernel<1, 1, kRope, true>) : m == 2 ? go(gemv_bf16_kernel<2, 1, kRope, true>)
                      : m == 3 ? go(gemv_bf16_kernel<3, 1, kRope, true>) : go(gemv_bf16_kernel<4, 1, kRope, true>);
  return e == cudaSuccess ? 0 : -300;
}
