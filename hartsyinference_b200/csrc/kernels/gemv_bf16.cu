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
#include "common.cuh"

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

constexpr int kGemvDepth = 4;     // 16-byte loads of a row in flight per lane

// kGlu: w holds the gate rows and, n rows on, the up rows; a warp takes kRows of both and writes act(gate) * up.
template <int kTokens, int kOut, bool kGlu = false>
__global__ void __launch_bounds__(256) gemv_bf16_kernel(const GemvBf16Params p) {
  constexpr int kRows = kGlu ? 2 * kOut : kOut;        // weight rows of a warp: with kGlu the up rows follow the gate rows
  __shared__ float part[8][kTokens * kRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = warp / p.share, slice = warp - group * p.share;
  const int row0 = (blockIdx.x * (8 / p.share) + group) * kOut;
  const int nvec = p.k >> 3, step = 32 * p.share;
  const uint4* wr[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r)      // rows past the end are not stored
    wr[r] = reinterpret_cast<const uint4*>(p.w + (min(row0 + r % kOut, p.n - 1) + (r >= kOut ? p.n : 0)) * p.ldw);
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
  pdl_wait();
  pdl_trigger();
  for (; v0 < nvec; v0 += kGemvDepth * step) {
#pragma unroll
    for (int u = 0; u < kGemvDepth; ++u) {
      const int v = v0 + u * step;
      const bool inside = v < nvec;                          // past the end both operands are zeros
#pragma unroll
      for (int t = 0; t < kTokens; ++t) {
        // plain loads: x may have been written by the kernel in front
        uint4 xr = make_uint4(0u, 0u, 0u, 0u);
        if (inside) xr = *reinterpret_cast<const uint4*>(p.x + t * p.ldx + static_cast<long long>(v) * 8);
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
  if (kGlu) {
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
#define GLU_ROWS(R) (m == 1 ? go(gemv_bf16_kernel<1, R, true>) : m == 2 ? go(gemv_bf16_kernel<2, R, true>) : m == 3 ? go(gemv_bf16_kernel<3, R, true>) : go(gemv_bf16_kernel<4, R, true>))
  e = rows == 2 ? GLU_ROWS(2) : GLU_ROWS(1);
#undef GLU_ROWS
  return e == cudaSuccess ? 0 : -300;
}
