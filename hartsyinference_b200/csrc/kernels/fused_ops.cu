// Bandwidth-bound fused row kernels: (residual add +) RMSNorm, LayerNorm + AdaLN modulation,
// SwiGLU / GEGLU, fp8 1x128 block quantisation (also fused as an optional second output of the
// norm and activation kernels), QK-norm + RoPE + paged-KV write, embedding gather, argmax,
// repetition penalty, CFG + Euler step, and the weight initialisers used by synthetic benchmarks.
//
// They replace the reference's scalar decode-step kernels (src/HartsyInference.Cuda/Kernels/lm/
// lm_f32.cu: lm_add_rmsnorm_f32:470, lm_qkv_rope_scatter_f32:393, lm_qknorm_rope_scatter_f32:1304,
// lm_glu_act_f32:357, lm_argmax_lastdim_f32:214, lm_embed_gather_decode_f32:1461,
// lm_repetition_penalty_f32:1500), its DiT row kernels (Kernels/dit/dit_f32.cu:
// dit_layernorm_modulate_f32:1323, dit_gated_residual_lastdim_f32:85, dit_cfg_euler_f32:182,
// dit_fp8emit.cu) and its two-pass per-tensor fp8 quantiser (Kernels/dequant/fp8_quant.cu).
// All rows are processed with 16-byte loads, one CTA per row (or several rows per CTA for short
// rows), fp32 math, bf16 storage.
#include "layer_ops.cuh"

namespace b200 {

int num_sms();      // of the current device, see gemm_tcgen05.cu

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < nw) ? red[l] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}

__device__ __forceinline__ uint8_t to_e4m3(float v) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}

// Eight values times `inv` as e4m3 bytes: one conversion instruction per pair.
__device__ __forceinline__ uint2 to_e4m3x8(const float (&y)[8], float inv) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    w[i] = __nv_cvt_float2_to_fp8x2(make_float2(y[2 * i] * inv, y[2 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3);
  return make_uint2(w[0] | w[1] << 16, w[2] | w[3] << 16);
}
__device__ __forceinline__ void unpack_bf16x8(const uint4& raw, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 pack_bf16x8(const float (&v)[8]) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
// Eight parameters from column c (a multiple of 8): one 16-byte load where the host found the array aligned.
__device__ __forceinline__ void load_param8(const __nv_bfloat16* w, long long c, bool vec, float (&v)[8]) {
  if (vec) {
    unpack_bf16x8(__ldg(reinterpret_cast<const uint4*>(w + c)), v);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __bfloat162float(w[c + i]);
  }
}

// Eight e4m3 values of vector `vi` of a row of `dim` values, whose 1x128 group has the largest magnitude
// `amax`; the group's first thread stores its scale.
__device__ __forceinline__ void store_fp8(const float (&y)[8], float amax, uint8_t* dst, float* scales, int row, int vi,
                                          int dim, int sf_tile_rows) {
  if (sf_tile_rows > 0) {
    uint32_t eb;
    const float inv = mx_scale_inv(amax, eb);
    *reinterpret_cast<uint2*>(dst) = to_e4m3x8(y, inv);
    if ((vi & 15) == 0) store_sf(reinterpret_cast<uint8_t*>(scales), row, vi >> 4, sf_tile_rows, (dim + 511) >> 9, eb);
  } else {
    const float sc = fmaxf(amax, 1e-12f) / kFp8Max;
    *reinterpret_cast<uint2*>(dst) = to_e4m3x8(y, 1.f / sc);
    if ((vi & 15) == 0) scales[static_cast<long long>(row) * (dim >> 7) + (vi >> 4)] = sc;
  }
}

struct NormParams {
  const __nv_bfloat16* x;         // [rows][dim]
  SplitPartials part;             // ws != null: x comes as unsummed K ranges of the producing GEMM
  const __nv_bfloat16* residual;  // optional [rows][dim]: h = x + residual
  __nv_bfloat16* residual_out;    // optional: receives h
  const __nv_bfloat16* weight;    // optional [dim]
  const __nv_bfloat16* bias;      // optional [dim] (LayerNorm affine)
  const __nv_bfloat16* shift;     // optional AdaLN shift [batch][mod_stride]
  const __nv_bfloat16* scale;     // optional AdaLN scale [batch][mod_stride]  -> y * (1 + scale) + shift
  __nv_bfloat16* out;             // optional bf16 output
  uint8_t* out_fp8;               // optional e4m3 output [rows][dim]
  float* out_scale;               // [rows][dim/128] fp32
  int rows, dim, rows_per_batch, mod_stride;
  float eps;
  int layernorm;                  // 0 = RMSNorm, 1 = LayerNorm (mean-centred)
  int weight_plus_one;            // Gemma-style (1 + w)
  int sf_tile_rows;               // > 0: out_scale is a blocked UE8M0 scale-factor array
  int vec_params;                 // weight, bias, shift and scale can be read in 16-byte pieces
};

// One block per row, dim % 8 == 0, the row kept in registers: kMaxVec 16-byte vectors a thread, all loads (the
// residual's too) in flight before the first use. Bound by HBM. Many rows take several vectors a thread, so that more
// rows share a processor and one row's loads run under another's reduction; few rows (decoding) take one
// vector a thread, where the latency of a single row is what counts. Residual + norm + fp8, one vector a
// thread before: 8192 x 8192 163.6 -> 112.5 us (5.4 TB/s), 14040 x 5120 160 -> 118 us; two vectors instead of
// four 123 and 118, so four start at rows of 8192. Unsummed K ranges are read by instances of their own (kParts):
// the branch alone kept the loads of the others apart (131 us).
template <int kMaxVec, bool kParts>
__global__ void __launch_bounds__(1024) norm_kernel(const NormParams p) {
  pdl_wait();
  pdl_trigger();   // a GEMM launched behind this kernel may start fetching its weights now
  __shared__ float red[32];
  const int row = blockIdx.x;
  const int nvec = p.dim >> 3;
  const long long base = static_cast<long long>(row) * p.dim;
  uint4 raw[kMaxVec], res[kMaxVec];
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int vi = threadIdx.x + it * blockDim.x;
    raw[it] = res[it] = make_uint4(0u, 0u, 0u, 0u);
    if (vi < nvec) {
      if (kParts) {
        float sum8[8];
        split_sum8(p.part, row, vi * 8, sum8);
        raw[it] = pack_bf16x8(sum8);
      } else {
        raw[it] = *reinterpret_cast<const uint4*>(p.x + base + vi * 8);
      }
      if (p.residual) res[it] = *reinterpret_cast<const uint4*>(p.residual + base + vi * 8);
    }
  }
  float v[kMaxVec][8];
  float sum = 0.f, sumsq = 0.f;
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int vi = threadIdx.x + it * blockDim.x;
    unpack_bf16x8(raw[it], v[it]);
    if (p.residual) {
      float r[8];
      unpack_bf16x8(res[it], r);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[it][i] += r[i];
    }
    if (p.residual_out) {
      const uint4 o = pack_bf16x8(v[it]);
      if (vi < nvec) *reinterpret_cast<uint4*>(p.residual_out + base + vi * 8) = o;
      // the norm must see the value that was stored (bf16-rounded), as the unfused path does
      unpack_bf16x8(o, v[it]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      sum += v[it][i];
      sumsq += v[it][i] * v[it][i];
    }
  }
  float mean = 0.f;
  if (p.layernorm) {
    mean = block_sum(sum, red) / p.dim;
    // second pass over registers for a numerically stable variance
    float var = 0.f;
#pragma unroll
    for (int it = 0; it < kMaxVec; ++it) {
      const int vi = threadIdx.x + it * blockDim.x;
      if (vi < nvec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float d = v[it][i] - mean;
          var += d * d;
        }
      }
    }
    sumsq = var;
  }
  const float total = block_sum(sumsq, red);
  const float rstd = rsqrtf(total / p.dim + p.eps);
  const long long mod = p.rows_per_batch > 0 ? static_cast<long long>(row / p.rows_per_batch) * p.mod_stride : 0;
#pragma unroll
  for (int it = 0; it < kMaxVec; ++it) {
    const int vi = threadIdx.x + it * blockDim.x;
    const bool active = vi < nvec;
    const int c = vi * 8;
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = active ? (v[it][i] - mean) * rstd : 0.f;
    if (active) {
      float t[8];
      if (p.weight) {
        load_param8(p.weight, c, p.vec_params, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] *= p.weight_plus_one ? (1.f + t[i]) : t[i];
      }
      if (p.bias) {
        load_param8(p.bias, c, p.vec_params, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] += t[i];
      }
      if (p.scale) {
        load_param8(p.scale, mod + c, p.vec_params, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] *= 1.f + t[i];
      }
      if (p.shift) {
        load_param8(p.shift, mod + c, p.vec_params, t);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] += t[i];
      }
    }
    const uint4 o = pack_bf16x8(y);
    if (p.out && active) *reinterpret_cast<uint4*>(p.out + base + c) = o;
    if (p.out_fp8) {
      // fp8 consumers see the bf16-rounded activations, exactly like the unfused path. All 32 lanes
      // take part in the half-warp shuffles; inactive lanes carry zeros and do not store. dim % 128 == 0
      // is required for the fp8 output, so a 16-lane group is all-active or all-inactive.
      unpack_bf16x8(o, y);
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(y[i]));
#pragma unroll
      for (int o2 = 8; o2 > 0; o2 >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o2));
      if (active) store_fp8(y, amax, p.out_fp8 + base + c, p.out_scale, row, vi, p.dim, p.sf_tile_rows);
    }
  }
}

// fp8 1x128 quantisation of a bf16 matrix [rows][dim] (dim % 128 == 0) with row pitch ld. A thread keeps its
// vector of eight columns and takes kRows rows, whose loads go out together; grid (column blocks, row groups).
// Bound by HBM: 14040 x 13824 202 -> 130 us (4.5 TB/s), 4608 x 15360 77 -> 51 us (one row a thread 145 and 56).
template <int kRows>
__global__ void __launch_bounds__(256) quant_fp8_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ out,
                                 float* __restrict__ scales, int rows, int dim, long long ld,
                                 int sf_tile_rows) {
  pdl_wait();
  pdl_trigger();
  const int vi = blockIdx.x * blockDim.x + threadIdx.x;
  const bool col = vi < (dim >> 3);            // dim % 128 == 0: a 16-lane group is uniform
  // whole warps make the same rounds: rows of one block lie together
  for (int base = blockIdx.y * blockDim.y * kRows; base < rows; base += gridDim.y * blockDim.y * kRows) {
    const int row0 = base + threadIdx.y * kRows;
    uint4 raw[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      raw[r] = make_uint4(0u, 0u, 0u, 0u);
      if (col && row0 + r < rows) raw[r] = *reinterpret_cast<const uint4*>(x + (row0 + r) * ld + vi * 8);
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      float v[8];
      unpack_bf16x8(raw[r], v);
      float amax = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(v[k]));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      if (col && row0 + r < rows)
        store_fp8(v, amax, out + static_cast<long long>(row0 + r) * dim + vi * 8, scales, row0 + r, vi, dim, sf_tile_rows);
    }
  }
}

// Weight quantisation to e4m3 with one scale per 128 x 128 block. w [n][k] bf16 -> out [n][k] u8,
// scales [ceil(n/128)][k/128] fp32. One CTA (256 threads) per block.
__global__ void quant_fp8_weight_kernel(const __nv_bfloat16* __restrict__ w,
                                        uint8_t* __restrict__ out, float* __restrict__ scales,
                                        int n, int k) {
  __shared__ float red[32];
  const int nb = blockIdx.x, kb = blockIdx.y;
  float amax = 0.f;
  for (int i = threadIdx.x; i < 128 * 16; i += blockDim.x) {
    const int r = nb * 128 + (i >> 4), c = kb * 128 + (i & 15) * 8;
    if (r < n) {
      uint4 raw = *reinterpret_cast<const uint4*>(w + static_cast<long long>(r) * k + c);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 f = __bfloat1622float2(h[q]);
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = 0.f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) amax = fmaxf(amax, red[i]);
  const float sc = fmaxf(amax, 1e-12f) / kFp8Max;
  const float inv = 1.f / sc;
  if (threadIdx.x == 0) scales[static_cast<long long>(nb) * gridDim.y + kb] = sc;
  for (int i = threadIdx.x; i < 128 * 16; i += blockDim.x) {
    const int r = nb * 128 + (i >> 4), c = kb * 128 + (i & 15) * 8;
    if (r < n) {
      uint4 raw = *reinterpret_cast<const uint4*>(w + static_cast<long long>(r) * k + c);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float2 f = __bfloat1622float2(h[q]);
        lo |= static_cast<uint32_t>(to_e4m3(f.x * inv)) << (16 * q);
        lo |= static_cast<uint32_t>(to_e4m3(f.y * inv)) << (16 * q + 8);
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float2 f = __bfloat1622float2(h[2 + q]);
        hi |= static_cast<uint32_t>(to_e4m3(f.x * inv)) << (16 * q);
        hi |= static_cast<uint32_t>(to_e4m3(f.y * inv)) << (16 * q + 8);
      }
      *reinterpret_cast<uint2*>(out + static_cast<long long>(r) * k + c) = make_uint2(lo, hi);
    }
  }
}

// Gated activation: out[r][c] = act(in[r][c]) * in[r][F + c] for in [rows][2F] (gate first, then up), act:
// 0 = SiLU, 1 = GELU-tanh. Optional fp8 1x128 output (F % 128 == 0). A thread keeps its vector of eight columns
// and takes kRows rows, whose loads go out together; grid (column blocks, row groups), so no index is divided.
// Arithmetic and HBM bind about equally: 8192 x 28672 with fp8 output 485 -> 365 us, bf16 338 -> 270 us
// (one row a thread 377 and 300, four 490 and 361: too many registers; blocks that walk rows with three in flight
// 383 and 256).
template <int kRows>
__global__ void __launch_bounds__(256) glu_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                           uint8_t* __restrict__ out_fp8, float* __restrict__ out_scale, int rows,
                           int f, int act, int sf_tile_rows, const SplitPartials part) {
  pdl_wait();
  pdl_trigger();
  constexpr bool kParts = kRows == 1;          // unsummed K ranges come from small batches only
  const int vi = blockIdx.x * blockDim.x + threadIdx.x;
  const bool col = vi < (f >> 3);              // f % 128 == 0 with the fp8 output: a 16-lane group is uniform
  // whole warps make the same rounds: rows of one block lie together
  for (int base = blockIdx.y * blockDim.y * kRows; base < rows; base += gridDim.y * blockDim.y * kRows) {
    const int row0 = base + threadIdx.y * kRows;
    uint4 graw[kRows], uraw[kRows];
    if (!(kParts && part.ws)) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        graw[r] = uraw[r] = make_uint4(0u, 0u, 0u, 0u);
        if (col && row0 + r < rows) {
          const __nv_bfloat16* g = in + static_cast<long long>(row0 + r) * 2 * f + vi * 8;
          graw[r] = *reinterpret_cast<const uint4*>(g);
          uraw[r] = *reinterpret_cast<const uint4*>(g + f);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int row = row0 + r;
      const bool active = col && row < rows;
      float gv[8], uv[8];
      if (kParts && part.ws) {
        // the producing GEMM left its K ranges unsummed: add them here (no reduce kernel in between)
#pragma unroll
        for (int k = 0; k < 8; ++k) gv[k] = uv[k] = 0.f;
        if (active) {
          split_sum8(part, row, vi * 8, gv);
          split_sum8(part, row, f + vi * 8, uv);
        }
      } else {
        unpack_bf16x8(graw[r], gv);
        unpack_bf16x8(uraw[r], uv);
      }
      float y[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) y[k] = (act == 0 ? silu(gv[k]) : gelu_tanh(gv[k])) * uv[k];
      const uint4 o = pack_bf16x8(y);
      if (out && active) *reinterpret_cast<uint4*>(out + static_cast<long long>(row) * f + vi * 8) = o;
      if (out_fp8) {
        unpack_bf16x8(o, y);
        float amax = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(y[k]));
#pragma unroll
        for (int o2 = 8; o2 > 0; o2 >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o2));
        if (active)
          store_fp8(y, amax, out_fp8 + static_cast<long long>(row) * f + vi * 8, out_scale, row, vi, f, sf_tile_rows);
      }
    }
  }
}

// QK-norm (optional) + rotary embedding + paged KV write for a packed qkv activation.
//   qkv  [T][(hq + 2*hkv) * d] bf16 (q heads, then k heads, then v heads)
//   q_out [T][hq][d] bf16 (rotated), k/v written to cache pages
//   cache layout [num_pages][hkv][page][d]; slot_mapping[t] = page_index * page + offset
//   rope: style 0 = split-half (pairs (i, i + rot/2)), 1 = interleaved (pairs (2i, 2i+1));
//   rotary dims = rot (<= d); angle = pos * theta^(-2i/rot) * freq_scale[i] (optional table)
// One warp per (token, head).
struct RopeParams {
  const __nv_bfloat16* qkv;
  __nv_bfloat16* q_out;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  __nv_bfloat16* k_out;   // optional contiguous [T][hkv][d] outputs (prefill attention reads these)
  __nv_bfloat16* v_out;
  const int* positions;
  const long long* slot_mapping;  // may be null (no cache write)
  const __nv_bfloat16* q_norm_w;  // optional [d]
  const __nv_bfloat16* k_norm_w;
  const float* inv_freq;          // optional [rot/2] precomputed (scaled) inverse frequencies
  int tokens, hq, hkv, d, rot, style, page;
  float theta, eps;
  SplitPartials part;             // ws != null: qkv comes as unsummed K ranges of the producing GEMM
};

__global__ void rope_kv_kernel(const RopeParams p) {
  pdl_wait();
  pdl_trigger();
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int heads = p.hq + 2 * p.hkv;
  if (warp_global >= p.tokens * heads) return;
  const int t = warp_global / heads, h = warp_global % heads;
  const __nv_bfloat16* src = p.qkv + (static_cast<long long>(t) * heads + h) * p.d;
  const int kind = h < p.hq ? 0 : (h < p.hq + p.hkv ? 1 : 2);
  // each lane owns elements lane, lane+32, ... (d <= 256)
  float v[8];
  const int per = (p.d + 31) / 32;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = lane + 32 * i;
    if (!(i < per && c < p.d)) v[i] = 0.f;
    else if (p.part.ws) v[i] = split_sum(p.part, t, h * p.d + c);
    else v[i] = __bfloat162float(src[c]);
  }
  const __nv_bfloat16* nw = kind == 0 ? p.q_norm_w : (kind == 1 ? p.k_norm_w : nullptr);
  if (nw) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / p.d + p.eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = lane + 32 * i;
      if (i < per && c < p.d) v[i] = v[i] * rstd * __bfloat162float(nw[c]);
    }
  }
  __nv_bfloat16* dst;
  __nv_bfloat16* dst2 = nullptr;
  if (kind == 0) {
    dst = p.q_out + (static_cast<long long>(t) * p.hq + h) * p.d;
  } else {
    const int hk = kind == 1 ? h - p.hq : h - p.hq - p.hkv;
    __nv_bfloat16* cache = kind == 1 ? p.k_cache : p.v_cache;
    __nv_bfloat16* lin = kind == 1 ? p.k_out : p.v_out;
    dst = nullptr;
    if (cache && p.slot_mapping) {
      const long long slot = p.slot_mapping[t];
      if (slot >= 0) {
        const long long pg = slot / p.page, off = slot % p.page;
        dst = cache + ((pg * p.hkv + hk) * p.page + off) * p.d;
      }
    }
    if (lin) dst2 = lin + (static_cast<long long>(t) * p.hkv + hk) * p.d;
  }
  if (kind != 2 && p.rot > 0) {
    // The partner element of a rotary pair is fetched from its owner lane with shuffles; every
    // lane executes every shuffle. Partner of element c: split-half -> c +- rot/2,
    // interleaved -> c ^ 1.
    const float pos = static_cast<float>(p.positions[t]);
    const int half = p.rot >> 1;
    float outv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = lane + 32 * i;
      const bool in_rot = (i < per) && (c < p.rot);
      int partner = c, pair_idx = 0;
      bool first = true;
      if (p.style == 0) {
        first = c < half;
        pair_idx = first ? c : c - half;
        partner = first ? c + half : c - half;
      } else {
        first = (c & 1) == 0;
        pair_idx = c >> 1;
        partner = c ^ 1;
      }
      // the partner may sit in another lane and another register slot (partial rotary with
      // rot / 2 < 32 keeps it in slot 0 of lane c +- rot/2): fetch every slot from the partner's
      // lane and keep the one that holds it
      float pv = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float cand = __shfl_sync(0xffffffffu, v[j], partner & 31);
        if (j == (partner >> 5)) pv = cand;
      }
      if (in_rot) {
        const float inv = p.inv_freq ? p.inv_freq[pair_idx]
                                     : __powf(p.theta, -2.f * pair_idx / static_cast<float>(p.rot));
        float sn, cs;
        sincosf(pos * inv, &sn, &cs);
        outv[i] = first ? (v[i] * cs - pv * sn) : (v[i] * cs + pv * sn);
      } else {
        outv[i] = v[i];
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = outv[i];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = lane + 32 * i;
    if (i < per && c < p.d) {
      const __nv_bfloat16 b = __float2bfloat16(v[i]);
      if (dst) dst[c] = b;
      if (dst2) dst2[c] = b;
    }
  }
}

// Eight values as bf16 to one or two places.
__device__ __forceinline__ void store_twice(__nv_bfloat16* a, __nv_bfloat16* b, const float (&v)[8]) {
  const uint4 o = pack_bf16x8(v);
  if (a) *reinterpret_cast<uint4*>(a) = o;
  if (b) *reinterpret_cast<uint4*>(b) = o;
}

// The same for heads of 16, 32, 64, 128 or 256 values with a rotated part that is a multiple of 16, everything on
// 16-byte boundaries. Angles are the tokens', not the heads': a block works out the sines and cosines of
// `block_tokens` tokens once (they were 80 sincosf a pair of a 64 + 16 head token, and bound the kernel) and
// keeps a token's in registers while it walks the heads. A unit of work is two 16-byte vectors of one head:
// with split halves the vectors whose elements turn together, otherwise two neighbours; d / 16 lanes share a
// head. Bound by HBM: 8192 tokens x 80 heads x 128 628 -> 86 us (3.9 TB/s), 1935 x 48 83 -> 20 us.
__global__ void __launch_bounds__(256) rope_kv_vec_kernel(const RopeParams p, int block_tokens, int unit_bits) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ float rope_table[];            // [block_tokens][cos of rot / 2 | sin of rot / 2]
  __shared__ long long cache_row[8];               // row of the token in a cache of one head's pages, -1: not stored
  const int heads = p.hq + 2 * p.hkv, half = p.rot >> 1;
  const int t0 = blockIdx.x * block_tokens, nt = min(block_tokens, p.tokens - t0);
  for (int i = threadIdx.x; i < nt * half; i += blockDim.x) {
    const int tt = i / half, j = i - tt * half;
    const float pos = static_cast<float>(p.positions[t0 + tt]);
    const float inv = p.inv_freq ? p.inv_freq[j] : __powf(p.theta, -2.f * j / static_cast<float>(p.rot));
    float sn, cs;
    sincosf(pos * inv, &sn, &cs);
    rope_table[tt * p.rot + j] = cs;
    rope_table[tt * p.rot + half + j] = sn;
  }
  if (threadIdx.x < nt) {
    const long long slot = p.slot_mapping ? p.slot_mapping[t0 + threadIdx.x] : -1;
    cache_row[threadIdx.x] = slot < 0 ? -1 : slot / p.page * p.hkv * p.page + slot % p.page;
  }
  __syncthreads();
  const int u = threadIdx.x & ((1 << unit_bits) - 1);
  const int step = blockDim.x >> unit_bits;
  const int first = blockIdx.y * step + (threadIdx.x >> unit_bits), stride = gridDim.y * step;
  const bool turns = u < p.rot >> 4;               // this unit's vectors are rotated (of q and k)
  const int va = turns && p.style == 0 ? u : 2 * u, vb = turns && p.style == 0 ? u + (p.rot >> 4) : 2 * u + 1;
  for (int tt = 0; tt < nt; ++tt) {
    const int t = t0 + tt;
    float cs[8], sn[8];
    if (turns) {
      // split halves: the eight pairs of vector u; neighbours: the four pairs of each of the two vectors
      const float* tab = rope_table + tt * p.rot + u * 8;
#pragma unroll
      for (int k = 0; k < 8; ++k) { cs[k] = tab[k]; sn[k] = tab[half + k]; }
    }
    // every lane of a warp makes the same rounds, since the norm's sum is exchanged between lanes
    for (int h0 = first; h0 - (first % (32 >> unit_bits)) < heads; h0 += stride) {
      const bool active = h0 < heads;
      const int h = active ? h0 : heads - 1;
      const int kind = h < p.hq ? 0 : (h < p.hq + p.hkv ? 1 : 2);
      const int ca = (kind == 2 ? 2 * u : va) * 8, cb = (kind == 2 ? 2 * u + 1 : vb) * 8;
      float a[8], b[8];
      if (p.part.ws) {
        split_sum8(p.part, t, h * p.d + ca, a);
        split_sum8(p.part, t, h * p.d + cb, b);
      } else {
        const __nv_bfloat16* src = p.qkv + (static_cast<long long>(t) * heads + h) * p.d;
        const uint4 ra = *reinterpret_cast<const uint4*>(src + ca), rb = *reinterpret_cast<const uint4*>(src + cb);
        unpack_bf16x8(ra, a);
        unpack_bf16x8(rb, b);
      }
      if (p.q_norm_w || p.k_norm_w) {
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) ss += a[k] * a[k] + b[k] * b[k];
        for (int o = 1 << unit_bits >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const __nv_bfloat16* nw = kind == 0 ? p.q_norm_w : (kind == 1 ? p.k_norm_w : nullptr);
        if (nw) {
          const float rstd = rsqrtf(ss / p.d + p.eps);
          float w[8];
          load_param8(nw, ca, true, w);
#pragma unroll
          for (int k = 0; k < 8; ++k) a[k] = a[k] * rstd * w[k];
          load_param8(nw, cb, true, w);
#pragma unroll
          for (int k = 0; k < 8; ++k) b[k] = b[k] * rstd * w[k];
        }
      }
      if (turns && kind != 2) {
        if (p.style == 0) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float x = a[k], y = b[k];
            a[k] = x * cs[k] - y * sn[k];
            b[k] = y * cs[k] + x * sn[k];
          }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float x = a[2 * k], y = a[2 * k + 1], z = b[2 * k], w = b[2 * k + 1];
            a[2 * k] = x * cs[k] - y * sn[k];
            a[2 * k + 1] = y * cs[k] + x * sn[k];
            b[2 * k] = z * cs[4 + k] - w * sn[4 + k];
            b[2 * k + 1] = w * cs[4 + k] + z * sn[4 + k];
          }
        }
      }
      if (!active) continue;
      __nv_bfloat16 *dst = nullptr, *dst2 = nullptr;
      if (kind == 0) {
        dst = p.q_out + (static_cast<long long>(t) * p.hq + h) * p.d;
      } else {
        const int hk = kind == 1 ? h - p.hq : h - p.hq - p.hkv;
        __nv_bfloat16* cache = kind == 1 ? p.k_cache : p.v_cache;
        __nv_bfloat16* lin = kind == 1 ? p.k_out : p.v_out;
        if (cache && cache_row[tt] >= 0) dst = cache + (cache_row[tt] + static_cast<long long>(hk) * p.page) * p.d;
        if (lin) dst2 = lin + (static_cast<long long>(t) * p.hkv + hk) * p.d;
      }
      store_twice(dst ? dst + ca : nullptr, dst2 ? dst2 + ca : nullptr, a);
      store_twice(dst ? dst + cb : nullptr, dst2 ? dst2 + cb : nullptr, b);
    }
  }
}

__global__ void embedding_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                 __nv_bfloat16* __restrict__ out, int tokens, int dim, int vocab,
                                 float scale) {
  const int t = blockIdx.x;
  int id = ids[t];
  id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
  const uint4* src = reinterpret_cast<const uint4*>(table + static_cast<long long>(id) * dim);
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<long long>(t) * dim);
  for (int i = threadIdx.x; i < (dim >> 3); i += blockDim.x) {
    uint4 raw = src[i];
    if (scale != 1.f) {
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float2 f = __bfloat1622float2(h[k]);
        h[k] = __floats2bfloat162_rn(f.x * scale, f.y * scale);
      }
    }
    dst[i] = raw;
  }
}

// The block's largest value and the lowest index that has it, in every thread; 0x7fffffff: no thread had one.
__device__ __forceinline__ void block_argmax(float& best, int& bi, float* sval, int* sidx) {
  auto warp_best = [&] {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
  };
  warp_best();
  if ((threadIdx.x & 31) == 0) { sval[threadIdx.x >> 5] = best; sidx[threadIdx.x >> 5] = bi; }
  __syncthreads();
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  best = lane < nw ? sval[lane] : -INFINITY;
  bi = lane < nw ? sidx[lane] : 0x7fffffff;
  warp_best();
}

// argmax over the last dim of bf16 / fp32 logits [rows][vocab]; ties -> lowest index. One block per row; from the row's
// first 16-byte boundary on a thread reads 16 bytes at a time, four in flight: one row of 151936 bf16 42 -> 8 us. Rows
// between boundaries one value at a time left a processor too few bytes in flight: 512 of 50257 fp32 90 us.
template <typename T>
__global__ void __launch_bounds__(1024) argmax_kernel(const T* __restrict__ logits, int* __restrict__ out, int vocab,
                              long long ld) {
  __shared__ float sval[32];
  __shared__ int sidx[32];
  const T* row = logits + blockIdx.x * ld;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  constexpr int kPer = 16 / sizeof(T);
  const int head = min(vocab, static_cast<int>((16 - (reinterpret_cast<uintptr_t>(row) & 15)) % 16 / sizeof(T)));
  const int nvec = (vocab - head) / kPer;
  const uint4* body = reinterpret_cast<const uint4*>(row + head);
  if (static_cast<int>(threadIdx.x) < head) {
    const float v = static_cast<float>(row[threadIdx.x]);
    if (v > best) { best = v; bi = threadIdx.x; }
  }
  for (int i0 = threadIdx.x; i0 < nvec; i0 += 4 * blockDim.x) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * blockDim.x < nvec) raw[u] = __ldg(body + i0 + u * blockDim.x);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i >= nvec) break;
      const T* e = reinterpret_cast<const T*>(&raw[u]);
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const float v = static_cast<float>(e[k]);
        if (v > best) { best = v; bi = head + i * kPer + k; }       // a thread's indices ascend
      }
    }
  }
  for (int i = head + nvec * kPer + threadIdx.x; i < vocab; i += blockDim.x) {
    const float v = static_cast<float>(row[i]);
    if (v > best) { best = v; bi = i; }
  }
  block_argmax(best, bi, sval, sidx);
  if (bi == 0x7fffffff) {
    // Nothing above -infinity: the first value that equals it (a mask that allows no token), 0 for a row of NaN. Apart
    // from the loops above, where the second comparison costs 1 to 2 us of 10.
    for (int i = threadIdx.x; i < vocab && bi == 0x7fffffff; i += blockDim.x)
      if (static_cast<float>(row[i]) == -INFINITY) bi = i;
    __syncthreads();
    block_argmax(best, bi, sval, sidx);
    if (bi == 0x7fffffff) bi = 0;
  }
  if (threadIdx.x == 0) out[blockIdx.x] = bi;
}

// logits[b][tok] /= penalty when > 0 else *= penalty, for every token in the row's history.
__global__ void repetition_penalty_kernel(float* __restrict__ logits, const int* __restrict__ history,
                                          const int* __restrict__ hist_len, int max_hist, int vocab,
                                          const float* __restrict__ penalty) {
  const int b = blockIdx.x;
  const float pen = penalty[b];
  if (pen == 1.f) return;
  const int n = hist_len[b];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int tok = history[static_cast<long long>(b) * max_hist + i];
    if (tok >= 0 && tok < vocab) {
      // duplicates in the history would race; resolve by letting only the first occurrence act
      bool first = true;
      for (int j = 0; j < i; ++j)
        if (history[static_cast<long long>(b) * max_hist + j] == tok) { first = false; break; }
      if (first) {
        float* l = logits + static_cast<long long>(b) * vocab + tok;
        *l = *l > 0.f ? *l / pen : *l * pen;
      }
    }
  }
}

// Classifier-free-guidance combine fused with the Euler / flow-match step:
//   v = g * cond + (1 - g) * uncond ; z += v * dt     (uncond may be null: v = cond)
__global__ void cfg_euler_kernel(float* __restrict__ z, const __nv_bfloat16* __restrict__ cond,
                                 const __nv_bfloat16* __restrict__ uncond, long long n, float g,
                                 float dt) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float c = __bfloat162float(cond[i]);
    const float v = uncond ? g * c + (1.f - g) * __bfloat162float(uncond[i]) : c;
    z[i] += v * dt;
  }
}

// out = x + gate[batch][c] * y   (gated residual of DiT blocks), bf16
__global__ void gated_residual_kernel(const __nv_bfloat16* __restrict__ x,
                                      const __nv_bfloat16* __restrict__ y,
                                      const __nv_bfloat16* __restrict__ gate,
                                      __nv_bfloat16* __restrict__ out, int rows, int dim,
                                      int rows_per_batch, int mod_stride) {
  const int nvec = dim >> 3;
  const long long total = static_cast<long long>(rows) * nvec;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int row = static_cast<int>(i / nvec), vi = static_cast<int>(i % nvec);
    const int batch = rows_per_batch > 0 ? row / rows_per_batch : 0;
    uint4 xr = *reinterpret_cast<const uint4*>(x + static_cast<long long>(row) * dim + vi * 8);
    uint4 yr = *reinterpret_cast<const uint4*>(y + static_cast<long long>(row) * dim + vi * 8);
    uint4 gr = *reinterpret_cast<const uint4*>(gate + static_cast<long long>(batch) * mod_stride + vi * 8);
    const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xr);
    const __nv_bfloat162* yh = reinterpret_cast<const __nv_bfloat162*>(&yr);
    const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gr);
    uint4 o;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 a = __bfloat1622float2(xh[k]), b = __bfloat1622float2(yh[k]), g = __bfloat1622float2(gh[k]);
      ow[k] = pack_bf16x2(a.x + g.x * b.x, a.y + g.y * b.y);
    }
    *reinterpret_cast<uint4*>(out + static_cast<long long>(row) * dim + vi * 8) = o;
  }
}

// Deterministic pseudo-random fill (hash of the element index) for synthetic weights: bf16
// N(0, std) approximated by a sum of uniforms, or raw e4m3 bytes with |value| <= 448 * amp.
__device__ __forceinline__ uint32_t hash32(uint64_t x) {
  x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
  return static_cast<uint32_t>(x);
}
__global__ void fill_random_bf16_kernel(__nv_bfloat16* out, long long n, uint64_t seed, float std) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const uint32_t a = hash32(seed * 0x9e3779b97f4a7c15ull + 2 * i);
    const uint32_t b = hash32(seed * 0x9e3779b97f4a7c15ull + 2 * i + 1);
    // sum of four 16-bit uniforms: variance 4/12, mean 2 -> scale to unit variance
    const float u = ((a & 0xffff) + (a >> 16) + (b & 0xffff) + (b >> 16)) * (1.f / 65536.f) - 2.f;
    out[i] = __float2bfloat16(u * 1.7320508f * std);
  }
}
__global__ void fill_random_fp8_kernel(uint8_t* out, long long n, uint64_t seed) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const uint32_t a = hash32(seed * 0x9e3779b97f4a7c15ull + 2 * i);
    const uint32_t b = hash32(seed * 0x9e3779b97f4a7c15ull + 2 * i + 1);
    const float u = ((a & 0xffff) + (a >> 16) + (b & 0xffff) + (b >> 16)) * (1.f / 65536.f) - 2.f;
    // unit-variance value scaled so that ~4 sigma maps to the e4m3 maximum
    out[i] = to_e4m3(u * 1.7320508f * 112.f);
  }
}

inline int grid_for(long long n, int block, int cap_mult = 8) {
  long long g = (n + block - 1) / block;
  const long long cap = 148ll * cap_mult;
  return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

// Launch shape of the kernels that give a thread one vector of columns: `most` rows a thread once that still
// leaves every processor several blocks, one row below. Narrow matrices share a block between rows (threadIdx.y) once there are
// blocks enough: one row of 64 values in a block of 32 threads took 9.2 us for 16384 of them, where several take 2.6; fp8
// groups of 16 lanes stay whole.
struct RowGrid {
  int rows_each;
  dim3 block, grid;
  RowGrid(int rows, int nvec, int most) {
    const int threads = nvec >= 256 ? 256 : nvec > 16 ? (nvec + 31) / 32 * 32 : nvec > 8 ? 16 : 8;
    const int cols = (nvec + threads - 1) / threads;
    int share = threads < 32 ? 32 / threads : 1;
    while (threads < 128 && threads * share <= 128 && rows >= 148 * 4 * 2 * share) share *= 2;
    rows_each = static_cast<long long>(rows) * cols >= 148ll * 8 * 4 * share ? most : 1;
    const int each = rows_each * share, groups = (rows + each - 1) / each;
    block = dim3(threads, share);
    grid = dim3(cols, groups < 65535 ? groups : 65535);
  }
};

template <typename... P>
inline bool aligned16(P... ptrs) {
  return ((reinterpret_cast<uintptr_t>(ptrs) | ... | uintptr_t{0}) & 15) == 0;
}

}  // namespace b200

using namespace b200;

#define CHECK_LAUNCH()                                            \
  do {                                                            \
    cudaError_t e__ = cudaGetLastError();                         \
    if (e__ != cudaSuccess) return -static_cast<int>(e__) - 300;  \
  } while (0)

// (residual +) RMSNorm / LayerNorm with optional affine, AdaLN modulation, bf16 and/or fp8 output. part_ws != null: x
// is ignored and the rows are read as unsummed K ranges (see b200_glu).
B200_API int b200_norm(const void* x, const void* residual, void* residual_out, const void* weight,
                       const void* bias, const void* shift, const void* scale, void* out,
                       void* out_fp8, float* out_scale, int rows, int dim, int rows_per_batch,
                       int mod_stride, float eps, int layernorm, int weight_plus_one,
                       int sf_tile_rows, const float* part_ws, int part_splits, int part_bn, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (dim % 8 != 0 || dim > 16384) return -2;
  if (out_fp8 && dim % 128 != 0) return -3;
  NormParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.part = SplitPartials{part_ws, part_splits, part_bn};
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.residual_out = static_cast<__nv_bfloat16*>(residual_out);
  p.weight = static_cast<const __nv_bfloat16*>(weight);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.shift = static_cast<const __nv_bfloat16*>(shift);
  p.scale = static_cast<const __nv_bfloat16*>(scale);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_fp8 = static_cast<uint8_t*>(out_fp8);
  p.out_scale = out_scale;
  p.rows = rows; p.dim = dim; p.rows_per_batch = rows_per_batch; p.mod_stride = mod_stride;
  p.eps = eps; p.layernorm = layernorm; p.weight_plus_one = weight_plus_one;
  p.sf_tile_rows = sf_tile_rows;
  p.vec_params = aligned16(weight, bias, shift, scale) && mod_stride % 8 == 0;
  const int nvec = dim / 8;
  auto go = [&](auto* kernel, int per, int smem = 0) {
    launch_pdl(kernel, dim3(rows), dim3(((nvec + per - 1) / per + 31) / 32 * 32), smem, stream, p);
  };
  if (part_ws != nullptr) {
    // Blocks of this launch start while the product runs, on the processors that it leaves free. Where those are few, they would
    // take most of the rows and read their ranges alone (144 of 148 processors busy: 33 x 3072 x 3072 13.9 us with the reduce
    // kernel, 15.9 so, 11.1 with one row a processor at a time). The shared memory is not used.
    constexpr int kAlone = 116 * 1024;
    static PerDeviceOnce configured;
    if (configured.first_time() &&
        (cudaFuncSetAttribute(norm_kernel<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlone) != cudaSuccess ||
         cudaFuncSetAttribute(norm_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAlone) != cudaSuccess))
      return -4;
    nvec > 1024 ? go(norm_kernel<2, true>, 2, kAlone) : go(norm_kernel<1, true>, 1, kAlone);
  }
  else if (rows > 296 && nvec >= 1024) go(norm_kernel<4, false>, 4);
  else if (nvec > 1024 || (rows > 296 && nvec >= 256)) go(norm_kernel<2, false>, 2);
  else go(norm_kernel<1, false>, 1);
  CHECK_LAUNCH();
  return 0;
}

// sf_tile_rows > 0: `scales` is a blocked UE8M0 scale-factor array (see store_sf) instead of fp32
// [rows][dim / 128]; the same convention applies to b200_norm and b200_glu.
B200_API int b200_quant_fp8(const void* x, void* out, float* scales, int rows, int dim,
                            long long ld, int sf_tile_rows, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (dim % 128 != 0 || ld % 8 != 0) return -2;
  const RowGrid g(rows, dim / 8, 4);
  launch_pdl(g.rows_each == 4 ? quant_fp8_kernel<4> : quant_fp8_kernel<1>, g.grid, g.block, 0, stream,
             static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(out), scales, rows, dim, ld, sf_tile_rows);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_quant_fp8_weight(const void* w, void* out, float* scales, int n, int k,
                                   cudaStream_t stream) {
  if (k % 128 != 0) return -2;
  dim3 grid((n + 127) / 128, k / 128);
  quant_fp8_weight_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(w),
                                                    static_cast<uint8_t*>(out), scales, n, k);
  CHECK_LAUNCH();
  return 0;
}

// part_ws != null: `in` is ignored and the [rows][2f] input is read as the unsummed K ranges a
// deferred small-token GEMM left unsummed (see SplitPartials; b200_gemm_deferred).
B200_API int b200_glu(const void* in, void* out, void* out_fp8, float* out_scale, int rows, int f,
                      int act, int sf_tile_rows, const float* part_ws, int part_splits, int part_bn,
                      cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (f % 8 != 0 || (out_fp8 && f % 128 != 0)) return -2;
  const RowGrid g(rows, f / 8, part_ws != nullptr ? 1 : 2);
  const SplitPartials part{part_ws, part_splits, part_bn};
  launch_pdl(g.rows_each == 2 ? glu_kernel<2> : glu_kernel<1>, g.grid, g.block, 0, stream, static_cast<const __nv_bfloat16*>(in),
             static_cast<__nv_bfloat16*>(out), static_cast<uint8_t*>(out_fp8), out_scale, rows, f, act, sf_tile_rows,
             part);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_rope_kv(const void* qkv, void* q_out, void* k_cache, void* v_cache, void* k_out,
                          void* v_out, const int* positions, const long long* slot_mapping,
                          const void* q_norm_w, const void* k_norm_w, const float* inv_freq,
                          int tokens, int hq, int hkv, int d, int rot, int style, int page,
                          float theta, float eps, const float* part_ws, int part_splits, int part_bn,
                          const void* part_bias, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (d > 256 || rot > d || (rot & 1)) return -2;
  RopeParams p{};
  p.part = SplitPartials{part_ws, part_splits, part_bn, static_cast<const __nv_bfloat16*>(part_bias)};
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.q_out = static_cast<__nv_bfloat16*>(q_out);
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.k_out = static_cast<__nv_bfloat16*>(k_out);
  p.v_out = static_cast<__nv_bfloat16*>(v_out);
  p.positions = positions;
  p.slot_mapping = slot_mapping;
  p.q_norm_w = static_cast<const __nv_bfloat16*>(q_norm_w);
  p.k_norm_w = static_cast<const __nv_bfloat16*>(k_norm_w);
  p.inv_freq = inv_freq;
  p.tokens = tokens; p.hq = hq; p.hkv = hkv; p.d = d; p.rot = rot; p.style = style; p.page = page;
  p.theta = theta; p.eps = eps;
  const int heads = hq + 2 * hkv;
  int unit_bits = 0;
  while (16 << unit_bits < d) ++unit_bits;
  if (16 << unit_bits == d && rot % 16 == 0 && (style == 0 || style == 1) &&
      aligned16(qkv, q_out, k_cache, v_cache, k_out, v_out, q_norm_w, k_norm_w, part_ws, part_bias)) {
    const int block_heads = 256 >> unit_bits;
    const int chunks = (heads + block_heads - 1) / block_heads;
    const int each = tokens >= 148 * 8 ? 4 : 1;      // more tokens a block once every processor has several
    launch_pdl(rope_kv_vec_kernel, dim3((tokens + each - 1) / each, each == 1 ? chunks : 1), dim3(256),
               static_cast<size_t>(each) * rot * sizeof(float), stream, p, each, unit_bits);
    CHECK_LAUNCH();
    return 0;
  }
  const long long warps = static_cast<long long>(tokens) * heads;
  const int block = 256;
  const long long blocks = (warps * 32 + block - 1) / block;
  launch_pdl(rope_kv_kernel, dim3(static_cast<unsigned>(blocks)), dim3(block), 0, stream, p);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_embedding(const int* ids, const void* table, void* out, int tokens, int dim,
                            int vocab, float scale, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (dim % 8 != 0) return -2;
  embedding_kernel<<<tokens, 128, 0, stream>>>(ids, static_cast<const __nv_bfloat16*>(table),
                                               static_cast<__nv_bfloat16*>(out), tokens, dim, vocab,
                                               scale);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_argmax(const void* logits, int* out, int rows, int vocab, long long ld,
                         int is_fp32, cudaStream_t stream) {
  if (rows <= 0) return 0;
  // The registers of a 1024-thread block fill a processor; with more rows than processors half of that lets the start and
  // the end of one row run under the reads of another: 512 rows of 50264 fp32 24.5 -> 16.7 us, of 1000 5.9 -> 3.7 us.
  // A short row needs fewer: 1 x 100 bf16 2.8 -> 2.5 us.
  const int threads = vocab <= 2048 ? 128 : rows > num_sms() ? 512 : 1024;
  if (is_fp32)
    argmax_kernel<float><<<rows, threads, 0, stream>>>(static_cast<const float*>(logits), out, vocab, ld);
  else
    argmax_kernel<__nv_bfloat16><<<rows, threads, 0, stream>>>(static_cast<const __nv_bfloat16*>(logits), out, vocab, ld);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_repetition_penalty(float* logits, const int* history, const int* hist_len,
                                     int max_hist, int rows, int vocab, const float* penalty,
                                     cudaStream_t stream) {
  if (rows <= 0) return 0;
  repetition_penalty_kernel<<<rows, 256, 0, stream>>>(logits, history, hist_len, max_hist, vocab,
                                                      penalty);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_cfg_euler(float* z, const void* cond, const void* uncond, long long n, float g,
                            float dt, cudaStream_t stream) {
  if (n <= 0) return 0;
  cfg_euler_kernel<<<grid_for(n, 256), 256, 0, stream>>>(z, static_cast<const __nv_bfloat16*>(cond),
                                                         static_cast<const __nv_bfloat16*>(uncond),
                                                         n, g, dt);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_gated_residual(const void* x, const void* y, const void* gate, void* out,
                                 int rows, int dim, int rows_per_batch, int mod_stride,
                                 cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (dim % 8 != 0 || mod_stride % 8 != 0) return -2;
  const long long n = static_cast<long long>(rows) * (dim / 8);
  gated_residual_kernel<<<grid_for(n, 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(y),
      static_cast<const __nv_bfloat16*>(gate), static_cast<__nv_bfloat16*>(out), rows, dim,
      rows_per_batch, mod_stride);
  CHECK_LAUNCH();
  return 0;
}

B200_API int b200_fill_random(void* out, long long n, unsigned long long seed, float std,
                              int is_fp8, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (is_fp8)
    fill_random_fp8_kernel<<<grid_for(n, 256, 16), 256, 0, stream>>>(static_cast<uint8_t*>(out), n, seed);
  else
    fill_random_bf16_kernel<<<grid_for(n, 256, 16), 256, 0, stream>>>(static_cast<__nv_bfloat16*>(out), n, seed, std);
  CHECK_LAUNCH();
  return 0;
}

// ------------------------------------------------------------------------------------------
// DiT: split a packed qkv activation into head-major-free [T][H][D] q, k, v with optional per-head
// RMSNorm on q and k and rotary embedding from per-token (cos, sin) tables. Pairs are interleaved
// (2i, 2i+1), as in the Flux and Wan rotary layouts (src/HartsyInference.Diffusion/Models/
// Denoisers/DiTBlocks/FluxRope.cs, WanRope.cs:18-25; kernels dit_qkv_split_norm_f32:1358,
// dit_rope_f32:514, wan/wan_rope.cu). One warp per (token, head); d <= 256.
//   qkv [T][q_cols + 2 * kv_cols] with q first, then k, then v (row pitch ld)
//   cos/sin [T][d/2] fp32 (null = no rotation)
// ------------------------------------------------------------------------------------------
namespace b200 {
struct DitQkvParams {
  const __nv_bfloat16* qkv;
  __nv_bfloat16 *q, *k, *v;
  const __nv_bfloat16 *q_norm_w, *k_norm_w;
  const float *cos, *sin;
  int tokens, hq, hkv, d;
  long long ld;
  float eps;
};

// Four neighbouring pairs times their (cos, sin).
__device__ __forceinline__ void turn_pairs(float (&v)[8], const float* cos, const float* sin) {
  const float4 c = __ldg(reinterpret_cast<const float4*>(cos)), s = __ldg(reinterpret_cast<const float4*>(sin));
  const float cs[4] = {c.x, c.y, c.z, c.w}, sn[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float x = v[2 * k], y = v[2 * k + 1];
    v[2 * k] = x * cs[k] - y * sn[k];
    v[2 * k + 1] = y * cs[k] + x * sn[k];
  }
}

__global__ void dit_qkv_kernel(const DitQkvParams p) {
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int heads = p.hq + 2 * p.hkv;
  if (warp_global >= p.tokens * heads) return;
  const int t = warp_global / heads, h = warp_global % heads;
  const int kind = h < p.hq ? 0 : (h < p.hq + p.hkv ? 1 : 2);
  const __nv_bfloat16* src = p.qkv + static_cast<long long>(t) * p.ld + static_cast<long long>(h) * p.d;
  // lane owns pairs (2 * (lane + 32 * i), +1): d / 2 pairs over 32 lanes
  const int pairs = p.d >> 1;
  float a[4], b[4];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int pi = lane + 32 * i;
    if (pi < pairs) {
      const __nv_bfloat162 v2 = *reinterpret_cast<const __nv_bfloat162*>(src + 2 * pi);
      const float2 f = __bfloat1622float2(v2);
      a[i] = f.x; b[i] = f.y;
      ss += f.x * f.x + f.y * f.y;
    } else { a[i] = b[i] = 0.f; }
  }
  const __nv_bfloat16* nw = kind == 0 ? p.q_norm_w : (kind == 1 ? p.k_norm_w : nullptr);
  if (nw) {
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / p.d + p.eps);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int pi = lane + 32 * i;
      if (pi < pairs) {
        a[i] *= rstd * __bfloat162float(nw[2 * pi]);
        b[i] *= rstd * __bfloat162float(nw[2 * pi + 1]);
      }
    }
  }
  __nv_bfloat16* dst;
  if (kind == 0) dst = p.q + (static_cast<long long>(t) * p.hq + h) * p.d;
  else if (kind == 1) dst = p.k + (static_cast<long long>(t) * p.hkv + (h - p.hq)) * p.d;
  else dst = p.v + (static_cast<long long>(t) * p.hkv + (h - p.hq - p.hkv)) * p.d;
  const bool rot = kind != 2 && p.cos != nullptr;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int pi = lane + 32 * i;
    if (pi < pairs) {
      float x = a[i], y = b[i];
      if (rot) {
        const float c = p.cos[static_cast<long long>(t) * pairs + pi], s = p.sin[static_cast<long long>(t) * pairs + pi];
        x = a[i] * c - b[i] * s;
        y = b[i] * c + a[i] * s;
      }
      *reinterpret_cast<__nv_bfloat162*>(dst + 2 * pi) = __floats2bfloat162_rn(x, y);
    }
  }
}

// The same for heads of 32, 64, 128 or 256 values with everything on 16-byte boundaries: a thread takes 16
// neighbouring values of one head (two vectors, eight rotary pairs), d / 16 lanes share a head's norm. Bound by
// HBM: 4608 tokens x 72 heads x 128 with norm and rotation, 66 -> 29 us.
__global__ void __launch_bounds__(256) dit_qkv_vec_kernel(const DitQkvParams p, int unit_bits) {
  const int heads = p.hq + 2 * p.hkv;
  const long long at = blockIdx.x * 256ll + threadIdx.x, total = static_cast<long long>(p.tokens) * heads << unit_bits;
  if ((at & ~31ll) >= total) return;               // whole warps leave: the norm exchanges sums between lanes
  const bool active = at < total;
  const unsigned i = static_cast<unsigned>(active ? at : total - 1);
  const int u = i & ((1 << unit_bits) - 1);
  const int t = (i >> unit_bits) / heads, h = (i >> unit_bits) - t * heads;
  const int kind = h < p.hq ? 0 : (h < p.hq + p.hkv ? 1 : 2);
  const uint4* src = reinterpret_cast<const uint4*>(p.qkv + t * p.ld + static_cast<long long>(h) * p.d + u * 16);
  uint4 ra = src[0], rb = src[1];
  __nv_bfloat16* dst = kind == 0 ? p.q + (static_cast<long long>(t) * p.hq + h) * p.d
                     : kind == 1 ? p.k + (static_cast<long long>(t) * p.hkv + (h - p.hq)) * p.d
                                 : p.v + (static_cast<long long>(t) * p.hkv + (h - p.hq - p.hkv)) * p.d;
  float a[8], b[8];
  unpack_bf16x8(ra, a);
  unpack_bf16x8(rb, b);
  if (p.q_norm_w || p.k_norm_w) {
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += a[k] * a[k] + b[k] * b[k];
    for (int o = 1 << unit_bits >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const __nv_bfloat16* nw = kind == 0 ? p.q_norm_w : (kind == 1 ? p.k_norm_w : nullptr);
    if (nw) {
      const float rstd = rsqrtf(ss / p.d + p.eps);
      float w[8];
      load_param8(nw, u * 16, true, w);
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] *= rstd * w[k];
      load_param8(nw, u * 16 + 8, true, w);
#pragma unroll
      for (int k = 0; k < 8; ++k) b[k] *= rstd * w[k];
    }
  }
  if (kind != 2 && p.cos != nullptr) {
    const long long pair = static_cast<long long>(t) * (p.d >> 1) + u * 8;
    turn_pairs(a, p.cos + pair, p.sin + pair);
    turn_pairs(b, p.cos + pair + 4, p.sin + pair + 4);
  }
  if (kind != 2) { ra = pack_bf16x8(a); rb = pack_bf16x8(b); }
  if (active) {
    uint4* out = reinterpret_cast<uint4*>(dst + u * 16);
    out[0] = ra;
    out[1] = rb;
  }
}

// Query and key normalised over the whole row (all heads), then the rotation, and the three parts apart: one block
// per token, hq * d and hkv * d up to 8 * 256 * kVec values. Bound by HBM; it takes the place of two copies, two
// norms, a concatenation and the kernel above: 14040 tokens of 3 x 5120 about 1600 -> 218 us.
template <int kVec>
__global__ void __launch_bounds__(256) dit_qkv_row_kernel(const DitQkvParams p) {
  __shared__ float red[2][8];
  const int t = blockIdx.x, nq = p.hq * p.d >> 3, nk = p.hkv * p.d >> 3, per_head = p.d >> 3;
  const uint4* src = reinterpret_cast<const uint4*>(p.qkv + t * p.ld);
  uint4 rq[kVec], rk[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int at = threadIdx.x + 256 * i;
    rq[i] = rk[i] = make_uint4(0u, 0u, 0u, 0u);
    if (at < nq) rq[i] = src[at];
    if (at < nk) rk[i] = src[nq + at];
  }
  float sq = 0.f, sk = 0.f;
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    float a[8], b[8];
    unpack_bf16x8(rq[i], a);
    unpack_bf16x8(rk[i], b);
#pragma unroll
    for (int k = 0; k < 8; ++k) { sq += a[k] * a[k]; sk += b[k] * b[k]; }
  }
  sq = warp_sum(sq);
  sk = warp_sum(sk);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = sq; red[1][threadIdx.x >> 5] = sk; }
  __syncthreads();
  sq = sk = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) { sq += red[0][w]; sk += red[1][w]; }
  const float fq = p.q_norm_w ? rsqrtf(sq / (p.hq * p.d) + p.eps) : 1.f, fk = p.k_norm_w ? rsqrtf(sk / (p.hkv * p.d) + p.eps) : 1.f;
  const long long pair0 = static_cast<long long>(t) * (p.d >> 1);
  auto part = [&](const uint4& raw, int at, const __nv_bfloat16* w, float f, __nv_bfloat16* dst) {
    float a[8];
    unpack_bf16x8(raw, a);
    if (w) {
      float c[8];
      load_param8(w, at * 8, true, c);
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] *= f * c[k];
    }
    if (p.cos) {
      const long long pair = pair0 + (at % per_head) * 4;
      turn_pairs(a, p.cos + pair, p.sin + pair);
    }
    reinterpret_cast<uint4*>(dst)[at] = pack_bf16x8(a);
  };
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int at = threadIdx.x + 256 * i;
    if (at < nq) part(rq[i], at, p.q_norm_w, fq, p.q + static_cast<long long>(t) * nq * 8);
    if (at < nk) part(rk[i], at, p.k_norm_w, fk, p.k + static_cast<long long>(t) * nk * 8);
  }
  for (int at = threadIdx.x; at < nk; at += 256)
    reinterpret_cast<uint4*>(p.v + static_cast<long long>(t) * nk * 8)[at] = src[nq + nk + at];
}
}  // namespace b200

B200_API int b200_dit_qkv(const void* qkv, void* q, void* k, void* v, const void* q_norm_w,
                          const void* k_norm_w, const float* cos, const float* sin, int tokens, int hq,
                          int hkv, int d, long long ld, float eps, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (d > 256 || (d & 1)) return -2;
  DitQkvParams p{};
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.q = static_cast<__nv_bfloat16*>(q);
  p.k = static_cast<__nv_bfloat16*>(k);
  p.v = static_cast<__nv_bfloat16*>(v);
  p.q_norm_w = static_cast<const __nv_bfloat16*>(q_norm_w);
  p.k_norm_w = static_cast<const __nv_bfloat16*>(k_norm_w);
  p.cos = cos; p.sin = sin;
  p.tokens = tokens; p.hq = hq; p.hkv = hkv; p.d = d; p.ld = ld; p.eps = eps;
  const long long warps = static_cast<long long>(tokens) * (hq + 2 * hkv);
  int unit_bits = 1;
  while (16 << unit_bits < d) ++unit_bits;
  if (16 << unit_bits == d && ld % 8 == 0 && aligned16(qkv, q, k, v, q_norm_w, k_norm_w, cos, sin) && warps << unit_bits < 1ll << 31) {
    dit_qkv_vec_kernel<<<static_cast<unsigned>(((warps << unit_bits) + 255) / 256), 256, 0, stream>>>(p, unit_bits);
    CHECK_LAUNCH();
    return 0;
  }
  const long long blocks = (warps * 32 + 255) / 256;
  dit_qkv_kernel<<<static_cast<int>(blocks), 256, 0, stream>>>(p);
  CHECK_LAUNCH();
  return 0;
}

// b200_dit_qkv with the norms taken over the whole rows of q and k (weights [hq * d] and [hkv * d]). Returns -2 for
// sizes or alignments that it does not take.
B200_API int b200_dit_qkv_row(const void* qkv, void* q, void* k, void* v, const void* q_norm_w,
                              const void* k_norm_w, const float* cos, const float* sin, int tokens, int hq,
                              int hkv, int d, long long ld, float eps, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  const int widest = (hq > hkv ? hq : hkv) * d;
  if (d % 8 != 0 || ld % 8 != 0 || widest > 8192 || !aligned16(qkv, q, k, v, q_norm_w, k_norm_w, cos, sin)) return -2;
  const DitQkvParams p{static_cast<const __nv_bfloat16*>(qkv), static_cast<__nv_bfloat16*>(q), static_cast<__nv_bfloat16*>(k),
                       static_cast<__nv_bfloat16*>(v), static_cast<const __nv_bfloat16*>(q_norm_w),
                       static_cast<const __nv_bfloat16*>(k_norm_w), cos, sin, tokens, hq, hkv, d, ld, eps};
  if (widest <= 4096) dit_qkv_row_kernel<2><<<tokens, 256, 0, stream>>>(p);
  else if (widest <= 6144) dit_qkv_row_kernel<3><<<tokens, 256, 0, stream>>>(p);
  else dit_qkv_row_kernel<4><<<tokens, 256, 0, stream>>>(p);
  CHECK_LAUNCH();
  return 0;
}
