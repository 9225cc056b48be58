// What the kernels of a dense product share: their parameters and the epilogue of 32 accumulator columns.
#pragma once
#include "comm.cuh"

namespace b200 {

// Fused GEMM -> all-reduce (+ residual add + RMSNorm + fp8 quantisation) for the row-parallel
// linears of a tensor-parallel group, token counts up to 128. One kernel per linear:
//   1. the tcgen05 tiles of this rank's partial product are stored as bf16 into the rank's OWN
//      `part` buffer of the symmetric heap ([K splits][tokens][features]; a K split is simply one
//      more addend of the reduction, so split tiles need no local fix-up);
//   2. the last CTA of the rank to finish its tiles raises the `ready` counter of every rank (one
//      multimem.red through the NVSwitch, or one red per peer);
//   3. token rows are dealt to the ranks in contiguous blocks; CTA i of the owning rank waits for
//      `ready`, pulls row i summed over all ranks (multimem.ld_reduce: the switch adds the ranks'
//      copies in fp32; without a multicast mapping: one peer load per rank), adds bias and the
//      rank-local residual row, applies RMSNorm and optionally quantises to e4m3 with 1x128 scales,
//      and stores the results into EVERY rank's output buffers (multimem.st or one store per peer);
//   4. the rank's last row raises `done` everywhere; CTA 0 leaves only after `done` shows that all
//      rows of all ranks have landed locally, so the next kernel in the stream may read them.
// The residual stream stays sharded by token row (each rank keeps the rows it owns up to date),
// the normalised activations come out replicated. Counters are cumulative over calls (no host
// resets: the kernel is capturable in CUDA graphs); every wait is bounded and reports through
// the status word.
struct AllReduceParams {
  int rank, world;
  int part_splits;                   // K splits the `part` buffer has room for
  int use_mc;                        // 1: entries [0] of the arrays below are multicast aliases
  __nv_bfloat16* part;               // local: [splits][tokens][features] bf16 partial products
  const __nv_bfloat16* part_src[8];  // where to read the partials of all ranks from
  __nv_bfloat16* res;                // local residual stream [tokens][features], updated in place (may be null)
  const __nv_bfloat16* norm_w;       // RMSNorm weight [features] (null: no normalisation)
  const __nv_bfloat16* bias;         // [features], may be null
  float eps;
  int weight_plus_one;
  __nv_bfloat16* out_bf16[8];        // [tokens][features] bf16 (may be null)
  uint8_t* out_q[8];                 // [tokens][features] e4m3 (may be null)
  uint32_t* out_sf[8];               // its scales: fp32 [tokens][features / 128] or blocked UE8M0 words
  int sf_tile_rows;                  // > 0: blocked UE8M0 layout with this many rows per block
  uint32_t* flags[8];                // per rank two counters: [0] ready, [1] done
  uint32_t* flags_local;
  uint32_t* ctr;                     // local: [0] calls completed, [1] CTAs past the GEMM, [2] row CTAs done, [3] CTAs finished
  long long wait_budget;             // cycles
  int debug_skip_ready;              // test aid: this rank never raises `ready`, so the waits on it run out
  // More than 128 tokens (prefill, DiT sequences): the GEMM runs in its large-token orientation
  // without K splits, `part` is [tokens][features], and the reduce phase is elementwise:
  //   out = res + gate * (sum over ranks + bias)      (res, gate optional; no norm, no fp8 emit)
  // `res` is then the replicated residual stream and is only read (the new stream is `out`).
  int large;
  const __nv_bfloat16* gate;         // [features], may be null
  // Reduce-scatter form of the large-token case (sequence-parallel regions): the result rows this
  // rank owns go to `out_local` ([owned rows][features], local memory) and nowhere else; `res` is
  // then the rank's block of the residual stream, indexed from the first owned row.
  __nv_bfloat16* out_local;
};

// All-gather -> GEMM for the column-parallel linears of a sequence-parallel region (more than 128
// tokens): every rank holds a contiguous block of ceil(m / world) token rows (activations, and for
// fp8 their scales). One kernel per linear:
//   1. the epilogue warps of all CTAs copy the rank's block into the same rows of EVERY rank's
//      gather buffer (multimem.st through the NVSwitch, or one store per peer), then the rank's last
//      CTA raises the rank's arrival counter on every rank;
//   2. the TMA producer waits for the arrival counters of the ranks whose rows a token tile covers
//      before it loads that tile from the LOCAL gather buffer; tiles are walked starting with the
//      rank's own rows, so the tensor core works on local data while the peers' rows arrive;
//   3. when the rank's last CTA is through, it raises `done` on every rank; the copy phase of the
//      next call waits for the `done` of all ranks before it overwrites the gather buffers.
// Counters are cumulative (capturable in CUDA graphs); every wait is bounded.
struct GatherParams {
  int rank, world;
  int use_mc;                         // 1: entries [0] of the destination arrays are multicast aliases
  int rows_total, rows_per_rank;      // rank r owns rows [r * rows_per_rank, ...) of rows_total
  const uint8_t* src;                 // local block [rows][row_bytes]
  long long row_bytes;                // bytes of one activation row (a multiple of 16)
  uint8_t* dst[8];                    // every rank's gather buffer [rows_total][row_bytes]
  // scales of an fp8 operand: fp32 [rows][k / 128] (sf_words = 0) or the blocked UE8M0 layout, one
  // 32-bit word per (row, group of four 128-wide K blocks) (sf_words = words per row = k groups)
  const uint32_t* src_scale;
  uint32_t* dst_scale[8];
  int scale_words;                    // fp32 scales per row (fp32 mode)
  int sf_words;                       // > 0: blocked UE8M0 layout
  uint32_t* flags[8];                 // per rank: [0, 8) arrival of source rank s, [8] done
  uint32_t* flags_local;
  uint32_t* ctr;                      // local: [0] calls completed, [1] CTAs past the copy, [2] CTAs finished
  long long wait_budget;
};
constexpr int kAgFlagDone = 8;

struct GemmParams {
  int rows_a;          // rows of the A operand (tiled by 128)
  int rows_b;          // rows of the B operand (tiled by BN)
  int k;               // reduction length in elements
  int stages;
  int swap_out;        // 0: C[a_row][b_row]; 1: C[b_row][a_row]
  // Grouped mode (MoE experts): A stacks `rows_a / group_n` weight matrices of group_n rows, B
  // stacks one BN-row token block per group; A tile t pairs with B block (t * 128) / group_n and
  // the output column is a_row % group_n. 0 = ordinary GEMM.
  int group_n;
  // Grouped mode: number of used slots per group (device memory, may be null). Groups with a zero
  // count are skipped by every role of every CTA, so idle experts cost no weight traffic.
  const int* group_counts;
  // Grouped "column-batched" variant (per-head projections): every group reads the SAME token rows
  // of B at column offset g * group_b_koff (elements) and writes output columns starting at
  // g * group_out_stride. 0 = stacked token blocks as described above.
  int group_b_koff;
  int group_out_stride;
  // Stacked grouped mode with several token blocks per weight group (`group_chunks` > 1): B block
  // e * chunks + c pairs with weight group e. Tiles are ordered (group, A tile, chunk) so that the
  // chunks of one weight tile run next to each other and the second read of the weights hits L2.
  int group_chunks;
  // Stacked grouped mode with a DEVICE-SIDE block list (variable tokens per group): B block b
  // belongs to weight group block_group[b] and *dyn_blocks blocks are in use; tile t is
  // (block t / tpg, A tile t % tpg). Null = the static layouts above.
  const int* block_group;
  const int* dyn_blocks;
  // MX mode (hardware block scaling): UE8M0 scale factors in the blocked layout
  // [row tile][k group of 512][128 x uint32], see quant_mx.cuh; sf_tile_b = B rows per SF block.
  const uint32_t* sf_a;
  const uint32_t* sf_b;
  int sf_kgroups;
  int sf_tile_b;
  // Shifted-row accumulation (convolutions as one GEMM): K is a sequence of taps of tap_kblocks
  // k-blocks each; tap t reads A rows shifted down by tap_shift[t] and A columns
  // [0, tap_kblocks * 64). 0 = ordinary GEMM.
  int tap_kblocks;
  int tap_shift[28];
  // 1: every tile is split over the CTAs of a thread-block cluster (cluster size = splits, one work
  // item per CTA); the partials stay in shared memory and are summed through distributed shared
  // memory, each CTA reducing its share of the tile. No scratch traffic, no second kernel.
  int cluster_reduce;
  // 1: every tile is split and a second kernel (splitk_reduce_kernel) sums the partials with the
  // whole machine; 0: the last CTA to arrive at a split tile sums them inside this kernel.
  int external_reduce;
  // K-split of the trailing tiles: tiles [0, first_split_tile) are whole, every later tile is
  // cut into `splits` ranges of `kblocks_per_split` k-blocks
  int first_split_tile;
  int num_tiles;
  int splits;
  int kblocks_per_split;
  // > 0: even shares (small-token orientation, more tiles than CTAs): CTA c takes the c-th of share_ctas equal parts of all tiles'
  // K groups in a row (share_groups a tile, share_kblocks k-blocks each). A share holds a tile at least, so a tile is cut by one
  // boundary between shares at most; its two pieces meet in slot c = the CTA of the first one
  int share_ctas, share_groups, share_kblocks;
  float* split_ws;          // [split tiles][splits][BN][128] fp32 partials
  uint32_t* split_counter;  // [split tiles], zero between launches
  long long ldc;            // leading dimension of C in elements
  __nv_bfloat16* out;
  const __nv_bfloat16* bias;      // per output feature (column of C), may be null
  const __nv_bfloat16* gate;      // per output feature multiplicative gate, may be null
  const __nv_bfloat16* residual;  // same layout as C, may be null
  int act;                        // 0 none, 1 gelu-tanh, 2 silu, 3 relu squared, 4 tanh
  int act_col;                    // first output feature that the activation applies to
  // fp8 block scales, K-contiguous: scale(row, kb) = s[(row / gran) * ld + kb], ld = K / 128.
  // A thread walks one row's scales along K, so consecutive k-blocks hit the same cache line.
  const float* scale_a;
  const float* scale_b;
  int sa_gran, sa_ld, sb_gran, sb_ld;
  DeviceStatus* status;
  AllReduceParams ar;   // ar.world == 0: plain GEMM
  GatherParams ag;      // ag.world == 0: the A operand is complete when the kernel starts
  int ta_rotate;        // plain GEMM: A tiles are walked starting with this one
  // Gated product (kGlu instances): w holds f gate rows, then f up rows; a tile's columns are 128 of either, and
  // act(gate) * up leaves as bf16 (out) or as e4m3 with 1x128 UE8M0 scales in the blocked layout (glu_q, glu_sf)
  int glu_f, glu_act;   // act: 0 = SiLU, 1 = GELU-tanh
  uint8_t* glu_q;
  uint8_t* glu_sf;
  int glu_sf_rows;      // rows per block of the scale layout
  // Quantised output (gemm_pair.cu): features from q_from on leave as e4m3 with 1x128 UE8M0 scales, in columns from q_col0 on of a
  // matrix with rows q_ld bytes apart and q_kgroups scale words a row; the ones in front as bf16 to out
  int q_from, q_col0, q_kgroups;
  long long q_ld;
  int row_stores;       // large-token orientation: C (and bias, gate, residual) can be reached in 16-byte pieces
  int band;             // > 0, plain GEMM: tiles are walked in bands of this many A tiles (see decode_item)
};

constexpr int kTileA = 128;
constexpr int kStageBytesA = kTileA * 128;
constexpr int kGemmThreads = 320;   // TMA warp, MMA warp, 8 epilogue warps

// Output column of weight row `a_row` in the small-token orientation.
__device__ __forceinline__ long long swap_col(const GemmParams& p, int a_row) {
  if (p.group_n <= 0) return a_row;
  const int g = a_row / p.group_n, c = a_row - g * p.group_n;
  return p.group_b_koff > 0 ? static_cast<long long>(g) * p.group_out_stride + c : c;
}

__device__ __forceinline__ float apply_epilogue(const GemmParams& p, float v, long long row,
                                                long long col) {
  // row = token index, col = output feature, both already bounds-checked
  if (p.bias) v += __bfloat162float(p.bias[col]);
  if (col < p.act_col) { /* features ahead of the activation's first */ }
  else if (p.act == 1) v = gelu_tanh(v);
  else if (p.act == 2) v = silu(v);
  else if (p.act == 3) v = relu2(v);
  else if (p.act == 4) v = tanhf(v);
  if (p.gate) v *= __bfloat162float(p.gate[col]);
  if (p.residual) v += __bfloat162float(p.residual[row * p.ldc + col]);
  return v;
}

// The activation of 32 values: chosen once, so that the others' code is not in the way
__device__ __forceinline__ void act_chunk(int act, float (&v)[32]) {
  if (act == 1) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
  } else if (act == 2) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
  } else if (act == 3) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = relu2(v[j]);
  } else if (act == 4) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = tanhf(v[j]);
  }
}

// Stores 32 consecutive accumulator columns (B rows b0..b0+31) of A row `a_row` of a whole tile
// to its destination: C, or (fused all-reduce) the staging buffer of the owning rank.
// `b_end` is the end of the tile's B rows (a 16-row tile fills only half of a 32-column chunk; the
// rest of the chunk is not this tile's data). kSwap: the small-token orientation (p.swap_out).
template <bool kSwap>
__device__ __forceinline__ void store_chunk(const GemmParams& p, float (&v)[32], int a_row,
                                            int b0, int b_end, int split = 0) {
  if (a_row >= p.rows_a) return;
  if (p.ar.world > 0) {
    // fused all-reduce: raw bf16 partial of this K split into the rank's own [split][token][feature]
    // buffer (always the small-token orientation: a_row is the feature, the chunk walks tokens)
    if constexpr (!kSwap) {
      // large-token orientation: a_row is the token, the chunk walks 32 features (whole chunks:
      // the feature count is a multiple of 128)
      if (b0 >= b_end) return;
      __nv_bfloat16* dst = p.ar.part + static_cast<long long>(a_row) * p.rows_b + b0;
#pragma unroll
      for (int j = 0; j < 32; j += 8)
        *reinterpret_cast<uint4*>(dst + j) =
            make_uint4(pack_bf16x2(v[j], v[j + 1]), pack_bf16x2(v[j + 2], v[j + 3]), pack_bf16x2(v[j + 4], v[j + 5]),
                       pack_bf16x2(v[j + 6], v[j + 7]));
      return;
    }
    __nv_bfloat16* dst = p.ar.part + (static_cast<long long>(split) * p.rows_b + b0) * p.rows_a + a_row;
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (b0 + j < b_end) dst[static_cast<long long>(j) * p.rows_a] = __float2bfloat16(v[j]);
    return;
  }
  if constexpr (!kSwap) {
    __nv_bfloat16* dst = p.out + static_cast<long long>(a_row) * p.ldc + b0;
    if (b0 + 32 <= b_end && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
      uint32_t w[16];
#pragma unroll
      for (int j = 0; j < 32; j += 2)
        w[j >> 1] = pack_bf16x2(apply_epilogue(p, v[j], a_row, b0 + j),
                                apply_epilogue(p, v[j + 1], a_row, b0 + j + 1));
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<uint4*>(dst + 2 * j) = make_uint4(w[j], w[j + 1], w[j + 2], w[j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (b0 + j < b_end)
          dst[j] = __float2bfloat16(apply_epilogue(p, v[j], a_row, b0 + j));
    }
  } else {
    // A lane holds one feature of 32 tokens, so bias, gate and the activation's choice are the same for all of them. One short
    // loop per step: with apply_epilogue in each of the 32 the code of every activation lay between two stores, and fetching
    // it the once or twice that a kernel comes by took 500 to 1400 cycles a token (a tile of 128 tokens 31000, of 6 8500).
    const long long col = swap_col(p, a_row);
    if (p.bias) {
      const float t = __bfloat162float(p.bias[col]);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] += t;
    }
    if (p.act != 0 && col >= p.act_col) act_chunk(p.act, v);
    if (p.gate) {
      const float t = __bfloat162float(p.gate[col]);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] *= t;
    }
    const int n = b_end - b0;
    const long long at = static_cast<long long>(b0) * p.ldc + col;
    if (p.residual) {
      const __nv_bfloat16* src = p.residual + at;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < n) v[j] += __bfloat162float(src[static_cast<long long>(j) * p.ldc]);
    }
    __nv_bfloat16* dst = p.out + at;
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < n) dst[static_cast<long long>(j) * p.ldc] = __float2bfloat16(v[j]);
  }
}

__device__ __forceinline__ void load_cols8(const __nv_bfloat16* src, float (&v)[8]) {
  const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src));
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

// Epilogue of 32 rows x 32 columns of a whole tile in the large-token orientation: lane l holds row
// row0 + l. The values go through a strip of shared memory that belongs to the warp, so that global
// memory sees 64-byte runs of a row instead of 16-byte pieces of 32 rows, whose half-written sectors held the
// tensor core up (fp8 4608 x 21504 x 3072 with the 128 x 256 tile: 1127 -> 326 us, bf16 579 -> 440 us).
constexpr int kStripPitch = 80;                        // 64 bytes + 16: rows of a strip start in different banks
constexpr int kStripBytes = 32 * kStripPitch;
__device__ __forceinline__ void store_chunk_rows(const GemmParams& p, float (&v)[32], int row0, int b0, uint8_t* strip) {
  const int lane = threadIdx.x & 31;
  const int pr = lane >> 2, pc = lane & 3;             // this lane's row of eight and 16-byte piece in global accesses
  const long long at = static_cast<long long>(row0 + pr) * p.ldc + b0 + pc * 8;
  if (p.residual) {
    uint4 raw[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      raw[i] = make_uint4(0u, 0u, 0u, 0u);
      if (row0 + i * 8 + pr < p.rows_a) raw[i] = *reinterpret_cast<const uint4*>(p.residual + at + i * 8 * p.ldc);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(strip + (i * 8 + pr) * kStripPitch + pc * 16) = raw[i];
    __syncwarp();
  }
  uint8_t* own = strip + lane * kStripPitch;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float t[8];
    if (p.bias) {
      load_cols8(p.bias + b0 + q * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[q * 8 + j] += t[j];
    }
    if (b0 + q * 8 < p.act_col) {
      // features ahead of the activation's first (a multiple of 8)
    } else if (p.act == 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[q * 8 + j] = gelu_tanh(v[q * 8 + j]);
    } else if (p.act == 2) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[q * 8 + j] = silu(v[q * 8 + j]);
    } else if (p.act == 3) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[q * 8 + j] = relu2(v[q * 8 + j]);
    } else if (p.act == 4) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[q * 8 + j] = tanhf(v[q * 8 + j]);
    }
    if (p.gate) {
      load_cols8(p.gate + b0 + q * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[q * 8 + j] *= t[j];
    }
    if (p.residual) {
      const uint4 raw = *reinterpret_cast<const uint4*>(own + q * 16);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        v[q * 8 + 2 * j] += f.x;
        v[q * 8 + 2 * j + 1] += f.y;
      }
    }
    *reinterpret_cast<uint4*>(own + q * 16) =
        make_uint4(pack_bf16x2(v[q * 8], v[q * 8 + 1]), pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]),
                   pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]), pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]));
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 o = *reinterpret_cast<const uint4*>(strip + (i * 8 + pr) * kStripPitch + pc * 16);
    if (row0 + i * 8 + pr < p.rows_a) *reinterpret_cast<uint4*>(p.out + at + i * 8 * p.ldc) = o;
  }
  __syncwarp();                                        // the strip is free for the next chunk
}

// 32 bytes a lane, one sector: what an epilogue of whole rows per lane writes without passing through shared memory, whose
// 128 bytes a cycle the operands take (64 in by TMA, 64 out to the tensor core).
__device__ __forceinline__ void store_words8(void* dst, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
               "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
__device__ __forceinline__ void load_words8(uint32_t* w, const void* src) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(src)
               : "memory");
}
// Largest magnitude of 32 features, bf16 pairs
__device__ __forceinline__ float words_max(const uint32_t (&y)[16], float mx) {
#pragma unroll
  for (int j = 0; j < 16; ++j) mx = fmaxf(mx, fmaxf(fabsf(__uint_as_float(y[j] << 16)), fabsf(__uint_as_float(y[j] & 0xffff0000u))));
  return mx;
}
// 32 features of act(gate) * up as bf16 pairs
__device__ __forceinline__ void glu_words(const GemmParams& p, const uint32_t (&gate)[32], const uint32_t (&up)[32], uint32_t (&y)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float g0 = __uint_as_float(gate[2 * j]), g1 = __uint_as_float(gate[2 * j + 1]);
    y[j] = pack_bf16x2((p.glu_act == 0 ? silu(g0) : gelu_tanh(g0)) * __uint_as_float(up[2 * j]),
                       (p.glu_act == 0 ? silu(g1) : gelu_tanh(g1)) * __uint_as_float(up[2 * j + 1]));
  }
}
// 32 features, bf16 pairs, as e4m3
__device__ __forceinline__ void fp8_words(const uint32_t (&y)[16], float inv, uint32_t* q) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t a = y[2 * j], b = y[2 * j + 1];
    q[j] = static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(__uint_as_float(a << 16) * inv, __uint_as_float(a & 0xffff0000u) * inv),
                                                          __NV_SATFINITE, __NV_E4M3)) |
           static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(__uint_as_float(b << 16) * inv, __uint_as_float(b & 0xffff0000u) * inv),
                                                          __NV_SATFINITE, __NV_E4M3)) << 16;
  }
}

// Epilogue of a gated tile: this warp's 32 rows and, of the tile's 128 output features, the half `hsel`. r holds
// the gate values of those 64 features, then the up values. The scale of a row's 128 features needs both halves, which
// sit in two warps: they exchange maxima through `amax` ([2][128], one of two buffers) behind a barrier of their
// own, which a warp whose accumulator did not come (got = false) still meets.
__device__ __forceinline__ void store_glu_tile(const GemmParams& p, uint32_t (&r)[4][32], int row0, int tb, int hsel, int quarter,
                                               float* amax, uint8_t* strip, bool got) {
  const int lane = threadIdx.x & 31, pr = lane >> 2, pc = lane & 3;
  uint32_t y[2][16];                                   // 64 features as bf16 pairs
#pragma unroll
  for (int c = 0; c < 2; ++c) glu_words(p, r[c], r[2 + c], y[c]);
  auto leave = [&](const uint32_t* words, uint8_t* dst, long long pitch) {      // 64 bytes per row through the strip
    uint8_t* own = strip + lane * kStripPitch;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4*>(own + q * 16) = make_uint4(words[4 * q], words[4 * q + 1], words[4 * q + 2], words[4 * q + 3]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 v = *reinterpret_cast<const uint4*>(strip + (i * 8 + pr) * kStripPitch + pc * 16);
      if (got && row0 + i * 8 + pr < p.rows_a) *reinterpret_cast<uint4*>(dst + (i * 8 + pr) * pitch + pc * 16) = v;
    }
    __syncwarp();
  };
  if (p.glu_q == nullptr) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
      leave(y[c], reinterpret_cast<uint8_t*>(p.out + static_cast<long long>(row0) * p.ldc + tb * 128 + hsel * 64 + c * 32), p.ldc * 2);
    return;
  }
  float mx = 0.f;
#pragma unroll
  for (int j = 0; j < 32; ++j)
    mx = fmaxf(mx, fmaxf(fabsf(__uint_as_float(y[j >> 4][j & 15] << 16)), fabsf(__uint_as_float(y[j >> 4][j & 15] & 0xffff0000u))));
  const int row = quarter * 32 + lane;
  amax[hsel * 128 + row] = mx;
  asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
  mx = fmaxf(mx, amax[(hsel ^ 1) * 128 + row]);
  uint32_t eb;
  const float inv = mx_scale_inv(mx, eb);
  uint32_t q[16];
#pragma unroll
  for (int c = 0; c < 2; ++c) fp8_words(y[c], inv, q + c * 8);
  leave(q, p.glu_q + static_cast<long long>(row0) * p.glu_f + tb * 128 + hsel * 64, p.glu_f);
  if (hsel == 0 && got && row0 + lane < p.rows_a) store_sf(p.glu_sf, row0 + lane, tb, p.glu_sf_rows, (p.glu_f + 511) >> 9, eb);
}

// Host side (gemm_tcgen05.cu)
int num_sms();                                         // of the current device
int make_kmajor_map(CUtensorMap* out, const void* base, int elem_bytes, long long rows, long long k, long long ld, int box_rows);

int make_sf_map(CUtensorMap* out, const void* base, long long blocks);   // scale-factor blocks of 128 words; a box is one block
// gemm_pair.cu: products on CTA pairs. p holds sizes, epilogue and scale factors; rows_a tokens, rows_b weight rows
bool pair_takes(long long tokens, long long rows_b, int k, int dtype, long long ldc, const void* out, const void* residual, bool fuses = false);
int gemm_pair(GemmParams p, const void* x, const void* w, long long ldx, long long ldw, int dtype, cudaStream_t stream, bool quant = false);

}  // namespace b200
