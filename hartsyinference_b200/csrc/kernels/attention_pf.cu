// Causal attention of prompt chunks over the paged K/V cache on the 5th-generation tensor cores: bf16, head
// dim 128, any number of sequences of any length in one launch, keys read in place through the block table.
//
// One CTA owns two tiles of 128 query rows: the same rows of two query heads that share a key head where the
// group has an even number of heads (both tiles then end at the same key), two neighbouring tiles of one
// head otherwise. It walks the keys up to its last row in tiles of 128:
//   warp 0       TMA producer: both Q tiles once, then per key tile one box of [page rows][64 columns] per page
//                and half head, K and V alike, one lane per box. Boxes of pages past the last key start past the
//                end of the pool and arrive as zeros
//   warp 1       one thread issues every tcgen05.mma; TMEM holds S0 | S1 | O0 | O1 as in attention_fa.cu, P is
//                written over S and read from TMEM. V is consumed as it lies in the pages ([key][dim], an
//                MN-major operand), so nothing is transposed or gathered beforehand
//   warp 2       clears the rows of V behind the last key of a page that is not full: their probabilities
//                are zero, but what a page held before may not be finite
//   warps 4..11  softmax of tile 0 and 1: one row per thread, lazy rescale (see attention_fa.cu); tiles that
//                the diagonal or the last key crosses are masked before the maximum
//
// Bound by the softmax warps' chain and the tensor core about equally; CTAs start with the longest rows, so
// that the last wave is made of short ones. 32 heads on 8, 2048 tokens behind 6144: 1585 us with the mma.sync kernel
// -> 257 us (937 TFLOP/s of what the mask leaves); 64 heads on 8, four prompts of 2048: 1821 -> 438 us.
//
// Replaces the per-sequence prefill attention of the reference's scheduler (src/HartsyInference.LLM/Generation/
// DynamicBatchScheduler.cs, AdmitAndPrefill:311-383).
#include "layer_ops.cuh"

namespace b200 {

int num_sms();      // of the current device, see gemm_tcgen05.cu
int make_kmajor_map(CUtensorMap* out, const void* base, int elem_bytes, long long rows, long long k, long long ld, int box_rows);

constexpr int kPfD = 128;
constexpr int kPfTile = 128;
constexpr int kPfThreads = 384;
constexpr int kPfStages = 2;
constexpr int kPfTileBytes = kPfTile * kPfD * 2;
constexpr float kPfRescaleGap = 8.f;      // raise the running maximum only beyond this many powers of two

struct PfBarriers {
  uint64_t q_full;
  uint64_t k_full[kPfStages], k_empty[kPfStages];
  uint64_t v_full[kPfStages], v_empty[kPfStages];
  uint64_t v_last, v_clean;  // the last V tile has landed; its rows behind the last key are cleared
  uint64_t s_full[2], p_ready[2], o_done[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
};

struct PfParams {
  __nv_bfloat16* out;        // [tokens][hq][128]
  const int* block_table;    // [sequences][max_pages]
  const int* kv_lens;        // [sequences]
  const int* cu_q;           // [sequences + 1]
  int hq, hkv, max_pages, page_shift, pair_heads;
  int pool_rows;             // rows of 128 values in the K (or V) pool
  float scale_log2;          // softmax scale * log2(e)
  DeviceStatus* status;
};

__device__ __forceinline__ float pf_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void __launch_bounds__(kPfThreads, 1)
attn_prefill_tc_kernel(const PfParams p, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sq = smem;                                   // two Q tiles, each [half head][128 rows][128 bytes]
  uint8_t* sk = sq + 2 * kPfTileBytes;
  uint8_t* sv = sk + kPfStages * kPfTileBytes;
  PfBarriers* bars = reinterpret_cast<PfBarriers*>(sv + kPfStages * kPfTileBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seq = blockIdx.z, qi = static_cast<int>(gridDim.y) - 1 - static_cast<int>(blockIdx.y);
  const int q_off = p.cu_q[seq], q_len = p.cu_q[seq + 1] - q_off, kv_len = p.kv_lens[seq];
  const int ctx = kv_len - q_len;                       // keys in front of the first query
  const int head0 = p.pair_heads ? 2 * blockIdx.x : blockIdx.x;
  const int row0 = p.pair_heads ? qi * kPfTile : qi * 2 * kPfTile;
  if (row0 >= q_len) return;
  const int row1 = p.pair_heads ? row0 : row0 + kPfTile;          // first row of the second tile
  const bool tile1 = row1 < q_len;
  const int last_row = min(q_len, (tile1 ? row1 : row0) + kPfTile) - 1;
  const int n_keys = min(kv_len, ctx + last_row + 1);
  const int n_tiles = n_keys > 0 ? (n_keys + kPfTile - 1) / kPfTile : 0;
  const int kv_head = head0 / (p.hq / p.hkv);
  // keys of the last tile, and whether a page of it is only partly filled
  const int last_valid = min(kv_len - (n_tiles - 1) * kPfTile, kPfTile);
  const bool clean = n_tiles > 0 && (last_valid & ((1 << p.page_shift) - 1)) != 0;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    mbar_init(&bars->v_last, 1);
    mbar_init(&bars->v_clean, 1);
    for (int i = 0; i < kPfStages; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&bars->s_full[t], 1);
      mbar_init(&bars->p_ready[t], 4);
      mbar_init(&bars->o_done[t], 1);
    }
    bars->abort_flag = 0;
    fence_mbar_init();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  volatile uint32_t* abort_flag = &bars->abort_flag;
  constexpr uint32_t kIdescS = make_idesc(128, 128, kFmtBf16, kFmtBf16);
  constexpr uint32_t kIdescPV = kIdescS | kIdescBMn;

  // launch: 168 registers a thread; the softmax groups take what the first group gives back
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      // ----------------------------------------------------------------------- TMA producer
      const int page = 1 << p.page_shift;
      const int boxes = 2 * kPfTile >> p.page_shift;    // per tile and operand: pages x half heads
      bool ok = true;
      if (lane == 0 && n_tiles > 0) {
        const int nq = tile1 ? 2 : 1;
        mbar_arrive_expect_tx(&bars->q_full, nq * kPfTileBytes);
        for (int t = 0; t < nq; ++t)
          for (int a = 0; a < 2; ++a)
            tma_load_2d(sq + t * kPfTileBytes + a * (kPfTileBytes / 2), &tm_q, &bars->q_full,
                        (head0 + (p.pair_heads ? t : 0)) * kPfD + a * 64, q_off + (t ? row1 : row0));
      }
      const int i = lane >> 1, half = lane & 1;         // this lane's page of the tile and half head
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int s = j % kPfStages;
        const uint32_t ph = static_cast<uint32_t>((j / kPfStages) & 1);
        const int key = j * kPfTile + (i << p.page_shift);
        int row = p.pool_rows;                          // past the pool: zeros
        if (lane < boxes && key < kv_len)
          row = (p.block_table[static_cast<long long>(seq) * p.max_pages + (key >> p.page_shift)] * p.hkv + kv_head) << p.page_shift;
        uint8_t* const at = sk + s * kPfTileBytes + half * (kPfTileBytes / 2) + i * page * 128;
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->k_empty[s], ph ^ 1, abort_flag));
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(&bars->k_full[s], kPfTileBytes);
        __syncwarp();
        if (lane < boxes) tma_load_2d(at, &tm_k, &bars->k_full[s], half * 64, row);
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->v_empty[s], ph ^ 1, abort_flag));
        if (!ok) break;
        if (lane == 0) mbar_arrive_expect_tx(&bars->v_full[s], kPfTileBytes);
        __syncwarp();
        if (lane < boxes) tma_load_2d(at + (sv - sk), &tm_v, &bars->v_full[s], half * 64, row);
      }
      if (!ok && lane == 0) report_status(p.status, kWaitTimeout, kKernelAttnPrefill, 31, blockIdx.x);
    } else if (warp == 1) {
      // ----------------------------------------------------------------------- MMA issuer
      if (lane == 0 && n_tiles > 0) {
        const int nq = tile1 ? 2 : 1;
        bool ok = mbar_wait(&bars->q_full, 0, abort_flag);
        // S_t(j) = Q_t K_j^T into TMEM columns [t * 128, t * 128 + 128)
        auto issue_s = [&](int t, int j) {
          const int s = j % kPfStages;
#pragma unroll
          for (int a = 0; a < 2; ++a) {
            const uint64_t ad = make_desc_sw128(smem_u32(sq + t * kPfTileBytes + a * (kPfTileBytes / 2)));
            const uint64_t bd = make_desc_sw128(smem_u32(sk + s * kPfTileBytes + a * (kPfTileBytes / 2)));
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_bf16_ss(tmem_base + t * 128, ad + 2 * k, bd + 2 * k, kIdescS, (a | k) != 0);
          }
          tc_commit(&bars->s_full[t]);
        };
        if (ok) ok = mbar_wait(&bars->k_full[0], 0, abort_flag);
        if (ok) {
          tc_fence_after_sync();
          for (int t = 0; t < nq; ++t) issue_s(t, 0);
          tc_commit(&bars->k_empty[0]);
        }
        for (int j = 0; j < n_tiles && ok; ++j) {
          const int s = j % kPfStages;
          const uint32_t ph = static_cast<uint32_t>((j / kPfStages) & 1);
          for (int t = 0; t < nq && ok; ++t) {
            if (!mbar_wait(&bars->p_ready[t], j & 1, abort_flag)) { ok = false; break; }
            if (t == 0 && !mbar_wait(&bars->v_full[s], ph, abort_flag)) { ok = false; break; }
            if (t == 0 && clean && j == n_tiles - 1) {
              mbar_arrive(&bars->v_last);
              if (!mbar_wait(&bars->v_clean, 0, abort_flag)) { ok = false; break; }
            }
            tc_fence_after_sync();
            // O_t += P_t V_j: A = P_t in TMEM (16 keys are 8 columns of bf16 pairs), B = 16 rows of the V tile
            const uint64_t bd = make_desc_sw128_mn(smem_u32(sv + s * kPfTileBytes), kPfTileBytes / 2);
#pragma unroll
            for (int k = 0; k < 8; ++k)
              mma_bf16_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + k * 8, bd + k * (2048 >> 4), kIdescPV, (j | k) != 0);
            tc_commit(&bars->o_done[t]);
            if (t == nq - 1) tc_commit(&bars->v_empty[s]);
            if (j + 1 < n_tiles) {
              const int s1 = (j + 1) % kPfStages;
              if (t == 0 && !mbar_wait(&bars->k_full[s1], static_cast<uint32_t>(((j + 1) / kPfStages) & 1), abort_flag)) {
                ok = false;
                break;
              }
              tc_fence_after_sync();
              issue_s(t, j + 1);     // executes after the P_t V_j above: it overwrites the columns P_t lives in
              if (t == nq - 1) tc_commit(&bars->k_empty[s1]);
            }
          }
        }
        if (!ok) report_status(p.status, kWaitTimeout, kKernelAttnPrefill, 32, blockIdx.x);
      }
    } else if (warp == 2 && clean) {
      // ----------------------------------------------------------------------- rows of V behind the last key
      // (told by the MMA thread: a waiter that has not seen every phase of v_full cannot tell which one it is in)
      const int s = (n_tiles - 1) % kPfStages;
      if (__all_sync(0xffffffffu, mbar_wait(&bars->v_last, 0, abort_flag))) {
        // whole 128-byte rows, so the swizzle inside a row does not matter
        for (int i = last_valid * 8 + lane; i < kPfTile * 8; i += 32)
          for (int a = 0; a < 2; ++a)
            *reinterpret_cast<uint4*>(sv + s * kPfTileBytes + a * (kPfTileBytes / 2) + i * 16) = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->v_clean);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // ------------------------------------------------------------------------- softmax warps
    const int t = (warp >> 2) - 1;                        // query tile of this warp group
    const int quarter = warp & 3;                         // TMEM lane quarter this warp may touch
    const int row = quarter * 32 + lane;                  // query row inside the tile = TMEM lane
    const int q_first = (t ? row1 : row0) + quarter * 32; // first query row of this warp
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t s_col = lane_base + t * 128, o_col = lane_base + 256 + t * 128;
    if (t == 0 || tile1) {
      const int lim = min(kv_len, ctx + q_first + lane + 1);            // keys this row sees
      const int lim_first = min(kv_len, ctx + q_first + 1);             // fewest keys of a row of this warp
      float m_run = -INFINITY, l_run = 0.f;
      const float c = p.scale_log2;
      bool ok = true;
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->s_full[t], j & 1, abort_flag))) { ok = false; break; }
        tc_fence_after_sync();
        uint32_t r[128];
        float mf[8];
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) tmem_ld_32x32(s_col + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[cc * 32]));
        tmem_ld_wait();
#pragma unroll
        for (int cc = 2; cc < 4; ++cc) tmem_ld_32x32(s_col + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[cc * 32]));
        if (lim_first >= (j + 1) * kPfTile) {
          // every row of the warp sees the whole tile; the second half is in flight while the maximum of
          // the first is taken
#pragma unroll
          for (int u = 0; u < 8; ++u) mf[u] = __uint_as_float(r[u]);
#pragma unroll
          for (int i = 8; i < 64; ++i) mf[i & 7] = fmaxf(mf[i & 7], __uint_as_float(r[i]));
          tmem_ld_wait();
        } else {
          tmem_ld_wait();
          const int valid = lim - j * kPfTile;
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i >= valid) r[i] = 0xff800000u;
#pragma unroll
          for (int u = 0; u < 8; ++u) mf[u] = __uint_as_float(r[u]);
#pragma unroll
          for (int i = 8; i < 64; ++i) mf[i & 7] = fmaxf(mf[i & 7], __uint_as_float(r[i]));
        }
#pragma unroll
        for (int i = 64; i < 128; ++i) mf[i & 7] = fmaxf(mf[i & 7], __uint_as_float(r[i]));
        const float mx = fmaxf(fmaxf(fmaxf(mf[0], mf[1]), fmaxf(mf[2], mf[3])), fmaxf(fmaxf(mf[4], mf[5]), fmaxf(mf[6], mf[7]))) * c;
        // raise the running maximum only when it would grow by more than the gap (or on the first tile);
        // a warp decides together because the O rescale below is a warp-wide TMEM access
        if (__any_sync(0xffffffffu, mx > m_run + kPfRescaleGap)) {
          const float m_new = fmaxf(m_run, mx);
          const float alpha = m_run == -INFINITY ? 0.f : pf_exp2(m_run - m_new);
          if (j > 0) {
            if (!__all_sync(0xffffffffu, mbar_wait(&bars->o_done[t], (j - 1) & 1, abort_flag))) { ok = false; break; }
            tc_fence_after_sync();
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
              uint32_t o[32];
              tmem_ld_32x32(o_col + cc * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32(o_col + cc * 32, o);
            }
            tmem_st_wait();
          }
          l_run *= alpha;
          m_run = m_new;
        }
        const float sub = m_run == -INFINITY ? 0.f : m_run;
        float sums[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t packed[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float a = pf_exp2(fmaf(__uint_as_float(r[cc * 64 + 2 * i]), c, -sub));
            const float b = pf_exp2(fmaf(__uint_as_float(r[cc * 64 + 2 * i + 1]), c, -sub));
            sums[i & 3] += a + b;
            packed[i] = pack_bf16x2(a, b);
          }
          tmem_st_32x32(s_col + cc * 32, packed);        // P_t: columns [0, 64) of S_t
        }
        tmem_st_wait();
        l_run += (sums[0] + sums[1]) + (sums[2] + sums[3]);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_ready[t]);
      }
      if (ok && n_tiles > 0) ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_done[t], (n_tiles - 1) & 1, abort_flag));
      if (!ok) {
        if (lane == 0) report_status(p.status, kWaitTimeout, kKernelAttnPrefill, 33, blockIdx.x);
      } else {
        tc_fence_after_sync();
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
        // The Q tile is no longer read: 32 rows of 128 bytes per warp turn the rows that the lanes hold into
        // 128-byte runs. 16-byte pieces are placed by (piece xor row), which keeps the banks apart.
        uint8_t* strip = sq + t * kPfTileBytes + quarter * 32 * 128;
        const int head = head0 + (p.pair_heads ? t : 0);
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
          uint32_t o[64];
          tmem_ld_32x32(o_col + hc * 64, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));
          tmem_ld_32x32(o_col + hc * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint32_t w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              w[u] = n_tiles > 0 ? pack_bf16x2(__uint_as_float(o[i * 8 + 2 * u]) * inv, __uint_as_float(o[i * 8 + 2 * u + 1]) * inv) : 0u;
            *reinterpret_cast<uint4*>(strip + lane * 128 + ((i ^ (lane & 7)) * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = i * 4 + (lane >> 3), piece = lane & 7;
            const uint4 v = *reinterpret_cast<const uint4*>(strip + rr * 128 + ((piece ^ (rr & 7)) * 16));
            if (q_first + rr < q_len)
              *reinterpret_cast<uint4*>(p.out + (static_cast<long long>(q_off + q_first + rr) * p.hq + head) * kPfD + hc * 64 + piece * 8) = v;
          }
          __syncwarp();
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200

using namespace b200;

// q, out [total_q][hq][128] bf16; k_pool, v_pool [pages][hkv][page][128] bf16; block_table [seqs][max_pages], kv_lens [seqs]
// and cu_q [seqs + 1] int32 on the device. Causal, scale > 0; page of 8, 16, 32 or 64 rows; max_kv_len: no sequence has
// more keys. Returns -2 .. -6 for what it does not take, 1 (nothing launched) where b200_attn_prefill is faster.
B200_API int b200_attn_prefill_tc(const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table,
                                  const int* kv_lens, const int* cu_q, int seqs, int total_q, int max_q_len, int hq, int hkv,
                                  int page, int max_pages, long long pages, int max_kv_len, float scale, void* status, cudaStream_t stream) {
  if (seqs <= 0 || max_q_len <= 0 || total_q <= 0) return 0;
  if (hkv <= 0 || hq % hkv != 0) return -3;
  PfParams p{};
  p.page_shift = page == 8 ? 3 : page == 16 ? 4 : page == 32 ? 5 : page == 64 ? 6 : -1;
  if (p.page_shift < 0) return -4;
  if (!(scale > 0.f) || seqs > 65535) return -5;
  const long long rows = pages * hkv * page;
  if (rows <= 0 || rows >= (1ll << 31)) return -6;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.block_table = block_table; p.kv_lens = kv_lens; p.cu_q = cu_q;
  p.hq = hq; p.hkv = hkv; p.max_pages = max_pages;
  p.pair_heads = (hq / hkv) % 2 == 0 ? 1 : 0;
  p.pool_rows = static_cast<int>(rows);
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = static_cast<DeviceStatus*>(status);
  const int rows_each = p.pair_heads ? kPfTile : 2 * kPfTile;
  const int q_tiles = (max_q_len + rows_each - 1) / rows_each;
  if (q_tiles > 65535) return -5;
  // A block fills a processor and starts up for 7.5 us before its keys (0.015 us each) count; b200_attn_prefill has several small
  // blocks of 64 rows and one head on a processor, 1.6 us each and 0.028 us a key, and takes at least 4.7 us and 0.045 us a
  // key. So it stays faster for short prompts (32 heads on 8, this / that: 17 tokens 11.4 / 6.6 us, 64 10.8 / 7.3, 100 of 5 behind
  // 10 98 / 53; 8 heads 64 of 64 behind 64 31 / 23) and slower from about 150 keys on (9 behind 400 17 / 24).
  const double sms = num_sms(), keys = max_kv_len;
  const double here = 2.5 + ((static_cast<long long>(p.pair_heads ? hq / 2 : hq) * q_tiles * seqs + num_sms() - 1) / num_sms()) * (7.5 + 0.015 * keys);
  const double rows_us = (static_cast<double>((max_q_len + 63) / 64) * hq * seqs / sms) * (1.6 + 0.028 * keys);
  if (fmax(4.7 + 0.045 * keys, rows_us) < here) return 1;
  CUtensorMap tq, tk, tv;
  int rc = make_kmajor_map(&tq, q, 2, total_q, static_cast<long long>(hq) * kPfD, static_cast<long long>(hq) * kPfD, kPfTile);
  if (rc == 0) rc = make_kmajor_map(&tk, k_pool, 2, rows, kPfD, kPfD, page);
  if (rc == 0) rc = make_kmajor_map(&tv, v_pool, 2, rows, kPfD, kPfD, page);
  if (rc) return rc;
  const int smem = (2 + 2 * kPfStages) * kPfTileBytes + static_cast<int>(sizeof(PfBarriers)) + 1024;
  static PerDeviceOnce configured;
  if (configured.first_time() &&
      cudaFuncSetAttribute(attn_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return -200;
  attn_prefill_tc_kernel<<<dim3(p.pair_heads ? hq / 2 : hq, q_tiles, seqs), kPfThreads, smem, stream>>>(p, tq, tk, tv);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -static_cast<int>(e) - 300;
}
