// Dense product of many tokens on CTA pairs (tcgen05 cta_group::2): C = A * B^T, tiles of 256 tokens x 256 features.
//
// Replaces the same calls of the reference as gemm_tcgen05.cu (src/HartsyInference.Cuda/CudaBackend.cs:1769-2425), for
// sizes that give most of the processors a tile.
//
// Why pairs: a 128 x 256 tile of one SM takes 48 KB of operands from L2 for every 512 cycles of its tensor core
// (96 bytes a cycle, more than an SM gets), so it ran at 0.6 of the core's rate in 8 and in 16 bits. Two SMs on one tile each
// keep 128 rows of A and 128 rows of B, and the tensor cores read the other half of B from the neighbour's shared
// memory: 32 KB for the same cycles, a third less.
//
// Structure of one CTA (320 threads; persistent, pair i takes tiles i, i + pairs, ...):
//   warp 0      one thread issues TMA loads of this CTA's 128 rows of either operand into its own shared memory; their
//               bytes are counted on the barrier of the pair's first CTA
//   warp 1      allocates TMEM; in the first CTA one thread issues tcgen05.mma (M = 256, N = 256) for both and
//               commits to the barriers of both
//   warps 2..9  epilogue of this CTA's 128 rows x 256 columns
// Bound by the tensor core and the power limit: fp8 4096 x 9216 x 3072 116 -> 92 us (one-SM tiles before), 8192 x 8192 x
// 28672 1691 -> 1317 us (2.9 PFLOP/s, then held by power), bf16 2048 x 28672 x 4096 gated 364 -> 300 us (1.6 PFLOP/s).
// Two accumulators: the epilogue of a tile runs beside the products of the next. With scale factors in TMEM (8 bits)
// 480 columns are left, so the two overlap by 32 columns, which the epilogue takes out first.
#include "gemm_common.cuh"

namespace b200 {

constexpr int kPairStages = 6;
constexpr int kPairBand = 8;                           // tiles of 256 tokens in a band: 74 tiles in flight cover 8 x 9 of them

__device__ __forceinline__ uint32_t map_to_rank(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
// Loads into this CTA's shared memory; the bytes are counted on `bar`, a shared::cluster address in either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t bar, int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
// Arrival at a barrier of either CTA. What it announces are reads of TMEM, which tcgen05.wait::ld has seen done; a release at
// cluster scope also waits for the thread's stores to global memory (1200 cycles behind the epilogue's).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void pair_commit(uint64_t* bar, uint16_t ctas) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(ctas)
               : "memory");
}
__device__ __forceinline__ void pair_cp_sf(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// The issuing thread bounded the 8-bit products in a first form, with waits that acquire at cluster scope and descriptors counted on
// in 64 bits: 690 cycles a K block of four 128-cycle instructions. With waits at CTA scope, the next stage asked for ahead of
// this one's instructions and the descriptors' upper halves as constants (only the lower ones change, see make_desc_sw128): 511.
#define B200_PAIR_DESCS                          \
  "{\n\t"                                        \
  ".reg .pred p;\n\t"                            \
  ".reg .b64 da, db;\n\t"                        \
  "mov.b64 da, {%1, 0x40004040};\n\t"            \
  "mov.b64 db, {%2, 0x40004040};\n\t"            \
  "setp.ne.b32 p, %4, 0;\n\t"
__device__ __forceinline__ void pair_mma_bf16(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(B200_PAIR_DESCS "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}" ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(acc)
               : "memory");
}
__device__ __forceinline__ void pair_mma_mx(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc, uint32_t sfa, uint32_t sfb) {
  asm volatile(B200_PAIR_DESCS "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], da, db, %3, [%5], [%6], p;\n\t}" ::"r"(d), "r"(a),
               "r"(b), "r"(idesc), "r"(acc), "r"(sfa), "r"(sfb)
               : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Epilogue of 32 columns from b0 on (all of them there) of one row: bias, activation, gate and residual, rounded to bf16 pairs.
__device__ __forceinline__ void finish_row32(const GemmParams& p, const uint32_t (&r)[32], int row, int b0, uint32_t (&out)[16]) {
  uint32_t res[16];
  const bool inside = row < p.rows_a;
  if (p.residual && inside) {
    const __nv_bfloat16* src = p.residual + static_cast<long long>(row) * p.ldc + b0;
    load_words8(res, src);
    load_words8(res + 8, src + 16);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float v[8], t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[q * 8 + j]);
    if (p.bias) {
      load_cols8(p.bias + b0 + q * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += t[j];
    }
    if (b0 + q * 8 < p.act_col) {
      // features ahead of the activation's first (a multiple of 8)
    } else if (p.act == 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = gelu_tanh(v[j]);
    } else if (p.act == 2) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = silu(v[j]);
    } else if (p.act == 3) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = relu2(v[j]);
    } else if (p.act == 4) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = tanhf(v[j]);
    }
    if (p.gate) {
      load_cols8(p.gate + b0 + q * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= t[j];
    }
    if (p.residual && inside) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[2 * j] += __uint_as_float(res[q * 4 + j] << 16);
        v[2 * j + 1] += __uint_as_float(res[q * 4 + j] & 0xffff0000u);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) out[q * 4 + j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
  }
}

struct alignas(16) PairBarriers {
  uint64_t full[kPairStages], empty[kPairStages];        // full: counted in the first CTA of the pair; empty: in each
  uint64_t tmem_full[2];             // in each
  uint64_t tmem_empty[2], shared_empty[2];   // in the first: accumulator read; its columns that the other one shares read
  uint64_t drain;
  uint32_t tmem_base, abort_flag;
  float amax[2][256];                // gated tiles: maxima of a row's two halves
};

template <int kMode>
constexpr int pair_stage_bytes() { return 2 * kStageBytesA + (kMode == 2 ? 2048 : 0); }

// kQuant: see GemmParams::q_from. A warp's 128 columns are one group of a row's scales.
template <int kMode, bool kGlu, bool kQuant = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const GemmParams p, const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_sfa, const __grid_constant__ CUtensorMap tm_sfb) {
  constexpr bool kMx = kMode == 2;
  constexpr int kStages = kPairStages, kStageBytes = pair_stage_bytes<kMode>();
  constexpr int kElems = kMx ? 128 : 64;               // K elements in one 128-byte swizzle atom
  constexpr int kAccStride = kMx ? 224 : 256;          // first column of the second accumulator
  constexpr uint32_t kSfCol = 480;
  constexpr uint32_t kIdesc = kMx ? make_idesc_mx(256, 256) : make_idesc(256, 256, kFmtBf16, kFmtBf16);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  PairBarriers* bars = reinterpret_cast<PairBarriers*>(smem + kStages * kStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int tiles_a = (p.rows_a + 255) / 256, kblocks = (p.k + kElems - 1) / kElems;
  const int first = static_cast<int>(blockIdx.x >> 1), step = static_cast<int>(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->tmem_full[b], 1);
      mbar_init(&bars->tmem_empty[b], 16);             // one arrival per epilogue warp of the pair
      mbar_init(&bars->shared_empty[b], 8);            // per warp that holds a shared chunk
    }
    mbar_init(&bars->drain, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
    prefetch_tensormap(&tm_a);
    prefetch_tensormap(&tm_b);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                  // the barriers of both CTAs are set up
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  volatile uint32_t* abort_flag = &bars->abort_flag;
  pdl_trigger();

  auto tile_of = [&](int w, int& ta, int& tb) {        // as in decode_item of gemm_tcgen05.cu
    const int per = kPairBand * (p.num_tiles / tiles_a), b = w / per, r = w - b * per;
    const int width = min(kPairBand, tiles_a - b * kPairBand);
    tb = r / width;
    ta = b * kPairBand + (r - tb * width);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      pdl_wait();
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      long long issued = 0;
      for (int w = first; w < p.num_tiles && ok; w += step) {
        int ta, tb;
        tile_of(w, ta, tb);
        const int a_row = ta * 256 + static_cast<int>(rank) * 128;
        const int b_row = kGlu ? tb * 128 + static_cast<int>(rank) * p.glu_f : tb * 256 + static_cast<int>(rank) * 128;
        const int sfa = (2 * ta + static_cast<int>(rank)) * p.sf_kgroups;
        const int sfb0 = (kGlu ? tb : 2 * tb) * p.sf_kgroups, sfb1 = (kGlu ? tb + (p.glu_f >> 7) : 2 * tb + 1) * p.sf_kgroups;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&bars->empty[s], ph ^ 1, abort_flag)) {
            report_status(p.status, kWaitTimeout, kKernelGemm, 21, blockIdx.x);
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * kStageBytes;
          const uint32_t bar = map_to_rank(&bars->full[s], 0);
          const bool with_sf = kMx && (kb & 3) == 0;   // a stage that starts a group of four K blocks carries their scale factors
          if (rank == 0) mbar_arrive_expect_tx(&bars->full[s], 2 * (2 * kStageBytesA + (with_sf ? 1536 : 0)));
          if (with_sf) {
            uint8_t* sf = sa + 2 * kStageBytesA;
            tma_load_2d_pair(sf, &tm_sfa, bar, 0, sfa + (kb >> 2));
            tma_load_2d_pair(sf + 512, &tm_sfb, bar, 0, sfb0 + (kb >> 2));
            tma_load_2d_pair(sf + 1024, &tm_sfb, bar, 0, sfb1 + (kb >> 2));
          }
          tma_load_2d_pair(sa, &tm_a, bar, kb * kElems, a_row);
          tma_load_2d_pair(sa + kStageBytesA, &tm_b, bar, kb * kElems, b_row);
          ++issued;
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
      if (!ok && rank == 0) {
        // let the copies in flight land before the CTAs leave
        for (int i = 0; i < kStages && i < issued; ++i) {
          int ss = s - 1 - i;
          uint32_t pp = ph;
          if (ss < 0) { ss += kStages; pp ^= 1; }
          uint32_t dummy = 0;
          mbar_wait(&bars->full[ss], pp, &dummy, 4000000ll);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0 && rank == 0) {
      pdl_wait();
      const uint32_t smem_base = smem_u32(smem);
      int s = 0, t = 0;
      uint32_t ph = 0;
      bool ok = true, issued_any = false;
      for (int w = first; w < p.num_tiles && ok; w += step, ++t) {
        const int b = t & 1;
        if (!mbar_wait(&bars->tmem_empty[b], ((t >> 1) & 1) ^ 1, abort_flag) ||
            (kMx && t > 0 && !mbar_wait(&bars->shared_empty[b ^ 1], ((t - 1) >> 1) & 1, abort_flag))) {
          report_status(p.status, kWaitTimeout, kKernelGemm, 22, blockIdx.x);
          ok = false;
          break;
        }
        const uint32_t d = tmem_base + b * kAccStride;
        bool ready = mbar_test(&bars->full[s], ph);
        for (int kg = 0; kg < kblocks && ok; kg += 4) {
          const uint32_t slot = tmem_base + kSfCol + ((kg >> 2) & 1) * 16;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (kg + j >= kblocks || !ok) break;
            if (!ready && !mbar_wait(&bars->full[s], ph, abort_flag)) {
              report_status(p.status, kWaitTimeout, kKernelGemm, 23, blockIdx.x);
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint32_t sa = smem_base + s * kStageBytes, lo = (sa >> 4) | 1u << 16;
            if (kMx && j == 0) {
              pair_cp_sf(slot, make_desc_sf(sa + 2 * kStageBytesA));
              pair_cp_sf(slot + 4, make_desc_sf(sa + 2 * kStageBytesA + 512));
              pair_cp_sf(slot + 8, make_desc_sf(sa + 2 * kStageBytesA + 1024));
            }
            uint64_t* const done = &bars->empty[s];
            if (++s == kStages) { s = 0; ph ^= 1; }
            ready = mbar_test(&bars->full[s], ph);     // asked here, needed behind the four instructions
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t acc = j > 0 || k > 0 || kg > 0;
              if (kMx)
                pair_mma_mx(d, lo + 2 * k, lo + (kStageBytesA >> 4) + 2 * k, kIdesc | (j << 29) | (j << 4), acc, slot, slot + 4);
              else
                pair_mma_bf16(d, lo + 2 * k, lo + (kStageBytesA >> 4) + 2 * k, kIdesc, acc);
            }
            issued_any = true;
            pair_commit(done, 3);
          }
        }
        if (ok) pair_commit(&bars->tmem_full[b], 3);
      }
      if (!ok && issued_any) {
        pair_commit(&bars->drain, 1);
        uint32_t dummy = 0;
        mbar_wait(&bars->drain, 0, &dummy, 4000000ll);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps 2..9
    pdl_wait();
    const int q = warp & 3, hsel = (warp - 2) >> 2;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    bool ok = true;
    int t = 0;
    for (int w = first; w < p.num_tiles; w += step, ++t) {
      int ta, tb;
      tile_of(w, ta, tb);
      const int b = t & 1, row0 = ta * 256 + static_cast<int>(rank) * 128 + q * 32;
      // the accumulator's chunk of 32 columns that it shares with the other one: 7 of the first, 0 of the second
      const bool holds_shared = kMx && hsel == (b ^ 1);
      const uint32_t acc = lane_base + b * kAccStride;
      if (ok && !__all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[b], (t >> 1) & 1, abort_flag))) {
        if (lane == 0) report_status(p.status, kWaitTimeout, kKernelGemm, 24, blockIdx.x);
        ok = false;
      }
      const int row = row0 + lane;
      auto taken = [&](bool shared) {                  // the columns loaded so far are in registers
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_rank(shared ? &bars->shared_empty[b] : &bars->tmem_empty[b], 0));
      };
      if constexpr (kGlu) {
        // 64 features in two runs of 32, gate and up, the run with the shared chunk first
        uint32_t y[2][16];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = hsel * 64 + (u ^ b ^ 1) * 32;
          if (ok) {
            uint32_t g[32], up[32];
            if (u == 0) tc_fence_after_sync();
            tmem_ld_32x32(acc + c, g);
            tmem_ld_32x32(acc + 128 + c, up);
            tmem_ld_wait();
            if (u == 0 && holds_shared) taken(true);
            if (u == 1) taken(false);
            glu_words(p, g, up, y[u]);
            if (!kMx && row < p.rows_a) {
              __nv_bfloat16* dst = p.out + static_cast<long long>(row) * p.ldc + tb * 128 + c;
              store_words8(dst, y[u]);
              store_words8(dst + 16, y[u] + 8);
            }
          }
        }
        if constexpr (kMx) {
          // the scale of a row's 128 features needs both halves, which sit in two warps: they exchange maxima behind a barrier of
          // their own, which a warp whose accumulator did not come still meets
          float mx = words_max(y[1], words_max(y[0], 0.f));
          bars->amax[b][hsel * 128 + q * 32 + lane] = mx;
          asm volatile("bar.sync %0, 64;" ::"r"(2 + q) : "memory");
          mx = fmaxf(mx, bars->amax[b][(hsel ^ 1) * 128 + q * 32 + lane]);
          uint32_t eb;
          const float inv = mx_scale_inv(mx, eb);
          if (ok && row < p.rows_a) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              uint32_t w[8];
              fp8_words(y[u], inv, w);
              store_words8(p.glu_q + static_cast<long long>(row) * p.glu_f + tb * 128 + hsel * 64 + (u ^ b ^ 1) * 32, w);
            }
            if (hsel == 0) store_sf(p.glu_sf, row, tb, p.glu_sf_rows, (p.glu_f + 511) >> 9, eb);
          }
        }
      } else if (ok) {
        tc_fence_after_sync();
        const int turn = holds_shared && b == 0 ? 3 : 0;
        if constexpr (kQuant) {
          const int group = tb * 256 + hsel * 128;
          if (group >= p.q_from) {
            uint32_t y[4][16];
            float mx = 0.f;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int c = hsel * 4 + ((u + turn) & 3);
              uint32_t r[32];
              tmem_ld_32x32(acc + c * 32, r);
              tmem_ld_wait();
              if (u == 0 && holds_shared) taken(true);
              if (u == 3) taken(false);
              if (group < p.rows_b) finish_row32(p, r, row, tb * 256 + c * 32, y[u]);
              if (group < p.rows_b) mx = words_max(y[u], mx);
            }
            if (group < p.rows_b && row < p.rows_a) {
              uint32_t eb;
              const float inv = mx_scale_inv(mx, eb);
              uint8_t* dst = p.glu_q + static_cast<long long>(row) * p.q_ld + p.q_col0 + (group - p.q_from);
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                uint32_t w[8];
                fp8_words(y[u], inv, w);
                store_words8(dst + ((u + turn) & 3) * 32, w);
              }
              store_sf(p.glu_sf, row, (p.q_col0 + group - p.q_from) >> 7, 128, p.q_kgroups, eb);
            }
            continue;
          }
        }
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {
          const int c = hsel * 4 + ((u + turn) & 3), b0 = tb * 256 + c * 32;
          uint32_t r[32];
          tmem_ld_32x32(acc + c * 32, r);
          tmem_ld_wait();
          if (u == 0 && holds_shared) taken(true);
          if (u == 3) taken(false);
          if (b0 + 32 <= p.rows_b) {
            uint32_t y[16];
            finish_row32(p, r, row, b0, y);
            if (row < p.rows_a) {
              __nv_bfloat16* dst = p.out + static_cast<long long>(row) * p.ldc + b0;
              store_words8(dst, y);
              store_words8(dst + 16, y + 8);
            }
          } else {
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            store_chunk<false>(p, v, row, b0, p.rows_b);
          }
        }
      }
    }
  }

  __syncwarp();                                        // the single-lane roles rejoin their warps
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                                  // no signal from the other CTA is on its way any more
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// ------------------------------------------------------------------------------------------ host side
template <int kMode, bool kGlu, bool kQuant = false>
static int launch_pair(const GemmParams& p, const CUtensorMap (&maps)[4], cudaStream_t stream) {
  const int smem = kPairStages * pair_stage_bytes<kMode>() + static_cast<int>(sizeof(PairBarriers)) + 1024;
  static PerDeviceOnce configured;
  if (configured.first_time()) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<kMode, kGlu, kQuant>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return -static_cast<int>(e) - 200;
  }
  const int pairs = num_sms() / 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * (p.num_tiles < pairs ? p.num_tiles : pairs));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = g_b200_pdl ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, gemm_pair_kernel<kMode, kGlu, kQuant>, p, maps[0], maps[1], maps[2], maps[3]) != cudaSuccess) return -300;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -static_cast<int>(e) - 300;
}

// Whether a product of `tokens` rows by `rows_b` weight rows runs here and not on the tiles of one SM (gemm_tcgen05.cu). Both sides
// measured over 1200 sizes of either type around the line (bf16 256 x 9216 x 3072 47.4 -> 23.7 us, 2600 x 28672 x 4096 gated 535 -> 417,
// fp8 600 x 4096 x 3072 56.5 -> 17.0, 8192 x 8192 x 8192 480 -> 377, 4096 x 9216 x 3072 116 -> 92):
//  - a wave of pair tiles takes 0.8 of the time of a wave of 128 x 256 tiles in bf16 and 0.6 to 0.7 in 8 bits, so tokens that leave
//    the last 256 rows half empty stay there where that costs more waves (bf16 five waves against four: 640 x 28672 x 1024 39.8 us there
//    and 36.0 here, k 4096 118 both, k 8192 230 and 237, 2600 x 7168 x 14336 382 and 403; fp8 300 x 12288 x 1024 14.4 and 15.3)
//  - few tiles of a long row are cut along K there: bf16 16 to 19 tiles k 3072 24.3 there and 21.8 here, k 4096 24.5 and 26.9, and where six
//    ranges of a tile fit (300 x 2048) 21.1 and 21.7, 22.1 and 26.2; in three ranges (300 x 4096) k 6144 38.1 and 37.5, k 8192 44.1 and 46.8,
//    k 14336 58 and 75; in two (512 x 4096) k 14336 76.6 and 75.7, k 18432 90.5 and 94.1. fp8 16 to 19 tiles k 8192 30.9 and 26.7,
//    k 12288 34.3 and 37.2, in six ranges k 6144 22.1 and 22.2, k 8192 24.8 and 26.7; ones of a short row are as fast there
//    (300 x 6144 x 1024 10.4 and 10.7, k 256 8.0 and 8.6)
// fuses: the epilogue here does the work of a kernel that would follow a product there, and the line lies further out (gated 300 x 1024
// of k 4096 24.7 there, 25.8 here; never slower over 264 sizes of either type otherwise).
// Rows of the output (and residual) start on 32-byte boundaries: the epilogue's accesses.
bool pair_takes(long long tokens, long long rows_b, int k, int dtype, long long ldc, const void* out, const void* residual, bool fuses) {
  if (tokens <= 128 || (dtype != 0 && dtype != 2)) return false;
  if (ldc % 16 != 0 || ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual)) & 31)) return false;
  const long long sms = num_sms(), cols = (rows_b + 255) / 256;
  const long long tiles = (tokens + 255) / 256 * cols, waves = (tiles + sms / 2 - 1) / (sms / 2);
  const long long one = (tokens + 127) / 128 * cols, waves_one = (one + sms - 1) / sms;      // 128 x 256 tiles
  if (tiles < 16 || tiles >= 1ll << 30) return false;
  if (dtype == 0) {
    if (4 * waves > 5 * waves_one || (tiles < 32 && k > 4096)) return false;
    if (fuses) return tiles >= 20 || k <= 3072 || 6 * one > sms;
    return (4 * waves < 5 * waves_one || k <= 4096) && (tiles >= 20 || k <= (6 * one <= sms ? 2048 : 3072)) &&
           (3 * one > sms || k <= 6144) && (2 * one > sms || k <= 14336);
  }
  if ((3 * waves > 5 * waves_one && k < 3072) || (k < 2048 && tiles <= 36) || (tiles < 32 && k > 12288)) return false;
  return fuses || ((k >= 2048 || 2 * one > sms) && (tiles >= 20 || k <= (6 * one <= sms ? 6144 : 8192)));
}

int gemm_pair(GemmParams p, const void* x, const void* w, long long ldx, long long ldw, int dtype, cudaStream_t stream, bool quant) {
  const bool mx = dtype == 2, gated = p.glu_f > 0;
  const int esz = mx ? 1 : 2;
  p.num_tiles = (p.rows_a + 255) / 256 * (gated ? p.glu_f / 128 : (p.rows_b + 255) / 256);
  CUtensorMap maps[4];
  int rc = make_kmajor_map(&maps[0], x, esz, p.rows_a, p.k, ldx, 128);
  if (rc == 0) rc = make_kmajor_map(&maps[1], w, esz, p.rows_b, p.k, ldw, 128);
  maps[2] = maps[3] = maps[0];
  if (rc == 0 && mx) rc = make_sf_map(&maps[2], p.sf_a, (p.rows_a + 127ll) / 128 * p.sf_kgroups);
  if (rc == 0 && mx) rc = make_sf_map(&maps[3], p.sf_b, (p.rows_b + 127ll) / 128 * p.sf_kgroups);
  if (rc) return rc;
  if (quant) return launch_pair<2, false, true>(p, maps, stream);
  if (mx) return gated ? launch_pair<2, true>(p, maps, stream) : launch_pair<2, false>(p, maps, stream);
  return gated ? launch_pair<0, true>(p, maps, stream) : launch_pair<0, false>(p, maps, stream);
}

}  // namespace b200

using namespace b200;

// Whether b200_gemm runs m tokens by n features of depth k on CTA pairs (operands and output dense).
B200_API int b200_gemm_on_pairs(int m, int n, int k, int dtype) { return pair_takes(m, n, k, dtype, n, nullptr, nullptr) ? 1 : 0; }

// Whether b200_gemm_quant takes m tokens by n features of depth k.
B200_API int b200_gemm_quant_fits(int m, int n, int k) {
  return m > 128 && n >= 128 && n % 128 == 0 && k >= 16 && k % 16 == 0 && pair_takes(m, n, k, 2, n, nullptr, nullptr, true) ? 1 : 0;
}

// Whether b200_gemm_quant is faster than b200_gemm and the quantisation of its output. The epilogue that quantises takes 3 to 6 us longer at
// the end of the last wave, the other kernel 3 us and what it reads and writes: measured over 67 sizes (the two / this, us) 512 x 12288 of k 3072
// 35.5 / 36.3, 256 x 13824 of k 5120 30 / 43, 1024 x 13824 69.6 / 72.0, 1024 x 12288 52.0 / 50.9, 1651 x 3072 of k 768 27.1 / 29.0, 1651 x 6144 of
// k 1536 42.7 / 41.7, 2560 x 3072 30.5 / 29.5, 4608 x 12288 186 / 157, 14040 x 13824 917 / 781.
B200_API int b200_gemm_quant_pays(int m, int n) { return m >= 1536 && static_cast<long long>(m) * n >= 7500000 ? 1 : 0; }

// act(x w^T + bias) of e4m3 operands with UE8M0 scales for a next product that reads e4m3: features from q_from on (a multiple of 128)
// leave as e4m3 with 1x128 scales (rounded to bf16 first, as a quantisation of the stored product would find them) in columns from q_col0
// on of out_q, rows q_ld bytes apart; scales in the blocked layout of q_kgroups words a row. The features in front leave as bf16 in
// out [m][ldc]. What the quantisation kernel read and wrote stays away from memory: 4096 x 12288 of k 3072 with GELU 133 + 36 us -> 144,
// 12288 features of 4608 x 21504 250 + 42 -> 259, 14040 x 13824 of k 5120 732 + 189 -> 827. act as in b200_gemm. -12: sizes or boundaries that it does not take.
B200_API int b200_gemm_quant(const void* x, const void* w, void* out, void* out_q, void* out_sf, int m, int n, int k, long long ldx, long long ldw,
                             long long ldc, const float* x_scale, const float* w_scale, const void* bias, int act, int q_from, long long q_ld,
                             int q_col0, int q_kgroups, void* status, cudaStream_t stream) {
  if (!b200_gemm_quant_fits(m, n, k) || q_from < 0 || q_from >= n || q_from % 128 != 0 || q_col0 < 0 || q_col0 % 128 != 0 || q_ld % 32 != 0 || !x_scale ||
      !w_scale || !out_q || !out_sf || (q_from > 0 && (!out || ldc % 16 != 0)) || ldx % 16 != 0 || ldw % 16 != 0 || (act >> 8) % 8 != 0)
    return -12;
  if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(out_q)) & 31) return -12;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(x_scale) |
       reinterpret_cast<uintptr_t>(w_scale)) & 15)
    return -12;
  GemmParams p{};
  p.k = k;
  p.rows_a = m;
  p.rows_b = n;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.ldc = ldc;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.act = act & 255;
  p.act_col = act >> 8;
  p.status = static_cast<DeviceStatus*>(status);
  p.glu_q = static_cast<uint8_t*>(out_q);
  p.glu_sf = static_cast<uint8_t*>(out_sf);
  p.q_from = q_from; p.q_ld = q_ld; p.q_col0 = q_col0; p.q_kgroups = q_kgroups;
  p.sf_a = reinterpret_cast<const uint32_t*>(x_scale);
  p.sf_b = reinterpret_cast<const uint32_t*>(w_scale);
  p.sf_kgroups = (k + 511) / 512;
  return gemm_pair(p, x, w, ldx, ldw, 2, stream, true);
}
