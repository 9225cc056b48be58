// Batched token sampling on the device: temperature -> top-k -> top-p -> min-p -> seeded draw, one
// thread block per request row, the vocabulary never sorted and never copied to the host.
//
// With w_i = exp((l_i - max l) / T) every filter of the chain keeps a set of the form {w_i >= tau}:
//   top-k   tau = the k-th largest w (ties at that value are all kept, like a mask "below the k-th");
//   top-p   over the survivors, in descending order, keep an element while the mass in front of it
//           is <= p of the survivors' mass: tau = the smallest w still kept;
//   min-p   tau = min_p * max w = min_p.
// The two order statistics are found by a radix search on the bit pattern of w (positive floats
// order like their bits): three passes of 11 + 11 + 10 bits, each one histogram of counts and of
// (fixed-point) masses in shared memory. The draw walks the vocabulary in index order with a block-wide prefix
// sum of the kept masses.
//
// A row of up to 262144 logits belongs to a cluster of eight blocks that keep it in registers: one read of
// the row, histograms and prefix sums met through distributed shared memory. Longer rows go through one block that makes
// eight passes over a row in L2, and so do short rows and many rows of moderate length, where the exchanges of a
// cluster cost more than the passes (see b200_sample_form). Both forms sum masses in 2^-40, so a row's token is the
// same whatever batch it comes in (fp32 sums in the one block drew another token than the cluster in two or three of 1000 flat rows of 100000).
//
// The reference applies the same chain on the host, one request at a time, after copying the logits
// back (src/HartsyInference.LLM/Sampling/SamplerChain.cs:26-85, TopKSampler.cs, TopPSampler.cs,
// MinPSampler.cs); a row with temperature <= 0 is an argmax (ties -> lowest id) like
// lm_argmax_lastdim_f32 (Kernels/lm/lm_f32.cu:214).
#include "common.cuh"

namespace b200 {

int num_sms();      // of the current device, see gemm_tcgen05.cu

constexpr int kSampleThreads = 1024;
constexpr int kSampleBins = 2048;

struct SampleParams {
  const void* logits;          // [rows][ld] fp32 or bf16
  int is_f32;
  long long ld;
  int vocab;
  const float* temperature;    // [rows]; <= 0: argmax
  const int* top_k;            // [rows]; <= 0 or >= vocab: off
  const float* top_p;          // [rows]; <= 0 or >= 1: off
  const float* min_p;          // [rows]; <= 0: off
  const unsigned long long* seed;     // [rows]
  const unsigned long long* counter;  // [rows]: position of the draw in the request's stream
  int* out;                    // [rows]
};

__device__ __forceinline__ float sample_logit(const SampleParams& p, long long row_off, int i) {
  return p.is_f32 ? static_cast<const float*>(p.logits)[row_off + i]
                  : __bfloat162float(static_cast<const __nv_bfloat16*>(p.logits)[row_off + i]);
}

// splitmix64 of (seed, counter) -> uniform in [0, 1)
__device__ __forceinline__ float sample_uniform(unsigned long long seed, unsigned long long counter) {
  unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (counter + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return static_cast<float>(z >> 40) * (1.f / 16777216.f);
}

// The row's uniform number (24 bits) times its whole mass: in [0, total).
__device__ __forceinline__ unsigned long long draw_point(const SampleParams& p, int row, unsigned long long total) {
  const unsigned long long bits = static_cast<unsigned long long>(sample_uniform(p.seed[row], p.counter[row]) * 16777216.f);
  return __umul64hi(total, bits << 40);
}

__device__ __forceinline__ float block_reduce_max(float v, float* red) {
  v = warp_max(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = threadIdx.x < 32 ? red[threadIdx.x] : -INFINITY;
  if (threadIdx.x < 32) {
    t = warp_max(t);
    if (threadIdx.x == 0) red[0] = t;
  }
  __syncthreads();
  t = red[0];
  __syncthreads();
  return t;
}

// One level of the radix search. Elements whose bits above `shift + bits` equal `prefix` (all
// elements at the first level) and whose w >= floor are binned by `bits` bits at `shift`. Walking
// the bins from the top, with `count_before` / `mass_before` already in front:
//   by_count: stop in the bin where the count reaches `k`
//   else:     stop in the bin that holds the first element whose mass in front exceeds `limit`
// Leaves the chosen bin in sh->bin (-1: the walk ran off the end, everything is kept) and adds what lies
// in front of that bin to the running totals in `sh`.
// Masses are accumulated in 2^-40 fixed point: integer shared-memory atomics are native and the sums do
// not depend on the order of arrival, so a (seed, counter) pair always draws the same token.
constexpr float kMassScale = 1099511627776.f;        // 2^40

struct RadixState {
  unsigned prefix;                      // bits above the current level (every thread keeps a copy)
};

// Block-wide state of the search (shared memory): what lies in front of the current prefix, the
// chosen bin, and the scratch of the scans.
struct RadixShared {
  unsigned count_before;
  unsigned long long mass_before;       // 2^-40 fixed point
  int bin;
  unsigned warp_cnt[kSampleThreads / 32];
  unsigned long long warp_mass[kSampleThreads / 32];
};

__device__ void radix_level(const SampleParams& p, long long row_off, float mx, float inv_t, float floor_w, int shift, int bits,
                            unsigned hi_mask, const RadixState& st, bool by_count, unsigned long long target, unsigned* hist_cnt,
                            unsigned long long* hist_mass, RadixShared* sh) {
  const int nb = 1 << bits;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    hist_cnt[b] = 0u;
    hist_mass[b] = 0ull;
  }
  if (threadIdx.x == 0) sh->bin = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < p.vocab; i += blockDim.x) {
    const float w = __expf((sample_logit(p, row_off, i) - mx) * inv_t);
    if (!(w >= floor_w)) continue;
    const unsigned u = __float_as_uint(w);
    if ((u & hi_mask) != st.prefix) continue;
    const int b = (u >> shift) & (nb - 1);
    atomicAdd(hist_cnt + b, 1u);
    atomicAdd(hist_mass + b, static_cast<unsigned long long>(w * kMassScale));
  }
  __syncthreads();
  // Walk from the top bin down, all bins at once: thread t owns bins 2t and 2t + 1; an inclusive scan
  // over the threads gives every bin what lies at and above it. By count the wanted bin is the
  // highest non-empty one at which the count from the top reaches the target; by mass the highest
  // non-empty one at which the mass from the top exceeds it.
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const unsigned c0 = 2 * t < nb ? hist_cnt[2 * t] : 0u, c1 = 2 * t + 1 < nb ? hist_cnt[2 * t + 1] : 0u;
  const unsigned long long m0 = 2 * t < nb ? hist_mass[2 * t] : 0ull, m1 = 2 * t + 1 < nb ? hist_mass[2 * t + 1] : 0ull;
  unsigned pc = c0 + c1;
  unsigned long long pm = m0 + m1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned vc = __shfl_up_sync(0xffffffffu, pc, o);
    const unsigned long long vm = __shfl_up_sync(0xffffffffu, pm, o);
    if (lane >= o) { pc += vc; pm += vm; }
  }
  if (lane == 31) { sh->warp_cnt[wid] = pc; sh->warp_mass[wid] = pm; }
  __syncthreads();
  unsigned base_c = 0, total_c = 0;
  unsigned long long base_m = 0, total_m = 0;
#pragma unroll 4
  for (int w = 0; w < kSampleThreads / 32; ++w) {
    const unsigned wc = sh->warp_cnt[w];
    const unsigned long long wm = sh->warp_mass[w];
    if (w < wid) { base_c += wc; base_m += wm; }
    total_c += wc;
    total_m += wm;
  }
  // inclusive prefix (ascending bins) up to and including this thread's pair -> what lies at and above
  const unsigned incl_c = base_c + pc;
  const unsigned long long incl_m = base_m + pm;
  const unsigned above_c = total_c - incl_c;                  // bins above 2t + 1
  const unsigned long long above_m = total_m - incl_m;
  const unsigned before_c = sh->count_before;
  const unsigned long long before_m = sh->mass_before;
  // bin 2t + 1, then bin 2t
  auto hit = [&](unsigned cnt, unsigned front_c, unsigned long long mass, unsigned long long front_m) {
    if (cnt == 0u) return false;
    return by_count ? (static_cast<unsigned long long>(before_c) + front_c + cnt >= target) : (before_m + front_m + mass > target);
  };
  int mine = -1;
  if (hit(c1, above_c, m1, above_m)) mine = 2 * t + 1;
  else if (hit(c0, above_c + c1, m0, above_m + m1)) mine = 2 * t;
  if (mine >= 0) atomicMax(&sh->bin, mine);
  __syncthreads();
  const int chosen = sh->bin;
  __syncthreads();
  if (chosen >= 0 && (chosen >> 1) == t) {
    // what lies in front of the chosen bin joins the running totals
    const bool upper = (chosen & 1) != 0;
    sh->count_before = before_c + above_c + (upper ? 0u : c1);
    sh->mass_before = before_m + above_m + (upper ? 0ull : m1);
  }
  __syncthreads();
}

// Sum of `x` over the threads of the block in front of this one; the block's sum in `total`. `sums` may be used again.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long x, unsigned long long* sums, unsigned long long& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto warp_scan = [&](unsigned long long incl) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    return incl;
  };
  const unsigned long long incl = warp_scan(x);
  __syncthreads();
  if (lane == 31) sums[wid] = incl;
  __syncthreads();
  const unsigned long long own = sums[lane], upto = warp_scan(own);      // 32 warps
  total = __shfl_sync(0xffffffffu, upto, 31);
  return __shfl_sync(0xffffffffu, upto - own, wid) + incl - x;
}

__global__ void __launch_bounds__(kSampleThreads) sample_kernel(const SampleParams p) {
  __shared__ float red[32];
  __shared__ unsigned hist_cnt[kSampleBins];
  __shared__ unsigned long long hist_mass[kSampleBins];
  __shared__ RadixShared rsh;
  __shared__ unsigned long long s_scan[kSampleThreads / 32];
  __shared__ int s_pick;
  const int row = blockIdx.x;
  const long long row_off = static_cast<long long>(row) * p.ld;
  const float temp = p.temperature[row];

  // ---- maximum (and its first index: the answer of a greedy row)
  float mx = -INFINITY;
  int arg = 0x7fffffff;
  for (int i = threadIdx.x; i < p.vocab; i += blockDim.x) {
    const float v = sample_logit(p, row_off, i);
    if (v > mx) { mx = v; arg = i; }
  }
  const float bmx = block_reduce_max(mx, red);
  if (temp <= 0.f || !(bmx > -INFINITY)) {
    // ties -> lowest index
    int cand = mx == bmx ? arg : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cand = min(cand, __shfl_xor_sync(0xffffffffu, cand, o));
    __shared__ int s_arg[32];
    if ((threadIdx.x & 31) == 0) s_arg[threadIdx.x >> 5] = cand;
    __syncthreads();
    if (threadIdx.x == 0) {
      int best = 0x7fffffff;
      for (int w = 0; w < kSampleThreads / 32; ++w) best = min(best, s_arg[w]);
      p.out[row] = best == 0x7fffffff ? 0 : best;
    }
    return;
  }
  const float inv_t = 1.f / fmaxf(temp, 1e-6f);
  float tau = 0.f;     // keep w >= tau

  // ---- top-k: the k-th largest w
  const int k = p.top_k[row];
  if (k > 0 && k < p.vocab) {
    RadixState st{0u};
    if (threadIdx.x == 0) { rsh.count_before = 0u; rsh.mass_before = 0ull; }
    __syncthreads();
    unsigned hi_mask = 0u;
    int shift = 21;
    const int level_bits[3] = {11, 11, 10};
    bool open_end = false;
    for (int lv = 0; lv < 3; ++lv) {
      shift = lv == 0 ? 21 : lv == 1 ? 10 : 0;
      radix_level(p, row_off, bmx, inv_t, 0.f, shift, level_bits[lv], hi_mask, st, true, static_cast<unsigned long long>(k),
                  hist_cnt, hist_mass, &rsh);
      const int b = rsh.bin;
      if (b < 0) { open_end = true; break; }
      st.prefix |= static_cast<unsigned>(b) << shift;
      hi_mask |= static_cast<unsigned>((1 << level_bits[lv]) - 1) << shift;
    }
    if (!open_end) tau = __uint_as_float(st.prefix);
  }

  // ---- top-p over the survivors: the smallest w whose mass in front is <= p * kept_mass
  const float tp = p.top_p[row];
  if (tp > 0.f && tp < 1.f) {
    unsigned long long kept = 0;
    for (int i = threadIdx.x; i < p.vocab; i += blockDim.x) {
      const float w = __expf((sample_logit(p, row_off, i) - bmx) * inv_t);
      if (w >= tau) kept += static_cast<unsigned long long>(w * kMassScale);
    }
    unsigned long long total;
    block_scan(kept, s_scan, total);
    const unsigned long long limit = static_cast<unsigned long long>(static_cast<double>(tp) * static_cast<double>(total));
    RadixState st{0u};
    if (threadIdx.x == 0) { rsh.count_before = 0u; rsh.mass_before = 0ull; }
    __syncthreads();
    unsigned hi_mask = 0u;
    const int level_bits[3] = {11, 11, 10};
    bool open_end = false;
    for (int lv = 0; lv < 3; ++lv) {
      const int shift = lv == 0 ? 21 : lv == 1 ? 10 : 0;
      radix_level(p, row_off, bmx, inv_t, tau, shift, level_bits[lv], hi_mask, st, false, limit, hist_cnt, hist_mass, &rsh);
      const int b = rsh.bin;
      if (b < 0) { open_end = true; break; }
      st.prefix |= static_cast<unsigned>(b) << shift;
      hi_mask |= static_cast<unsigned>((1 << level_bits[lv]) - 1) << shift;
    }
    // the chosen value is the first one with MORE than the limit in front of its last copy: it is
    // still kept when the mass in front of its first copy is within the limit (the usual case of a
    // value that occurs once), so the threshold is that value itself
    if (!open_end) tau = fmaxf(tau, __uint_as_float(st.prefix));
  }

  // ---- min-p relative to the largest probability (w = 1)
  const float mp = p.min_p[row];
  if (mp > 0.f) tau = fmaxf(tau, fminf(mp, 1.f));

  // ---- draw: index-ordered prefix sums of the kept masses, in 2^-40 as in sample_row_kernel: the token of a row does not
  // depend on which of the two its batch takes
  const int per = (p.vocab + kSampleThreads - 1) / kSampleThreads;
  const int i0 = threadIdx.x * per, i1 = min(p.vocab, i0 + per);
  unsigned long long local = 0;
  for (int i = i0; i < i1; ++i) {
    const float w = __expf((sample_logit(p, row_off, i) - bmx) * inv_t);
    if (w >= tau) local += static_cast<unsigned long long>(w * kMassScale);
  }
  unsigned long long total;
  unsigned long long front = block_scan(local, s_scan, total);
  if (threadIdx.x == 0) s_pick = -1;
  __syncthreads();
  const unsigned long long u = draw_point(p, row, total);
  if (u >= front && u < front + local) {
    // walk this thread's chunk
    for (int i = i0; i < i1; ++i) {
      const float w = __expf((sample_logit(p, row_off, i) - bmx) * inv_t);
      if (w >= tau) {
        front += static_cast<unsigned long long>(w * kMassScale);
        if (u < front) { s_pick = i; break; }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int pick = s_pick;
    if (pick < 0) {
      // no finite mass: the most probable token
      pick = 0;
      float best = -INFINITY;
      for (int i = 0; i < p.vocab; ++i) {
        const float v = sample_logit(p, row_off, i);
        if (v > best) { best = v; pick = i; }
      }
    }
    p.out[row] = pick;
  }
}

// ---- one row per cluster -------------------------------------------------------------------------
constexpr int kRowBlocks = 8;          // blocks of a row's cluster (the portable size)
constexpr int kRowThreads = 512;

__device__ __forceinline__ uint32_t dsmem_addr(const void* local, int block) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(local)), "r"(block));
  return r;
}
__device__ __forceinline__ unsigned long long ld_dsmem_u64(uint32_t addr) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_dsmem_u32(uint32_t addr) {
  unsigned v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_dsmem_u32x4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// A block's histogram: counts in `lo`, or masses (up to 2^41 each, 2^15 of them) as three 32-bit sums of 14-bit
// pieces, because 32-bit adds are what shared memory does by itself; 64-bit ones are compare-and-swap loops that
// the few bins of a peaked row keep failing.
struct RowHist {
  unsigned lo[kSampleBins], mid[kSampleBins], hi[kSampleBins];
};
constexpr int kRowRun = 32, kRowRuns = kSampleBins / kRowRun;      // bins whose sum a block gives its peers, and how many such runs
struct RowShared {
  RowHist hist[2];                                    // levels alternate
  unsigned long long runs[2][kRowRuns];               // sums of this block's runs of bins
  unsigned long long part[kSampleBins];               // the draw's masses per step and warp
  unsigned long long scan[kRowThreads / 32];
  unsigned long long front;                           // what lies in front of the chosen bin
  unsigned long long meet[3];                         // this block's words of the exchanges: (max, index), kept mass, drawn mass
  unsigned long long all[kRowBlocks];
  int bin;
};

// All blocks' words of exchange `n` in sh.all (thread 0 has written sh.meet[n], which is used once).
__device__ __forceinline__ void row_exchange(RowShared& sh, int n) {
  cluster_sync_all();
  if (threadIdx.x < kRowBlocks) sh.all[threadIdx.x] = ld_dsmem_u64(dsmem_addr(&sh.meet[n], threadIdx.x));
  __syncthreads();
}

// Sum of `x` over the threads in front of this one; the block's sum in `total`.
__device__ __forceinline__ unsigned long long row_scan(RowShared& sh, unsigned long long x, unsigned long long& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();
  if (lane == 31) sh.scan[wid] = incl;
  __syncthreads();
  unsigned long long base = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kRowThreads / 32; ++w) {
    const unsigned long long y = sh.scan[w];
    if (w < wid) base += y;
    total += y;
  }
  return base + incl - x;
}

// Order statistic of the row's values >= floor_w (see radix_level): by count the `target`-th largest value, by
// mass the first value, from the largest down, with more than `target` up to and including it. 0 when there is
// no such value.
template <int V>
__device__ __forceinline__ float row_select(RowShared& sh, int& level, const float (&v)[V], float floor_w, bool by_count,
                                            unsigned long long target) {
  unsigned prefix = 0u, hi_mask = 0u;
  unsigned long long before = 0;
#pragma unroll 1
  for (int lv = 0; lv < 3; ++lv) {
    const int shift = lv == 0 ? 21 : lv == 1 ? 10 : 0, bits = lv == 2 ? 10 : 11, nb = 1 << bits;
    const int parity = level & 1;
    RowHist& hist = sh.hist[parity];
    ++level;
    for (int b = threadIdx.x; b < kSampleBins; b += kRowThreads) {
      hist.lo[b] = 0u;
      if (!by_count) hist.mid[b] = hist.hi[b] = 0u;
    }
    if (threadIdx.x == 0) sh.bin = -1;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const unsigned u = __float_as_uint(v[i]);
      if (v[i] >= floor_w && (u & hi_mask) == prefix) {
        const int b = (u >> shift) & (nb - 1);
        if (by_count) {
          atomicAdd(hist.lo + b, 1u);
        } else {
          const unsigned long long m = static_cast<unsigned long long>(v[i] * kMassScale);
          if (m & 0x3fffu) atomicAdd(hist.lo + b, static_cast<unsigned>(m) & 0x3fffu);
          if (m >> 14) atomicAdd(hist.mid + b, static_cast<unsigned>(m >> 14) & 0x3fffu);
          if (m >> 28) atomicAdd(hist.hi + b, static_cast<unsigned>(m >> 28));
        }
      }
    }
    __syncthreads();
    // Sums of runs of bins first: the peers read 64 words of each block, and then the bins of the one run that the walk ends in. (All
    // blocks' bins, 24 KB of each, took 12000 cycles a level and kept the blocks waiting for one another for as long.)
    auto bin_of = [&](const RowHist& h, int at) {
      unsigned long long m = h.lo[at];
      if (!by_count) m += (static_cast<unsigned long long>(h.mid[at]) << 14) + (static_cast<unsigned long long>(h.hi[at]) << 28);
      return m;
    };
    unsigned long long* const runs = sh.runs[parity];
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < kRowRuns; r += kRowThreads / 32) {
      unsigned long long m = bin_of(hist, r * kRowRun + lane);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      if (lane == 0) runs[r] = m;
    }
    cluster_sync_all();
    // one warp walks, the top run first: a lane takes two runs, then one bin
    if (threadIdx.x < 32) {
      unsigned long long c[2] = {0ull, 0ull};
      const int r0 = kRowRuns - 2 - 2 * lane;
#pragma unroll
      for (int k = 0; k < kRowBlocks; ++k) {
        const uint4 x = ld_dsmem_u32x4(dsmem_addr(runs + r0, k));
        c[0] += x.x | static_cast<unsigned long long>(x.y) << 32;
        c[1] += x.z | static_cast<unsigned long long>(x.w) << 32;
      }
      auto in_front = [&](unsigned long long x) {            // sum over the lanes in front
        unsigned long long incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        return incl - x;
      };
      // what lies in front has not reached the target, with this it has: of one run and one bin at most
      auto ends = [&](unsigned long long front, unsigned long long x) {
        return x != 0ull && (by_count ? front < target && front + x >= target : front <= target && front + x > target);
      };
      unsigned long long front = before + in_front(c[0] + c[1]);
      int run = -1;
      if (ends(front, c[1])) run = r0 + 1;
      else if (ends(front + c[1], c[0])) { run = r0; front += c[1]; }
      const unsigned who = __ballot_sync(0xffffffffu, run >= 0);
      if (who) {
        run = __shfl_sync(0xffffffffu, run, __ffs(who) - 1);
        front = __shfl_sync(0xffffffffu, front, __ffs(who) - 1);
        const int at = run * kRowRun + kRowRun - 1 - lane;
        unsigned long long m = 0;
#pragma unroll
        for (int k = 0; k < kRowBlocks; ++k) {
          m += ld_dsmem_u32(dsmem_addr(hist.lo + at, k));
          if (!by_count) m += (static_cast<unsigned long long>(ld_dsmem_u32(dsmem_addr(hist.mid + at, k))) << 14) +
                              (static_cast<unsigned long long>(ld_dsmem_u32(dsmem_addr(hist.hi + at, k))) << 28);
        }
        front += in_front(m);
        if (ends(front, m)) { sh.bin = at; sh.front = front; }
      }
    }
    __syncthreads();
    const int chosen = sh.bin;
    if (chosen < 0) return 0.f;
    before = sh.front;
    prefix |= static_cast<unsigned>(chosen) << shift;
    hi_mask |= static_cast<unsigned>(nb - 1) << shift;
    __syncthreads();
  }
  return __uint_as_float(prefix);
}

// The filter chain and the draw of sample_kernel with the row in registers: thread t of block b holds the values
// (b * V + i) * 512 + t. Masses are 2^-40 fixed point throughout, so sums do not depend on their order.
// Bound by the adds into the first histogram of a search, whose bins are few, and by the chain of exchanges, not by
// memory. 64 rows of 128256 (a block per row / every block reading all bins of its peers / the run's bins only): top-p 393 / 205 /
// 74 us, top-k and top-p 484 / 257 / 86, neither 66 / 42 / 32; one row with both 470 / 73 / 34 us.
template <int V>
__global__ void __launch_bounds__(kRowThreads, V <= 40 ? 2 : 1) sample_row_kernel(const SampleParams p) {
  extern __shared__ __align__(16) uint8_t row_smem[];
  RowShared& sh = *reinterpret_cast<RowShared*>(row_smem);
  const int row = blockIdx.x / kRowBlocks, block = blockIdx.x % kRowBlocks;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long row_off = static_cast<long long>(row) * p.ld;
  const int first = block * V * kRowThreads + threadIdx.x;
  float v[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int at = first + i * kRowThreads;
    v[i] = at < p.vocab ? sample_logit(p, row_off, at) : -INFINITY;
  }
  // ---- maximum and its first index: ordered so that the largest word is the largest logit, then the lowest index
  float mx = -INFINITY;
  int arg = 0x7fffffff;
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (v[i] > mx) { mx = v[i]; arg = first + i * kRowThreads; }
  auto word = [](float f, int i) {
    const unsigned u = __float_as_uint(f), key = u & 0x80000000u ? ~u : u | 0x80000000u;
    return static_cast<unsigned long long>(key) << 32 | static_cast<unsigned>(0x7fffffff - i);
  };
  if (mx == 0.f) mx = 0.f;                     // -0 and +0 tie
  unsigned long long best = word(mx, arg);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long y = __shfl_xor_sync(0xffffffffu, best, o);
    best = y > best ? y : best;
  }
  if (lane == 0) sh.scan[wid] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kRowThreads / 32; ++w) best = sh.scan[w] > best ? sh.scan[w] : best;
    sh.meet[0] = best;
  }
  row_exchange(sh, 0);
  best = sh.all[0];
#pragma unroll
  for (int k = 1; k < kRowBlocks; ++k) best = sh.all[k] > best ? sh.all[k] : best;
  const unsigned key = static_cast<unsigned>(best >> 32);
  const float bmx = __uint_as_float(key & 0x80000000u ? key & 0x7fffffffu : ~key);
  const int top = 0x7fffffff - static_cast<int>(static_cast<unsigned>(best));
  const float temp = p.temperature[row];
  if (temp <= 0.f || !(bmx > -INFINITY)) {
    if (block == 0 && threadIdx.x == 0) p.out[row] = top == 0x7fffffff ? 0 : top;
    cluster_sync_all();                        // nobody leaves while a peer may still read its words
    return;
  }
  const float inv_t = 1.f / fmaxf(temp, 1e-6f);
#pragma unroll
  for (int i = 0; i < V; ++i)
    v[i] = first + i * kRowThreads < p.vocab ? __expf((v[i] - bmx) * inv_t) : -1.f;      // below every threshold

  int level = 0;
  float tau = 0.f;
  const int k = p.top_k[row];
  if (k > 0 && k < p.vocab) tau = row_select<V>(sh, level, v, 0.f, true, static_cast<unsigned long long>(k));
  const float tp = p.top_p[row];
  if (tp > 0.f && tp < 1.f) {
    unsigned long long mine = 0, total;
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (v[i] >= tau) mine += static_cast<unsigned long long>(v[i] * kMassScale);
    row_scan(sh, mine, total);
    if (threadIdx.x == 0) sh.meet[1] = total;
    row_exchange(sh, 1);
    total = 0;
#pragma unroll
    for (int b = 0; b < kRowBlocks; ++b) total += sh.all[b];
    const unsigned long long limit = static_cast<unsigned long long>(static_cast<double>(tp) * static_cast<double>(total));
    tau = fmaxf(tau, row_select<V>(sh, level, v, tau, false, limit));
  }
  const float mp = p.min_p[row];
  if (mp > 0.f) tau = fmaxf(tau, fminf(mp, 1.f));

  // ---- draw: index-ordered prefix sums of the kept masses, per warp and step first
  __syncthreads();
  unsigned long long* part = sh.part;                      // [V steps][16 warps]
#pragma unroll
  for (int i = 0; i < V; ++i) {
    unsigned long long m = v[i] >= tau ? static_cast<unsigned long long>(v[i] * kMassScale) : 0ull;
    // 41 bits in two pieces whose sums over a warp fit 32: one instruction each
    m = __reduce_add_sync(0xffffffffu, static_cast<unsigned>(m) & 0xfffffu) +
        (static_cast<unsigned long long>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(m >> 20))) << 20);
    if (lane == 0) part[i * (kRowThreads / 32) + wid] = m;
  }
  __syncthreads();
  constexpr int kParts = V * (kRowThreads / 32), kEach = (kParts + kRowThreads - 1) / kRowThreads;
  unsigned long long mine = 0, total;
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const int at = threadIdx.x * kEach + e;
    if (at < kParts) mine += part[at];
  }
  const unsigned long long own = row_scan(sh, mine, total);      // parts in front of this thread's
  if (threadIdx.x == 0) { sh.meet[2] = total; sh.bin = -1; }
  row_exchange(sh, 2);
  unsigned long long before = 0, all = 0;
#pragma unroll
  for (int b = 0; b < kRowBlocks; ++b) {
    if (b < block) before += sh.all[b];
    all += sh.all[b];
  }
  const unsigned long long u = draw_point(p, row, all);
  unsigned long long run = before + own;
#pragma unroll
  for (int e = 0; e < kEach; ++e) {
    const int at = threadIdx.x * kEach + e;
    const unsigned long long m = at < kParts ? part[at] : 0ull;
    if (m != 0ull && u >= run && u < run + m) { sh.bin = at; sh.front = run; }
    run += m;
  }
  __syncthreads();
  const int at = sh.bin;
  if (at >= 0 && wid == at % (kRowThreads / 32)) {
    const int step = at / (kRowThreads / 32);
    float w = -1.f;
#pragma unroll
    for (int i = 0; i < V; ++i)
      if (i == step) w = v[i];
    const unsigned long long m = w >= tau ? static_cast<unsigned long long>(w * kMassScale) : 0ull;
    unsigned long long incl = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    incl += sh.front;
    if (m != 0ull && u >= incl - m && u < incl) p.out[row] = first + step * kRowThreads;
  }
  if (all == 0ull && block == 0 && threadIdx.x == 0) p.out[row] = top;      // no finite mass: the most probable token
  cluster_sync_all();
}

template <int V>
static int launch_rows(const SampleParams& p, int rows, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * kRowBlocks);
  cfg.blockDim = dim3(kRowThreads);
  cfg.dynamicSmemBytes = sizeof(RowShared);
  cfg.stream = stream;
  static PerDeviceOnce configured;
  if (configured.first_time() &&
      cudaFuncSetAttribute(sample_row_kernel<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(RowShared)) != cudaSuccess)
    return -200;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kRowBlocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, sample_row_kernel<V>, p) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -300;
}

}  // namespace b200

using namespace b200;

static int row_values(int vocab) { return (vocab + kRowBlocks * kRowThreads - 1) / (kRowBlocks * kRowThreads); }      // that a thread holds

// Whether b200_sample gives a row to a cluster (1) or to one block (0). Which filters a row asks for is known on the device only. Every filter
// asked for, a block takes 28 us + a us per 290 logits, all rows of a wave at once; a cluster 21 to 44 us, twice that when they fill the
// machine, and from there 0.8 to 2.9 us a row by the values that a thread holds. Without filters a block takes 4 us + a us per 1950 to 2400
// logits and 0.7 of that for each further wave; a cluster 7 to 18 us, a fifth more from 16 rows and nearly twice that from 37 on, where a
// second wave starts, and 0.2 to 0.7 us a row beyond 49. A cluster has to be a fifth faster in the full chain and at most an eighth slower
// without one (us, block / cluster: without filters, with all):
//   1 x 2048      5.0 / 6.5, 30 / 21      8 x 8192      7.5 / 6.9, 47 / 22      37 x 8192     7.6 / 12.4, 47 / 45     48 x 16384    11.2 / 13.5, 69 / 47
//   64 x 32000    22 / 16, 116 / 52       96 x 50257    26 / 27, 159 / 91       64 x 128256   64 / 37, 433 / 92      128 x 128256  65 / 71, 437 / 181
//   148 x 128256  64 / 82, 435 / 214      200 x 202048  206 / 415, 1367 / 771   256 x 151936  152 / 235, 1033 / 480  512 x 100352  266 / 395, 1258 / 819
// Rows of more than 163840 logits, one block of a cluster on a processor: there the full chain decides, with 105 us for 18 of them.
B200_API int b200_sample_form(int rows, int vocab) {
  const int each = row_values(vocab), sms = num_sms();
  if (rows < 1 || rows >= (1 << 27) || sms < kRowBlocks || each > 64) return 0;
  const int waves = (rows + sms - 1) / sms;
  if (each > 40) return 105. * ((rows + 17) / 18) <= (24. + vocab / 350.) * waves ? 1 : 0;
  const int width = each <= 8 ? 0 : each <= 16 ? 1 : each <= 32 ? 2 : 3;
  constexpr double kRowUs[4] = {0.76, 0.93, 1.33, 1.6};                                        // with every filter
  const double block_us = (28. + vocab / 290.) * waves, cluster_us = kRowUs[width] * (rows <= 8 ? 28. : rows <= 18 ? 36. : rows <= 49 ? 55. : rows + 6.);
  constexpr double kFirst[4] = {6.9, 8., 15., 18.4}, kMore[4] = {0.205, 0.25, 0.52, 0.67}, kBase[4] = {1.5, 3., 4., 2.5};      // without
  constexpr double kLogitsUs[4] = {2400., 2400., 2150., 1950.};
  const double block_plain = 4.2 + vocab / kLogitsUs[width] * (1. + 0.72 * (waves - 1));
  const double cluster_plain = rows <= 12 ? kFirst[width] : rows <= 36 ? 1.22 * kFirst[width] : rows <= 49 ? 1.9 * kFirst[width] : kBase[width] + kMore[width] * rows;
  return cluster_us <= 0.8 * block_us && cluster_plain <= 1.12 * block_plain ? 1 : 0;
}

// logits [rows][ld] (fp32 when is_f32, else bf16); per-row device arrays as in SampleParams; out int32 [rows].
B200_API int b200_sample(const void* logits, int is_f32, long long ld, int rows, int vocab, const float* temperature,
                         const int* top_k, const float* top_p, const float* min_p, const unsigned long long* seed,
                         const unsigned long long* counter, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0 || vocab > (1 << 24)) return -2;
  SampleParams p{};
  p.logits = logits; p.is_f32 = is_f32; p.ld = ld; p.vocab = vocab;
  p.temperature = temperature; p.top_k = top_k; p.top_p = top_p; p.min_p = min_p;
  p.seed = seed; p.counter = counter; p.out = out;
  if (b200_sample_form(rows, vocab)) {
    const int each = row_values(vocab);
    if (each <= 8) return launch_rows<8>(p, rows, stream);
    if (each <= 16) return launch_rows<16>(p, rows, stream);
    if (each <= 32) return launch_rows<32>(p, rows, stream);
    if (each <= 40) return launch_rows<40>(p, rows, stream);
    if (each <= 64) return launch_rows<64>(p, rows, stream);
  }
  sample_kernel<<<rows, kSampleThreads, 0, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -300;
}
