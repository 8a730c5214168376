// Token selection on the device: arg-max, and sampling with temperature, top-k and
// top-p in the order of the reference (src/sampler/mod.rs:194-222): logits / T, top-k
// on the scaled logits, softmax, top-p on the probabilities, inverse-CDF draw.
//
// A cluster of blocks per row of logits holds the row in registers (vocabularies of up to
// 262,144 entries; one block per row walks longer ones through memory).  Probabilities are kept
// as 40-bit fixed-point integers of exp(z - max): integer sums do not depend on the order of
// addition, so every threshold and the draw are the same from run to run, the same from both
// kernels and equal to a sequential pass in index order.  The uniform number of each row comes from the
// host, which derives it from (seed, sequence, step).
//
// Ties: arg-max keeps the highest index among equal maxima, as the reference's max_by does
// (src/sampler/mod.rs:60-68); at a top-k or top-p threshold the tied entries of lowest
// index are kept (top-k: as the reference, :108-117; top-p: the reference's unstable
// sort leaves it open, :147).
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"

#define SAMPLE_THREADS 1024
#define FIX_ONE 1099511627776.0f  // 2^40

typedef unsigned long long u64;

__device__ __forceinline__ uint32_t float_key(float f) {
  // larger float -> larger key; NaN is pushed below everything
  if (f != f) return 0u;
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// --------------------------------------------------------------------------
// arg-max
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(SAMPLE_THREADS)
argmax_kernel(const float* __restrict__ logits, int ld, int V, int* __restrict__ out) {
  __shared__ uint32_t sk[32];
  __shared__ int si[32];
  pdl_wait();
  pdl_launch_dependents();
  const float* row = logits + (size_t)blockIdx.x * ld;
  uint32_t best = 0u;
  int best_i = -1;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const uint32_t k = float_key(row[i]);
    if (k > best || (k == best && i > best_i)) { best = k; best_i = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint32_t ok = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ok > best || (ok == best && oi > best_i)) { best = ok; best_i = oi; }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sk[warp] = best; si[warp] = best_i; }
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    best = lane < nw ? sk[lane] : 0u;
    best_i = lane < nw ? si[lane] : -1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const uint32_t ok = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
      if (ok > best || (ok == best && oi > best_i)) { best = ok; best_i = oi; }
    }
    if (lane == 0) out[blockIdx.x] = (best_i >= 0 && best_i < V) ? best_i : 0;
  }
}

// The same with several blocks per row, for the few rows of a decode step (one block per row
// leaves most SMs idle and takes as long as its one chain of loads).  A block folds its part
// of the row into one 64-bit word per row with atomicMax: key in the high half, the index
// plus one in the low half, so that among equal keys the highest index wins.  The
// block that finishes a row last writes the result and clears the row's word and counter for
// the next launch (they are static: launches on one stream at a time).
#define ARGMAX_ROWS 4096
#define ARGMAX_THREADS 256
__device__ unsigned long long tl_argmax_word[ARGMAX_ROWS];
__device__ unsigned int tl_argmax_count[ARGMAX_ROWS];

__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_parts_kernel(const float* __restrict__ logits, int ld, int V, int per_block, int* __restrict__ out) {
  TL_TRACE_SCOPE(6, V, 6);
  __shared__ unsigned long long sw[ARGMAX_THREADS / 32];
  pdl_wait();
  TL_TRACE_RELEASED();
  pdl_launch_dependents();
  const int r = blockIdx.y;
  const float* row = logits + (size_t)r * ld;
  const int begin = blockIdx.x * per_block, end = min(V, begin + per_block);
  unsigned long long best = 0ull;
#pragma unroll 4
  for (int i = begin + threadIdx.x; i < end; i += ARGMAX_THREADS) {
    const unsigned long long w = ((unsigned long long)float_key(row[i]) << 32) | (uint32_t)(i + 1);
    best = w > best ? w : best;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long ow = __shfl_xor_sync(0xffffffffu, best, o);
    best = ow > best ? ow : best;
  }
  if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < ARGMAX_THREADS / 32; ++w) best = sw[w] > best ? sw[w] : best;
    atomicMax(&tl_argmax_word[r], best);
    __threadfence();
    if (atomicAdd(&tl_argmax_count[r], 1u) == gridDim.x - 1) {   // every part of the row is in
      __threadfence();
      const unsigned long long w = atomicExch(&tl_argmax_word[r], 0ull);
      const uint32_t low = (uint32_t)(w & 0xffffffffull);   // index + 1; 0: nothing was folded in
      out[r] = (low != 0u && low <= (uint32_t)V) ? (int)(low - 1u) : 0;
      tl_argmax_count[r] = 0u;
    }
  }
}

extern "C" int tl_argmax(const float* logits, int ld, int rows, int V, int* out,
                         cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0) return -1;
  // few rows: spread each over several blocks, about 148 blocks in all
  const int parts = rows >= 64 ? 1 : min(16, max(1, min(148 / rows, (V + 2047) / 2048)));
  if (parts > 1 && rows <= ARGMAX_ROWS) {
    const int per_block = (V + parts - 1) / parts;
    return tl_launch(argmax_parts_kernel, dim3(parts, rows), dim3(ARGMAX_THREADS), 0, stream, logits, ld, V,
                     per_block, out);
  }
  return tl_launch(argmax_kernel, dim3(rows), dim3(SAMPLE_THREADS), 0, stream, logits, ld, V, out);
}

// --------------------------------------------------------------------------
// sampling
// --------------------------------------------------------------------------
struct SampleShared {
  u64 wsum[256];
  uint32_t cnt[256];
  u64 warp_tot[32];
  float red[33];
  u64 bcast_u64[2];
  int bcast_int[2];
};

__device__ __forceinline__ float blk_max(float v, SampleShared& sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) sm.red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < (int)(blockDim.x >> 5) ? sm.red[lane] : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
    if (lane == 0) sm.red[32] = t;
  }
  __syncthreads();
  return sm.red[32];
}

// Inclusive scan of one value per thread over the block, in thread order.
// Returns the inclusive prefix; *total receives the block total.
__device__ __forceinline__ u64 blk_scan(u64 v, SampleShared& sm, u64* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u64 n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  __syncthreads();
  if (lane == 31) sm.warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {
    u64 t = lane < (int)(blockDim.x >> 5) ? sm.warp_tot[lane] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 n = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += n;
    }
    sm.warp_tot[lane] = t;  // inclusive totals of the warps
  }
  __syncthreads();
  const u64 off = warp ? sm.warp_tot[warp - 1] : 0ull;
  *total = sm.warp_tot[(blockDim.x >> 5) - 1];
  return v + off;
}

// Histogram updates of a whole warp: lanes that hit the same bin are found with match_any and
// one of them adds for all (most logits share their leading bits, so plain atomics would
// queue a thousand threads on two or three bins).  Every lane of the warp must call these;
// `bin` < 0 takes no part.
__device__ __forceinline__ void warp_count(uint32_t* cnt, int bin) {
  if (!__any_sync(0xffffffffu, bin >= 0)) return;   // after the first digits few entries still carry the prefix
  const unsigned peers = __match_any_sync(0xffffffffu, bin);
  if (bin >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[bin], (uint32_t)__popc(peers));
}
__device__ __forceinline__ void warp_count_weight(uint32_t* cnt, u64* wsum, int bin, u64 w) {
  if (!__any_sync(0xffffffffu, bin >= 0)) return;   // (as above: most warps have nothing to add in the later passes)
  const unsigned peers = __match_any_sync(0xffffffffu, bin);
  // the weights have 41 bits: three sums of 16-bit (and 9-bit) pieces cannot overflow 32 bits
  const uint32_t a = __reduce_add_sync(peers, (uint32_t)(w & 0xffffull));
  const uint32_t b = __reduce_add_sync(peers, (uint32_t)((w >> 16) & 0xffffull));
  const uint32_t c = __reduce_add_sync(peers, (uint32_t)(w >> 32));
  if (bin >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) {
    atomicAdd(&cnt[bin], (uint32_t)__popc(peers));
    atomicAdd(&wsum[bin], (u64)a + ((u64)b << 16) + ((u64)c << 32));
  }
}

// Calls f(i, row[i], valid) for every entry of the row, every lane of a warp the same number
// of times (entries past the end come with valid = false).  Four consecutive entries per
// thread and 16-byte loads when the row allows it, so that a pass is not a chain of single
// loads that each wait for L2.
template <typename F>
__device__ __forceinline__ void for_each_entry(const float* row, int V, F f) {
  const int tid = threadIdx.x;
  const int V4 = (((uintptr_t)row & 15) == 0) ? (V & ~3) : 0;
  for (int i0 = 0; i0 < V4; i0 += blockDim.x * 4) {
    const int i = i0 + tid * 4;
    const bool valid = i < V4;
    const float4 x = valid ? *reinterpret_cast<const float4*>(row + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    f(i, x.x, valid); f(i + 1, x.y, valid); f(i + 2, x.z, valid); f(i + 3, x.w, valid);
  }
  for (int i0 = V4; i0 < V; i0 += blockDim.x) {
    const int i = i0 + tid;
    const bool valid = i < V;
    f(i, valid ? row[i] : 0.0f, valid);
  }
}

struct RowView {
  const float* row;
  int V;
  float T;
  float m;            // max of z
  // top-k state
  bool use_k;
  uint32_t k_thr;     // key of the k-th largest z
  int k_cut;          // entries equal to k_thr are kept up to this index
  // top-p state
  bool use_p;
  u64 p_thr;
  int p_cut;
};

__device__ __forceinline__ float z_from(const RowView& rv, float x) { return x / rv.T; }

__device__ __forceinline__ bool kept_k(const RowView& rv, float z, int i) {
  if (!rv.use_k) return true;
  const uint32_t k = float_key(z);
  return k > rv.k_thr || (k == rv.k_thr && i <= rv.k_cut);
}

__device__ __forceinline__ u64 fix_of(const RowView& rv, float z) {
  return (u64)(expf(z - rv.m) * FIX_ONE);
}

// The first index, in index order, at which the running sum of weight(i) exceeds `target`
// (`fallback` if the whole sum does not).  Each thread takes SCAN_E consecutive entries per
// round, so a round of the block covers 8192 entries with one scan.
#define SCAN_E 8
template <typename Weight>
__device__ int first_exceeding(const float* row, int V, u64 target, SampleShared& sm, int fallback,
                               Weight weight) {
  u64 carry = 0;
  int found = fallback;
  const bool vec = ((uintptr_t)row & 15) == 0;
  for (int base = 0; base < V; base += blockDim.x * SCAN_E) {
    const int i0 = base + threadIdx.x * SCAN_E;
    float x[SCAN_E];
    if (vec && i0 + SCAN_E <= V) {
      const float4 a = *reinterpret_cast<const float4*>(row + i0), b = *reinterpret_cast<const float4*>(row + i0 + 4);
      x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
      for (int e = 0; e < SCAN_E; ++e) x[e] = i0 + e < V ? row[i0 + e] : 0.0f;
    }
    u64 w[SCAN_E], mine = 0;
#pragma unroll
    for (int e = 0; e < SCAN_E; ++e) {
      w[e] = i0 + e < V ? weight(i0 + e, x[e]) : 0ull;
      mine += w[e];
    }
    u64 total;
    const u64 inc = blk_scan(mine, sm, &total) + carry;
    u64 run = inc - mine;
    if (mine && inc > target && run <= target) {   // the crossing lies in this thread's entries
#pragma unroll
      for (int e = 0; e < SCAN_E; ++e) {
        const bool before = run <= target;
        run += w[e];
        if (before && run > target) sm.bcast_int[0] = i0 + e;
      }
    }
    const bool done = carry + total > target;
    carry += total;
    __syncthreads();
    if (done) { found = sm.bcast_int[0]; break; }
  }
  __syncthreads();
  return found;
}

// Index of the `need`-th entry (1-based, in index order) for which pred holds.
template <typename Pred>
__device__ int nth_in_order(const float* row, int V, int need, SampleShared& sm, Pred pred) {
  return first_exceeding(row, V, (u64)(need - 1), sm, V - 1,
                         [&](int i, float x) { return pred(i, x) ? 1ull : 0ull; });
}

// One row by one block, walking it through memory.
__device__ __noinline__ void sample_row(const float* row, int V, float temperature, int top_k, float top_p, float r,
                                        int* out, SampleShared& sm) {
  const int tid = threadIdx.x;
  RowView rv;
  rv.row = row;
  rv.V = V;
  rv.T = temperature;
  rv.use_k = top_k > 0 && top_k < V;
  rv.use_p = top_p > 0.0f && top_p < 1.0f;
  rv.k_thr = 0u; rv.k_cut = V; rv.p_thr = 0ull; rv.p_cut = V;

  // ---- max of the scaled logits
  float m = -INFINITY;
  for_each_entry(rv.row, V, [&](int, float x, bool valid) {
    const float z = z_from(rv, x);
    if (valid && z == z) m = fmaxf(m, z);
  });
  rv.m = blk_max(m, sm);

  // ---- top-k: key of the k-th largest scaled logit by radix selection
  if (rv.use_k) {
    uint32_t prefix = 0u, mask = 0u;
    int remaining = top_k;
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (int b = tid; b < 256; b += blockDim.x) sm.cnt[b] = 0u;
      __syncthreads();
      for_each_entry(rv.row, V, [&](int, float x, bool valid) {   // whole warps: see warp_count
        const uint32_t k = float_key(z_from(rv, x));
        warp_count(sm.cnt, (valid && (k & mask) == prefix) ? (int)((k >> shift) & 255u) : -1);
      });
      __syncthreads();
      if (tid == 0) {
        int rem = remaining, b = 255;
        for (; b > 0; --b) {
          if ((int)sm.cnt[b] >= rem) break;
          rem -= (int)sm.cnt[b];
        }
        sm.bcast_int[0] = b;
        sm.bcast_int[1] = rem;
      }
      __syncthreads();
      prefix |= ((uint32_t)sm.bcast_int[0]) << shift;
      mask |= 255u << shift;
      remaining = sm.bcast_int[1];
      __syncthreads();
    }
    rv.k_thr = prefix;
    // `remaining` entries equal to the threshold are kept, lowest indices first
    const uint32_t thr = prefix;
    const RowView rvc = rv;
    rv.k_cut = nth_in_order(rv.row, V, remaining, sm,
                            [&](int, float x) { return float_key(z_from(rvc, x)) == thr; });
  }

  // ---- sum of the kept fixed-point weights
  u64 part = 0;
  for_each_entry(rv.row, V, [&](int i, float x, bool valid) {
    const float z = z_from(rv, x);
    if (valid && z == z && kept_k(rv, z, i)) part += fix_of(rv, z);
  });
  u64 S;
  blk_scan(part, sm, &S);
  __syncthreads();

  // ---- top-p: smallest weight that still belongs to the nucleus
  if (rv.use_p) {
    u64 target = (u64)ceil((double)top_p * (double)S);
    if (target > S) target = S;
    if (target < 1ull) target = 1ull;
    u64 prefix = 0ull, mask = 0ull, above = 0ull;  // `above` = weight strictly above the prefix
    for (int shift = 40; shift >= 0; shift -= 8) {
      for (int b = tid; b < 256; b += blockDim.x) { sm.cnt[b] = 0u; sm.wsum[b] = 0ull; }
      __syncthreads();
      for_each_entry(rv.row, V, [&](int i, float x, bool valid) {   // whole warps: see warp_count
        int b = -1;
        u64 w = 0;
        const float z = z_from(rv, x);
        if (valid && z == z && kept_k(rv, z, i)) {
          w = fix_of(rv, z);
          if ((w & mask) == prefix) b = (int)((w >> shift) & 255ull);
        }
        warp_count_weight(sm.cnt, sm.wsum, b, w);
      });
      __syncthreads();
      if (tid == 0) {
        u64 acc = above;
        int b = 255;
        for (; b > 0; --b) {
          if (acc + sm.wsum[b] >= target) break;
          acc += sm.wsum[b];
        }
        sm.bcast_int[0] = b;
        sm.bcast_u64[0] = acc;
      }
      __syncthreads();
      prefix |= ((u64)sm.bcast_int[0]) << shift;
      mask |= 255ull << shift;
      above = sm.bcast_u64[0];
      __syncthreads();
    }
    rv.p_thr = prefix;
    int need = 1;
    if (prefix > 0ull && target > above) {
      const u64 n = (target - above + prefix - 1ull) / prefix;
      need = n > (u64)V ? V : (int)n;
      if (need < 1) need = 1;
    }
    const RowView rvc = rv;
    const u64 thr = prefix;
    rv.p_cut = nth_in_order(rv.row, V, need, sm, [&](int i, float x) {
      const float z = z_from(rvc, x);
      return z == z && kept_k(rvc, z, i) && fix_of(rvc, z) == thr;
    });
    S = above + (u64)need * prefix;
  }

  // ---- draw: first kept index whose running weight exceeds floor(r * S)
  r = r < 0.0f ? 0.0f : (r >= 1.0f ? 0.99999994f : r);
  u64 target = (u64)((double)r * (double)S);
  if (target >= S) target = S ? S - 1ull : 0ull;
  const RowView rvd = rv;
  const int chosen = first_exceeding(rv.row, V, target, sm, -1, [&](int i, float x) {
    const float z = z_from(rvd, x);
    if (!(z == z) || !kept_k(rvd, z, i)) return 0ull;
    const u64 w = fix_of(rvd, z);
    if (rvd.use_p && !(w > rvd.p_thr || (w == rvd.p_thr && i <= rvd.p_cut))) return 0ull;
    return w;
  });
  if (tid == 0) *out = chosen >= 0 ? chosen : V - 1;  // the reference's fallback, :237
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int ld, int V, float temperature, int top_k,
              float top_p, const float* __restrict__ uniform, int* __restrict__ out) {
  __shared__ SampleShared sm;
  pdl_wait();
  pdl_launch_dependents();
  sample_row(logits + (size_t)blockIdx.x * ld, V, temperature, top_k, top_p, uniform[blockIdx.x], out + blockIdx.x, sm);
}

// --------------------------------------------------------------------------
// The same by a cluster of blocks per row, each thread with EPT consecutive entries of the row
// in registers.  The kernel above is bound by its passes over the row: ten to fifteen, 128 entries
// per thread of its one block at 131,072 entries, with the division, the exponential and the
// fixed-point weight again in each.  Here an entry is read, divided and turned into its weight
// once, a pass touches EPT registers, and what the blocks have to add up (histograms, sums,
// counts of ties) goes through distributed shared memory.  Measured, temperature / top-k 50 / top-p 0.95 / both,
// with the launch from Python: 8 rows of 131,072 entries 74 / 178 / 916 / 378 us by one block, 10 / 29 / 30 / 47 us
// here; 8 x 32,000: 21 / 63 / 306 / 145 and 9 / 18 / 22 / 32 us; 64 x 131,072: 80 / 202 / 968 / 407 and 31 / 100 / 78 /
// 138 us; 64 x 1000: 7 / 33 / 81 / 93 and 7 / 13 / 13 / 20 us.  What is left at top-p is the atomics of its first
// pass on shared memory and seven cluster barriers.
// --------------------------------------------------------------------------
// A block holds at most 32 x 1024 entries, so the sums of 16-bit pieces of its weights fit 32 bits, whose atomics
// on shared memory are single instructions (64-bit ones are loops: with them a top-k pass took twice as long).
// The first digit of top-k's selection is little more than the exponent: a warp's lanes share a few bins, and one of them
// adds for all that share its bin.  Later digits are spread, and every lane adds for itself.  Top-p's first digit is spread
// too: of the exponentials that have a weight, 2^-40 to 1, it is the exponent and five bits more, so that no lane has to
// look for others of its bin (finding them and adding three sums for each group of lanes was half of the kernel), and two
// digits of nine bits are left (8 x 131,072 69 -> 32 us, 64 x 131,072 250 -> 79, 64 x 32,000 67 -> 23, launched by a graph).  Its many
// bins are what small vocabularies pay for after top-k, whose few entries never crowded a bin: the sums of the
// blocks come over two bins to a load (8 x 32,000, both: 32 us with four digits of eight bits, 37 with a load per bin, 32).
#define SAMPLE_BINS 1312      // of the first digit of top-p: 41 powers of two in 32 parts
template <int ROOM>
__device__ __forceinline__ void part_add(uint32_t (*part)[ROOM], int bin, u64 w) {
  atomicAdd(&part[0][bin], (uint32_t)(w & 0xffffull));
  atomicAdd(&part[1][bin], (uint32_t)((w >> 16) & 0xffffull));
  atomicAdd(&part[2][bin], (uint32_t)(w >> 32));
}
template <bool SHARED_BINS, int ROOM>
__device__ __forceinline__ void part_count(uint32_t (*part)[ROOM], int bin) {
  if (SHARED_BINS) {
    if (!__any_sync(0xffffffffu, bin >= 0)) return;
    const unsigned peers = __match_any_sync(0xffffffffu, bin);
    if (bin >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&part[0][bin], (uint32_t)__popc(peers));
  } else if (bin >= 0) {
    atomicAdd(&part[0][bin], 1u);
  }
}

template <int ROOM>
struct ClusterShared {
  uint32_t part[3][ROOM];// the block's histogram as it grows: counts, or weights in pieces of 16, 16 and 9 bits
  alignas(16) u64 hist[2][ROOM];  // of this block; two in turn, so that one cluster barrier per exchange is enough
  u64 word[2][2];       // two numbers of this block, in turn likewise
  u64 pick[2];
  SampleShared blk;
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ u64 ld_peer_u64(const u64* local, uint32_t rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
  uint32_t r;
  u64 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(r) : "memory");
  return v;
}
__device__ __forceinline__ void ld_peer_2u64(const u64* local, uint32_t rank, u64& x, u64& y) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(local);
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(r) : "memory");
}

// What the blocks of a row exchange.  `turn` counts the exchanges of either kind: a buffer is written
// again two exchanges later, when the barrier between has seen every block past its reads.
template <int ROOM>
struct RowCluster {
  ClusterShared<ROOM>& sm;
  uint32_t rank, size;
  int turn;

  // The sums over the row's blocks of two numbers, and of the first one over the blocks before this one.
  // Every thread of a block passes the same numbers.
  __device__ void sums(u64 a, u64 b, u64* before_a, u64* total_a, u64* total_b) {
    u64* w = sm.word[turn & 1];
    ++turn;
    if (threadIdx.x == 0) { w[0] = a; w[1] = b; }
    cluster_barrier();
    u64 before = 0, ta = 0, tb = 0;
    for (uint32_t r = 0; r < size; ++r) {
      const u64 x = ld_peer_u64(w, r), y = ld_peer_u64(w + 1, r);
      if (r < rank) before += x;
      ta += x;
      tb += y;
    }
    *before_a = before; *total_a = ta; *total_b = tb;
  }
  __device__ float max(float m) {
    u64* w = sm.word[turn & 1];
    ++turn;
    if (threadIdx.x == 0) w[0] = (u64)__float_as_uint(m);
    cluster_barrier();
    for (uint32_t r = 0; r < size; ++r) m = fmaxf(m, __uint_as_float((uint32_t)ld_peer_u64(w, r)));
    return m;
  }
  template <int BINS>
  __device__ void clear() {
    if constexpr (BINS <= SAMPLE_THREADS) {
      if (threadIdx.x < BINS) sm.part[0][threadIdx.x] = sm.part[1][threadIdx.x] = sm.part[2][threadIdx.x] = 0u;
    } else {
      for (int b = threadIdx.x; b < BINS; b += SAMPLE_THREADS) sm.part[0][b] = sm.part[1][b] = sm.part[2][b] = 0u;
    }
    __syncthreads();
  }
  // The highest bin at which the sum from the top bin down, on top of `above`, reaches `target` (bin 0 if none
  // does); `above` then holds what lies above that bin.  With `share` the target is that share of the whole.
  template <int BINS>
  __device__ int choose(u64& above, u64& target, float share, bool share_given) {
    constexpr int PER = BINS <= SAMPLE_THREADS ? 1 : 2;       // bins per thread, from the top bin down
    static_assert(BINS <= 2 * SAMPLE_THREADS && (PER == 1 || BINS % 2 == 0), "a thread has one bin or a pair of them");
    u64* h = sm.hist[turn & 1];
    ++turn;
    __syncthreads();
    for (int b = threadIdx.x; b < BINS; b += SAMPLE_THREADS)
      h[b] = (u64)sm.part[0][b] + ((u64)sm.part[1][b] << 16) + ((u64)sm.part[2][b] << 32);
    cluster_barrier();
    const bool has = (int)threadIdx.x * PER < BINS;
    const int low = BINS - PER - (int)threadIdx.x * PER;      // the lower one of a thread's bins
    u64 v = 0, lower = 0;
    if (has)
      for (uint32_t r = 0; r < size; ++r) {
        if constexpr (PER == 1) {
          v += ld_peer_u64(h + low, r);
        } else {
          u64 x, y;
          ld_peer_2u64(h + low, r, x, y);
          lower += x;
          v += y;
        }
      }
    u64 total;
    const u64 over = above + blk_scan(v + lower, sm.blk, &total) - v - lower;
    if (share_given) {
      target = (u64)ceil((double)share * (double)total);
      if (target > total) target = total;
      if (target < 1ull) target = 1ull;
    }
    if (has && low == 0) { sm.pick[0] = 0ull; sm.pick[1] = over + (PER == 2 ? v : 0ull); }   // bin 0 unless another one takes it
    __syncthreads();
    if (has && over < target) {
      if (low + PER > 1 && over + v >= target) {
        sm.pick[0] = (u64)(low + PER - 1);
        sm.pick[1] = over;
      } else if (PER == 2 && low > 0 && over + v < target && over + v + lower >= target) {
        sm.pick[0] = (u64)low;
        sm.pick[1] = over + v;
      }
    }
    __syncthreads();
    above = sm.pick[1];
    const int bin = (int)sm.pick[0];
    __syncthreads();
    return bin;
  }
};

template <int EPT, bool TOP_K, bool TOP_P>
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_cluster_kernel(const float* __restrict__ logits, int ld, int V, float temperature, int top_k,
                      float top_p, const float* __restrict__ uniform, int* __restrict__ out) {
  constexpr int ROOM = TOP_P ? SAMPLE_BINS : 256;
  __shared__ ClusterShared<ROOM> sm;
  uint32_t rank, size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  RowCluster<ROOM> rc{sm, rank, size, 0};
  const int tid = threadIdx.x;
  const int r = blockIdx.x / size;
  const float* row = logits + (size_t)r * ld;
  const int i0 = ((int)rank * SAMPLE_THREADS + tid) * EPT;
  pdl_wait();

  // ---- the scaled logits, and their maximum
  float z[EPT];
  if (((uintptr_t)row & 15) == 0 && i0 + EPT <= V) {
#pragma unroll
    for (int e = 0; e < EPT; e += 4) {
      const float4 x = *reinterpret_cast<const float4*>(row + i0 + e);
      z[e] = x.x; z[e + 1] = x.y; z[e + 2] = x.z; z[e + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < EPT; ++e) z[e] = i0 + e < V ? row[i0 + e] : 0.0f;
  }
  pdl_launch_dependents();
  const int valid = min(max(V - i0, 0), EPT);     // this thread's entries
  float m = -INFINITY;
#pragma unroll
  for (int e = 0; e < EPT; ++e) {
    z[e] = z[e] / temperature;
    if (e < valid && z[e] == z[e]) m = fmaxf(m, z[e]);
  }
  m = rc.max(blk_max(m, sm.blk));
  if (!(m - m == 0.0f)) {
    // no finite maximum (an infinite logit, or none that is a number): the weights are no numbers; one block
    // walks the row, so that what comes out does not depend on the kernel
    if (rank == 0) sample_row(row, V, temperature, top_k, top_p, uniform[r], out + r, sm.blk);
    cluster_barrier();   // no block leaves while another reads its shared memory
    return;
  }

  // ---- top-k: key of the k-th largest scaled logit by radix selection
  const bool use_k = TOP_K && top_k > 0 && top_k < V;
  uint32_t dropped = 0;                           // bit e: not among the k largest
  if constexpr (TOP_K) if (use_k) {
    uint32_t prefix = 0u, mask = 0u;
    u64 above = 0, target = (u64)top_k;
    for (int shift = 24; shift >= 0; shift -= 8) {
      rc.template clear<256>();
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const uint32_t k = float_key(z[e]);
        const int bin = (e < valid && (k & mask) == prefix) ? (int)((k >> shift) & 255u) : -1;
        if (shift == 24) part_count<true>(sm.part, bin);
        else part_count<false>(sm.part, bin);
      }
      prefix |= (uint32_t)rc.template choose<256>(above, target, 0.0f, false) << shift;
      mask |= 255u << shift;
    }
    // target - above entries equal to the threshold are kept, lowest indices first
    u64 equal = 0, total, before, all, unused;
#pragma unroll
    for (int e = 0; e < EPT; ++e) equal += (e < valid && float_key(z[e]) == prefix) ? 1ull : 0ull;
    u64 inc = blk_scan(equal, sm.blk, &total);
    rc.sums(total, 0ull, &before, &all, &unused);
    u64 at = before + inc - equal;
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const uint32_t k = float_key(z[e]);
      if (k < prefix || (k == prefix && e < valid && at >= target - above)) dropped |= 1u << e;
      if (k == prefix && e < valid) ++at;
    }
  }

  // ---- weights of the kept entries; from here z[e] is exp(z - max), 0 where nothing is kept
#pragma unroll
  for (int e = 0; e < EPT; ++e) z[e] = (e < valid && z[e] == z[e] && !(dropped >> e & 1)) ? expf(z[e] - m) : 0.0f;
  auto weight = [](float e) { return (u64)(e * FIX_ONE); };

  // ---- top-p: the largest weight w such that the weights of w and above reach the share, by radix selection on
  // the bits of exp(z - max), which are in the order of the weights
  u64 S = 0;
  const bool use_p = TOP_P && top_p > 0.0f && top_p < 1.0f;
  if constexpr (TOP_P) if (use_p) {
    constexpr uint32_t least = 87u << 23;      // 2^-40: what lies below has no weight
    u64 above = 0, target = 0;
    rc.template clear<SAMPLE_BINS>();
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const uint32_t k = __float_as_uint(z[e]);
      if (k >= least) part_add(sm.part, (int)((k - least) >> 18), weight(z[e]));
    }
    uint32_t prefix = (uint32_t)rc.template choose<SAMPLE_BINS>(above, target, top_p, true);
#pragma unroll (EPT == 4 ? 1 : 2)      // (top-k at 8 x 32,000: 17.7 us with the loop, 18.9 without)
    for (int shift = 9; shift >= 0; shift -= 9) {
      rc.template clear<512>();
#pragma unroll
      for (int e = 0; e < EPT; ++e) {
        const uint32_t k = __float_as_uint(z[e]);
        if (k >= least && (k - least) >> (shift + 9) == prefix)
          part_add(sm.part, (int)((k - least) >> shift & 511u), weight(z[e]));
      }
      prefix = prefix << 9 | (uint32_t)rc.template choose<512>(above, target, 0.0f, false);
    }
    prefix += least;
    // small exponentials share a weight: ties are ties of the weight
    const u64 thr = weight(__uint_as_float(prefix));
    u64 over = 0, equal = 0, total, before, all, over_all;
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const u64 w = weight(z[e]);
      over += w > thr ? w : 0ull;
      equal += (w == thr && thr != 0ull) ? 1ull : 0ull;
    }
    blk_scan(over, sm.blk, &over_all);
    const u64 inc = blk_scan(equal, sm.blk, &total);
    rc.sums(total, over_all, &before, &all, &above);
    u64 need = 0;
    if (thr > 0ull) {
      need = target > above ? (target - above + thr - 1ull) / thr : 1ull;
      if (need < 1ull) need = 1ull;
    }
    u64 at = before + inc - equal;
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const u64 w = weight(z[e]);
      if (w < thr || (w == thr && at >= need)) z[e] = 0.0f;
      if (w == thr && thr != 0ull) ++at;
    }
    S = above + need * thr;
  }

  // ---- draw: first kept index whose running weight exceeds floor(u * S)
  u64 mine = 0, total, before, all, unused;
#pragma unroll
  for (int e = 0; e < EPT; ++e) mine += weight(z[e]);
  const u64 inc = blk_scan(mine, sm.blk, &total);
  rc.sums(total, 0ull, &before, &all, &unused);
  if (!use_p) S = all;
  float u = uniform[r];
  u = u < 0.0f ? 0.0f : (u >= 1.0f ? 0.99999994f : u);
  u64 target = (u64)((double)u * (double)S);
  if (target >= S) target = S ? S - 1ull : 0ull;
  u64 run = before + inc - mine;
  if (mine && run + mine > target && run <= target) {   // the crossing lies in this thread's entries
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const bool ahead = run <= target;
      run += weight(z[e]);
      if (ahead && run > target) out[r] = i0 + e;
    }
  }
  cluster_barrier();   // no block leaves while another reads its shared memory
}

template <int EPT, bool TOP_K, bool TOP_P>
static int launch_sample_cluster(int blocks_per_row, const float* logits, int ld, int rows, int V, float temperature,
                                 int top_k, float top_p, const float* uniform, int* out, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows * blocks_per_row);
  cfg.blockDim = dim3(SAMPLE_THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = blocks_per_row;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, sample_cluster_kernel<EPT, TOP_K, TOP_P>, logits, ld, V, temperature, top_k, top_p,
                                     uniform, out);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// One block per row, any vocabulary.  temperature must be > 0.
extern "C" int tl_sample_walk(const float* logits, int ld, int rows, int V, float temperature, int top_k,
                              float top_p, const float* uniform, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0 || !(temperature > 0.0f)) return -1;
  return tl_launch(sample_kernel, dim3(rows), dim3(SAMPLE_THREADS), 0, stream, logits, ld, V,
                   temperature, top_k, top_p, uniform, out);
}

// Whether walking the rows with one block each is faster than clusters of `blocks` blocks, `per` entries per thread.  What more
// clusters than run at once cost, they cost in rounds, while a row's walk takes its SM as long whatever the others do;
// top-p alone, whose walk takes many passes, always gains, and so do 16 entries per thread and fewer.  us (temperature alone /
// top-k / both): a round of clusters 17 / 55 / 84; a walk 5 + 0.00058 V / 22 + 0.00138 V / 78 + 0.00254 V, some more per row beyond
// 148 rows and beyond what the L2 cache holds.  Measured, clusters / walk: 148 rows of 200,000 entries 185 / 153, 609 / 382 and
// 928 / 740 us, 100 rows 130 / 125, 423 / 295, 643 / 586, 64 rows 92 / 122, 294 / 294, 452 / 591; 148 rows of 131,072 77 / 86, 268 /
// 206, 410 / 416; 300 of 32,000 53 / 49, 135 / 160, 222 / 399; 1000 of 5000 45 / 54, 116 / 213, 203 / 615.
static bool sample_walks(int rows, int V, int blocks, int per, bool use_k, bool use_p) {
  if ((use_p && !use_k) || per <= 16) return false;
  const int kind = use_p ? 2 : use_k ? 1 : 0;
  static const double round[3] = {17, 55, 84}, fixed[3] = {5, 22, 78}, entry[3] = {0.58e-3, 1.38e-3, 2.54e-3};
  const int at_once = blocks == 1 ? 148 : blocks == 2 ? 74 : blocks == 4 ? 33 : 15;
  double clusters = blocks == 1 && kind == 1 ? 50.0 : round[kind];
  clusters *= (rows + at_once - 1) / at_once * (blocks == 8 ? 1.08 : blocks == 4 ? 0.96 : 1.0);
  double walk = fixed[kind] + entry[kind] * V;
  if (rows > 148) walk *= kind == 0 ? 0.35 + 0.9 * rows / 148 : 0.47 + 0.95 * rows / 148;
  if ((double)rows * V > 2.2e7) walk *= 1.2;
  return walk < clusters;
}

#define SAMPLE_MAX_CLUSTER 8   // portable cluster size
// The blocks per row and the entries per thread, or false if the rows are walked.
// As many blocks per row as give a thread four entries, at most 8 and no more than run at once (a block fills an
// SM), but enough that 32 entries per thread cover the row: a pass costs what a thread holds, a barrier of eight
// blocks little more than one of two, and a second round of blocks as much as the first.
static bool sample_plan(int rows, int V, int top_k, float top_p, int* blocks, int* per) {
  int n = 1;
  while (n < SAMPLE_MAX_CLUSTER && n * SAMPLE_THREADS * 4 < V &&
         (n * SAMPLE_THREADS * 32 < V || (long long)rows * n * 2 <= 148))
    n *= 2;
  *blocks = n;
  *per = (V + n * SAMPLE_THREADS - 1) / (n * SAMPLE_THREADS);
  return *per <= 32 && !sample_walks(rows, V, n, *per, top_k > 0 && top_k < V, top_p > 0.0f && top_p < 1.0f);
}

// temperature must be > 0; rows with temperature <= 0 go through tl_argmax.
extern "C" int tl_sample(const float* logits, int ld, int rows, int V, float temperature,
                         int top_k, float top_p, const float* uniform, int* out,
                         cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (V <= 0 || !(temperature > 0.0f)) return -1;
  int blocks, per;
  if (!sample_plan(rows, V, top_k, top_p, &blocks, &per))
    return tl_sample_walk(logits, ld, rows, V, temperature, top_k, top_p, uniform, out, stream);
#define SAMPLE_CLUSTER(EPT_, K_, P_) \
  return launch_sample_cluster<EPT_, K_, P_>(blocks, logits, ld, rows, V, temperature, top_k, top_p, uniform, out, stream)
  // A kernel that can do everything, but for two: the registers that a digit's sums take from top-k and temperature cost top-k 4 % at
  // 16 entries per thread (8 x 70,000: 30.8 us, 29.9 without top-p) and temperature 3 % at 32 (64 x 131,072: 31.6 and 30.8).
  const bool use_k = top_k > 0 && top_k < V, use_p = top_p > 0.0f && top_p < 1.0f;
  if (per <= 4) SAMPLE_CLUSTER(4, true, true);
  if (per <= 8) SAMPLE_CLUSTER(8, true, true);
  if (per <= 16 && use_p) SAMPLE_CLUSTER(16, true, true);
  if (per <= 16) SAMPLE_CLUSTER(16, true, false);
  if (use_k || use_p) SAMPLE_CLUSTER(32, true, true);
  SAMPLE_CLUSTER(32, false, false);
#undef SAMPLE_CLUSTER
}

// Blocks per row, or 0 if the rows are walked (for the test of the rule).
extern "C" int tl_sample_route(int rows, int V, int top_k, float top_p) {
  int blocks, per;
  return sample_plan(rows, V, top_k, top_p, &blocks, &per) ? blocks : 0;
}

TL_TRACE_EXPORT(sampling)
