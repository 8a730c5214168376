// Attention over the paged cache in 32-bit, on CUDA cores, for head sizes 16, 32, 64 and 128
// (reference: scores, softmax and weighted sum of src/model/modules/attention.rs:78-121; window inequality of
// src/model/models/gpt_oss.rs:168-176).  A query at position p sees the keys i in [max(0, p - W + 1), p] with a window W,
// else [0, p].  Everything is 32-bit: products, sums, running maximum and sum of the softmax.
//
// The kernel for every head size (attention_generic.cu) gives a block to each (token, query head); every block reads
// its keys and values by itself, the values (transposed in their pages) 32 bytes for 4.  Both kernels here bring whole
// pages into shared memory with 16-byte copies and use them for all query heads that share them:
//   prompts  64 rows per block, (tokens) x (query heads of one key/value head), in tiles of 64 keys: the two products as
//            register tiles of 4 x 4 and 4 x (head size / 16) per thread, operands by 16-byte loads along the contracted
//            dimension.  The next page's keys arrive during the softmax and P.V, its values during Q.K^T.  Bound by the
//            multiply-adds and the shared memory reads that feed them (2 of 16 bytes per 16 multiply-adds).
//   decode   a run of pages of one sequence and key/value head per block, two pages in flight, all query heads of the
//            group; blocks of one sequence merge through a second kernel.  Bound by the pages' bytes.
// Measured, 32 heads over 8 of 128, by the kernel for every head size / here: prompts of 400 and 131 tokens 1770 / 99 us, one
// of 2000 tokens 38,086 / 1152 us (28 of some 70 TFLOP/s); one token each of four sequences of 500 to 2000 tokens 244 / 26 us
// with the merge (5.5 at the copy rate), of eight of 4000 tokens 760 / 100 us (40); 20 tokens after 980 440 / 161 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "per_device.cuh"

#define PAGE 64
static_assert(TL_PAGE == PAGE, "the tiles are pages of 64 keys");

__device__ __forceinline__ void cp16(void* smem, const void* gmem, int bytes) {   // the rest of the 16 bytes become zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Row strides in shared memory: one 16-byte unit more than the row, so that rows of neighbouring lanes fall on
// different banks.
template <int HD> struct Sizes {
  static constexpr int KLD = HD + 4, VLD = PAGE + 4;
  static constexpr int K = PAGE * KLD, V = HD * VLD;      // floats of a page's keys and of its values
};

// Copies the keys (rows) or values (columns) of a page up to the place `last` in it; what lies beyond becomes zero.
template <int HD, int THREADS>
__device__ __forceinline__ void load_keys(float* dst, const float* page, int last) {
  for (int i = threadIdx.x; i < PAGE * (HD / 4); i += THREADS) {
    const int key = i / (HD / 4), c = i % (HD / 4);
    cp16(dst + key * Sizes<HD>::KLD + 4 * c, page + key * HD + 4 * c, key <= last ? 16 : 0);
  }
}
template <int HD, int THREADS>
__device__ __forceinline__ void load_values(float* dst, const float* page, int last) {
  for (int i = threadIdx.x; i < HD * (PAGE / 4); i += THREADS) {
    const int d = i / (PAGE / 4), c = i % (PAGE / 4);
    const int n = min(max(last + 1 - 4 * c, 0), 4);
    cp16(dst + d * Sizes<HD>::VLD + 4 * c, page + d * PAGE + 4 * c, 4 * n);
  }
}

struct AttnArgs {
  const float* q;          // [tokens, nh * HD]
  const float* k_pages;    // [pages, nkv, 64, HD]
  const float* v_pages;    // [pages, nkv, HD, 64]
  float* out;
  const int* seq_start;
  const int* seq_len;
  const int* seq_slot;
  const int* page_table;
  int table_stride, nh, nkv, window;
  float scale;
  float* part;             // decode: [sequences, nkv, splits, group, HD + 2]
  int pages_per_block, splits;
};

#define P_THREADS 256
#define P_ROWS 64

template <int HD>
__global__ void __launch_bounds__(P_THREADS)
attn_f32_prompt_kernel(const AttnArgs a, int tokens_per_block) {
  constexpr int DJ = HD / 16;     // dimensions per thread
  constexpr int KLD = Sizes<HD>::KLD, VLD = Sizes<HD>::VLD;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                       // [64][KLD]
  float* Ks = Qs + P_ROWS * KLD;        // [64][KLD]
  float* Vs = Ks + Sizes<HD>::K;        // [HD][VLD]
  float* Ps = Vs + Sizes<HD>::V;        // [64][VLD]
  pdl_wait();
  const int b = blockIdx.z, kvh = blockIdx.y, group = a.nh / a.nkv;
  const int tile = gridDim.x - 1 - blockIdx.x;      // the tiles with most keys first
  const int first = a.seq_start[b], n_new = a.seq_start[b + 1] - first;
  const int t0 = tile * tokens_per_block;
  if (t0 >= n_new) return;
  const int tokens = min(tokens_per_block, n_new - t0), rows = tokens * group;
  const int p0 = a.seq_len[b] - n_new + t0, p_last = p0 + tokens - 1;     // positions of the block's tokens
  const int lo = a.window > 0 ? max(p0 - a.window + 1, 0) : 0;
  const int pg0 = lo / PAGE, n_pg = p_last / PAGE - pg0 + 1;
  const int* table = a.page_table + (size_t)a.seq_slot[b] * a.table_stride + pg0;
  const size_t page_floats = (size_t)a.nkv * PAGE * HD, head_off = (size_t)kvh * PAGE * HD;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;

  for (int i = tid; i < P_ROWS * (HD / 4); i += P_THREADS) {
    const int r = i / (HD / 4), c = i % (HD / 4);
    const bool live = r < rows;
    const float* src = a.q + ((size_t)(first + t0 + (live ? r / group : 0)) * a.nh + kvh * group + (live ? r % group : 0)) * HD + 4 * c;
    cp16(Qs + r * KLD + 4 * c, src, live ? 16 : 0);
  }
  auto keys = [&](int i) {
    if (i < n_pg) load_keys<HD, P_THREADS>(Ks, a.k_pages + (size_t)table[i] * page_floats + head_off, p_last - (pg0 + i) * PAGE);
    cp_commit();
  };
  auto values = [&](int i) {
    if (i < n_pg) load_values<HD, P_THREADS>(Vs, a.v_pages + (size_t)table[i] * page_floats + head_off, p_last - (pg0 + i) * PAGE);
    cp_commit();
  };
  keys(0);
  values(0);

  int pos[4];
  float m_run[4], l_run[4], acc[4][DJ];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    pos[i] = p0 + (ty * 4 + i) / group;
    m_run[i] = -INFINITY;
    l_run[i] = 0.0f;
#pragma unroll
    for (int j = 0; j < DJ; ++j) acc[i][j] = 0.0f;
  }
  for (int pg = 0; pg < n_pg; ++pg) {
    const int key0 = (pg0 + pg) * PAGE;
    const bool masked = key0 + PAGE - 1 > p0 || (a.window > 0 && key0 < p_last - a.window + 1);
    cp_wait<1>();          // the page's keys (and the queries); its values may still be on their way
    __syncthreads();
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 4
    for (int d = 0; d < HD; d += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(Qs + (ty * 4 + i) * KLD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * KLD + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(qv[i].x, kv[j].x, s[i][j]);
          s[i][j] = fmaf(qv[i].y, kv[j].y, s[i][j]);
          s[i][j] = fmaf(qv[i].z, kv[j].z, s[i][j]);
          s[i][j] = fmaf(qv[i].w, kv[j].w, s[i][j]);
        }
    }
    __syncthreads();       // the keys are used up
    keys(pg + 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float m = m_run[i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = key0 + tx + 16 * j;
        const bool seen = !masked || (key <= pos[i] && (a.window <= 0 || key > pos[i] - a.window));
        s[i][j] = seen ? s[i][j] * a.scale : -INFINITY;
        m = fmaxf(m, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      const float base = m == -INFINITY ? 0.0f : m;     // (no key seen yet: every weight is 0)
      const float alpha = expf(m_run[i] - base);
      m_run[i] = m;
      l_run[i] *= alpha;
#pragma unroll
      for (int j = 0; j < DJ; ++j) acc[i][j] *= alpha;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = expf(s[i][j] - base);
        l_run[i] += p;
        Ps[(ty * 4 + i) * VLD + tx + 16 * j] = p;
      }
    }
    if (masked) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = key0 + tx + 16 * j;
          if (key > pos[i] || (a.window > 0 && key <= pos[i] - a.window)) Ps[(ty * 4 + i) * VLD + tx + 16 * j] = -1.0f;
        }
    }
    cp_wait<1>();          // the page's values
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < PAGE; k += 4) {
      float4 pv[4], vv[DJ];
#pragma unroll
      for (int i = 0; i < 4; ++i) pv[i] = *reinterpret_cast<const float4*>(Ps + (ty * 4 + i) * VLD + k);
#pragma unroll
      for (int j = 0; j < DJ; ++j) vv[j] = *reinterpret_cast<const float4*>(Vs + (tx + 16 * j) * VLD + k);
      if (masked) {
        // a value that a row does not see (weight -1) must not reach it, whatever it is; one that it does see counts, however
        // small its weight
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < DJ; ++j) {
            if (!(pv[i].x < 0.0f)) acc[i][j] = fmaf(pv[i].x, vv[j].x, acc[i][j]);
            if (!(pv[i].y < 0.0f)) acc[i][j] = fmaf(pv[i].y, vv[j].y, acc[i][j]);
            if (!(pv[i].z < 0.0f)) acc[i][j] = fmaf(pv[i].z, vv[j].z, acc[i][j]);
            if (!(pv[i].w < 0.0f)) acc[i][j] = fmaf(pv[i].w, vv[j].w, acc[i][j]);
          }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < DJ; ++j) {
            acc[i][j] = fmaf(pv[i].x, vv[j].x, acc[i][j]);
            acc[i][j] = fmaf(pv[i].y, vv[j].y, acc[i][j]);
            acc[i][j] = fmaf(pv[i].z, vv[j].z, acc[i][j]);
            acc[i][j] = fmaf(pv[i].w, vv[j].w, acc[i][j]);
          }
      }
    }
    __syncthreads();       // the values and the weights are used up
    values(pg + 1);
  }
  pdl_launch_dependents();
  cp_wait<0>();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float l = l_run[i];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const int r = ty * 4 + i;
    if (r < rows) {
      float* o = a.out + ((size_t)(first + t0 + r / group) * a.nh + kvh * group + r % group) * HD;
#pragma unroll
      for (int j = 0; j < DJ; ++j) o[tx + 16 * j] = acc[i][j] / l;
    }
  }
}

#define D_THREADS 128

// GM: query heads per key/value head, rounded up.
template <int HD, int GM>
__global__ void __launch_bounds__(D_THREADS)
attn_f32_decode_kernel(const AttnArgs a) {
  constexpr int KLD = Sizes<HD>::KLD, VLD = Sizes<HD>::VLD;
  constexpr int PARTS = D_THREADS / HD;               // threads that share a dimension of P.V, each some of the keys
  extern __shared__ __align__(16) float sm[];
  float* Ks = sm;                                     // [2][64][KLD]
  float* Vs = Ks + 2 * Sizes<HD>::K;                  // [2][HD][VLD]
  float* Qs = Vs + 2 * Sizes<HD>::V;                  // [GM][HD]
  float* Ss = Qs + GM * HD;                           // [2][GM][64] halves of the scores; then the weights in the first
  float* Os = Ss + 2 * GM * PAGE;                     // [GM][128] partial outputs
  float* alpha_s = Os + GM * D_THREADS;               // [GM], then the running maximum and sum of each head
  float* m_s = alpha_s + GM;
  float* l_s = m_s + GM;
  pdl_wait();
  pdl_launch_dependents();   // (at once: in a small model's step the next kernel's launch is what this one hides)
  const int b = blockIdx.z, kvh = blockIdx.y, split = blockIdx.x, group = a.nh / a.nkv;
  const int pos = a.seq_len[b] - 1;
  const int lo = a.window > 0 ? max(pos - a.window + 1, 0) : 0;
  const int n_pg = pos / PAGE - lo / PAGE + 1;
  const int begin = split * a.pages_per_block, end = min(begin + a.pages_per_block, n_pg);
  if (begin >= end) return;
  const int pg0 = lo / PAGE;
  const int* table = a.page_table + (size_t)a.seq_slot[b] * a.table_stride + pg0;
  const size_t page_floats = (size_t)a.nkv * PAGE * HD, head_off = (size_t)kvh * PAGE * HD;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int token = a.seq_start[b];
  auto fetch = [&](int i, int at) {
    if (i < end) {
      const size_t off = (size_t)table[i] * page_floats + head_off;
      const int last = pos - (pg0 + i) * PAGE;
      load_keys<HD, D_THREADS>(Ks + at * Sizes<HD>::K, a.k_pages + off, last);
      load_values<HD, D_THREADS>(Vs + at * Sizes<HD>::V, a.v_pages + off, last);
    }
    cp_commit();
  };
  fetch(begin, 0);
  fetch(begin + 1, 1);
  for (int i = tid; i < GM * HD; i += D_THREADS)
    Qs[i] = i < group * HD ? a.q[((size_t)token * a.nh + kvh * group) * HD + i] : 0.0f;
  if (tid < GM) { m_s[tid] = -INFINITY; l_s[tid] = 0.0f; }
  float acc[GM];
#pragma unroll
  for (int g = 0; g < GM; ++g) acc[g] = 0.0f;
  const int key = tid & 63, half = tid >> 6;
  const int d = tid % HD, part = tid / HD;
  for (int i = begin; i < end; ++i) {
    const int at = (i - begin) & 1, key0 = (pg0 + i) * PAGE;
    cp_wait<1>();
    __syncthreads();
    // values that have left the window must not reach the sum, whatever they are: 0 x NaN is NaN
    for (int e = part; e < lo - key0; e += PARTS) Vs[at * Sizes<HD>::V + d * VLD + e] = 0.0f;
    {
      // a key and half of the dimensions per thread
      float s[GM];
#pragma unroll
      for (int g = 0; g < GM; ++g) s[g] = 0.0f;
      const float* kr = Ks + at * Sizes<HD>::K + key * KLD + half * (HD / 2);
#pragma unroll 4
      for (int e = 0; e < HD / 2; e += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(kr + e);
#pragma unroll
        for (int g = 0; g < GM; ++g) {
          const float4 qv = *reinterpret_cast<const float4*>(Qs + g * HD + half * (HD / 2) + e);
          s[g] = fmaf(qv.x, kv.x, s[g]);
          s[g] = fmaf(qv.y, kv.y, s[g]);
          s[g] = fmaf(qv.z, kv.z, s[g]);
          s[g] = fmaf(qv.w, kv.w, s[g]);
        }
      }
#pragma unroll
      for (int g = 0; g < GM; ++g) Ss[(half * GM + g) * PAGE + key] = s[g];
    }
    __syncthreads();
    for (int g = warp; g < GM; g += D_THREADS / 32) {   // a warp per head, two keys per lane
      float s[2], m = m_s[g];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h, at_key = key0 + k;
        s[h] = at_key <= pos && at_key >= lo ? (Ss[g * PAGE + k] + Ss[(GM + g) * PAGE + k]) * a.scale : -INFINITY;
        m = fmaxf(m, s[h]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      float p[2], sum;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        p[h] = s[h] == -INFINITY ? 0.0f : expf(s[h] - m);
        Ss[g * PAGE + lane + 32 * h] = p[h];
      }
      sum = p[0] + p[1];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      __syncwarp();
      if (lane == 0) {
        const float alpha = m_s[g] == -INFINITY ? 0.0f : expf(m_s[g] - m);
        alpha_s[g] = alpha;
        l_s[g] = l_s[g] * alpha + sum;
        m_s[g] = m;
      }
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < GM; ++g) acc[g] *= alpha_s[g];
    const float* vr = Vs + at * Sizes<HD>::V + d * VLD + part * (PAGE / PARTS);
#pragma unroll 4
    for (int e = 0; e < PAGE / PARTS; e += 4) {
      const float4 vv = *reinterpret_cast<const float4*>(vr + e);
#pragma unroll
      for (int g = 0; g < GM; ++g) {
        const float4 pv = *reinterpret_cast<const float4*>(Ss + g * PAGE + part * (PAGE / PARTS) + e);
        acc[g] = fmaf(pv.x, vv.x, acc[g]);
        acc[g] = fmaf(pv.y, vv.y, acc[g]);
        acc[g] = fmaf(pv.z, vv.z, acc[g]);
        acc[g] = fmaf(pv.w, vv.w, acc[g]);
      }
    }
    __syncthreads();       // the page and its weights are used up
    fetch(i + 2, at);
  }
  cp_wait<0>();
#pragma unroll
  for (int g = 0; g < GM; ++g) Os[g * D_THREADS + tid] = acc[g];
  __syncthreads();
  for (int i = tid; i < group * HD; i += D_THREADS) {
    const int g = i / HD, e = i % HD;
    float o = 0.0f;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) o += Os[g * D_THREADS + p * HD + e];
    if (a.splits == 1) {
      a.out[((size_t)token * a.nh + kvh * group + g) * HD + e] = o / l_s[g];
    } else {
      float* dst = a.part + ((((size_t)b * a.nkv + kvh) * a.splits + split) * group + g) * (HD + 2);
      dst[e] = o;
      if (e == 0) { dst[HD] = m_s[g]; dst[HD + 1] = l_s[g]; }
    }
  }
}

// A block per (head, sequence), a thread per dimension: the splits in their order.
template <int HD>
__global__ void __launch_bounds__(HD)
attn_f32_merge_kernel(const AttnArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.x, b = blockIdx.y, group = a.nh / a.nkv, kvh = h / group, g = h % group, e = threadIdx.x;
  const int pos = a.seq_len[b] - 1;
  const int lo = a.window > 0 ? max(pos - a.window + 1, 0) : 0;
  const int n_pg = pos / PAGE - lo / PAGE + 1;
  const int n = (n_pg + a.pages_per_block - 1) / a.pages_per_block;
  const float* src = a.part + (((size_t)b * a.nkv + kvh) * a.splits * group + g) * (HD + 2);
  const size_t step = (size_t)group * (HD + 2);
  float m = -INFINITY;
  for (int s = 0; s < n; ++s) m = fmaxf(m, src[s * step + HD]);
  float o = 0.0f, l = 0.0f;
#pragma unroll 4
  for (int s = 0; s < n; ++s) {
    const float f = src[s * step + HD] == -INFINITY ? 0.0f : expf(src[s * step + HD] - m);
    o = fmaf(f, src[s * step + e], o);
    l = fmaf(f, src[s * step + HD + 1], l);
  }
  a.out[((size_t)a.seq_start[b] * a.nh + h) * HD + e] = o / l;
}

template <int HD>
static int run_prompt(const AttnArgs& a, int seqs, int max_new, cudaStream_t stream) {
  const int smem = (2 * P_ROWS * Sizes<HD>::KLD + Sizes<HD>::V + P_ROWS * Sizes<HD>::VLD) * 4;
  const cudaError_t set = tl_allow_smem<attn_f32_prompt_kernel<HD>>(smem);
  if (set != cudaSuccess) return (int)set;
  const int per = P_ROWS / (a.nh / a.nkv);
  return tl_launch(attn_f32_prompt_kernel<HD>, dim3((max_new + per - 1) / per, a.nkv, seqs), dim3(P_THREADS), (size_t)smem, stream, a, per);
}
template <int HD, int GM>
static int run_decode(const AttnArgs& a, int seqs, cudaStream_t stream) {
  const int smem = (2 * Sizes<HD>::K + 2 * Sizes<HD>::V + GM * (HD + 2 * PAGE + D_THREADS + 3)) * 4;
  const cudaError_t set = tl_allow_smem<attn_f32_decode_kernel<HD, GM>>(smem);
  if (set != cudaSuccess) return (int)set;
  int rc = tl_launch(attn_f32_decode_kernel<HD, GM>, dim3(a.splits, a.nkv, seqs), dim3(D_THREADS), (size_t)smem, stream, a);
  if (rc == 0 && a.splits > 1) rc = tl_launch(attn_f32_merge_kernel<HD>, dim3(a.nh, seqs), dim3(HD), 0, stream, a);
  return rc;
}
template <int HD>
static int run_heads(const AttnArgs& a, int seqs, int max_new, int decode, cudaStream_t stream) {
  const int group = a.nh / a.nkv;
  if (!decode) return group <= P_ROWS ? run_prompt<HD>(a, seqs, max_new, stream) : -2;
  if (group <= 1) return run_decode<HD, 1>(a, seqs, stream);
  if (group <= 2) return run_decode<HD, 2>(a, seqs, stream);
  if (group <= 4) return run_decode<HD, 4>(a, seqs, stream);
  if (group <= 8) return run_decode<HD, 8>(a, seqs, stream);
  return -2;
}

// `decode`: every sequence brings one token; the keys of a sequence are then shared out over blocks of
// `pages_per_block` pages, at most `splits` of them (what the longest sequence needs), and `part` holds
// sequences * nh * splits * (hd + 2) floats if splits > 1.  Returns 0, a CUDA error, or -2 for sizes that are not taken.
extern "C" int tl_attn_f32(const float* q, const float* k_pages, const float* v_pages, float* out, const int* seq_start,
                           const int* seq_len, const int* seq_slot, const int* page_table, int table_stride, int seqs,
                           int max_new, int nh, int nkv, int hd, int window, float scale, int decode, float* part,
                           int pages_per_block, int splits, cudaStream_t stream) {
  if (seqs <= 0 || max_new <= 0) return 0;
  if (nkv <= 0 || nh % nkv || (decode && (pages_per_block < 1 || splits < 1 || (splits > 1 && !part)))) return -1;
  if (seqs > 65535 || nkv > 65535) return -2;
  if (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) return -2;
  AttnArgs a = {q, k_pages, v_pages, out, seq_start, seq_len, seq_slot, page_table, table_stride, nh, nkv, window,
                scale, part, pages_per_block, splits};
  switch (hd) {
    case 16: return run_heads<16>(a, seqs, max_new, decode, stream);
    case 32: return run_heads<32>(a, seqs, max_new, decode, stream);
    case 64: return run_heads<64>(a, seqs, max_new, decode, stream);
    case 128: return run_heads<128>(a, seqs, max_new, decode, stream);
  }
  return -2;
}
