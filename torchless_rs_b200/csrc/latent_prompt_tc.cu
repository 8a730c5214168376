// Latent attention (latent_attention.cu says what it computes) of steps whose sequences all start with them, with every
// head's keys and values formed: k_h = [W_uk,h c | r], v_h = W_uv,h c, for heads of 128 plain entries, at most 64 rotated
// ones and values of 128.
//
// Against the positions' vectors [c | r] a query costs 576 + 512 multiply-adds per key and head (latents of 512), and all
// heads' sums of 512 columns have to go through tensor memory and a product per head after it.  With the keys formed it is
// 192 + 128, and forming them costs two small products per token, which a prompt's queries share.  They are formed from
// the step's own latents, which `latent_prep` leaves in token order, so a step that continues a sequence, and would have
// to form the keys of all it has seen, runs on the kernels of [c | r].  Measured, 16 heads, one prompt, the whole mixer on
// [c | r] / here: 300 tokens 107 / 73 us, 2048 390 / 157, 4096 960 / 289; of that this kernel 22, 55 and 128 us.
//
// A block owns 128 consecutive queries of one head and walks over the keys they see, 64 at a time:
//   warps 0-3  softmax, a row per thread
//   warp 4     TMA: a chunk's k_h and r beside it (one slot, free again after Q . K^T), v_h (two slots)
//   warp 5     issues Q . K^T, up to two chunks ahead (two S buffers)
//   warp 6     issues P . V: P from tensor memory, V's rows read across (the positions are the contracted dimension)
// and the blocks of an SM, two of them, fill each other's waits.  What bounds it is the chain of a chunk: at 2048 tokens and 16 heads
// all 256 blocks run at once, and the longest takes some 1.5 us for each of its 32 chunks (scores out of tensor memory, the
// exponentials, O times what the maximum moved by, the weights back) while the tensor pipe is busy for 20 % of the cycles, the issue
// slots for 35 and the loads from shared memory for 3.  (Two slots of keys and
// one of values: 74 us instead of 66 for 2048 tokens and 16 heads, both as first written.  One block an SM of two tiles
// that share their keys: 68 us against 52 then, because at 2048 tokens the longest blocks are left alone.)  The queries are turned,
// scaled and rounded on their way into shared memory, and O / l leaves through it, gated, a warp per row.
//
// l sums the weights as they were rounded, so that where few keys count their rounding cancels.
//
// Every wait on an mbarrier is bounded; when a bound is hit the block records a code in tl_latent_prompt_error, stops,
// frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "per_device.cuh"
#include "umma.cuh"

#include <mutex>

#define LP_THREADS 224
#define LP_ROWS 128
#define LP_KEYS 64
#define LP_DIM 128                          // plain entries of a head's query and key
#define LP_ROT 64                           // room for rotated entries
#define LP_VDIM 128
#define LP_QSUB (LP_ROWS * 128)             // bytes of 64 columns of a tile's queries
#define LP_KSUB (LP_KEYS * 128)             // bytes of 64 columns of a chunk
#define LP_Q (3 * LP_QSUB)
#define LP_K (3 * LP_KSUB)
#define LP_V (2 * LP_KSUB)
#define LP_VSLOTS 2
#define LP_OLD (LP_VDIM + 4)                // floats of a row of the result in shared memory (over the queries and keys)
#define LP_BATCH 6                          // rows whose loads a warp has in flight

// The block's memory starts where it is declared to, on the swizzle's boundary.  (Rounded up at run time, as the other kernels do
// it, the addresses are no constants any more: 512 tokens 29.9 us instead of 26.4, 2048 tokens 59 instead of 55.)  The kernel
// looks all the same: a block whose memory lay elsewhere would say so in tl_latent_prompt_error, which the host raises.
#define LP_SMEM (LP_Q + LP_K + LP_VSLOTS * LP_V + 256)
static_assert(LP_ROWS * LP_OLD * 4 <= LP_Q + LP_K, "the results lie where the queries and keys lay");
#define LP_COL_O (2 * LP_KEYS)              // tensor memory: two S buffers, then O
#define LP_TMEM 256

__device__ int tl_latent_prompt_error = 0;

__device__ __forceinline__ bool lp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  return tl_mbar_park(bar, parity, abort_flag, code, &tl_latent_prompt_error);
}
__device__ __forceinline__ void lp_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void lp_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void lp_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void lp_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void lp_umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ float lp_ex2(float x) {   // 2^x, one instruction; tiny results flush to zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t lp_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float lp_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
// Two 32-bit floats in one 64-bit register, and the packed addition of sm_100 on them.
__device__ __forceinline__ uint64_t lp_pack2(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void lp_unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t lp_add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float lp_max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
// Rows of 64 positions read across them: 64 columns contiguous (128 bytes, 128-byte swizzle), the next 64 columns a
// sub-tile further, eight positions 1024 bytes further.
__device__ __forceinline__ uint64_t lp_desc_v(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)(LP_KSUB >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// The tensor core multiplies a weight of 0 like any other, and 0 x NaN is NaN.  So in a chunk that not every row of the block
// sees whole, the numbers of positions outside [seen_lo, seen_hi] (what all rows see) that are not finite are set to zero
// before P . V.  By the 128 softmax threads, eight to a position; true if this thread cleared one of a position that some row
// does see, in [some_lo, some_hi]: the caller adds it to that row's result.
__device__ __forceinline__ bool lp_clear_unseen(uint8_t* v, int key0, int seen_lo, int seen_hi, int some_lo, int some_hi) {
  bool found = false;
#pragma unroll
  for (int k = (int)(threadIdx.x >> 3); k < LP_KEYS; k += LP_ROWS / 8) {
    const int key = key0 + k;
    if (key >= seen_lo && key <= seen_hi) continue;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint4* at = reinterpret_cast<uint4*>(v + u * LP_KSUB + k * 128 + (threadIdx.x & 7) * 16);
      const uint4 x = *at;
      // an exponent of all ones carries into the bit above it
      auto bad = [](uint32_t w) { return (((w & 0x7f807f80u) + 0x00800080u) >> 15 & 0x00010001u) * 0xffffu; };
      const uint4 m = make_uint4(bad(x.x), bad(x.y), bad(x.z), bad(x.w));
      if (m.x | m.y | m.z | m.w) {
        *at = make_uint4(x.x & ~m.x, x.y & ~m.y, x.z & ~m.z, x.w & ~m.w);
        found |= key >= some_lo && key <= some_hi;
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor core reads the chunk as it is now
  return found;
}

struct LatentPromptArgs {
  const float* q;             // [T, ldq]: head h's entries at column h * (LP_DIM + rot)
  const float2* turn;         // [T, dims / 2] cosine and sine of every token's angles
  const __nv_bfloat16* kv;    // [T, 2 * heads * 128]: all heads' keys, then all heads' values
  __nv_bfloat16* out;         // [T, heads * 128]
  const float* gate;          // null, [T, ldg] per entry, or per head
  const float* sink;          // [heads] or null
  const int* seq_start;
  int ldq, ldg, gate_one, heads, rot, dims, window;
  float scale_log2;
};

__global__ void __launch_bounds__(LP_THREADS, 2)
latent_prompt_tc_kernel(const __grid_constant__ CUtensorMap tm_kv, const __grid_constant__ CUtensorMap tm_r,
                        const LatentPromptArgs a) {
  extern __shared__ __align__(1024) uint8_t lp_smem[];
  uint8_t* q_s = lp_smem;
  float* o_s = reinterpret_cast<float*>(lp_smem);
  uint8_t* k_s = q_s + LP_Q;
  uint8_t* v_s = k_s + LP_K;
  uint64_t* k_full = (uint64_t*)(v_s + LP_VSLOTS * LP_V);
  uint64_t* k_empty = k_full + 1;
  uint64_t* v_full = k_empty + 1;    // [LP_VSLOTS]
  uint64_t* s_full = v_full + LP_VSLOTS;   // [2]
  uint64_t* p_full = s_full + 2;     // [2]
  uint64_t* pv_done = p_full + 2;    // [2]: P . V of the chunk whose P lies in S buffer u is done
  uint64_t* o_done = pv_done + 2;
  uint32_t* tmem_slot = (uint32_t*)(o_done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile int* cleared = abort_flag + 1;           // values that some row sees were set to zero (lp_clear_unseen)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.z;
  pdl_wait();
  const int tok0 = a.seq_start[b], n = a.seq_start[b + 1] - tok0;
  const int first = (int)(gridDim.y - 1 - blockIdx.y) * LP_ROWS;    // the blocks with most keys first
  if (first >= n) return;
  if (smem_u32(lp_smem) & 1023u) {       // the swizzle's alignment; nothing has been taken yet
    if (threadIdx.x == 0) atomicCAS(&tl_latent_prompt_error, 0, 9);
    return;
  }
  const int rows = min(LP_ROWS, n - first), last = first + rows - 1;
  const int lo_all = a.window > 0 ? max(first - a.window + 1, 0) : 0;   // what some row sees starts here,
  const int lo_last = a.window > 0 ? max(last - a.window + 1, 0) : 0;   // and what every row sees is [lo_last, first]
  const int c0 = lo_all / LP_KEYS, n_ch = last / LP_KEYS - c0 + 1;

  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    mbar_init(k_empty, 1);
    for (int u = 0; u < LP_VSLOTS; ++u) mbar_init(&v_full[u], 1);
    for (int u = 0; u < 2; ++u) { mbar_init(&s_full[u], 1); mbar_init(&p_full[u], LP_ROWS); mbar_init(&pv_done[u], 1); }
    mbar_init(o_done, 1);
    *abort_flag = 0;
    *cleared = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) { tmem_alloc(tmem_slot, LP_TMEM); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (threadIdx.x == 0) pdl_launch_dependents();

  if (warp == 4) {
    if (elect_one()) {
      // ---- TMA; rows past the step's end come as zeros, those of the next sequence are masked like any unseen one
      for (int i = 0; i <= n_ch; ++i) {
        if (i < n_ch) {
          const int y = tok0 + (c0 + i) * LP_KEYS;
          if (!lp_wait(k_empty, ((uint32_t)i & 1u) ^ 1u, abort_flag, 1)) break;
          mbar_expect_tx(k_full, 2 * LP_KSUB + (a.rot > 0 ? LP_KSUB : 0));
          tma_load_2d(k_s, &tm_kv, k_full, h * LP_DIM, y);
          tma_load_2d(k_s + LP_KSUB, &tm_kv, k_full, h * LP_DIM + 64, y);
          if (a.rot > 0) tma_load_2d(k_s + 2 * LP_KSUB, &tm_r, k_full, 0, y);
        }
        if (i > 0) {
          const int j = i - 1, s = j % LP_VSLOTS, y = tok0 + (c0 + j) * LP_KEYS, x = a.heads * LP_DIM + h * LP_VDIM;
          // the slot holds V(j - 2) until P(j - 2) . V(j - 2) has read it
          if (j >= LP_VSLOTS && !lp_wait(&pv_done[s], (uint32_t)((j - LP_VSLOTS) >> 1) & 1u, abort_flag, 2)) break;
          uint8_t* dst = v_s + s * LP_V;
          mbar_expect_tx(&v_full[s], LP_V);
          tma_load_2d(dst, &tm_kv, &v_full[s], x, y);
          tma_load_2d(dst + LP_KSUB, &tm_kv, &v_full[s], x + 64, y);
        }
      }
    }
  } else {
    // ---- the queries: turned, times scale and log2(e), rounded.  A warp per row, LP_BATCH rows' loads issued before any is
    // used, entries 2l and 2l + 1 of the rotated part with lane l.  What a lane does with its entries is selected, not
    // branched on: a branch that depends on the lane alone splits the warp for the whole loop (29 us a block against 4).
    // Rows past the last stay as they are; nobody reads what comes of them.
    const int me = warp < 4 ? warp : warp - 1, head_w = LP_DIM + a.rot, pairs = a.dims >> 1;
    const float f = a.scale_log2;
    const float* q0 = a.q + (size_t)(tok0 + first) * a.ldq + (size_t)h * head_w;
    int own[2], other[2], angle[2];
    float keep[2], turns[2], sign[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int e = 2 * lane + j;
      own[j] = LP_DIM + min(e, a.rot - 1);
      angle[j] = min(e < pairs ? e : e - pairs, max(pairs - 1, 0));
      other[j] = LP_DIM + (e < pairs ? e + pairs : angle[j]);
      keep[j] = e < a.rot ? f : 0.0f;
      turns[j] = e < a.dims ? 1.0f : 0.0f;
      sign[j] = e < pairs ? -1.0f : 1.0f;
    }
#pragma unroll 1
    for (int r0 = me; r0 < rows; r0 += 6 * LP_BATCH) {
      float4 x[LP_BATCH];
      float v[LP_BATCH][2], o[LP_BATCH][2];
      float2 cs[LP_BATCH][2];
#pragma unroll
      for (int k = 0; k < LP_BATCH; ++k) {
        const int r = min(r0 + 6 * k, rows - 1);
        const float* src = q0 + (size_t)r * a.ldq;
        x[k] = __ldg(reinterpret_cast<const float4*>(src) + lane);
        if (a.rot > 0) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            v[k][j] = __ldg(src + own[j]);
            if (pairs > 0) {
              o[k][j] = __ldg(src + other[j]);
              cs[k][j] = __ldg(a.turn + (size_t)(tok0 + first + r) * pairs + angle[j]);
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < LP_BATCH; ++k) {
        const int r = min(r0 + 6 * k, rows - 1);      // (the last row more than once: the same numbers)
        uint8_t* row = q_s + r * 128;
        *reinterpret_cast<uint2*>(row + (lane >> 4) * LP_QSUB + ((((lane & 15) >> 1) ^ (r & 7)) << 4) + (lane & 1) * 8) =
            make_uint2(lp_pack(x[k].x * f, x[k].y * f), lp_pack(x[k].z * f, x[k].w * f));
        if (a.rot > 0) {
          float y[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            y[j] = v[k][j];
            if (pairs > 0) {
              const float turned = v[k][j] * cs[k][j].x + (sign[j] * o[k][j]) * cs[k][j].y;
              y[j] = turns[j] != 0.0f ? turned : y[j];
            }
          }
          *reinterpret_cast<uint32_t*>(row + 2 * LP_QSUB + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4) =
              lp_pack(y[0] * keep[0], y[1] * keep[1]);
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync 1, 192;" ::: "memory");
    if (warp == 5) {
      if (elect_one()) {
        // ---- S(j) = Q . K(j)^T into buffer j & 1
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LP_KEYS >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t dq = smem_desc_k128(smem_u32(q_s)), dk = smem_desc_k128(smem_u32(k_s));
        const int subs = a.rot > 0 ? 3 : 2;
        for (int j = 0; j < n_ch; ++j) {
          // the buffer holds P(j - 2) until P(j - 2) . V(j - 2) has read it
          if (j >= 2 && !lp_wait(&pv_done[j & 1], (uint32_t)((j - 2) >> 1) & 1u, abort_flag, 4)) break;
          if (!lp_wait(k_full, (uint32_t)j & 1u, abort_flag, 3)) break;
          tc_fence_after();
          const uint32_t acc = tmem + (uint32_t)(j & 1) * LP_KEYS;
          for (int u = 0; u < subs; ++u) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_bf16(acc, dq + (uint64_t)(u * (LP_QSUB >> 4) + 2 * k), dk + (uint64_t)(u * (LP_KSUB >> 4) + 2 * k), idesc,
                        (u > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit(&s_full[j & 1]);
          umma_commit(k_empty);
        }
      }
    } else if (warp == 6) {
      if (elect_one()) {
        // ---- O (+)= P(j) . V(j)
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(LP_VDIM >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        for (int j = 0; j < n_ch; ++j) {
          if (!lp_wait(&v_full[j % LP_VSLOTS], (uint32_t)(j / LP_VSLOTS) & 1u, abort_flag, 3)) break;
          if (!lp_wait(&p_full[j & 1], (uint32_t)(j >> 1) & 1u, abort_flag, 4)) break;
          tc_fence_after();
          const uint64_t dv = lp_desc_v(smem_u32(v_s + (j % LP_VSLOTS) * LP_V));
#pragma unroll
          for (int k = 0; k < LP_KEYS / 16; ++k)   // 16 positions: 8 columns of P, 2048 bytes of each sub-tile
            lp_umma_ts(tmem + LP_COL_O, tmem + (uint32_t)(j & 1) * LP_KEYS + k * 8, dv + (uint64_t)(k * (2048 >> 4)), idesc,
                       (j > 0 || k > 0) ? 1u : 0u);
          umma_commit(o_done);
          umma_commit(&pv_done[j & 1]);
        }
      }
    } else {
      // ---- softmax: one thread per row
      const int r = threadIdx.x;
      const bool valid = r < rows;
      const int pos = first + min(r, rows - 1);
      const int lo = a.window > 0 ? max(pos - a.window + 1, 0) : 0;
      const uint32_t lanes = (uint32_t)(warp * 32) << 16, t_o = tmem + LP_COL_O + lanes;
      float m = -INFINITY, l = 0.0f;
      bool ok = true;
      for (int i = 0; i < n_ch; ++i) {
        const uint32_t u = (uint32_t)i & 1u, t_s = tmem + u * LP_KEYS + lanes;
        ok = lp_wait(&s_full[u], (uint32_t)(i >> 1) & 1u, abort_flag, 5);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        tc_fence_after();
        uint32_t sa[32], sb[32];
        lp_ld32(t_s, sa);
        lp_ld32(t_s + 32, sb);
        tmem_ld_wait();
        const int key0 = (c0 + i) * LP_KEYS;
        const bool whole = __all_sync(0xffffffffu, valid && key0 >= lo && key0 + LP_KEYS - 1 <= pos);
        if (!whole) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int ka = key0 + j, kb = key0 + 32 + j;
            if (!(valid && ka >= lo && ka <= pos)) sa[j] = 0xff800000u;
            if (!(valid && kb >= lo && kb <= pos)) sb[j] = 0xff800000u;
          }
        }
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 32; ++j) mx = lp_max3(mx, __uint_as_float(sa[j]), __uint_as_float(sb[j]));
        // The reference is the running maximum itself: the weight of the key that stands out is then 1, which bfloat16 holds
        // exactly.  (One that moves only when a score exceeds it by 2^8 spares most of the rescaling of O, 49.6 us instead of
        // 55.0 for 2048 tokens, but rounds that weight too: where few keys count the weights' part of the error is 1.8 times
        // as large, and a result 7 % further from 64 bits.)
        const float m_new = fmaxf(m, mx);
        const float ref = m_new == -INFINITY ? 0.0f : m_new;
        // (a row without a token, or that sees no key so far, must not ask for rescaling)
        const float alpha = valid && m_new != -INFINITY ? exp2f(m - ref) : 1.0f;
        m = m_new;
        uint32_t pk[32];   // the row of P as bfloat16 pairs
        const uint64_t nref = lp_pack2(-ref, -ref);
        uint64_t sum_a = 0, sum_b = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float x0, x1, x2, x3;
          lp_unpack2(lp_add2(lp_pack2(__uint_as_float(sa[2 * j]), __uint_as_float(sa[2 * j + 1])), nref), x0, x1);
          lp_unpack2(lp_add2(lp_pack2(__uint_as_float(sb[2 * j]), __uint_as_float(sb[2 * j + 1])), nref), x2, x3);
          pk[j] = lp_pack(lp_ex2(x0), lp_ex2(x1));
          pk[16 + j] = lp_pack(lp_ex2(x2), lp_ex2(x3));
          sum_a = lp_add2(sum_a, lp_pack2(__uint_as_float(pk[j] << 16), __uint_as_float(pk[j] & 0xffff0000u)));
          sum_b = lp_add2(sum_b, lp_pack2(__uint_as_float(pk[16 + j] << 16), __uint_as_float(pk[16 + j] & 0xffff0000u)));
        }
        float sum, sum_hi;
        lp_unpack2(lp_add2(sum_a, sum_b), sum, sum_hi);
        l = l * alpha + (sum + sum_hi);
        // O is touched only when some row's maximum moved; every warp waits for P(i - 1) . V(i - 1) on every chunk all
        // the same, so that no phase of its barrier is taken for another
        if (i > 0) {
          ok = lp_wait(o_done, (uint32_t)(i - 1) & 1u, abort_flag, 7);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          tc_fence_after();
          if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll 1
            for (int c = 0; c < LP_VDIM; c += 32) {
              uint32_t ov[32];
              lp_ld32(t_o + c, ov);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * alpha);
              lp_st32(t_o + c, ov);
            }
            lp_wait_st();
          }
        }
        if (key0 < lo_last || key0 + LP_KEYS - 1 > first) {
          const int s = i % LP_VSLOTS;
          ok = lp_wait(&v_full[s], (uint32_t)(i / LP_VSLOTS) & 1u, abort_flag, 3);     // what TMA wrote is visible
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          if (lp_clear_unseen(v_s + s * LP_V, key0, lo_last, first, lo_all, last)) *cleared = 1;
        }
        lp_st32(t_s, pk);   // this lane's row of P, keys 2c and 2c + 1 in column c
        lp_wait_st();
        tc_fence_before();
        lp_arrive(&p_full[u]);
      }
      if (ok) ok = lp_wait(o_done, (uint32_t)(n_ch - 1) & 1u, abort_flag, 8);
      // `cleared` by any of these threads; the last product is done, so O / l may take the queries' and the keys' place
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (__all_sync(0xffffffffu, ok)) {
        tc_fence_after();
        // a sink is in the denominator and has no value
        const float inv = 1.0f / (a.sink != nullptr ? l + exp2f(a.sink[h] * 1.4426950408889634f - m) : l);
        float* row = o_s + r * LP_OLD;
#pragma unroll 1
        for (int c = 0; c < LP_VDIM; c += 32) {
          uint32_t ov[32];
          lp_ld32(t_o + c, ov);
          tmem_ld_wait();
          float y[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(ov[j]) * inv;
          if (*cleared) {
            for (int key = lo_all; key <= last; ++key) {
              if (key >= lo_last && key <= first) { key = first; continue; }     // these were multiplied as they are
              if (key < lo || key > pos) continue;
              const __nv_bfloat16* v = a.kv + ((size_t)(tok0 + key) * 2 + 1) * a.heads * LP_VDIM + h * LP_VDIM + c;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (!(fabsf(__bfloat162float(v[j])) < INFINITY)) y[j] += __bfloat162float(v[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(row + c + j) = make_float4(y[j], y[j + 1], y[j + 2], y[j + 3]);
        }
      }
    }
  }
  __syncwarp();
  __syncthreads();
  if (!*abort_flag) {
    // ---- the gate and the way out, a warp per row
    const bool each = a.gate != nullptr && !a.gate_one;
#pragma unroll 1
    for (int r0 = warp; r0 < rows; r0 += 7 * LP_BATCH) {
      float4 g[LP_BATCH];
#pragma unroll
      for (int k = 0; k < LP_BATCH; ++k) {
        const int r = min(r0 + 7 * k, rows - 1);
        const float* src = a.gate + (size_t)(tok0 + first + r) * a.ldg;
        if (each) g[k] = __ldg(reinterpret_cast<const float4*>(src + h * LP_VDIM) + lane);
        else if (a.gate != nullptr) g[k].x = g[k].y = g[k].z = g[k].w = __ldg(src + h);
      }
#pragma unroll
      for (int k = 0; k < LP_BATCH; ++k) {
        const int r = min(r0 + 7 * k, rows - 1);
        float4 y = *reinterpret_cast<const float4*>(o_s + r * LP_OLD + 4 * lane);
        if (a.gate != nullptr) {
          y.x *= lp_sigmoid(g[k].x);
          y.y *= lp_sigmoid(g[k].y);
          y.z *= lp_sigmoid(g[k].z);
          y.w *= lp_sigmoid(g[k].w);
        }
        *reinterpret_cast<uint2*>(a.out + ((size_t)(tok0 + first + r) * a.heads + h) * LP_VDIM + 4 * lane) =
            make_uint2(lp_pack(y.x, y.y), lp_pack(y.z, y.w));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, LP_TMEM);
}

typedef CUresult (*LpEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static LpEncodeFn lp_encode() {
  static LpEncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (LpEncodeFn)p;
  });
  return fn;
}

// `latents`: [T, rank + rot] bfloat16, the tokens' [c | r]; of them r alone is read here.  Returns 0, a CUDA error, or -2 for
// sizes or alignments that are not taken.
extern "C" int tl_latent_prompt_tc(const float* q, int ldq, const float* turn, const void* kv, const void* latents, void* out,
                                   const float* gate, int ldg, int gate_one, const float* sink, const int* seq_start,
                                   int T, int seqs, int max_new, int heads, int dim, int vdim, int rank, int rot, int dims,
                                   int window, float scale, cudaStream_t stream) {
  if (T <= 0 || seqs <= 0 || max_new <= 0) return 0;
  if (dim != LP_DIM || vdim != LP_VDIM || rot < 0 || rot > LP_ROT || rot % 8 || rank <= 0 || rank % 8 || dims < 0 || dims > rot ||
      (dims & 1) || heads < 1 || seqs > 65535)
    return -2;
  if (dims > 0 && !turn) return -1;
  if (ldq % 4 || (((uintptr_t)q | (uintptr_t)kv | (uintptr_t)latents | (uintptr_t)out) & 15) || ((uintptr_t)turn & 7)) return -2;
  if (gate != nullptr && !gate_one && (ldg % 4 || ((uintptr_t)gate & 15))) return -2;
  const int tiles = (max_new + LP_ROWS - 1) / LP_ROWS;
  if (tiles > 65535) return -2;
  LpEncodeFn fn = lp_encode();
  if (!fn) return -2;
  CUtensorMap tm_kv, tm_r;
  auto make = [&](CUtensorMap* m, const void* at, long long cols, long long ld) {
    const cuuint64_t dim2[2] = {(cuuint64_t)cols, (cuuint64_t)T}, stride[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, LP_KEYS}, estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(at), dim2, stride, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  const long long cols = (long long)heads * (LP_DIM + LP_VDIM);
  if (!make(&tm_kv, kv, cols, cols)) return -2;
  // the columns from `rank` on; what lies past them in a box is zero
  if (rot > 0 && !make(&tm_r, (const __nv_bfloat16*)latents + rank, rot, rank + rot)) return -2;
  if (rot == 0) tm_r = tm_kv;
  const cudaError_t set = tl_allow_smem<latent_prompt_tc_kernel>(LP_SMEM);
  if (set != cudaSuccess) return (int)set;
  LatentPromptArgs a = {q, (const float2*)turn, (const __nv_bfloat16*)kv, (__nv_bfloat16*)out, gate, sink, seq_start, ldq, ldg,
                        gate_one, heads, rot, dims, window, scale * 1.4426950408889634f};
  return tl_launch(latent_prompt_tc_kernel, dim3(heads, tiles, seqs), dim3(LP_THREADS), LP_SMEM, stream, tm_kv, tm_r, a);
}

// Reads and clears the error word that a kernel sets when one of its bounded waits ran out.  Synchronises the device.
extern "C" int tl_latent_prompt_take_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, tl_latent_prompt_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(tl_latent_prompt_error, &zero, sizeof(int));
  return v;
}
