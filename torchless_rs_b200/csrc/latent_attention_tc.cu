// Prompts of the latent attention (latent_attention.cu says what it computes) on the fifth-generation tensor cores, for
// latents of 512 numbers and a rotated part of at most 64.
//
// All heads share a position's vector [c | r], so the rows of a tile are (tokens of one sequence) x (heads), 128 of them,
// and a page of 64 positions serves as K (rows, contracted over [c | r]) and as V (columns c, contracted over the
// positions: the same bytes read through a descriptor whose leading dimension is the other one).  The weighted sum of
// 512 columns in 32 bits would fill the tensor memory and leave none for the scores, and the queries of 576 columns most
// of the shared memory.  So two blocks of a cluster share a tile: each holds the queries' and the pages' half of c (the
// first also r), multiplies its half for scores that are half sums, hands them to the other through distributed shared
// memory, and after the softmax, which both compute from the same sums, sums its own half of c.
//   warps 0-3  softmax, a row per thread; exchange of the half scores; output
//   warp 4     TMA of the pages, four in flight
//   warp 5     issues Q . K^T (the queries' half of c from tensor memory), up to two pages ahead (two S buffers)
//   warp 6     issues P . V, P from tensor memory
// Bound by the chain of a page, 2 us where the GPU is otherwise idle: the scores' way out of tensor memory and to the other
// block, the exponentials, the weights' way back (the tensor core's part of a page is some 1100 cycles and overlaps it).
// It is the exchange and not the exponentials: with two threads per row, each half of a page's keys, it took as long (before
// the maximum below moved with every page).
// Measured, 16 heads, on mma.sync with a token's heads per tile / here: one prompt of 2048 tokens 582 / 254 us, of 4096
// 1941 / 723 us; 32 heads, 2048 tokens 1025 / 479 us.
//
// Every wait on an mbarrier is bounded; when a bound is hit the block records a code in tl_latent_tc_error, stops, frees
// its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "per_device.cuh"
#include "umma.cuh"

#include <mutex>

#define PAGE 64
static_assert(TL_PAGE == PAGE, "a chunk of keys is a page");
#define LT_THREADS 224
#define LT_ROWS 128
#define LT_RANK 512
#define LT_HALF 256                        // columns of c per block
#define LT_SUBS 4                          // tiles of 64 columns of the half of c
#define LT_ROT 32                          // columns of r per block
#define LT_QR (LT_ROWS * LT_ROT * 2)       // bytes of the queries' part of r
#define LT_KR (PAGE * LT_ROT * 2)          // bytes of a page's part of r
#define LT_K (LT_SUBS * PAGE * 128 + LT_KR)
#define LT_PAGES 4                         // pages in flight
#define LT_X (PAGE * LT_ROWS * 4)          // bytes of the other block's half scores of a page
#define LT_SMEM (1024 + LT_QR + LT_PAGES * LT_K + 2 * LT_X + 256)
// tensor memory: two S buffers of 64 columns, O, the queries' half of c (two numbers per column)
#define LT_COL_O 128
#define LT_COL_Q 384

__device__ int tl_latent_tc_error = 0;

__device__ __forceinline__ bool lt_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  return tl_mbar_park(bar, parity, abort_flag, code, &tl_latent_tc_error);
}
// The same for a barrier at which the other block's threads arrive: what they wrote before is visible after it.
__device__ __forceinline__ bool lt_wait_peer(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  const uint32_t a = smem_u32(bar);
  for (uint32_t i = 0; i < TL_WAIT_LIMIT / 16; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 63u) == 63u && *abort_flag) return false;
  }
  *abort_flag = code;
  atomicCAS(&tl_latent_tc_error, 0, code);
  return false;
}
__device__ __forceinline__ uint32_t lt_mapa(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void lt_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void lt_st32(uint32_t taddr, const uint32_t (&r)[32]) {
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
__device__ __forceinline__ void lt_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void lt_umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ float lt_ex2(float x) {   // 2^x, one instruction; tiny results flush to zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t lt_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Operand tile of 64-position rows read across them: 64 columns of c contiguous (128 bytes, 128-byte swizzle), the next
// 64 columns a tile further, eight positions 1024 bytes further.
__device__ __forceinline__ uint64_t lt_desc_v(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)((PAGE * 128) >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

// K-major tile whose rows are 64 bytes with the 64-byte swizzle: 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t lt_desc_k64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

// The tensor core multiplies a weight of 0 like any other, and 0 x NaN is NaN.  So in a page that not every row of the tile sees
// whole, a position outside [seen_lo, seen_hi] (what all rows see) whose values are not all finite is set to zero before P . V.
// By the 128 softmax threads, eight to a position's 512 bytes; true if this thread cleared one that some row does see, in
// [some_lo, some_hi].  Such a row's score of it is NaN or infinite, so its weight is NaN, which reaches the row's sum l, or 0,
// and the caller puts in what 0 x the value gives.
__device__ __forceinline__ bool lt_clear_unseen(uint8_t* page, int key0, int seen_lo, int seen_hi, int some_lo, int some_hi) {
  const int row0 = (int)(threadIdx.x >> 3), chunk = (int)(threadIdx.x & 7);
  bool found = false;
#pragma unroll
  for (int k = row0; k < PAGE; k += LT_ROWS / 8) {
    const int key = key0 + k;
    uint4* at = reinterpret_cast<uint4*>(page + k * 128 + chunk * 16);
    uint32_t carry = 0;                    // an exponent of all ones carries into the bit above it
    const bool look = key < seen_lo || key > seen_hi;
    if (look) {
#pragma unroll
      for (int u = 0; u < LT_SUBS; ++u) {
        const uint4 x = at[u * (PAGE * 128 / 16)];
        carry |= ((x.x & 0x7f807f80u) + 0x00800080u) | ((x.y & 0x7f807f80u) + 0x00800080u) |
                 ((x.z & 0x7f807f80u) + 0x00800080u) | ((x.w & 0x7f807f80u) + 0x00800080u);
      }
    }
    const uint32_t any = __ballot_sync(0xffffffffu, (carry & 0x80008000u) != 0u) >> (threadIdx.x & 24u) & 0xffu;
    if (look && any) {
#pragma unroll
      for (int u = 0; u < LT_SUBS; ++u) at[u * (PAGE * 128 / 16)] = make_uint4(0u, 0u, 0u, 0u);
      found |= key >= some_lo && key <= some_hi;
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor core reads the page as it is now
  return found;
}

struct LatentArgs {
  const float* qa;
  const float* q;
  const __nv_bfloat16* pages;
  float* o;                 // [tokens, heads, 512]
  const int* seq_start;
  const int* token_pos;
  const int* seq_slot;
  const int* page_table;
  const float* inv_freq;    // [dims / 2]
  const float* sink;        // [heads] or null
  int ld_qa, qa_head, ldq, q_head, q_off, table_stride, heads, rot, dims, window, tokens;   // `tokens` per tile
  float scale_log2, amp;
};

__global__ void __launch_bounds__(LT_THREADS, 1)
latent_attn_tc_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_r, const LatentArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* qr_s = smem;
  uint8_t* k_s = qr_s + LT_QR;
  uint8_t* x_s = k_s + LT_PAGES * LT_K;
  uint64_t* k_full = (uint64_t*)(x_s + 2 * LT_X);   // [LT_PAGES]
  uint64_t* k_empty = k_full + LT_PAGES;            // [LT_PAGES]
  uint64_t* s_full = k_empty + LT_PAGES;            // [2]
  uint64_t* x_full = s_full + 2;     // [2]: the other block's half scores
  uint64_t* p_full = x_full + 2;     // [2]
  uint64_t* pv_done = p_full + 2;    // [2]: P . V of the page whose P lies in S buffer u is done
  uint64_t* o_done = pv_done + 2;
  uint32_t* tmem_slot = (uint32_t*)(o_done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile int* cleared = abort_flag + 1;   // values that some row sees were set to zero (lt_clear_unseen)

  const int warp = threadIdx.x >> 5, tid = threadIdx.x;
  const uint32_t half = cluster_rank();
  pdl_wait();
  const int b = blockIdx.y, first = a.seq_start[b], n_new = a.seq_start[b + 1] - first;
  const int t0 = (int)(gridDim.x / 2 - 1 - (blockIdx.x >> 1)) * a.tokens;   // the tiles with most keys first
  if (t0 >= n_new) return;                                                  // (both blocks)
  const int tokens = min(a.tokens, n_new - t0), rows = tokens * a.heads;
  const int p0 = a.token_pos[first + t0], p_last = p0 + tokens - 1;
  const int lo_all = a.window > 0 ? max(p0 - a.window + 1, 0) : 0;
  const int lo_last = a.window > 0 ? max(p_last - a.window + 1, 0) : 0;     // [lo_last, p0]: what every row of the tile sees
  const int pg0 = lo_all / PAGE, n_pg = p_last / PAGE - pg0 + 1;
  const int* table = a.page_table + (size_t)a.seq_slot[b] * a.table_stride + pg0;

  if (tid == 0) {
    for (int u = 0; u < LT_PAGES; ++u) { mbar_init(&k_full[u], 1); mbar_init(&k_empty[u], 1); }
    for (int u = 0; u < 2; ++u) {
      mbar_init(&s_full[u], 1);
      mbar_init(&x_full[u], 1);
      mbar_init(&p_full[u], LT_ROWS);
      mbar_init(&pv_done[u], 1);
    }
    mbar_init(o_done, 1);
    *abort_flag = 0;
    *cleared = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int u = 0; u < 2 && u < n_pg; ++u) mbar_expect_tx(&x_full[u], LT_X);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }

  // ---- the queries: times scale and log2(e), rounded.  Each of the first 128 threads brings its row: the half of c into
  // tensor memory, the half of r, turned at the token's position, into shared memory (cosines and sines once per token, in
  // the exchange buffers, which are free until the first page).
  const int pairs = a.dims >> 1;
  float2* turn = reinterpret_cast<float2*>(x_s);           // [tokens][pairs] <= 128 x 32
  for (int i = tid; i < tokens * pairs; i += LT_THREADS) {
    float sn, cs;
    sincosf((float)(p0 + i / pairs) * a.inv_freq[i % pairs], &sn, &cs);
    turn[i] = make_float2(cs * a.amp, sn * a.amp);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp < 4) {
    const int r = tid, token = r / a.heads, head = r % a.heads;
    const bool live = r < rows;
    const float f = a.scale_log2;
    const float* src = a.qa + (size_t)(first + t0 + (live ? token : 0)) * a.ld_qa + (size_t)(live ? head : 0) * a.qa_head + half * LT_HALF;
#pragma unroll 1
    for (int c = 0; c < LT_HALF; c += 64) {
      float4 x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = *reinterpret_cast<const float4*>(src + c + 4 * j);
      uint32_t v[32];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        v[2 * j] = live ? lt_pack(x[j].x * f, x[j].y * f) : 0u;
        v[2 * j + 1] = live ? lt_pack(x[j].z * f, x[j].w * f) : 0u;
      }
      lt_st32(tmem + ((uint32_t)(warp * 32) << 16) + LT_COL_Q + c / 2, v);
    }
    lt_wait_st();
    const float* rs = a.q + (size_t)(first + t0 + (live ? token : 0)) * a.ldq + (size_t)(live ? head : 0) * a.q_head + a.q_off;
#pragma unroll
    for (int g = 0; g < LT_ROT / 8; ++g) {
      uint32_t v[4];
      float e8[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int e = (int)half * LT_ROT + 8 * g + j;
        float y = 0.0f;
        if (live && e < a.rot) {
          if (e < a.dims) {
            const int p = e < pairs ? e : e - pairs;
            const float2 t = turn[token * pairs + p];
            const float u = rs[p], w = rs[p + pairs];
            y = e < pairs ? u * t.x - w * t.y : w * t.x + u * t.y;
          } else {
            y = rs[e];
          }
        }
        e8[j] = y * f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = lt_pack(e8[2 * j], e8[2 * j + 1]);
      *reinterpret_cast<uint4*>(qr_s + r * (LT_ROT * 2) + ((g ^ ((r >> 1) & 3)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // both blocks' barriers exist, and nobody reads the exchange buffers as a table any more
  tc_fence_after();
  if (tid == 0) pdl_launch_dependents();

  if (warp == 4 && elect_one()) {
    // ---- TMA: this block's columns of the pages
    const bool rot = a.rot > 0;
    for (int i = 0; i < n_pg; ++i) {
      const int s = i % LT_PAGES;
      if (!lt_wait(&k_empty[s], ((uint32_t)(i / LT_PAGES) & 1u) ^ 1u, abort_flag, 1)) break;
      const int y = table[i] * PAGE;
      uint8_t* dst = k_s + s * LT_K;
      mbar_expect_tx(&k_full[s], LT_SUBS * (PAGE * 128) + (rot ? LT_KR : 0));
      for (int u = 0; u < LT_SUBS; ++u)
        tma_load_2d(dst + u * (PAGE * 128), &tm, &k_full[s], (int)half * LT_HALF + u * 64, y);
      if (rot) tma_load_2d(dst + LT_SUBS * (PAGE * 128), &tm_r, &k_full[s], LT_RANK + (int)half * LT_ROT, y);
    }
  } else if (warp == 5 && elect_one()) {
    // ---- S(j) = this block's part of Q . K(j)^T into buffer j & 1
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(PAGE >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const uint64_t dqr = lt_desc_k64(smem_u32(qr_s));
    for (int j = 0; j < n_pg; ++j) {
      // the buffer holds P(j - 2) until P(j - 2) . V(j - 2) has read it
      if (j >= 2 && !lt_wait(&pv_done[j & 1], (uint32_t)((j - 2) >> 1) & 1u, abort_flag, 4)) break;
      if (!lt_wait(&k_full[j % LT_PAGES], (uint32_t)(j / LT_PAGES) & 1u, abort_flag, 3)) break;
      tc_fence_after();
      const uint32_t ka = smem_u32(k_s + (j % LT_PAGES) * LT_K);
      const uint64_t dk = smem_desc_k128(ka), dkr = lt_desc_k64(ka + LT_SUBS * (PAGE * 128));
      const uint32_t acc = tmem + (uint32_t)(j & 1) * PAGE;
#pragma unroll
      for (int u = 0; u < LT_SUBS; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          lt_umma_ts(acc, tmem + LT_COL_Q + u * 32 + k * 8, dk + (uint64_t)(u * ((PAGE * 128) >> 4) + 2 * k), idesc,
                     (u > 0 || k > 0) ? 1u : 0u);
      if (a.rot > 0) {
#pragma unroll
        for (int k = 0; k < LT_ROT / 16; ++k) umma_bf16(acc, dqr + 2 * k, dkr + 2 * k, idesc, 1u);
      }
      umma_commit(&s_full[j & 1]);
    }
  } else if (warp == 6 && elect_one()) {
    // ---- O (+)= P(j) . V(j), V the positions' own columns of c
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(LT_HALF >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    for (int j = 0; j < n_pg; ++j) {
      if (!lt_wait(&p_full[j & 1], (uint32_t)(j >> 1) & 1u, abort_flag, 4)) break;
      tc_fence_after();
      const uint64_t dv = lt_desc_v(smem_u32(k_s + (j % LT_PAGES) * LT_K));
#pragma unroll
      for (int k = 0; k < PAGE / 16; ++k)   // 16 positions: 8 columns of P, 2048 bytes of the page
        lt_umma_ts(tmem + LT_COL_O, tmem + (uint32_t)(j & 1) * PAGE + k * 8, dv + (uint64_t)(k * (2048 >> 4)), idesc,
                   (j > 0 || k > 0) ? 1u : 0u);
      umma_commit(o_done);
      umma_commit(&pv_done[j & 1]);
      umma_commit(&k_empty[j % LT_PAGES]);
    }
  } else if (warp < 4) {
    // ---- softmax: one thread per row
    const int r = tid;
    const bool valid = r < rows;
    const int pos = valid ? p0 + r / a.heads : p_last;
    const int lo = a.window > 0 ? max(pos - a.window + 1, 0) : 0;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16, t_s = tmem + lanes, t_o = tmem + LT_COL_O + lanes;
    float m = -INFINITY, l = 0.0f;
    const uint32_t mine = smem_u32(x_s) + (uint32_t)r * 16u, theirs = lt_mapa(mine, half ^ 1u);
    const uint32_t bar_theirs = lt_mapa(smem_u32(x_full), half ^ 1u);
    bool ok = true;
    for (int i = 0; i < n_pg; ++i) {
      const uint32_t u = (uint32_t)i & 1u;
      ok = lt_wait(&s_full[u], (uint32_t)(i >> 1) & 1u, abort_flag, 5);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after();
      uint32_t sa[32], sb[32];
      lt_ld32(t_s + u * PAGE, sa);
      lt_ld32(t_s + u * PAGE + 32, sb);
      tmem_ld_wait();
      // the half sums go to the other block, 16 bytes of a row beside the next row's; their bytes count at its barrier (plain
      // stores and an arrival that waits for them took 0.6 us more a page)
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        const uint32_t* v = g < 8 ? sa + 4 * g : sb + 4 * (g - 8);
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                         theirs + u * LT_X + (uint32_t)g * (LT_ROWS * 16)),
                     "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar_theirs + 8u * u)
                     : "memory");
      }
      ok = lt_wait_peer(&x_full[u], (uint32_t)(i >> 1) & 1u, abort_flag, 6);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      // the other block sends page i + 2 only when it has page i + 1 of this one, which is sent below
      if (r == 0 && i + 2 < n_pg) mbar_expect_tx(&x_full[u], LT_X);
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        uint32_t* v = g < 8 ? sa + 4 * g : sb + 4 * (g - 8);
        const float4 x = *reinterpret_cast<const float4*>(x_s + u * LT_X + g * (LT_ROWS * 16) + r * 16);
        v[0] = __float_as_uint(__uint_as_float(v[0]) + x.x);
        v[1] = __float_as_uint(__uint_as_float(v[1]) + x.y);
        v[2] = __float_as_uint(__uint_as_float(v[2]) + x.z);
        v[3] = __float_as_uint(__uint_as_float(v[3]) + x.w);
      }
      const int key0 = (pg0 + i) * PAGE;
      const bool whole = __all_sync(0xffffffffu, valid && key0 >= lo && key0 + PAGE - 1 <= pos);
      float mx = -INFINITY;
      if (!whole) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int ka = key0 + j, kb = key0 + 32 + j;
          if (!(valid && ka >= lo && ka <= pos)) sa[j] = 0xff800000u;
          if (!(valid && kb >= lo && kb <= pos)) sb[j] = 0xff800000u;
        }
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) mx = fmaxf(mx, fmaxf(__uint_as_float(sa[j]), __uint_as_float(sb[j])));
      // The reference is the running maximum itself: the weight of the key that stands out is then 1, which bfloat16 holds
      // exactly.  (A reference that moves only when a score exceeds it by 2^8 spares most of the rescaling of O, but rounds
      // that weight too while l sums weights as they are: 235 us instead of 251 for 2048 tokens (then), and up to 7 % further from 64
      // bits where few keys count.)
      const float m_new = fmaxf(m, mx);
      const float ref = m_new == -INFINITY ? 0.0f : m_new;
      // (a row without a token, or that sees no key so far, must not ask for rescaling)
      const float alpha = valid && m_new != -INFINITY ? exp2f(m - ref) : 1.0f;
      m = m_new;
      uint32_t pk[32];   // the row of P as bfloat16 pairs
      float sum = 0.0f, sum_hi = 0.0f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float w0 = lt_ex2(__uint_as_float(sa[2 * j]) - ref), w1 = lt_ex2(__uint_as_float(sa[2 * j + 1]) - ref);
        const float w2 = lt_ex2(__uint_as_float(sb[2 * j]) - ref), w3 = lt_ex2(__uint_as_float(sb[2 * j + 1]) - ref);
        sum += w0 + w1;
        sum_hi += w2 + w3;
        pk[j] = lt_pack(w0, w1);
        pk[16 + j] = lt_pack(w2, w3);
      }
      l = l * alpha + (sum + sum_hi);
      // O is touched only when some row's maximum moved; every warp waits for P(i - 1) . V(i - 1) on every page all the
      // same, so that no phase of its barrier is taken for another
      if (i > 0) {
        ok = lt_wait(o_done, (uint32_t)(i - 1) & 1u, abort_flag, 7);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        tc_fence_after();
        if (__any_sync(0xffffffffu, alpha != 1.0f)) {
#pragma unroll 2
          for (int c = 0; c < LT_HALF; c += 32) {
            uint32_t ov[32];
            lt_ld32(t_o + c, ov);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * alpha);
            lt_st32(t_o + c, ov);
          }
          lt_wait_st();
        }
      }
      if (key0 < lo_last || key0 + PAGE - 1 > p0) {   // (the page's scores are done: nobody else reads it now)
        ok = lt_wait(&k_full[i % LT_PAGES], (uint32_t)(i / LT_PAGES) & 1u, abort_flag, 3);   // what TMA wrote is visible
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        if (lt_clear_unseen(k_s + (i % LT_PAGES) * LT_K, key0, lo_last, p0, lo_all, p_last)) *cleared = 1;
      }
      lt_st32(t_s + u * PAGE, pk);   // this lane's row of P, keys 2c and 2c + 1 in column c
      lt_wait_st();
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&p_full[u])) : "memory");
    }
    if (ok) ok = lt_wait(o_done, (uint32_t)(n_pg - 1) & 1u, abort_flag, 8);
    asm volatile("bar.sync 1, 128;" ::: "memory");   // `cleared` by any of these warps
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      // a sink only enters the denominator
      const float inv = 1.0f / (a.sink != nullptr && valid ? l + exp2f(a.sink[r % a.heads] * 1.4426950408889634f - m) : l);
      float* orow = a.o + ((size_t)(first + t0) * a.heads + r) * LT_RANK + half * LT_HALF;
#pragma unroll 2
      for (int c = 0; c < LT_HALF; c += 32) {
        uint32_t ov[32];
        lt_ld32(t_o + c, ov);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(orow + c + j) =
                make_float4(__uint_as_float(ov[j]) * inv, __uint_as_float(ov[j + 1]) * inv, __uint_as_float(ov[j + 2]) * inv,
                            __uint_as_float(ov[j + 3]) * inv);
        }
      }
      if (valid && *cleared) {
        for (int key = lo_all; key <= p_last; ++key) {
          if (key >= lo_last && key <= p0) { key = p0; continue; }     // these were multiplied as they are
          if (key < lo || key > pos) continue;
          const __nv_bfloat16* v = a.pages + ((size_t)table[key / PAGE - pg0] * PAGE + key % PAGE) * (LT_RANK + a.rot) + half * LT_HALF;
          for (int c = 0; c < LT_HALF; ++c)
            if (!(fabsf(__bfloat162float(v[c])) < INFINITY)) orow[c] = NAN;
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // nobody leaves while the other may still write into its shared memory
  if (warp == 0) tmem_dealloc(tmem, 512);
}

typedef CUresult (*LtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static LtEncodeFn lt_encode() {
  static LtEncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (LtEncodeFn)p;
  });
  return fn;
}

// Steps whose tokens follow one another in each of `seqs` sequences (at most `max_new` of one).  Returns 0, a CUDA error,
// or -2 for sizes or alignments that are not taken.
extern "C" int tl_latent_attn_tc(const float* qa, int ld_qa, int qa_head, const float* q, int ldq, int q_head, int q_off,
                                 const void* pages, long long n_pages, float* o, const int* seq_start, const int* token_pos,
                                 const int* seq_slot, const int* page_table, int table_stride, const float* inv_freq,
                                 const float* sink, int seqs, int max_new, int heads, int rank, int rot, int dims,
                                 int window, float scale, float amp, cudaStream_t stream) {
  if (seqs <= 0 || max_new <= 0) return 0;
  if (rank != LT_RANK || rot < 0 || rot > 64 || rot % 8 || dims < 0 || dims > rot || (dims & 1) || heads < 1 || heads > LT_ROWS)
    return -2;
  if (dims > 0 && !inv_freq) return -1;
  if (ld_qa % 4 || qa_head % 4 || (((uintptr_t)qa | (uintptr_t)pages | (uintptr_t)o) & 15) || seqs > 65535) return -2;
  if (n_pages * PAGE > 0x7fffffffll) return -2;
  LtEncodeFn fn = lt_encode();
  if (!fn) return -2;
  // c in boxes of 64 columns, r in boxes of 32 (what lies past the row's end is zero)
  CUtensorMap tm, tm_r;
  const cuuint64_t dim[2] = {(cuuint64_t)(rank + rot), (cuuint64_t)n_pages * PAGE}, stride[1] = {(cuuint64_t)(rank + rot) * 2};
  const cuuint32_t box[2] = {64, PAGE}, box_r[2] = {LT_ROT, PAGE}, estr[2] = {1, 1};
  auto make = [&](CUtensorMap* m, const cuuint32_t* bx, CUtensorMapSwizzle swizzle) {
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(pages), dim, stride, bx, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (!make(&tm, box, CU_TENSOR_MAP_SWIZZLE_128B) || !make(&tm_r, box_r, CU_TENSOR_MAP_SWIZZLE_64B)) return -2;
  const cudaError_t set = tl_allow_smem<latent_attn_tc_kernel>(LT_SMEM);
  if (set != cudaSuccess) return (int)set;
  LatentArgs a = {qa, q, (const __nv_bfloat16*)pages, o, seq_start, token_pos, seq_slot, page_table, inv_freq, sink, ld_qa, qa_head, ldq, q_head, q_off,
                  table_stride, heads, rot, dims, window, LT_ROWS / heads, scale * 1.4426950408889634f, amp};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * ((max_new + a.tokens - 1) / a.tokens), seqs);
  cfg.blockDim = dim3(LT_THREADS);
  cfg.dynamicSmemBytes = LT_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, latent_attn_tc_kernel, tm, tm_r, a);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// Reads and clears the error word that a kernel sets when one of its bounded waits ran out.  Synchronises the device.
extern "C" int tl_latent_tc_take_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, tl_latent_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(tl_latent_tc_error, &zero, sizeof(int));
  return v;
}
