// The experts' products of the bfloat16 path on the fifth-generation tensor cores, over rows grouped by expert (moe.cu
// groups them):
//   UP:    C[row, n] (bfloat16) = act( X[row] . Wg_e[n], X[row] . Wu_e[n] ),  W_e = [2 N, K]: N gate rows, then N up rows
//   DOWN:  C[row, n] (32-bit)   = X[row] . W_e[n],                             W_e = [N, K]
// X lies in the grouped order (moe_gather_kernel brings the tokens' rows there), so that an expert's rows are a range
// that TMA reads as it is.
//
// Persistent blocks walk over tiles of 128 rows of W (the M operand of tcgen05.mma; UP: 64 gate and the 64 up rows of the
// same columns) times up to 256 rows of one expert.  How many rows an expert has is known on the device only: every
// block reads the offsets and finds its tiles itself, and an expert's rows are cut into tiles of equal height, a
// multiple of 16.  Roles as in gemm_tc.cu: warps 0-3 epilogue, warp 4 TMA, warp 5 issues; the accumulator is
// double-buffered in tensor memory.
//
// Bound by the tensor cores on prompts and by the experts' weights on decode steps.  On mma.sync, 64 x 64 tiles (which this
// replaces), 3000 tokens of four choices among 16 experts of 1408 at width 2048 took 529 us up and 316 us down; here 157 and 78
// us (87 and 43 at the bfloat16 rate).  Four tokens: 59 and 32 us; here 24 and 13 (19 and 10 at the copy rate of the experts
// that are chosen).  Width 4096, experts of 3584, 16 tokens: 262 and 150 us; here 147 and 76 (143 and 72).  256 experts of 256 at
// width 1024, one token of eight choices: 38 and 62 us; here 10 and 6.  Only where a few experts of some fifty at widths of some
// fifty get thousands of rows was that faster (four of 48 at 64, 3000 tokens of two choices: 6.8 and 3.7 us; here 9.0 and 6.8).
//
// Every wait on an mbarrier is bounded; when a bound is hit the kernel records a code in tl_moe_tc_error, stops waiting
// everywhere, frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "per_device.cuh"
#include "umma.cuh"

#include <mutex>

#define MT_THREADS 192
#define MT_ROWS 128              // rows of W per tile
#define MT_K 64                  // K elements per stage (128 bytes)
#define MT_W (MT_ROWS * 128)     // bytes of a stage's rows of W
#define MT_BN 256                // most rows of X per tile
#define MT_BOX 32                // rows of X per TMA copy
#define MT_MAX_EXPERTS 1024
#define MT_XCHG 8192             // UP: two buffers in which the gate and up halves of a tile exchange values
#define MT_TAIL 256
#define MT_MAX_STAGES 10

#define MOE_ACT_SILU 0
#define MOE_ACT_CLAMPED 2

__device__ int tl_moe_tc_error = 0;

__device__ __forceinline__ bool mt_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  return tl_mbar_park(bar, parity, abort_flag, code, &tl_moe_tc_error);
}
__device__ __forceinline__ void mt_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// rows[r] = X[row_token[r]] for the grouped rows r < offsets[E]; 16 bytes per thread, 1 << row_log threads per row.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const uint4* __restrict__ X, int ldx16, const int* __restrict__ row_token, const int* __restrict__ offsets,
                  int E, int per_row, int row_log, uint4* __restrict__ rows) {
  pdl_wait();
  pdl_launch_dependents();
  const int n = offsets[E], threads = 1 << row_log, per_block = 256 >> row_log;
  for (int r = blockIdx.x * per_block + (threadIdx.x >> row_log); r < n; r += gridDim.x * per_block) {
    const uint4* src = X + (size_t)row_token[r] * ldx16;
    for (int i = threadIdx.x & (threads - 1); i < per_row; i += threads) rows[(size_t)r * per_row + i] = src[i];
  }
}

struct MoeArgs {
  void* C;
  const int* offsets;
  int ldc, E, N, K, bn_cap, stages, kind;
  float limit, alpha;
};

// What the gate and up sums of an expert go through (as in moe.cu).
__device__ __forceinline__ float mt_act(const MoeArgs& a, float g, float u) {
  if (a.kind == MOE_ACT_SILU) return g / (1.0f + expf(-g)) * u;
  g = fminf(g, a.limit);
  u = fminf(fmaxf(u, -a.limit), a.limit);
  return g / (1.0f + expf(-a.alpha * g)) * (u + 1.0f);
}

// The tiles of a block, in order: expert by expert, inside an expert all row tiles of one strip of W, then the next
// strip.  `first[e]`: the number of expert e's first tile, for e <= E.  (Walking from expert to expert with a division each
// took 40 us of 48 with 300 experts.)
struct MoeWalk {
  const int* off;
  const int* first;
  int E, cap;
  int e = 0;                       // expert
  int r0 = 0, rows = 0, bn = 0, strip = 0;
  __device__ bool find(int tile) {
    if (tile >= first[E]) return false;
    int hi = E;                    // the last expert whose first tile is not beyond; tiles rise, so it is not before e
    while (hi - e > 1) {
      const int mid = (e + hi) >> 1;
      if (first[mid] <= tile) e = mid;
      else hi = mid;
    }
    const int n = off[e + 1] - off[e], t = tile - first[e];
    int m_tiles = 1, m = 0;
    strip = t;
    bn = n;
    if (n > cap) {
      m_tiles = (n + cap - 1) / cap;
      m = t % m_tiles;
      strip = t / m_tiles;
      bn = (n + m_tiles - 1) / m_tiles;
    }
    bn = (bn + 15) / 16 * 16;
    r0 = off[e] + m * bn;
    rows = min(bn, off[e + 1] - r0);      // (0 or less: the tiles before took all rows)
    return true;
  }
};

template <bool UP>
__global__ void __launch_bounds__(MT_THREADS)
moe_tc_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const MoeArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int stages = args.stages;
  const uint32_t stage_bytes = MT_W + (uint32_t)args.bn_cap * 128u;
  float* xchg = (float*)(smem + (size_t)stages * stage_bytes);
  uint64_t* full = (uint64_t*)((uint8_t*)xchg + MT_XCHG);
  uint64_t* empty = full + MT_MAX_STAGES;
  uint64_t* acc_full = empty + MT_MAX_STAGES;   // [2]
  uint64_t* acc_empty = acc_full + 2;           // [2]
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  int* off = (int*)((uint8_t*)full + MT_TAIL);  // [E + 1]
  int* first = off + args.E + 1;                // [E + 1]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int TILE_N = UP ? 64 : 128;         // columns of C per tile
  const int n_tiles = (args.N + TILE_N - 1) / TILE_N;
  const int k_stages = (args.K + MT_K - 1) / MT_K;
  const int w_rows = (UP ? 2 : 1) * args.N;     // of one expert

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 128); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  pdl_wait();
  for (int i = threadIdx.x; i <= args.E; i += MT_THREADS) off[i] = args.offsets[i];
  __syncthreads();
  if (warp == 1) {
    int before = 0;
    for (int e0 = 0; e0 < args.E; e0 += 32) {
      const int e = e0 + lane;
      int v = e < args.E ? (off[e + 1] - off[e] + args.bn_cap - 1) / args.bn_cap * n_tiles : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (e < args.E) first[e + 1] = before + v;
      before += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) first[0] = 0;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (threadIdx.x == 0) pdl_launch_dependents();
  MoeWalk walk{off, first, args.E, args.bn_cap};

  if (warp == 4 && elect_one()) {
    // ---- TMA
    uint32_t it = 0;
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int tile = blockIdx.x; ok && walk.find(tile); tile += gridDim.x) {
      if (walk.rows <= 0) continue;
      const int boxes = (walk.bn + MT_BOX - 1) / MT_BOX;
      const int w0 = walk.e * w_rows + walk.strip * TILE_N;
      for (int k = 0; k < k_stages; ++k, ++it) {
        ok = mt_wait(&empty[s], ph ^ 1u, abort_flag, 1);
        if (!ok) break;
        uint8_t* st = smem + (size_t)s * stage_bytes;
        mbar_expect_tx(&full[s], MT_W + (uint32_t)boxes * (MT_BOX * 128u));
        tma_load_2d(st, &tm_w, &full[s], k * MT_K, w0);
        tma_load_2d(st + MT_W / 2, &tm_w, &full[s], k * MT_K, w0 + (UP ? args.N : 64));
        for (int b = 0; b < boxes; ++b)
          tma_load_2d(st + MT_W + b * (MT_BOX * 128), &tm_x, &full[s], k * MT_K, walk.r0 + b * MT_BOX);
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 5 && elect_one()) {
    // ---- MMA issuer
    uint32_t local = 0, ph = 0;
    int s = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && walk.find(tile); tile += gridDim.x) {
      if (walk.rows <= 0) continue;
      const uint32_t buf = local & 1u;
      ok = mt_wait(&acc_empty[buf], ((local >> 1) & 1u) ^ 1u, abort_flag, 4);
      if (!ok) break;
      ++local;
      tc_fence_after();
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(walk.bn >> 3) << 17) | ((uint32_t)(MT_ROWS >> 4) << 24);
      const uint32_t acc = tmem + buf * MT_BN;
      for (int k = 0; k < k_stages; ++k) {
        ok = mt_wait(&full[s], ph, abort_flag, 2);
        if (!ok) break;
        tc_fence_after();
        const uint64_t dw = smem_desc_k128(smem_u32(smem + (size_t)s * stage_bytes));
        const uint64_t dx = dw + (MT_W >> 4);
#pragma unroll
        for (int q = 0; q < MT_K / 16; ++q) umma_bf16(acc, dw + 2 * q, dx + 2 * q, idesc, (k > 0 || q > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
      if (ok) umma_commit(&acc_full[buf]);
    }
  } else if (warp < 4) {
    // ---- epilogue: thread = one row of W = one column of C
    const int row = warp * 32 + lane;
    uint32_t local = 0;
    for (int tile = blockIdx.x; walk.find(tile); tile += gridDim.x) {
      if (walk.rows <= 0) continue;
      const uint32_t buf = local & 1u;
      const bool ok = mt_wait(&acc_full[buf], (local >> 1) & 1u, abort_flag, 3);
      uint32_t all;
      asm volatile(
          "{\n\t.reg .pred p, q;\n\t"
          "setp.ne.b32 p, %1, 0;\n\t"
          "barrier.cta.red.and.pred q, 1, 128, p;\n\t"
          "selp.u32 %0, 1, 0, q;\n\t}"
          : "=r"(all)
          : "r"((uint32_t)ok)
          : "memory");
      if (!all) break;
      ++local;
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + buf * MT_BN;
      const int n0 = walk.strip * TILE_N;
      if (UP) {
        // rows 0-63 hold the gate, rows 64-127 the up value of a column; the gate half writes the first eight of
        // each 16 rows of X, the up half the others
        const int col = row & 63, up_half = row >> 6, n = n0 + col;
        for (int c0 = 0, i = 0; c0 < walk.rows; c0 += 16, ++i) {
          uint32_t r[16];
          tmem_ld16(taddr + c0, r);
          tmem_ld_wait();
          float* mine = xchg + (i & 1) * 1024 + (up_half ? 512 : 0);     // what this thread gives away
          float* theirs = xchg + (i & 1) * 1024 + (up_half ? 0 : 512);
#pragma unroll
          for (int j = 0; j < 8; ++j) mine[j * 64 + col] = __uint_as_float(r[up_half ? j : 8 + j]);
          asm volatile("bar.sync 1, 128;" ::: "memory");
          if (n < args.N) {
            const int first = c0 + (up_half ? 8 : 0), valid = walk.rows - first;
            __nv_bfloat16* c = (__nv_bfloat16*)args.C + (size_t)(walk.r0 + first) * args.ldc + n;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (j >= valid) break;
              const float other = theirs[j * 64 + col];
              const float g = up_half ? other : __uint_as_float(r[j]);
              const float u = up_half ? __uint_as_float(r[8 + j]) : other;
              c[(size_t)j * args.ldc] = __float2bfloat16_rn(mt_act(args, g, u));
            }
          }
        }
      } else {
        const int n = n0 + row;
        for (int c0 = 0; c0 < walk.rows; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(taddr + c0, r);
          tmem_ld_wait();
          if (n < args.N) {
            const int valid = walk.rows - c0;
            float* c = (float*)args.C + (size_t)(walk.r0 + c0) * args.ldc + n;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (j < valid) c[(size_t)j * args.ldc] = __uint_as_float(r[j]);
          }
        }
      }
      tc_fence_before();
      mt_arrive(&acc_empty[buf]);   // 128 arrivals free the accumulator
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

typedef CUresult (*MtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static MtEncodeFn mt_encode() {
  static MtEncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (MtEncodeFn)p;
  });
  return fn;
}
// [rows, K] bfloat16 with rows of ld elements; boxes of 64 K-elements x box_rows rows, 128-byte swizzle.
static bool mt_map(CUtensorMap* m, const void* ptr, long long rows, int K, long long ld, int box_rows) {
  MtEncodeFn fn = mt_encode();
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {MT_K, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  return fn && fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool UP>
static int run_moe(const CUtensorMap& tw, const CUtensorMap& tx, const MoeArgs& a, int smem, int blocks, cudaStream_t stream) {
  const cudaError_t set = tl_allow_smem<moe_tc_kernel<UP>>(227 * 1024);
  if (set != cudaSuccess) return (int)set;
  return tl_launch(moe_tc_kernel<UP>, dim3(blocks), dim3(MT_THREADS), (size_t)smem, stream, tw, tx, a);
}

// X [rows, K] in the grouped order; or, with row_token (UP), [tokens, K], whose rows go to `grouped` [max_rows, K] first.
// `most`: no expert has more rows.  Returns 0, a CUDA error, or -2 for sizes or alignments that are not taken.
extern "C" int tl_moe_tc(const void* X, int ldx, const int* row_token, void* grouped, const void* W, void* C, int ldc,
                         const int* offsets, int E, int max_rows, int most, int N, int K, int up, int kind, float limit,
                         float alpha, int num_sms, cudaStream_t stream) {
  if (max_rows <= 0 || E <= 0) return 0;
  if (N < 1 || K < 1 || most < 1 || (up && (!row_token || !grouped))) return -1;
  if (E > MT_MAX_EXPERTS || K % 8 || ldx % 8 || ((uintptr_t)X & 15) || ((uintptr_t)W & 15) || ((uintptr_t)grouped & 15))
    return -2;
  if ((long long)E * N * (up ? 2 : 1) > 0x7fffffffll) return -2;
  MoeArgs a = {C, offsets, ldc, E, N, K, 0, 0, kind, limit, alpha};
  const int tile_n = up ? 64 : 128, n_tiles = (N + tile_n - 1) / tile_n;
  a.bn_cap = most >= MT_BN ? MT_BN : (most + MT_BOX - 1) / MT_BOX * MT_BOX;
  if ((long long)E * n_tiles < num_sms) {
    // few experts with small matrices: tiles of as few rows as give every SM one (6000 rows, four experts of 48 at width 64: 9.0
    // us up and 6.8 down; with tiles of 256 rows 22.7 and 13.4)
    const long long share = ((long long)max_rows * n_tiles + num_sms - 1) / num_sms;
    if (share < a.bn_cap) a.bn_cap = (int)((share + MT_BOX - 1) / MT_BOX * MT_BOX);
  }
  const int stage = MT_W + a.bn_cap * 128, fixed = 1024 + MT_XCHG + MT_TAIL + 2 * (E + 1) * 4;
  a.stages = (227 * 1024 - fixed) / stage;
  if (a.stages > MT_MAX_STAGES) a.stages = MT_MAX_STAGES;
  CUtensorMap tw, tx;
  if (!mt_map(&tw, W, (long long)E * N * (up ? 2 : 1), K, K, 64)) return -2;
  if (!mt_map(&tx, up ? grouped : X, max_rows, K, up ? K : ldx, MT_BOX)) return -2;
  if (up) {
    int row_log = 0;
    while (row_log < 8 && (1 << row_log) < K / 8) ++row_log;
    const int want = (max_rows + (256 >> row_log) - 1) / (256 >> row_log);
    const int rc = tl_launch(moe_gather_kernel, dim3(want < 4096 ? want : 4096), dim3(256), 0, stream, (const uint4*)X,
                             ldx / 8, row_token, offsets, E, K / 8, row_log, (uint4*)grouped);
    if (rc != 0) return rc;
  }
  // no more blocks than there can be tiles
  const long long tiles = ((long long)max_rows / 16 + E) * n_tiles;
  const int blocks = tiles < num_sms ? (int)tiles : num_sms, smem = fixed + a.stages * stage;
  return up ? run_moe<true>(tw, tx, a, smem, blocks, stream) : run_moe<false>(tw, tx, a, smem, blocks, stream);
}

// Reads and clears the error word that a kernel sets when one of its bounded waits ran out.  Synchronises the device.
extern "C" int tl_moe_tc_take_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, tl_moe_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(tl_moe_tc_error, &zero, sizeof(int));
  return v;
}
