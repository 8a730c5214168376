// Matrix products of the true 32-bit path on the fifth-generation tensor cores.
//
//   C[M, N] (op)= X[M, K] * W[N, K]^T        X, W, C 32-bit, K contiguous in X and W
//
// A 32-bit number is the sum of three bfloat16 numbers exactly (24 bits of mantissa in three times eight; what is lost
// lies below the smallest bfloat16 number, 2^-133): x = x1 + x2 + x3, each the rounding of what the ones before leave.
// Of the nine products of two such sums the six largest are taken,
//   x1 w1  +  x1 w2 + x2 w1  +  x1 w3 + x2 w2 + x3 w1,
// each exact in the tensor core (8 x 8 bits); the other three are below 2^-26 of the product.  The tensor core adds
// in 32 bits but cuts what falls off instead of rounding, so the order of the sums decides the error: x1 w1 is summed
// over 64 or 256 K-elements in tensor memory, then added, rounded, to a sum in registers; the other five products, 2^-8 of it
// and less, have an accumulator of their own that runs over all of K.  Measured against 64 bits (root mean square over the
// results', K of 512 / 4096 / 14336): 2.3e-7 / 2.4e-7 / 3.3e-7 with many tokens, where one 32-bit fused multiply-add after another, which
// the kernel for many rows in gemm_generic.cu does (and the reference: src/loader/parameters.rs:551-594), is at
// 4e-7 / 1.15e-6 / 2.15e-6.
//
// A result that is not finite (an infinity or a NaN in an operand, a number that rounds to infinity in bfloat16, an
// overflow of one of the products) is computed again as the plain sequence of multiply-adds, so such operands give what
// they give there.  So is one below 2^-90 that is not 0: what a number below 2^-117 loses, up to 2^-134, counts in results
// that small (operands of size 2^-118 and 1 were 9e-6 off, of 2^-124 6e-4).  In larger results it counts only where numbers
// below 2^-117 meet some above 2^20.  A product whose results are all of these kinds takes some four times what the
// CUDA-core kernel does.
//
// One block computes 128 rows of W (the M operand of tcgen05.mma) times up to 192 tokens.
//   warps 0-3   sums in registers, epilogue
//   warps 4-11  take W as stored from shared memory, a row per thread, and write its three pieces into tensor memory;
//               two groups of four warps in turn
//   warp 12     TMA of W as stored (four tiles in flight)
//   warp 13     issues the instructions (with few tokens warp 15 those of the leading products)
//   warp 14     TMA of the pieces of X, which a kernel before has made
// W's pieces are operands from tensor memory because an instruction that reads both operands from shared memory is
// bound by that: with W's pieces there a stage of 192 tokens took 2900 cycles where its arithmetic takes 1152.  While
// the sum of the leading products is read, the instructions of the other five run.
//
// Products with few tiles split K over a cluster of blocks, which add their partial tiles in the order of the splits
// through distributed shared memory (the same bits every run).
//
// What bounds it: the tensor core's six products per multiply-add with many tokens (265 TFLOP/s at the bfloat16 rate;
// 231 at 531 x 6144 x 4096, whose tiles fill one round of blocks), with few W's way through a block (struct Sp).
// Measured, from the CUDA-core kernels to this: 16 tokens 356 / 282 / 826 / 1275 us -> 25 /
// 18 / 94 / 45 us for 6144 x 4096, 4096 x 4096, 14336 x 4096 with the SiLU-gate and 4096 x 14336 (W at the copy rate: 15 /
// 10 / 72 / 36), 531 tokens 1192 / 1061 / 4355 / 3705 -> 116 / 91 / 579 / 303 us, 5 tokens 75 / 40 / 200 / 287 ->
// 25 / 18 / 92 / 44 us.
//
// Output modes as in gemm_generic.cu: 0 store, 1 add into C, 2 SiLU-gate (W holds N gate rows, then N up rows; a tile
// is 64 rows of each, and the halves of the rows exchange values through shared memory), 3 store.
//
// Every wait on an mbarrier is bounded; when a bound is hit the kernel records a code in tl_gemm_split_error, stops
// waiting everywhere, frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pdl.cuh"
#include "per_device.cuh"
#include "umma.cuh"

#include <mutex>

#define SP_THREADS 512
#define SP_ROWS 128             // rows of W per tile
#define SP_BN 192               // most tokens per tile
#define SP_K 32                 // K elements per block of a stage
#define SP_RAW_BYTES (SP_ROWS * SP_K * 4)
#define SP_TAIL 512
#define SP_FEW 32               // most tokens of a tile that leaves its room to W

// What a block's memory is shared out to.  A tile of many tokens: four stages of X's pieces and of W as stored, two of W's pieces
// in tensor memory.  A tile of few, whose time is W's way through the block: 780 cycles for 16 KB of W so, of which the
// splitting is 700 for either group of warps and the issuing thread's waits and hand-overs 700 too (clock64 stamps); a
// stage of 64 K-elements halves what is paid per stage and puts twice the bytes under way, and the leading products have an
// issuing thread of their own.  4 tokens, before / now: 6144 x 4096 31 / 25 us, 4096 x 4096 20.8 / 17.8, 14336 x 4096 with the
// SiLU-gate 113 / 92, 4096 x 14336 52 / 44; 32 tokens 33 / 26, 21 / 18.5, 117 / 96, 55 / 46.  The bits are the same.  What is left
// of the SiLU-gate's is its second round of blocks, which fills half of the SMs.
template <bool FEW>
struct Sp {
  static constexpr int BN = FEW ? SP_FEW : SP_BN, GROUPS = BN / 16;
  static constexpr int SUBS = FEW ? 2 : 1;        // blocks of SP_K elements per stage
  static constexpr int XSTAGES = 4, RAW = 4, WSTAGES = FEW ? 4 : 2;
  static constexpr int XSUB = BN * 192;           // bytes of X's three pieces of SP_K elements, each rows of 32 bfloat16
  static constexpr int TWO = FEW ? BN : BN / 2;   // tiles of up to this many tokens have two accumulators for the leading sums
  // tensor memory columns: the leading sums, the small products' sums, W's pieces of 16 columns each
  static constexpr int COL_SMALL = FEW ? 2 * BN : BN, COL_W = FEW ? 3 * BN : 2 * BN;
  static constexpr int SMEM = 1024 + SUBS * (XSTAGES * XSUB + RAW * SP_RAW_BYTES) + SP_TAIL;
  static_assert(COL_W + 48 * SUBS * WSTAGES <= 512 && XSTAGES >= WSTAGES, "W's pieces fit, and a stage of X outlives them");
  // A group of warps takes every second stage, and a wait for a barrier's phase means that phase only to one who has waited
  // for the one before: a slot has to stay with its group.
  static_assert(RAW % 2 == 0 && WSTAGES % 2 == 0 && XSTAGES % 2 == 0, "a slot belongs to one group of the splitting warps");
  static_assert(8 * (2 * RAW + 2 * XSTAGES + 5) + 16 <= SP_TAIL, "the barriers fit");
};
#define SP_MAX_SPLITS 8         // portable cluster size

// What a block of SP_K elements, a round of blocks and a reduction take, in cycles, for the choice of tiles (sp_plan).  All ways of
// cutting twelve products of 4 to 96 tokens were timed: up to 32 tokens the choice was the fastest each time; with 750 cycles for the narrow
// tiles too, which were the tiles of many tokens' when this was drawn, 33 to 96 tokens of small matrices took wide tiles that
// are slower (us, then / now): 2048 x 2048 at 64 tokens 13.7 / 12.3, 2048 x 5632 22.2 / 20.8, 1024 x 4096 15.6 / 14.2.
#define SP_COST_TOKEN 6.5
#define SP_COST_STAGE 750.0
#define SP_COST_FEW 500.0
#define SP_COST_ROUND 8000.0
#define SP_COST_REDUCE 40.0

#define SP_LEAST ((127u - 90u) << 23)   // 2^-90 as its bits

#define MODE_ACCUM_F32 1
#define MODE_SWIGLU 2

__device__ int tl_gemm_split_error = 0;

__device__ __forceinline__ bool sp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  return tl_mbar_park(bar, parity, abort_flag, code, &tl_gemm_split_error);
}
__device__ __forceinline__ void sp_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// Descriptor of a K-major tile whose rows are 64 bytes with the 64-byte swizzle: 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

// Two numbers as three pairs of bfloat16, the first number in the low half.
__device__ __forceinline__ void split3(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(b), "f"(a));
  a -= __uint_as_float(p1 << 16);
  b -= __uint_as_float(p1 & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(b), "f"(a));
  a -= __uint_as_float(p2 << 16);
  b -= __uint_as_float(p2 & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p3) : "f"(b), "f"(a));
}
__device__ __forceinline__ void split8(const float4& u, const float4& v, uint4& p1, uint4& p2, uint4& p3) {
  split3(u.x, u.y, p1.x, p2.x, p3.x);
  split3(u.z, u.w, p1.y, p2.y, p3.y);
  split3(v.x, v.y, p1.z, p2.z, p3.z);
  split3(v.z, v.w, p1.w, p2.w, p3.w);
}

// planes[p][m][Kp]: the three pieces of X.  Eight elements per thread.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ X, int ldx, int M, int K, int Kp, uint4* __restrict__ planes) {
  pdl_wait();
  pdl_launch_dependents();
  const int per_row = Kp >> 3;
  const long long n = (long long)M * per_row;
  const bool vec = (ldx & 3) == 0 && ((uintptr_t)X & 15) == 0;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const int m = (int)(i / per_row), k = (int)(i - (long long)m * per_row) * 8;
    const float* x = X + (size_t)m * ldx + k;
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
    if (vec && k + 8 <= K) {
      u = *reinterpret_cast<const float4*>(x);
      v = *reinterpret_cast<const float4*>(x + 4);
    } else {
      float t[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) t[j] = k + j < K ? x[j] : 0.0f;
      u = make_float4(t[0], t[1], t[2], t[3]);
      v = make_float4(t[4], t[5], t[6], t[7]);
    }
    uint4 p1, p2, p3;
    split8(u, v, p1, p2, p3);
    planes[i] = p1;
    planes[n + i] = p2;
    planes[2 * n + i] = p3;
  }
}

struct SplitArgs {
  const float* X;
  const float* W;
  float* C;
  int ldx, ldw, ldc, M, N, K, mode, bn, m_tiles;
  int splits, k_per_split;   // K in blocks of SP_K
};

__device__ __forceinline__ float sp_silu(float g) { return g / (1.0f + expf(-g)); }

// All 128 threads of a group learn whether every one of them passed its wait.
__device__ __forceinline__ bool sp_group_all(bool ok, int group) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)ok), "r"(group + 1)
      : "memory");
  return r != 0;
}

// 16 columns (32 K elements of one piece) of this warp's 32 rows of tensor memory.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// The M operand from tensor memory.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Writes 16 tokens of one column of C.  All 128 threads of the group call it together; `turn` alternates.
template <bool SWIGLU>
__device__ __forceinline__ void sp_write(const SplitArgs& a, float (&v)[16], int n0, int row, int m, int tokens, float* xch,
                                         int turn, int group) {
  const bool up = SWIGLU && row >= 64;
  const int n = n0 + (SWIGLU ? (row & 63) : row);
  uint32_t bad = 0;   // results that are not finite, or so small that the operands may have lost bits: the plain sequence of multiply-adds
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const uint32_t size = __float_as_uint(v[j]) & 0x7fffffffu;       // ordered as the absolute values are, infinities and NaN last
    if (size != 0u && size - SP_LEAST >= 0x7f800000u - SP_LEAST && n < a.N && j < tokens) bad |= 1u << j;
  }
  if (bad) {            // (a branch and no function: the callers' register budgets differ)
    const float* x = a.X + (size_t)m * a.ldx;
    const float* w = a.W + (size_t)(up ? a.N + n : n) * a.ldw;
    // a walk along K for GROUP of them (one after the other an activation tensor of NaN took 27 ms at 300 x 4096 x 4096, 45 times
    // what the CUDA-core kernel takes; more than two under the SiLU-gate spill, which cost finite products 2 %); K, W and
    // its rows allow 16-byte loads
    constexpr int GROUP = SWIGLU ? 2 : 8;
#pragma unroll
    for (int j0 = 0; j0 < 16; j0 += GROUP) {
      if (!(bad >> j0 & ((1u << GROUP) - 1u))) continue;
      float sum[GROUP];
#pragma unroll
      for (int j = 0; j < GROUP; ++j) sum[j] = 0.0f;
#pragma unroll (SWIGLU ? 2 : 1)
      for (int k = 0; k < a.K; k += 4) {
        const float4 wv = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
        for (int j = 0; j < GROUP; ++j)
          if (bad >> (j0 + j) & 1) {
            const float* xj = x + (size_t)(j0 + j) * a.ldx + k;
            sum[j] = fmaf(xj[3], wv.w, fmaf(xj[2], wv.z, fmaf(xj[1], wv.y, fmaf(xj[0], wv.x, sum[j]))));
          }
      }
#pragma unroll
      for (int j = 0; j < GROUP; ++j)
        if (bad >> (j0 + j) & 1) v[j0 + j] = sum[j];
    }
  }
  float* c = a.C + (size_t)m * a.ldc + n;
  if (SWIGLU) {
    float* x = xch + (turn & 1) * 1024 + (row & 63);
    if (up) {
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j * 64] = v[j];
    }
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
    if (!up && n < a.N) {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < tokens) c[(size_t)j * a.ldc] = sp_silu(v[j]) * x[j * 64];
    }
  } else if (n < a.N) {
    if (a.mode == MODE_ACCUM_F32) {
      float prev[16];   // all loads first, so that they are in flight together
#pragma unroll
      for (int j = 0; j < 16; ++j) prev[j] = j < tokens ? c[(size_t)j * a.ldc] : 0.0f;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < tokens) c[(size_t)j * a.ldc] = prev[j] + v[j];
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < tokens) c[(size_t)j * a.ldc] = v[j];
    }
  }
}

template <bool SWIGLU, bool FEW>
__global__ void __launch_bounds__(SP_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                  const SplitArgs args) {
  typedef Sp<FEW> P;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* raw = smem + P::XSTAGES * P::SUBS * P::XSUB;
  uint64_t* raw_full = (uint64_t*)(raw + P::RAW * P::SUBS * SP_RAW_BYTES);   // [RAW]
  uint64_t* raw_empty = raw_full + P::RAW;                         // [RAW]
  uint64_t* full = raw_empty + P::RAW;      // [XSTAGES]: X's pieces (their bytes) and W's (a warp each) are there
  uint64_t* empty = full + P::XSTAGES;      // [XSTAGES]: the stage's instructions are done
  uint64_t* main_full = empty + P::XSTAGES;   // [2]
  uint64_t* main_empty = main_full + 2;       // [2]
  uint64_t* small_full = main_empty + 2;
  uint32_t* tmem_slot = (uint32_t*)(small_full + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bn = args.bn;                               // tokens of the tile
  const int split = (int)(blockIdx.x % args.splits), tile = (int)(blockIdx.x / args.splits);
  const int m0 = (tile % args.m_tiles) * bn;
  constexpr int TILE_N = SWIGLU ? 64 : 128;             // columns of C per tile
  const int n0 = (tile / args.m_tiles) * TILE_N;
  const int k_all = (args.K + SP_K - 1) / SP_K;
  const int k_first = split * args.k_per_split;
  const int n_blocks = min(args.k_per_split, k_all - k_first);       // blocks of SP_K elements
  const int n_k = (n_blocks + P::SUBS - 1) / P::SUBS;               // stages of this block; the last may not be full
  // Stages whose leading products are summed in tensor memory.  A narrow tile has two accumulators, so that handing a
  // sum over costs the instructions nothing, and takes 64 elements (error of 1024 / 4096 / 14336 elements: 0.9e-7 / 1.1e-7 /
  // 1.7e-7; the kernel for few rows of gemm_generic.cu, which sums K / 32 in a row, 1.2e-7 / 2.1e-7 / 3.8e-7); a wide one
  // takes 256 (2.4e-7 at 4096, where the kernel for many rows is at 1.15e-6).
  const bool two = bn <= P::TWO;
  const int chunk = (two ? 2 : 8) / P::SUBS;
  auto hands_over = [&](int i) { return i == n_k - 1 || (i + 1) % chunk == 0; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < P::RAW; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 4); }
    for (int s = 0; s < P::XSTAGES; ++s) { mbar_init(&full[s], 5); mbar_init(&empty[s], FEW ? 2 : 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&main_full[b], 1); mbar_init(&main_empty[b], 128); }
    mbar_init(small_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (threadIdx.x == 0) pdl_launch_dependents();
  const int row = threadIdx.x & 127, group = warp >> 2;
  float* xch = (float*)(raw + (size_t)group * 8192);      // free once all tiles of W are used up

  // Adds the partial tiles of the cluster's blocks and writes: the groups of 16 tokens go round the blocks of the
  // cluster, and in a block round its first three groups of warps.  (A tile of one block goes through shared memory too:
  // the epilogue written out for every register group of the sums is 300 KB of instructions, which took 30 us a tile
  // to fetch.)
  auto reduce = [&]() {
    if (args.splits > 1) cluster_sync_all();   // every block's partial tile is in its shared memory
    else asm volatile("bar.sync 5, 384;" ::: "memory");
    pdl_wait();           // C may be read and written by earlier kernels
    const int tokens = min(bn, args.M - m0);
    const bool live = !*abort_flag;
    int turn = 0;
    for (int g = split + args.splits * group; g * 16 < tokens && live; g += 3 * args.splits, ++turn) {
      const uint32_t at = smem_u32((float*)smem + (size_t)g * 16 * SP_ROWS + row);
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0.0f;
      for (int sp = 0; sp < args.splits; ++sp) {
        float p[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) p[j] = ld_remote_f32(at + j * SP_ROWS * 4, (uint32_t)sp);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += p[j];
      }
      sp_write<SWIGLU>(args, v, n0, row, m0 + g * 16, tokens - g * 16, xch, turn, group);
    }
    __syncwarp();
    if (args.splits > 1) cluster_sync_all();   // nobody leaves while others still read its shared memory
  };

  // Registers per thread of a tile of many tokens: 240 + 2 x 96 + 80 = 512 = 4 x the 128 that the block was launched with.  Those
  // suffice every role of a tile of few.
  if (warp < 4) {
    if (!FEW) asm volatile("setmaxnreg.inc.sync.aligned.u32 240;");
    const uint32_t t_main = tmem + ((uint32_t)(warp * 32) << 16);
    float acc[P::GROUPS][16];
#pragma unroll
    for (int g = 0; g < P::GROUPS; ++g)
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[g][j] = 0.0f;
    bool ok = true;
    uint32_t sums = 0;
    for (int i = 0; i < n_k; ++i) {
      if (!hands_over(i)) continue;
      const uint32_t buf = two ? sums & 1u : 0u, use = two ? sums >> 1 : sums;
      ok = sp_wait(&main_full[buf], use & 1u, abort_flag, 4);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      ++sums;
      tc_fence_after();
      const uint32_t t_sum = t_main + buf * P::TWO;
#pragma unroll
      for (int g = 0; g < P::GROUPS; g += 2) {
        if (g * 16 < bn) {
          uint32_t r[16], q[16];       // (the second may lie past the tile: what it holds is not used)
          tmem_ld16(t_sum + g * 16, r);
          tmem_ld16(t_sum + g * 16 + 16, q);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            acc[g][j] += __uint_as_float(r[j]);
            acc[g + 1][j] += __uint_as_float(q[j]);
          }
        }
      }
      tc_fence_before();
      sp_arrive(&main_empty[buf]);
    }
    ok = ok && sp_wait(small_full, 0, abort_flag, 5);
    ok = sp_group_all(ok, group);
    if (ok) {
      tc_fence_after();
      const int tokens = min(bn, args.M - m0);
#pragma unroll
      for (int g = 0; g < P::GROUPS; ++g) {
        const int c0 = g * 16;
        if (c0 < tokens) {
          uint32_t r[16];
          tmem_ld16(t_main + P::COL_SMALL + c0, r);
          tmem_ld_wait();
          float* part = (float*)smem + (size_t)c0 * SP_ROWS + row;   // [tokens][128 rows]; X's stages are free by now
#pragma unroll
          for (int j = 0; j < 16; ++j) part[j * SP_ROWS] = acc[g][j] + __uint_as_float(r[j]);
        }
      }
    }
    __syncwarp();
    reduce();
  } else if (warp < 12) {
    // ---- W as stored -> its pieces, a row per thread, the two groups of warps in turn
    if (!FEW) asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    const uint32_t t_w = tmem + ((uint32_t)((warp & 3) * 32) << 16) + P::COL_W;
    const uint8_t* own = raw + row * 128;
    for (int i = group - 1; i < n_k; i += 2) {
      const int r = i % P::RAW, before = i - P::WSTAGES;
      bool ok = sp_wait(&raw_full[r], (i / P::RAW) & 1, abort_flag, 1);
      if (!__all_sync(0xffffffffu, ok)) break;
      const uint8_t* src = own + r * (P::SUBS * SP_RAW_BYTES);
      const uint32_t at = t_w + (i % P::WSTAGES) * (48 * P::SUBS);
#pragma unroll
      for (int b = 0; b < P::SUBS; ++b) {
        float4 x[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = *reinterpret_cast<const float4*>(src + b * SP_RAW_BYTES + ((c ^ (row & 7)) << 4));
        uint32_t p1[16], p2[16], p3[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          split3(x[c].x, x[c].y, p1[2 * c], p2[2 * c], p3[2 * c]);
          split3(x[c].z, x[c].w, p1[2 * c + 1], p2[2 * c + 1], p3[2 * c + 1]);
        }
        if (b == P::SUBS - 1) {
          __syncwarp();
          if (lane == 0) sp_arrive(&raw_empty[r]);
        }
        if (b == 0) {      // the stage that had this place in tensor memory
          ok = before < 0 || sp_wait(&empty[before % P::XSTAGES], (before / P::XSTAGES) & 1, abort_flag, 2);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st16(at + 48 * b, p1);       // (of a stage that is not full, the last block is not used)
        tmem_st16(at + 48 * b + 16, p2);
        tmem_st16(at + 48 * b + 32, p3);
      }
      if (!ok) break;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) sp_arrive(&full[i % P::XSTAGES]);
    }
    __syncwarp();
    reduce();
  } else {
    if (!FEW) asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp == 12 && elect_one()) {
      // ---- TMA of W, which does not depend on earlier kernels
      for (int i = 0; i < n_k; ++i) {
        const int r = i % P::RAW;
        if (!sp_wait(&raw_empty[r], ((i / P::RAW) & 1) ^ 1, abort_flag, 3)) break;
        mbar_expect_tx(&raw_full[r], P::SUBS * SP_RAW_BYTES);     // (past K: zeros)
#pragma unroll
        for (int b = 0; b < P::SUBS; ++b) {
          const int k = (k_first + i * P::SUBS + b) * SP_K;
          uint8_t* dst = raw + (r * P::SUBS + b) * SP_RAW_BYTES;
          tma_load_2d(dst, &tm_w, &raw_full[r], k, n0);
          if (SWIGLU) tma_load_2d(dst + SP_RAW_BYTES / 2, &tm_w, &raw_full[r], k, args.N + n0);
        }
      }
    } else if (warp == 14 && elect_one()) {
      // ---- TMA of X's pieces, all three of a stage at once
      pdl_wait();
      for (int i = 0; i < n_k; ++i) {
        const int s = i % P::XSTAGES;
        if (!sp_wait(&empty[s], ((i / P::XSTAGES) & 1) ^ 1, abort_flag, 2)) break;
        mbar_expect_tx(&full[s], (uint32_t)(bn * 192 * P::SUBS));
#pragma unroll
        for (int b = 0; b < P::SUBS; ++b)
          tma_load_3d(smem + (s * P::SUBS + b) * P::XSUB, &tm_x, &full[s], (k_first + i * P::SUBS + b) * SP_K, m0, 0);
      }
    } else if ((warp == 13 || (FEW && warp == 15)) && elect_one()) {
      // ---- MMA issuer.  Of a tile of few tokens the leading products have a thread of their own: the waits for a stage and for
      // a free accumulator cost some 250 cycles each even where nothing is left to wait for.
      const bool smalls = !FEW || warp == 13, leading = !FEW || warp == 15;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(SP_ROWS >> 4) << 24);
      const uint32_t d_small = tmem + P::COL_SMALL;
      bool ok = true;
      uint32_t handed = 0;   // sums handed over so far
      bool fresh = true;     // the next leading product starts a sum
      for (int i = 0; i < n_k && ok; ++i) {
        const int s = i % P::XSTAGES, ws = i % P::WSTAGES;
        ok = sp_wait(&full[s], (i / P::XSTAGES) & 1, abort_flag, 6);
        if (!ok) break;
        tc_fence_after();
        const int subs = min(P::SUBS, n_blocks - i * P::SUBS);
        const uint64_t x0 = smem_desc_k64(smem_u32(smem + s * (P::SUBS * P::XSUB)));
        const uint32_t w0 = tmem + P::COL_W + ws * (48 * P::SUBS);
        if (smalls) {
#pragma unroll
          for (int b = 0; b < P::SUBS; ++b) {
            if (b >= subs) break;
            const uint64_t x1 = x0 + (uint64_t)(b * (P::XSUB >> 4)), x2 = x1 + (uint64_t)bn * 4, x3 = x2 + (uint64_t)bn * 4;
            const uint32_t w1 = w0 + 48 * b, w2 = w1 + 16, w3 = w2 + 16;
#pragma unroll
            for (int k = 0; k < SP_K / 16; ++k) {
              const uint64_t o = (uint64_t)k * 2;   // 32 bytes of shared memory, 8 columns of tensor memory
              umma_bf16_ts(d_small, w3 + 8 * k, x1 + o, idesc, (i == 0 && b == 0 && k == 0) ? 0u : 1u);
              umma_bf16_ts(d_small, w2 + 8 * k, x2 + o, idesc, 1u);
              umma_bf16_ts(d_small, w1 + 8 * k, x3 + o, idesc, 1u);
              umma_bf16_ts(d_small, w2 + 8 * k, x1 + o, idesc, 1u);
              umma_bf16_ts(d_small, w1 + 8 * k, x2 + o, idesc, 1u);
            }
          }
        }
        if (leading) {
          const uint32_t buf = two ? handed & 1u : 0u, use = two ? handed >> 1 : handed;
          if (fresh && use > 0) {
            ok = sp_wait(&main_empty[buf], (use - 1) & 1, abort_flag, 8);
            if (!ok) break;
            tc_fence_after();
          }
          const uint32_t d_main = tmem + buf * P::TWO;
#pragma unroll
          for (int b = 0; b < P::SUBS; ++b) {
            if (b >= subs) break;
#pragma unroll
            for (int k = 0; k < SP_K / 16; ++k)
              umma_bf16_ts(d_main, w0 + 48 * b + 8 * k, x0 + (uint64_t)(b * (P::XSUB >> 4) + k * 2), idesc,
                           (fresh && b == 0 && k == 0) ? 0u : 1u);
          }
          umma_commit(&empty[s]);
          fresh = hands_over(i);
          if (fresh) { umma_commit(&main_full[buf]); ++handed; }
        } else {
          umma_commit(&empty[s]);
        }
      }
      if (ok && smalls) umma_commit(small_full);
    }
  }
  __syncwarp();
  if (args.splits > 1 && warp >= 12) { cluster_sync_all(); cluster_sync_all(); }   // (the other warps' reduction)
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
typedef CUresult (*SpEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static SpEncodeFn sp_encode() {
  static SpEncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (SpEncodeFn)p;
  });
  return fn;
}

template <bool SWIGLU, bool FEW>
static cudaError_t sp_configure(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&attr)[2], int splits) {
  const cudaError_t set = tl_allow_smem<gemm_split_kernel<SWIGLU, FEW>>(Sp<FEW>::SMEM);
  cfg.blockDim = dim3(SP_THREADS);
  cfg.dynamicSmemBytes = Sp<FEW>::SMEM;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return set;
}
// How many clusters of `splits` blocks run at once on this device (the GPCs differ in size: not the SMs divided by it); a block
// takes an SM either way.
template <bool SWIGLU>
static int sp_clusters(int splits, int num_sms) {
  static int known_on[TL_DEVICES][SP_MAX_SPLITS + 1];
  static std::mutex mu;
  if (splits == 1) return num_sms;
  const int device = tl_device();
  int unknown[SP_MAX_SPLITS + 1] = {};
  std::lock_guard<std::mutex> lock(mu);
  int* known = device >= 0 ? known_on[device] : unknown;
  if (known[splits] == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    int n = 0;
    cudaError_t e = sp_configure<SWIGLU, false>(cfg, attr, splits);
    cfg.gridDim = dim3(splits);
    cfg.numAttrs = 1;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, gemm_split_kernel<SWIGLU, false>, &cfg);
    if (e != cudaSuccess) { cudaGetLastError(); n = 0; }
    known[splits] = n > 0 ? n : -1;
  }
  return known[splits];
}

template <bool SWIGLU, bool FEW>
static int run_split(const CUtensorMap& tw, const CUtensorMap& tx, const SplitArgs& a, int tiles, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cudaError_t e = sp_configure<SWIGLU, FEW>(cfg, attr, a.splits);
  if (e != cudaSuccess) return (int)e;
  cfg.gridDim = dim3((unsigned)tiles * a.splits);
  cfg.stream = stream;
  e = cudaLaunchKernelEx(&cfg, gemm_split_kernel<SWIGLU, FEW>, tw, tx, a);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// Tokens per tile and splits of K into `a`: the choice that takes the fewest cycles.  A block of SP_K elements takes SP_COST_TOKEN
// per token for its instructions and SP_COST_STAGE for splitting W at the least, SP_COST_FEW in tiles of few tokens, whose stages are
// paid for whole; a round of blocks SP_COST_ROUND besides, and the reduction over a cluster SP_COST_REDUCE per token of the
// tile.  Returns the tiles along N.
static int sp_plan(SplitArgs& a, int num_sms) {
  const bool swiglu = a.mode == MODE_SWIGLU;
  const int n_tiles = (a.N + (swiglu ? 64 : 128) - 1) / (swiglu ? 64 : 128), k_all = (a.K + SP_K - 1) / SP_K, M = a.M;
  double best = -1.0;
  for (int mt = (M + SP_BN - 1) / SP_BN, tries = 0; tries < 8 && mt <= M; ++mt, ++tries) {
    const int bn = ((M + mt - 1) / mt + 15) / 16 * 16;
    const long long tiles = (long long)n_tiles * ((M + bn - 1) / bn);
    for (int sp = 1; sp <= SP_MAX_SPLITS && (sp == 1 || sp * 8 <= k_all); ++sp) {
      const int at_once = swiglu ? sp_clusters<true>(sp, num_sms) : sp_clusters<false>(sp, num_sms);
      if (at_once <= 0 || (sp > 1 && tiles > at_once)) continue;    // K is split only over blocks that would idle
      const int per = (k_all + sp - 1) / sp;
      if (per * (sp - 1) >= k_all) continue;                        // no empty split
      const bool few = bn <= SP_FEW;
      const double least = few ? SP_COST_FEW : SP_COST_STAGE, block = SP_COST_TOKEN * bn > least ? SP_COST_TOKEN * bn : least;
      const int paid = few ? (per + Sp<true>::SUBS - 1) / Sp<true>::SUBS * Sp<true>::SUBS : per;
      const double cost = (double)((tiles + at_once - 1) / at_once) * (paid * block + SP_COST_ROUND) +
                          (sp > 1 ? SP_COST_REDUCE * bn : 0.0);
      if (best < 0.0 || cost < best) { best = cost; a.bn = bn; a.splits = sp; a.k_per_split = per; }
    }
  }
  a.m_tiles = (M + a.bn - 1) / a.bn;
  return n_tiles;
}

// Tokens per tile, splits of K and tiles of a product, for the tests.
extern "C" void tl_gemm_split_plan(int M, int N, int K, int mode, int num_sms, int* bn, int* splits, int* tiles) {
  SplitArgs a = {nullptr, nullptr, nullptr, 0, 0, 0, M, N, K, mode, 0, 0, 1, 0};
  *tiles = sp_plan(a, num_sms) * a.m_tiles;
  *bn = a.bn;
  *splits = a.splits;
}

// Bytes of scratch that tl_gemm_split needs for X's pieces.
extern "C" long long tl_gemm_split_scratch(int M, int K) { return 6ll * M * ((K + 7) / 8 * 8); }

// Returns 0, a CUDA error, or -2 when these sizes or alignments are not taken (the caller then uses the CUDA-core
// kernel).  N counts output columns; in mode 2 W has 2N rows.  `scratch`: tl_gemm_split_scratch bytes, on 16 bytes.
extern "C" int tl_gemm_split(const float* X, int ldx, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                             int mode, int num_sms, void* scratch, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (mode < 0 || mode > 3) return -1;
  if (K <= 0 || K % 4 || ldw % 4 || ((uintptr_t)W & 15) || ((uintptr_t)scratch & 15)) return -2;
  const bool swiglu = mode == MODE_SWIGLU;
  const int Kp = (K + 7) / 8 * 8;
  SplitArgs a = {X, W, C, ldx, ldw, ldc, M, N, K, mode, 0, 0, 1, 0};
  const int n_tiles = sp_plan(a, num_sms);
  const long long tiles = (long long)n_tiles * a.m_tiles;
  if (tiles * a.splits > 0x7fffffffll) return -2;
  SpEncodeFn fn = sp_encode();
  if (!fn) return -2;
  CUtensorMap tw, tx;
  {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N * (swiglu ? 2 : 1)}, strides[1] = {(cuuint64_t)ldw * 4};
    const cuuint32_t box[2] = {SP_K, swiglu ? 64u : 128u}, estr[2] = {1, 1};
    if (fn(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -2;
  }
  {
    const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)M, 3},
                     strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)Kp * 2 * (cuuint64_t)M};
    const cuuint32_t box[3] = {SP_K, (cuuint32_t)a.bn, 3}, estr[3] = {1, 1, 1};
    if (fn(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, scratch, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -2;
  }
  const long long n8 = (long long)M * (Kp / 8);
  const int rc = tl_launch(split_rows_kernel, dim3((unsigned)((n8 + 255) / 256 < 4096 ? (n8 + 255) / 256 : 4096)), dim3(256),
                           0, stream, X, ldx, M, K, Kp, (uint4*)scratch);
  if (rc != 0) return rc;
  if (a.bn <= SP_FEW)
    return swiglu ? run_split<true, true>(tw, tx, a, (int)tiles, stream) : run_split<false, true>(tw, tx, a, (int)tiles, stream);
  return swiglu ? run_split<true, false>(tw, tx, a, (int)tiles, stream) : run_split<false, false>(tw, tx, a, (int)tiles, stream);
}

// Reads and clears the error word that a kernel sets when one of its bounded waits ran out.  Synchronises the device.
extern "C" int tl_gemm_split_take_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, tl_gemm_split_error, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(tl_gemm_split_error, &zero, sizeof(int));
  return v;
}
