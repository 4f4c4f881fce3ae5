// 32-bit matrix product on the tensor cores: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) (+ R), fp32 in and out.
//
// A float is the sum of three bf16 numbers, x = x0 + x1 + x2, exactly: each takes the next eight bits of what is left (24 in
// all).  The product of two such sums has nine terms; the three with i + j > 2 are below 2^-25 of it and left out, the other
// six are bf16 products, which the tensor cores take exactly and add in fp32.  Those sums are cut off, not rounded, so they stay
// short: 32 k at a time, the five small terms before the large one, and each such sum is added to a running fp32 sum in
// registers, rounded to nearest.  Norm of the error against 64 bits, normal data, here / by multiply-adds: K = 1,024 5.6e-8 / 2.2e-7,
// 4,096 2.0e-7 / 8.1e-7, 12,288 1.8e-7 / 1.3e-6 (cut along K in four).
//
// An output's operations and their order depend on its column, N and K alone: on no other row, on no number of rows and on no tile
// width, so a row's bits do not change with the batch.
//
// Layout.  Weights are the M side of the MMA: clusters of two CTAs own 256 features (cta_group::2, 128 lanes of tensor memory
// each), tokens are its columns, up to 192 a tile.
//   warp 0      weights, fp32, by TMA: 128 rows x 32 k a stage (128-byte swizzle)
//   warp 1      (leader) issues the MMAs: per 32 k 6 terms x 2
//   warp 2      the activations' pieces by TMA, 64 k of all three a stage; each CTA holds half of the tile's tokens
//   warps 4-7   a thread per weight row: 32 fp32 to three bf16 pieces, into tensor memory (the A operand): shared memory would
//               have to give them back six times, more than it can beside the activations
//   warps 8-15  a thread per feature and half of the tokens: takes the sum of 32 k out of tensor memory into its
//               running sums, and writes the tile
// Tensor memory: a ring of two to four slots, an accumulator and a weight buffer of 48 columns each.
// The activations are cut into pieces by a kernel of its own before it ([3, M, K] bf16 in scratch): every tile reads all of them.
//
// Tiles that fill no whole round of 74 pairs are cut along K, each into the same number of parts (by N and K alone); a part's sums go to
// scratch and the part that arrives last adds them in order.
//
// What the pieces cannot hold: a product that is not finite is taken again by plain multiply-adds (infinities, and rows beyond the
// bf16 range); rows of A smaller than 2^-64 throughout are cut at 2^64 times their size; weights below 2^-110 lose bits under 2^-133.
//
// What bounds it: many rows, the tensor cores' 6 x 2 M N K at bf16 rates (1,152 clocks per 32 k of a tile of 192 tokens; it takes about
// 1,300, behind the weights' way through registers); few rows, the weights' bytes and 64 clocks an MMA for its A operand.  Measured, us,
// tiles of multiply-adds before / this: 185 x 24,576 x 4,096 871 / 169 (221 TFLOP/s), 185 x 4,096 x 12,288 683 / 105, 185 x 151,936 x 4,096
// 5,550 / 979, 1,024 x 24,576 x 4,096 4,735 / 902; one row: 24,576 x 4,096 143 / 89, 151,936 x 4,096 785 / 473 (5,260 GB/s).
//
// Every wait is bounded: after two to three seconds the role whose wait ran out records its code in `status`, all roles leave, tensor memory is
// freed.
#include <cuda.h>
#include <float.h>

#include "common.cuh"

#define BF 128                    // features per CTA (a tile has 256)
#define KC 32                     // k per step: the weights' stage, and the sum that leaves tensor memory
#define KB 64                     // k per stage of the activations
#define MAX_BN 192                // tokens per tile
#define RAW_BYTES (BF * KC * 4)
#define MAX_STAGES 12
#define WARPS 16
#define THREADS (WARPS * 32)
#define A_COLS 48                 // tensor memory columns of a weight buffer: 3 pieces x 16
#define MAX_RING 4
// registers a thread of the four warpgroups: 40 + 104 + 176 + 176 of the 4 x 128 that the block is launched with
#define REGS_ISSUE 40
#define REGS_CONVERT 104
#define REGS_EPILOGUE 176
#define PAIRS 74                  // pairs that the cut along K is made for (148 multiprocessors): part of the order of the sums
#ifndef ODI_WAIT_CYCLES
#define ODI_WAIT_CYCLES 4000000000ll   // about two seconds of SM clock; a self-test build makes it milliseconds
#endif
// How long a role waits for a copy, for the role that waits for that copy, and for those that wait for it in turn: a copy that never comes is
// reported by the role that missed it, in either CTA.
#define WAIT_CYCLES ((long long)ODI_WAIT_CYCLES)
#define WAIT_CYCLES_2 (WAIT_CYCLES + WAIT_CYCLES / 4)
#define WAIT_CYCLES_3 (WAIT_CYCLES + WAIT_CYCLES / 2)

#define ERR_WEIGHTS 41
#define ERR_MMA 42
#define ERR_TOKENS 43
#define ERR_CONVERT 44
#define ERR_EPILOGUE 45

struct F32SplitArgs {
  const float* x;          // [M, ldx]
  const float* w;          // [N, ldw]
  float* out;              // [M, ldo]
  const float* res;        // null, or [M, ldr]; may be out
  const float* bias;       // null, or [N]
  const float* row_scale;  // [M]: 1; 2^-64 for rows cut at 2^64 times their size; NaN for rows that hold one
  float* partial;          // [rest tiles, splits, M, 256]
  int* tickets;            // [rest tiles, m_tiles, 2], zero on entry
  int* status;
  int M, N, K, ldx, ldw, ldo, ldr;
  int bn, m_tiles;         // tokens a tile (a multiple of 32), tiles of tokens
  int full, rest, splits;  // feature tiles in one piece, those behind them, and their parts along K
  int raw_stages, tok_stages;
  int ring;                // slots in tensor memory (at most MAX_RING): ring * (bn + A_COLS) <= 512
  int withheld;            // self-test of the bounded waits: 1, the weights' producers request nothing; 2, the activations'
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait.  False when it gave up or when another role of the CTA did.  The role whose own wait ran out records its code before it raises
// the flag, so that `status` names it and not one that merely left after it.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code, long long limit) {
  if (mbar_test(bar, parity)) return true;
  const long long start = clock64();
  for (uint32_t i = 0;; ++i) {
    if (mbar_test(bar, parity)) return true;
    if ((i & 0xf) == 0xf) {
      if (*abort_flag) return false;
      if (clock64() - start > limit) break;
    }
  }
  atomicCAS(status, 0, code);
  *abort_flag = 1;
  return false;
}
// The same by a whole warp, with one answer for all of its lanes.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status, int code, long long limit) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, code, limit));
}
// After a role gave up: the copies that are still on their way to the stages of the last `stages` uses before `issued` (bounded).
__device__ __forceinline__ void drain(uint32_t full, int stages, int issued) {
  for (int i = max(0, issued - stages); i < issued; ++i)
    for (int n = 0; n < 100000 && !mbar_test(full + 8 * (i % stages), (uint32_t)(i / stages) & 1u); ++n) {}
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t local, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t cluster_bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// Into this CTA's shared memory, its bytes counted on a barrier of the pair's leader.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D += A B over both CTAs: A (each CTA's 128 rows x 16 k, two bf16 a column) in tensor memory, B in shared memory.
__device__ __forceinline__ void umma_pair_a_tmem(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives, once the MMAs issued so far have completed, on the barrier at this offset in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  const uint16_t both = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(both) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// The loads so far have arrived: r as well.
__device__ __forceinline__ void tmem_wait16(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}
// K-major tile written by TMA with the 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3ffff) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// kind::f16: fp32 accumulator, bf16 A and B, both K-major.
__device__ __forceinline__ uint32_t instr_desc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Two floats' next eight bits as a pair of bf16 (a in the low half), and what is left of them.
__device__ __forceinline__ uint32_t take_piece(float& a, float& b) {
  uint32_t p;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(b), "f"(a));
  a -= __uint_as_float(p << 16);
  b -= __uint_as_float(p & 0xffff0000u);
  return p;
}

// ------------------------------------------------------------------------------ the activations' pieces

#define CUT_THREADS 256
// A block per row: pieces[p, m, k], the row's scale; block 0 clears the tickets.
__global__ void __launch_bounds__(CUT_THREADS)
f32_cut_kernel(const float* __restrict__ x, bf16* __restrict__ pieces, float* __restrict__ row_scale, int* __restrict__ tickets,
               int n_tickets, int M, int K, int ldx, int pitch) {
  __shared__ float scratch[33];
  pdl_wait();
  pdl_launch_dependents();      // not earlier: the product reads weights before it waits, and those may be the work of a kernel before this one
  const int m = blockIdx.x;
  if (m == 0)
    for (int i = threadIdx.x; i < n_tickets; i += CUT_THREADS) tickets[i] = 0;
  const float4* row = (const float4*)(x + (size_t)m * ldx);
  float most = 0.f;
  bool nan = false;
  for (int i = threadIdx.x; i < K / 4; i += CUT_THREADS) {
    const float4 v = row[i];
    most = fmaxf(fmaxf(most, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    nan |= v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
  }
  nan = __syncthreads_or(nan);
  most = warp_max(most);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = most;
  __syncthreads();
  most = scratch[0];
#pragma unroll
  for (int i = 1; i < CUT_THREADS / 32; ++i) most = fmaxf(most, scratch[i]);
  const bool small = most < 5.421010862427522e-20f;      // 2^-64
  const float up = small ? 1.8446744073709552e19f : 1.f;
  if (threadIdx.x == 0) row_scale[m] = nan ? __uint_as_float(0x7fffffffu) : small ? 5.421010862427522e-20f : 1.f;
  for (int i = threadIdx.x; i < K / 4; i += CUT_THREADS) {
    float4 v = row[i];
    v.x *= up; v.y *= up; v.z *= up; v.w *= up;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint32_t lo = take_piece(v.x, v.y), hi = take_piece(v.z, v.w);
      *(uint2*)(pieces + ((size_t)p * M + m) * pitch + 4 * i) = make_uint2(lo, hi);
    }
  }
}

// ------------------------------------------------------------------------------ the product

// The u-th piece of work: feature tile, token tile, its steps of 32 k, and of a tile that is cut, which one and which part.
struct Unit { int n0, t0, k0, steps, cut, part; };
__device__ __forceinline__ bool unit_of(const F32SplitArgs& a, int u, Unit& t) {
  const int full_units = a.full * a.m_tiles;
  int k1 = a.K, tile;
  t.k0 = 0; t.cut = -1; t.part = 0;
  if (u < full_units) {
    tile = u / a.m_tiles;
    t.t0 = u % a.m_tiles * a.bn;
  } else {
    const int v = u - full_units, ts = v / a.m_tiles;
    if (ts >= a.rest * a.splits) return false;
    t.t0 = v % a.m_tiles * a.bn;
    t.cut = ts % a.rest;
    t.part = ts / a.rest;
    tile = a.full + t.cut;
    const int blocks = (a.K + KB - 1) / KB;
    t.k0 = blocks * t.part / a.splits * KB;
    k1 = min(blocks * (t.part + 1) / a.splits * KB, a.K);
  }
  t.n0 = tile * 2 * BF;
  t.steps = (k1 - t.k0 + KC - 1) / KC;
  return true;
}

// x . w by a warp in plain multiply-adds, for a product that is not finite: lane l takes the k with k % 32 = l.
__device__ __forceinline__ float plain_dot(const float* x, const float* w, int K) {
  float s = 0.f;
  for (int k = threadIdx.x & 31; k < K; k += 32) s = fmaf(x[k], w[k], s);
  return warp_sum(s);
}

__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const F32SplitArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // raw_full, raw_empty (this CTA's), tok_full (leader's), tok_empty (each CTA's); of a slot ready (leader's): weights written,
  // accumulator read; done (each CTA's): its products are
  __shared__ __align__(8) uint64_t bars[4 * MAX_STAGES + 2 * MAX_RING];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int last_part;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int half = a.bn >> 1;                                // tokens whose pieces this CTA holds
  const uint32_t tok_bytes = 3 * half * 128;
  const uint32_t raw0 = smem_u32(smem), tok0 = raw0 + a.raw_stages * RAW_BYTES;
  const uint32_t raw_full = smem_u32(bars), raw_empty = raw_full + 8 * MAX_STAGES, tok_full = raw_empty + 8 * MAX_STAGES,
                 tok_empty = tok_full + 8 * MAX_STAGES, ready = tok_empty + 8 * MAX_STAGES, done = ready + 8 * MAX_RING;
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(raw_full + 8 * s, 1);
      mbar_init(raw_empty + 8 * s, 4);          // the converting warps
      mbar_init(tok_full + 8 * s, 2);           // both CTAs' producers
      mbar_init(tok_empty + 8 * s, 1);
    }
    for (int b = 0; b < MAX_RING; ++b) {
      mbar_init(ready + 8 * b, 24);             // of both CTAs 4 converting and 8 epilogue warps each
      mbar_init(done + 8 * b, 1);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();               // both CTAs' barriers exist before anybody signals across
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_slot, 0), tmem_a = tmem + a.ring * a.bn;
  pdl_launch_dependents();

  Unit t;
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
    if (warp == 0 && lane == 0) {
      bool ok = a.withheld != 1;
      int it = 0, s = 0;
      uint32_t phase = 1;
      for (int u = pair; ok && unit_of(a, u, t); u += n_pairs)
        for (int st = 0; st < t.steps; ++st, ++it) {
          if (it >= a.raw_stages && !mbar_wait(raw_empty + 8 * s, phase, abort_ptr, a.status, ERR_WEIGHTS, WAIT_CYCLES_3)) { ok = false; break; }
          mbar_expect_tx(raw_full + 8 * s, RAW_BYTES);
          tma_load_2d(raw0 + s * RAW_BYTES, &map_w, t.k0 + st * KC, t.n0 + (int)rank * BF, raw_full + 8 * s);
          if (++s == a.raw_stages) { s = 0; phase ^= 1u; }
        }
      if (!ok) drain(raw_full, a.raw_stages, it);
    } else if (warp == 1 && rank == 0) {
      // the whole warp goes through the loop (see elect_one)
      const bool issues = elect_one();
      const uint32_t idesc = instr_desc_bf16(2 * BF, a.bn);
      const int piece = half * 128 >> 4;          // from one piece of the activations to the next, in the descriptor's units
      bool ok = true;
      int s = 0, slot = 0;
      uint32_t phase = 0, tok_phase = 0;
      uint64_t db = 0;
      for (int u = pair; ok && unit_of(a, u, t); u += n_pairs)
        for (int st = 0; st < t.steps; ++st) {
          if ((st & 1) == 0) {
            if (!warp_wait(tok_full + 8 * s, tok_phase, abort_ptr, a.status, ERR_MMA, WAIT_CYCLES)) { ok = false; break; }
            db = smem_desc_k_sw128(tok0 + s * tok_bytes);
          }
          if (!warp_wait(ready + 8 * slot, phase, abort_ptr, a.status, ERR_MMA, WAIT_CYCLES_2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem + slot * a.bn, wa = tmem_a + slot * A_COLS;
          const uint64_t b = db + (st & 1) * 4;
          // the small terms first: what the sum cuts off is in proportion to what it holds
          constexpr int wi[6] = {2, 0, 1, 1, 0, 0}, xi[6] = {0, 2, 1, 0, 1, 0};
          if (issues) {
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
              for (int j = 0; j < 2; ++j)
                umma_pair_a_tmem(d, wa + 16 * wi[i] + 8 * j, b + xi[i] * piece + 2 * j, idesc, i + j > 0 ? 1u : 0u);
          }
          if (issues) umma_commit_pair(done + 8 * slot);
          if (++slot == a.ring) { slot = 0; phase ^= 1u; }
          if ((st & 1) == 1 || st + 1 == t.steps) {
            if (issues) umma_commit_pair(tok_empty + 8 * s);
            if (++s == a.tok_stages) { s = 0; tok_phase ^= 1u; }
          }
        }
    } else if (warp == 2 && lane == 0) {
      pdl_wait();                     // the pieces come from the kernel before
      const uint32_t leader_full = map_to_rank(tok_full, 0);
      bool ok = a.withheld != 2;
      int it = 0, s = 0;
      uint32_t phase = 1;
      for (int u = pair; ok && unit_of(a, u, t); u += n_pairs)
        for (int b = 0; 2 * b < t.steps; ++b, ++it) {
          if (it >= a.tok_stages && !mbar_wait(tok_empty + 8 * s, phase, abort_ptr, a.status, ERR_TOKENS, WAIT_CYCLES_3)) { ok = false; break; }
          mbar_expect_tx_cluster(leader_full + 8 * s, tok_bytes);
          for (int p = 0; p < 3; ++p)
            tma_load_2d_pair(tok0 + s * tok_bytes + p * half * 128, &map_x, t.k0 + b * KB, p * a.M + t.t0 + (int)rank * half, leader_full + 8 * s);
          if (++s == a.tok_stages) { s = 0; phase ^= 1u; }
        }
      if (!ok && rank == 0) drain(tok_full, a.tok_stages, it);
    }
  } else if (warp < 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_CONVERT));
    const int row = (warp & 3) * 32 + lane;
    const uint32_t leader_ready = map_to_rank(ready, 0);
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true, first = true;
    int s = 0, slot = 0;
    uint32_t raw_phase = 0, phase = 1;
    for (int u = pair; ok && unit_of(a, u, t); u += n_pairs)
      for (int st = 0; st < t.steps; ++st) {
        if (!warp_wait(raw_full + 8 * s, raw_phase, abort_ptr, a.status, ERR_CONVERT, WAIT_CYCLES)) { ok = false; break; }
        const uint8_t* mine = smem + s * RAW_BYTES + row * 128;
        float v[32];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 f = *(const float4*)(mine + ((q ^ (row & 7)) << 4));
          v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
        }
        uint32_t w[3][16];
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int i = 0; i < 16; ++i) w[p][i] = take_piece(v[2 * i], v[2 * i + 1]);
        __syncwarp();
        if (lane == 0) mbar_arrive(raw_empty + 8 * s);
        if (++s == a.raw_stages) { s = 0; raw_phase ^= 1u; }
        // the products that read the slot's weights a round ago
        if (!first && !warp_wait(done + 8 * slot, phase, abort_ptr, a.status, ERR_CONVERT, WAIT_CYCLES_3)) { ok = false; break; }
        tc_fence_after();
        const uint32_t dst = tmem_a + lanes + slot * A_COLS;
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_st16(dst + 16 * p, w[p]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_ready + 8 * slot);
        if (++slot == a.ring) { slot = 0; phase ^= 1u; first = false; }
      }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_EPILOGUE));
    pdl_wait();                       // the residual, the scales and the tickets
    const int lane_group = warp & 3, part_of_tile = (warp - 8) >> 2;
    const uint32_t leader_ready = map_to_rank(ready, 0);
    const uint32_t src = tmem + ((uint32_t)(lane_group * 32) << 16) + part_of_tile * half;
    const int feature = (int)rank * BF + lane_group * 32 + lane;       // within the tile's 256
    float acc[MAX_BN / 2];
    bool ok = true;
    int slot = 0;
    uint32_t phase = 0;
    if (lane == 0)
      for (int b = 0; b < a.ring; ++b) mbar_arrive_cluster(leader_ready + 8 * b);      // the accumulators are free
    for (int u = pair; unit_of(a, u, t); u += n_pairs) {
#pragma unroll
      for (int c = 0; c < MAX_BN / 2; ++c) acc[c] = 0.f;
      // a warp whose wait gave up still walks its units: the others count on it at the barriers below
      for (int st = 0; ok && st < t.steps; ++st) {
        if (!warp_wait(done + 8 * slot, phase, abort_ptr, a.status, ERR_EPILOGUE, WAIT_CYCLES_3)) { ok = false; break; }
        tc_fence_after();
        const uint32_t from = src + slot * a.bn;
#pragma unroll
        for (int c = 0; c < MAX_BN / 2; c += 32)
          if (c < half) {
            uint32_t r[32];
            tmem_ld16(from + c, r);
            if (c + 16 < half) tmem_ld16(from + c + 16, r + 16);
            tmem_wait16(r);
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(r[i]);
            if (c + 16 < half) {
              tmem_wait16(r + 16);
#pragma unroll
              for (int i = 16; i < 32; ++i) acc[c + i] += __uint_as_float(r[i]);
            }
          }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(leader_ready + 8 * slot);
        if (++slot == a.ring) { slot = 0; phase ^= 1u; }
      }
      const int m0 = t.t0 + part_of_tile * half, cols = min(half, a.M - m0);      // this warp's tokens: m0 .. m0 + cols - 1
      const float* parts = nullptr;
      if (t.cut >= 0) {
        if (ok) {
          float* mine = a.partial + ((size_t)(t.cut * a.splits + t.part) * a.M + m0) * (2 * BF) + feature;
#pragma unroll
          for (int c = 0; c < MAX_BN / 2; ++c)
            if (c < cols) mine[(size_t)c * (2 * BF)] = acc[c];
          __threadfence();
        }
        epilogue_sync();
        if (threadIdx.x == 8 * 32)
          last_part = *abort_ptr ? -1 : atomicAdd(a.tickets + (t.cut * a.m_tiles + t.t0 / a.bn) * 2 + (int)rank, 1) == a.splits - 1 ? 1 : 0;
        epilogue_sync();
        const int last = last_part;
        epilogue_sync();
        if (last < 0) ok = false;
        if (last <= 0) continue;
        __threadfence();
        parts = a.partial + ((size_t)t.cut * a.splits * a.M + m0) * (2 * BF) + feature;
      }
      if (!ok || cols <= 0) continue;
      const int n = t.n0 + feature;
      const bool has = n < a.N;
      const float b = a.bias != nullptr && has ? a.bias[n] : 0.f;
      uint32_t bad[MAX_BN / 64] = {};
#pragma unroll
      for (int g = 0; g < MAX_BN / 2; g += 16) {
        const int left = cols - g;
        if (left <= 0) break;
        float v[16];
        const float scale = a.row_scale[m0 + g + min(lane & 15, left - 1)];      // a lane per token, handed around below
        if (parts != nullptr) {      // in the parts' order
          const float* from = parts + (size_t)g * (2 * BF);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = i < left ? __ldcg(from + i * (2 * BF)) : 0.f;
#pragma unroll 2
          for (int p = 1; p < a.splits; ++p) {
            from += (size_t)a.M * (2 * BF);
            float more[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) more[i] = i < left ? __ldcg(from + i * (2 * BF)) : 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += more[i];
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = acc[g + i];
        }
        uint32_t off = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          v[i] *= __shfl_sync(0xffffffffu, scale, i);
          if (!(fabsf(v[i]) <= FLT_MAX)) off |= 1u << i;
        }
        off &= has ? (left < 16 ? (1u << left) - 1 : 0xffffu) : 0;
        bad[g >> 5] |= off << (g & 31);
        if (a.bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] += b;
        }
        if (a.res != nullptr && has) {
          const float* from = a.res + (size_t)(m0 + g) * a.ldr + n;
          float r[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) { r[i] = i < left ? *from : 0.f; from += a.ldr; }
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] += r[i];
        }
        if (has) {
          float* to = a.out + (size_t)(m0 + g) * a.ldo + n;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (i < left && !((off >> i) & 1u)) *to = v[i];
            to += a.ldo;
          }
        }
      }
      if (__any_sync(0xffffffffu, (bad[0] | bad[1] | bad[2]) != 0)) {
        for (int c = 0; c < cols; ++c) {
          const int m = m0 + c;
          uint32_t left = __ballot_sync(0xffffffffu, ((c < 32 ? bad[0] : c < 64 ? bad[1] : bad[2]) >> (c & 31)) & 1u);
          while (left) {
            const int l = __ffs(left) - 1;
            left &= left - 1;
            const float scale = a.row_scale[m];
            float v = scale != scale ? scale : plain_dot(a.x + (size_t)m * a.ldx, a.w + (size_t)(t.n0 + (int)rank * BF + lane_group * 32 + l) * a.ldw, a.K);
            if (lane == l) {
              if (a.bias != nullptr) v += b;
              if (a.res != nullptr) v += a.res[(size_t)m * a.ldr + n];
              a.out[(size_t)m * a.ldo + n] = v;
            }
          }
        }
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();               // nobody leaves while its barriers or tensor memory may still be used by the peer
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// ------------------------------------------------------------------------------ host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}
// A row-major matrix in boxes of box_rows x 128 bytes with the 128-byte swizzle.
static int make_map(CUtensorMap* map, CUtensorMapDataType type, int elem_bytes, const void* base, long rows, int K, long pitch, int box_rows) {
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr) return ODI_ERR_UNSUPPORTED;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch * elem_bytes};
  cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = fn(map, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : ODI_ERR_ARGUMENT;
}

struct F32SplitPlan { int bn, m_tiles, full, rest, splits, pitch; size_t scale_at, ticket_at, partial_at, bytes; };
static F32SplitPlan plan_of(int M, int N, int K) {
  F32SplitPlan p;
  p.m_tiles = (M + MAX_BN - 1) / MAX_BN;
  p.bn = ((M + p.m_tiles - 1) / p.m_tiles + 31) / 32 * 32;
  const int tiles = (N + 2 * BF - 1) / (2 * BF), blocks = (K + KB - 1) / KB;
  p.full = tiles / PAIRS * PAIRS;
  p.rest = tiles - p.full;
  // parts of the tiles behind the whole rounds: the number that leaves the shortest walk; a part costs about a hundredth of a tile (its sums'
  // way through scratch) and keeps at least 256 k
  p.splits = 1;
  double least = 1e30;
  for (int s = 1; p.rest > 0 && s <= 16 && (s == 1 || blocks / s >= 4); ++s) {
    const double cost = (double)((p.rest * s + PAIRS - 1) / PAIRS) / s + (s > 1 ? 0.01 * s : 0.0);
    if (cost < least) { least = cost; p.splits = s; }
  }
  if (p.splits == 1) { p.full = tiles; p.rest = 0; }
  p.pitch = (K + 7) / 8 * 8;
  const size_t align = 255;
  p.scale_at = ((size_t)3 * M * p.pitch * 2 + align) & ~align;
  p.ticket_at = (p.scale_at + (size_t)M * 4 + align) & ~align;
  p.partial_at = (p.ticket_at + (size_t)p.rest * p.m_tiles * 2 * 4 + align) & ~align;
  p.bytes = p.partial_at + (size_t)p.rest * p.splits * M * 2 * BF * 4;
  return p;
}

extern "C" long odi_gemm_f32_split_scratch(int M, int N, int K) { return M <= 0 || N <= 0 || K <= 0 ? 0 : (long)plan_of(M, N, K).bytes; }

// x [M, ldx], w [N, ldw], out [M, ldo], res null or [M, ldr] (may be out), bias null or [N], all fp32; K, ldx and ldw multiples of 4,
// x and w on 16-byte boundaries; scratch: odi_gemm_f32_split_scratch bytes, 256-byte aligned; status: receives a code if a wait gives up.
// withheld: 0, or a self-test of that (F32SplitArgs).
extern "C" int odi_gemm_f32_split(const float* x, const float* w, float* out, const float* res, const float* bias, int M, int N,
                                  int K, int ldx, int ldw, int ldo, int ldr, void* scratch, long scratch_bytes, int* status,
                                  int withheld, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || status == nullptr) return ODI_ERR_ARGUMENT;
  if (K % 4 || ldx % 4 || ldw % 4 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)scratch & 255)) return ODI_ERR_UNSUPPORTED;
  const F32SplitPlan p = plan_of(M, N, K);
  if (scratch == nullptr || (size_t)scratch_bytes < p.bytes) return ODI_ERR_ARGUMENT;
  const long units = (long)p.full * p.m_tiles + (long)p.rest * p.splits * p.m_tiles;
  if (units > 0x3fffffffL || 3L * M > 0x7fffffffL) return ODI_ERR_UNSUPPORTED;
  static thread_local int sms = 0, known = -1;      // of the device that this thread launched on last: the attribute is the device's
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess && device != known) {
    known = -1;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 1024);
    if (e == cudaSuccess) known = device;
  }
  if (e != cudaSuccess) return (int)e;
  uint8_t* base = (uint8_t*)scratch;
  F32SplitArgs a;
  a.x = x; a.w = w; a.out = out; a.res = res; a.bias = bias; a.status = status; a.withheld = withheld;
  a.row_scale = (float*)(base + p.scale_at); a.tickets = (int*)(base + p.ticket_at); a.partial = (float*)(base + p.partial_at);
  a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldo = ldo; a.ldr = ldr;
  a.bn = p.bn; a.m_tiles = p.m_tiles; a.full = p.full; a.rest = p.rest; a.splits = p.splits;
  const int tok_bytes = 3 * (p.bn / 2) * 128, room = 224 * 1024 - 2048;
  a.tok_stages = p.bn > 64 ? 3 : 6;
  a.raw_stages = (room - a.tok_stages * tok_bytes) / RAW_BYTES;
  if (a.raw_stages > MAX_STAGES) a.raw_stages = MAX_STAGES;
  a.ring = 512 / (p.bn + A_COLS);
  if (a.ring > MAX_RING) a.ring = MAX_RING;
  CUtensorMap mx, mw;
  int rc = make_map(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, 3L * M, K, p.pitch, p.bn / 2);
  if (rc == 0) rc = make_map(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, w, N, K, ldw, BF);
  if (rc != 0) return rc;
  odi_rc = launch_pdl(f32_cut_kernel, dim3(M), dim3(CUT_THREADS), 0, stream, x, (bf16*)base, (float*)(base + p.scale_at), a.tickets,
                      p.rest * p.m_tiles * 2, M, K, ldx, p.pitch);
  const int pairs = units < sms / 2 ? (int)units : sms / 2;
  odi_rc = launch_pdl(gemm_f32_split_kernel, dim3(2 * pairs), dim3(THREADS), (size_t)a.raw_stages * RAW_BYTES + a.tok_stages * tok_bytes + 1024,
                      stream, mx, mw, a);
  return launch_status();
}
