// bf16 products of many rows, one weight matrix per expert, on the 5th-generation tensor cores: rows offsets[e] .. offsets[e + 1] - 1 of x
// (sorted by expert; the ranges stay on the device) go through weights e,
//   out[row, n] = epilogue( sum_k x[row, k] * w[e, n, k] ),  fp32 accumulation.
//
// The output features lie on the tensor core's lanes and the rows on its columns, in steps of 32 up to 256, so that an expert of a few
// dozen rows costs no more products than it has.  Persistent clusters of two CTAs, the two-CTA form of the MMA: a tile is 256 weight rows
// (128 a CTA, 64 + 64 of them gate and up rows for the gated epilogue) and an expert's rows, cut evenly where it has more than 256; each
// CTA's shared memory holds half of the tile's rows.
//   warp 0      weights and rows by TMA, 64 k a stage (128-byte swizzle)
//   warp 1      (leader) issues the MMAs; two accumulators in tensor memory
//   warps 4-11  a thread per weight row and half of the tile's rows: epilogue.  Gated, the gates' warps and the up rows' exchange half of
//               their columns through shared memory, so that each finishes half
// The tiles are dealt out in turn, an expert's together: those that run side by side share its weights and rows in L2.
//
// What bounds it: few rows an expert, the weights' bytes (64 rows 0.72 of the copy bandwidth); many, no one pipe: 41 % of the tensor pipe and
// 34 % of L2 at 273 rows.  Measured, us, operands from memory, 30 experts of 2,048 -> 2 x 1,024 gated (sums rounded first) and 1,024 -> 2,048, this against
// the vendor library's grouped product and the gate's kernel behind it, rows an expert 64: 68 + 40 / 85 + 51, 256: 84 + 47 / 91 + 50, 533:
// 147 + 78 / 153 + 76.  Without a gate the first product of 533 rows takes 137, with the rounded GELU 158.
#include <cuda.h>

#include "common.cuh"

#define EPI_STORE_BF16 0
#define EPI_GELU 1         // the exact (erf) form
#define EPI_GELU_TANH 2
#define EPI_RELU2 3
#define EPI_STORE_F32 5
#define EPI_GATED_CLAMP 4  // g sigmoid(alpha g) (u + shift) of g <= limit, |u| <= limit
// The same of the sums as bf16 holds them: the bits of a product that stores bf16 and the activation's kernel behind it
#define EPI_RELU2_ROUNDED 6
#define EPI_GATED_CLAMP_ROUNDED 7
#define EPI_GELU_ROUNDED 8
#define EPI_GELU_TANH_ROUNDED 9
#define EPI_IS_GATED(e) ((e) == EPI_GATED_CLAMP || (e) == EPI_GATED_CLAMP_ROUNDED)

#define BF 128             // weight rows per CTA
#define BK 64              // k per stage
#define MAX_BN 256         // rows per tile
#define BOX 32             // rows that one TMA copy brings
#define A_BYTES (BF * BK * 2)
#define STAGE_BYTES (2 * A_BYTES)
#define STAGES 6
#define THREADS 384
#define MAX_GROUPS 2048
#ifndef ODI_WAIT_CYCLES
#define ODI_WAIT_CYCLES 4000000000ll   // about two seconds of SM clock; a self-test build makes it milliseconds
#endif
// How long a role waits for a copy, and the longer wait for the role that waits for it: a copy that never comes is reported by the role that
// missed it.
#define WAIT_CYCLES ((long long)ODI_WAIT_CYCLES)
#define WAIT_CYCLES_2 (WAIT_CYCLES + WAIT_CYCLES / 4)

#define ERR_PRODUCER 51
#define ERR_MMA 52
#define ERR_EPILOGUE 53

struct ExpertsArgs {
  void* out;               // [rows, N] bf16, or fp32 for EPI_STORE_F32
  int* status;
  const int* offsets;      // [groups + 1]: the experts' row ranges
  int N, K;                // N: output features
  int w_rows, groups;      // weight rows an expert
  int n_tiles;             // feature tiles
  float limit, alpha, shift;
  int withheld;            // self-test of the bounded waits: the producers request nothing
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
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t cluster_bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_bar), "r"(bytes) : "memory");
}
// Into this CTA's shared memory, its bytes counted on a barrier of the pair's leader.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D += A B over both CTAs' shared memory (M = 256).
__device__ __forceinline__ void umma_pair_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
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

// 0.5 g (1 + tanh y) = g sigmoid(2 y), y = sqrt(2/pi) (g + 0.044715 g^3)
__device__ __forceinline__ float gelu_tanh_f(float g) { return quotient(g, 1.f + expf(-1.5957691216057308f * fmaf(0.044715f * g * g, g, g))); }
__device__ __forceinline__ float gelu_erf_f(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f)); }
// In the activation kernel's form.
__device__ __forceinline__ float gelu_tanh_kernel_f(float z) { return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z))); }
__device__ __forceinline__ float rounded(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
template <int EPI>
__device__ __forceinline__ float gated(const ExpertsArgs& a, float g, float u) {
  if (EPI == EPI_GATED_CLAMP_ROUNDED) { g = rounded(g); u = rounded(u); }
  g = fminf(g, a.limit);
  u = fminf(fmaxf(u, -a.limit), a.limit);
  return quotient(g, 1.f + expf(-a.alpha * g)) * (u + a.shift);
}
template <int EPI>
__device__ __forceinline__ float plain(float v) {
  if (EPI == EPI_GELU) return gelu_erf_f(v);
  if (EPI == EPI_GELU_TANH) return gelu_tanh_f(v);
  if (EPI == EPI_RELU2) { const float r = fmaxf(v, 0.f); return r * r; }
  if (EPI == EPI_RELU2_ROUNDED) { const float r = fmaxf(rounded(v), 0.f); return r * r; }
  if (EPI == EPI_GELU_ROUNDED) return gelu_erf_f(rounded(v));
  if (EPI == EPI_GELU_TANH_ROUNDED) return gelu_tanh_kernel_f(rounded(v));
  return v;
}

// The u-th tile; `group` is the expert of the last one (tiles only go forward).
struct Unit { int w0, n0, t0, cols, bn; };
template <bool GATE>
__device__ __forceinline__ bool unit_of(const ExpertsArgs& a, const int* first, int u, int& group, Unit& t) {
  if (u >= first[a.groups]) return false;
  while (u >= first[group + 1]) ++group;
  const int begin = a.offsets[group], rows = a.offsets[group + 1] - begin, tiles = (rows + MAX_BN - 1) / MAX_BN;
  const int idx = u - first[group];
  t.bn = ((rows + tiles - 1) / tiles + 31) / 32 * 32;
  t.t0 = begin + idx % tiles * t.bn;
  t.cols = min(t.bn, begin + rows - t.t0);
  t.n0 = idx / tiles * (GATE ? BF : 2 * BF);
  t.w0 = group * a.w_rows + t.n0;
  return true;
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
grouped_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const ExpertsArgs a) {
  constexpr bool GATE = EPI_IS_GATED(EPI);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  // full (leader's), empty (each CTA's), acc_full (each CTA's), acc_empty (leader's)
  __shared__ __align__(8) uint64_t bars[2 * STAGES + 4];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;
  __shared__ int first[MAX_GROUPS + 1];                      // tiles before each expert
  __shared__ float swap[GATE ? 2 * 4 * 2 * 8 * 32 : 1];      // [turn][column half, lane group & 1][direction][column][lane]

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const uint32_t ring = smem_u32(smem);
  const uint32_t full = smem_u32(bars), empty = full + 8 * STAGES, acc_full = empty + 8 * STAGES, acc_empty = acc_full + 16;
  volatile int* abort_ptr = &abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full + 8 * s, 2); mbar_init(empty + 8 * s, 1); }      // both CTAs' producers
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full + 8 * b, 1); mbar_init(acc_empty + 8 * b, 16); }       // the epilogue warps of both
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(2 * MAX_BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  pdl_wait();                       // the ranges come from a kernel before
  if (warp == 2) {
    int before = 0;
    for (int g0 = 0; g0 < a.groups; g0 += 32) {
      const int g = g0 + lane;
      int mine = 0;
      if (g < a.groups) mine = (a.offsets[g + 1] - a.offsets[g] + MAX_BN - 1) / MAX_BN * a.n_tiles;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
      if (g < a.groups) first[g] = before + sum - mine;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) first[a.groups] = before;
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();               // both CTAs' barriers exist before anybody signals across
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
  pdl_launch_dependents();

  Unit t = {};
  int group = 0;
  const int blocks = (a.K + BK - 1) / BK;
  if (warp == 0) {
    if (lane == 0) {
      const uint32_t leader_full = map_to_rank(full, 0);
      bool ok = !a.withheld;
      int it = 0, s = 0;
      uint32_t phase = 1;
      for (int u = pair; ok && unit_of<GATE>(a, first, u, group, t); u += n_pairs) {
        const int row = t.w0 + (int)rank * (GATE ? BF / 2 : BF), row2 = GATE ? row + a.N : row + BF / 2;
        const int tok0 = t.t0 + (int)rank * (t.bn / 2), boxes = (t.bn / 2 + BOX - 1) / BOX;
        for (int kb = 0; kb < blocks; ++kb, ++it) {
          if (it >= STAGES && !mbar_wait(empty + 8 * s, phase, abort_ptr, a.status, ERR_PRODUCER, WAIT_CYCLES_2)) { ok = false; break; }
          const uint32_t dst = ring + s * STAGE_BYTES, bar = leader_full + 8 * s;
          mbar_expect_tx_cluster(bar, A_BYTES + boxes * BOX * 128);
          tma_load_2d_pair(dst, &map_w, kb * BK, row, bar);
          tma_load_2d_pair(dst + A_BYTES / 2, &map_w, kb * BK, row2, bar);
          for (int b = 0; b < boxes; ++b) tma_load_2d_pair(dst + A_BYTES + b * BOX * 128, &map_x, kb * BK, tok0 + b * BOX, bar);
          if (++s == STAGES) { s = 0; phase ^= 1u; }
        }
      }
      if (!ok && rank == 0) drain(full, STAGES, it);
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const bool issues = elect_one();
      bool ok = true;
      int s = 0, local = 0;
      uint32_t phase = 0;
      for (int u = pair; ok && unit_of<GATE>(a, first, u, group, t); u += n_pairs, ++local) {
        const int buf = local & 1;
        const uint32_t idesc = instr_desc_bf16(2 * BF, t.bn), d = tmem + buf * MAX_BN;
        if (local >= 2 && !warp_wait(acc_empty + 8 * buf, ((uint32_t)(local >> 1) & 1u) ^ 1u, abort_ptr, a.status, ERR_MMA, WAIT_CYCLES)) { ok = false; break; }
        for (int kb = 0; kb < blocks; ++kb) {
          if (!warp_wait(full + 8 * s, phase, abort_ptr, a.status, ERR_MMA, WAIT_CYCLES)) { ok = false; break; }
          tc_fence_after();
          const uint64_t dw = smem_desc_k_sw128(ring + s * STAGE_BYTES), dx = smem_desc_k_sw128(ring + s * STAGE_BYTES + A_BYTES);
          if (issues) {
#pragma unroll
            for (int j = 0; j < BK / 16; ++j) umma_pair_bf16(d, dw + 2 * j, dx + 2 * j, idesc, kb > 0 || j > 0 ? 1u : 0u);
            umma_commit_pair(empty + 8 * s);
          }
          if (++s == STAGES) { s = 0; phase ^= 1u; }
        }
        if (ok && issues) umma_commit_pair(acc_full + 8 * buf);
      }
    }
  } else if (warp >= 4) {
    const int lane_group = warp & 3, side = (warp - 4) >> 2;          // which half of the tile's rows
    const int row = lane_group * 32 + lane;                           // weight row of the CTA's 128
    const uint32_t leader_empty = map_to_rank(acc_empty, 0);
    const int exchange = side * 2 + (lane_group & 1);                 // gate warp and up warp of the same features and rows
    bool ok = true;
    int local = 0, turn = 0;
    for (int u = pair; unit_of<GATE>(a, first, u, group, t); u += n_pairs, ++local) {
      // a warp whose wait gave up still walks its units: the others count on it at the barriers below
      const int buf = local & 1, half = t.bn / 2, c0 = side * half;
      const int n = GATE ? t.n0 + (int)rank * (BF / 2) + (row & 63) : t.n0 + (int)rank * BF + row;
      if (ok && !warp_wait(acc_full + 8 * buf, (uint32_t)(local >> 1) & 1u, abort_ptr, a.status, ERR_EPILOGUE, WAIT_CYCLES_2)) ok = false;
      tc_fence_after();
      const uint32_t src = tmem + ((uint32_t)(lane_group * 32) << 16) + buf * MAX_BN + c0;
      // columns that hold rows: no more are loaded than are waited for, so that no load lands in registers that have another use by then
      const int mine_cols = min(half, t.cols - c0);      // the same for the warps that exchange
      uint32_t next[16];                       // the next 16 columns: on their way while these are worked on
      if (mine_cols > 0) tmem_ld16(src, next);
      for (int c = 0; c < mine_cols; c += 16) {
        const int left = mine_cols - c;        // rows of these 16 (and more)
        float v[16];
        tmem_wait16(next);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(next[i]);
        if (c + 16 < mine_cols) tmem_ld16(src + c + 16, next);
        if (EPI == EPI_STORE_F32) {
          float* to = (float*)a.out + (size_t)(t.t0 + c0 + c) * a.N + n;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            if (ok && n < a.N && i < left) *to = v[i];
            to += a.N;
          }
          continue;
        }
        constexpr int COUNT = GATE ? 8 : 16;
        int from = 0;                        // the first of this thread's rows
        if (GATE) {
          // gate warps keep rows 0-7 and hand their gates of 8-15 over for the up values of 0-7; up warps the other way round
          float* give = swap + (((turn & 1) * 4 + exchange) * 2 + (lane_group >> 1)) * 256 + lane;
          const float* take = swap + (((turn & 1) * 4 + exchange) * 2 + (1 - (lane_group >> 1))) * 256 + lane;
          ++turn;
          if (lane_group < 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) give[32 * i] = v[8 + i];
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) give[32 * i] = v[i];
          }
          asm volatile("bar.sync %0, 64;" ::"r"(2 + exchange) : "memory");
          if (lane_group < 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = gated<EPI>(a, v[i], take[32 * i]);
          } else {
            from = 8;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = gated<EPI>(a, take[32 * i], v[8 + i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = plain<EPI>(v[i]);
        }
        // neighbouring lanes hold neighbouring features: of two rows a lane stores one, as a pair
        const bool odd = lane & 1;
        const int even = n - (odd ? 1 : 0);
        bf16* to = (bf16*)a.out + (size_t)(t.t0 + c0 + c + from + (odd ? 1 : 0)) * a.N + even;
        const bool both = (a.N & 1) == 0;
        int mine = ok && even < a.N ? left - from - (odd ? 1 : 0) : 0;      // this lane stores while its row lies below
#pragma unroll
        for (int i = 0; i < COUNT; i += 2) {
          const float other = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
          const __nv_bfloat162 p = odd ? __floats2bfloat162_rn(other, v[i + 1]) : __floats2bfloat162_rn(v[i], other);
          if (i < mine) {
            if (both) *(__nv_bfloat162*)to = p;
            else { to[0] = p.x; if (even + 1 < a.N) to[1] = p.y; }
          }
          to += 2 * (size_t)a.N;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_empty + 8 * buf);
    }
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();               // nobody leaves while its barriers or tensor memory may still be used by the peer
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * MAX_BN));
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

// Of the current device; what is known is of the device that this thread asked for last.
static int device_pairs(int* device, int* pairs) {
  static thread_local int known = -1, sms = 0;
  cudaError_t e = cudaGetDevice(device);
  if (e == cudaSuccess && *device != known) {
    known = -1;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, *device);
    if (e == cudaSuccess) known = *device;
  }
  *pairs = sms / 2;
  return (int)e;
}

template <int EPI>
static int launch(const CUtensorMap& mx, const CUtensorMap& mw, const ExpertsArgs& a, int device, int pairs, cudaStream_t stream) {
  auto kernel = grouped_tcgen05_kernel<EPI>;
  constexpr int SMEM = STAGES * STAGE_BYTES + 1024;
  static thread_local int configured = -1;      // the attribute is the device's
  if (device != configured) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = device;
  }
  odi_rc = launch_pdl(kernel, dim3(2 * pairs), dim3(THREADS), SMEM, stream, mx, mw, a);
  return launch_status();
}

// x [rows, K] bf16, w [groups, w_rows, K] bf16 (gated: the gate rows, then the up rows; n_out = w_rows / 2), out [rows, n_out] in bf16, or fp32 for EPI_STORE_F32,
// offsets [groups + 1] ints on the device, rising from 0 to at most `rows`; rows beyond the last are not touched.  K a multiple of 8, x and w on
// 16-byte boundaries.  status: receives a code if a wait gives up; withheld: 0, or 1 for a self-test of that.
extern "C" int odi_grouped_tcgen05(const void* x, const void* w, void* out, const int* offsets, int rows, int groups, int n_out, int K,
                                   int w_rows, int epi, float limit, float alpha, float shift, int* status, int withheld, cudaStream_t stream) {
  if (rows <= 0 || n_out <= 0) return 0;
  const bool gate = EPI_IS_GATED(epi);
  if (K <= 0 || status == nullptr || offsets == nullptr || groups < 1 || (gate ? w_rows != 2 * n_out : w_rows != n_out)) return ODI_ERR_ARGUMENT;
  if (K % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15) || ((uintptr_t)out & 3) || groups > MAX_GROUPS) return ODI_ERR_UNSUPPORTED;
  int device = 0, pairs = 0;
  int rc = device_pairs(&device, &pairs);
  if (rc != 0) return rc;
  ExpertsArgs a = {};
  a.out = out; a.status = status; a.offsets = offsets; a.N = n_out; a.K = K; a.w_rows = w_rows; a.groups = groups;
  a.n_tiles = (n_out + (gate ? BF : 2 * BF) - 1) / (gate ? BF : 2 * BF);
  a.limit = limit; a.alpha = alpha; a.shift = shift; a.withheld = withheld;
  if ((long)groups * w_rows > 0x7fffffffL || ((long)rows / MAX_BN + groups) * a.n_tiles > 0x3fffffffL) return ODI_ERR_UNSUPPORTED;
  CUtensorMap mx, mw;
  rc = make_map(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, rows, K, K, BOX);
  if (rc == 0) rc = make_map(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w, (long)groups * w_rows, K, K, BF / 2);
  if (rc != 0) return rc;
  switch (epi) {
    case EPI_STORE_BF16: return launch<EPI_STORE_BF16>(mx, mw, a, device, pairs, stream);
    case EPI_GELU: return launch<EPI_GELU>(mx, mw, a, device, pairs, stream);
    case EPI_GELU_TANH: return launch<EPI_GELU_TANH>(mx, mw, a, device, pairs, stream);
    case EPI_RELU2: return launch<EPI_RELU2>(mx, mw, a, device, pairs, stream);
    case EPI_RELU2_ROUNDED: return launch<EPI_RELU2_ROUNDED>(mx, mw, a, device, pairs, stream);
    case EPI_GATED_CLAMP_ROUNDED: return launch<EPI_GATED_CLAMP_ROUNDED>(mx, mw, a, device, pairs, stream);
    case EPI_GELU_ROUNDED: return launch<EPI_GELU_ROUNDED>(mx, mw, a, device, pairs, stream);
    case EPI_GELU_TANH_ROUNDED: return launch<EPI_GELU_TANH_ROUNDED>(mx, mw, a, device, pairs, stream);
    case EPI_STORE_F32: return launch<EPI_STORE_F32>(mx, mw, a, device, pairs, stream);
    case EPI_GATED_CLAMP: return launch<EPI_GATED_CLAMP>(mx, mw, a, device, pairs, stream);
  }
  return ODI_ERR_ARGUMENT;
}
