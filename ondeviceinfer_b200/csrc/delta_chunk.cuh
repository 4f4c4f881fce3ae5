// The gated delta rule over runs of tokens, 16 tokens at a time (delta.cu, with a decay per key channel; delta_head.cu, with one
// per head, which is then every channel's).
//
// Per sequence and head, with S [D, dv] the state before the chunk, g_t [D] the decays of token t, G_t = g_0 .. g_t and
// D_ts = g_(s+1) .. g_t (products lane by lane, with one decay a head once for all and rounded once; nothing is divided, so no decay
// is too small), the recurrence
//     S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// unrolls over the chunk to
//     u_t = beta_t (v_t - (G_t k_t)^T S - sum_(s<t) A_ts u_s),      A_ts = k_t . (D_ts k_s)
//     o_t = (G_t q_t)^T S + sum_(s<=t) B_ts u_s,                    B_ts = q_t . (D_ts k_s)
//     S  <- diag(G_15) S + sum_s (D_15,s k_s) u_s^T.
// The triangular system is linear in S: u_t = wv_t - wk_t^T S with wv and wk its solutions for v and for G k.  So
//  parts  (every chunk and head at once) leaves wk, q' = G q - B wk, k^ = D_15 k, G_15, wv and B wv;
//  scan   (a block per sequence, head and COLS value columns) goes through a sequence's chunks in order:
//             u = wv - wk S;   o = B wv + q' S;   S <- diag(G_15) S + k^T u
//         the 32 sums of a column over D rows lie on 16 lanes and are halved side by side, so that a chunk costs one
//         chain of shuffles where token by token costs 32.
// Everything is fp32, as token by token.  A last chunk of fewer tokens is filled with tokens that do nothing (k, q, v
// and beta 0, g 1).
//
// What bounds it: the scan, one sequence with heads of 64 by its chain of latencies (0.8 us a chunk), else by the pipe of shared memory
// (1.6 us a chunk of one sequence with heads of 128).  The scratch has a slot per chunk (run_chunks.cuh).
#pragma once
#include "run_chunks.cuh"

#define DC 16                                      // tokens of a chunk
#define DC_WORDS(D) ((3 * DC + 1) * (D))           // floats per slot and head: wk, q', k^ [16][D] each, G_15 [D]

struct DeltaChunkArgs {
  float* wq;              // [slots, heads, DC_WORDS(D)]
  float* vo;              // [slots, heads, 2, DC, dv]: wv, B wv
  float* state;           // [cache slots, heads, D, dv]
  float* o;               // [n_tokens, heads, dv]: the read-outs
  const int* cu_q;
  const int* slots;
  int n_seqs, heads, dv;
};

template <int D, bool HEAD>
struct DeltaChunkShared {
  float q[DC][D], k[DC][D];
  float g[HEAD ? DC + 1 : DC][HEAD ? DC : D];      // decays per token and channel; HEAD: dc_head_decays
  __align__(16) float A[DC][DC];
  __align__(16) float B[DC][DC];
  float beta[DC];
  int found[3];
};

// One decay a head: row s the products D_ts of the tokens behind s (1 at s, 0 before), the last row G_t.  By the block's first warp,
// whose lanes hold a token's decay each (1 from lane DC on).
template <typename Shared>
__device__ __forceinline__ void dc_head_decays(Shared& sh, float own) {
  const int s = threadIdx.x;
  DecayProduct run;
#pragma unroll
  for (int t = 0; t < DC; ++t) {
    const float g = __shfl_sync(0xffffffffu, own, t);
    if (t > s || s == DC) run.times(g);
    if (s <= DC) sh.g[s][t] = t < s && s < DC ? 0.f : run.value();
  }
}

// The parts of a chunk from its unit vectors, decays and step sizes in shared memory (written before a barrier) and
// its values; by all threads of a block of whole warps, D + dv columns in turn.
template <int D, bool HEAD, typename Value>
__device__ __forceinline__ void dc_parts(DeltaChunkShared<D, HEAD>& sh, const DeltaChunkArgs& a, int b, int h, Value value) {
  static_assert(D % 32 == 0, "lanes own whole channels");
  constexpr int NI = D / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  // A and B: a warp takes a token s, its lanes carry D_ts k_s on over the tokens behind it; the 32 sums over the lanes (A's and
  // B's column s) are halved side by side
  for (int s = warp; s < DC; s += n_warps) {
    float w[NI], r[2 * DC];
#pragma unroll
    for (int e = 0; e < NI; ++e) w[e] = sh.k[s][lane + 32 * e];
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      r[t] = r[DC + t] = 0.f;
      if (t >= s) {
#pragma unroll
        for (int e = 0; e < NI; ++e) {
          if (!HEAD && t > s) w[e] *= sh.g[t][lane + 32 * e];
          r[t] = fmaf(w[e], sh.k[t][lane + 32 * e], r[t]);
          r[DC + t] = fmaf(w[e], sh.q[t][lane + 32 * e], r[DC + t]);
        }
      }
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      const bool up = lane & m;
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const float keep = up ? r[m + i] : r[i], give = up ? r[i] : r[m + i];
        r[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
      }
    }
    const float decayed = HEAD ? r[0] * sh.g[s][lane & (DC - 1)] : r[0];
    (lane < DC ? sh.A : sh.B)[lane & (DC - 1)][s] = decayed;      // column s; A's diagonal and what lies above are not read
  }
  __syncthreads();
  const size_t item = (size_t)b * a.heads + h;
  float* wk = a.wq + item * DC_WORDS(D);
  float* vo = a.vo + item * 2 * DC * a.dv;
  for (int c = threadIdx.x; c < D + a.dv; c += blockDim.x) {
    const bool is_k = c < D;
    float w[DC], decay = 1.f;
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      if (is_k) decay = HEAD ? sh.g[HEAD ? DC : 0][t] : decay * sh.g[t][c];
      float x = 0.f;      // summed before it is taken off: one rounding of the larger number
#pragma unroll
      for (int s = 0; s < t; ++s) x = fmaf(sh.A[t][s], w[s], x);
      w[t] = sh.beta[t] * (is_k ? fmaf(sh.k[t][c], decay, -x) : value(t, c - D) - x);
    }
    float run = 1.f, tail = 1.f;
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      float x = 0.f;
#pragma unroll
      for (int s = 0; s <= t; ++s) x = fmaf(sh.B[t][s], w[s], x);
      if (is_k) {
        run = HEAD ? sh.g[HEAD ? DC : 0][t] : run * sh.g[t][c];
        wk[t * D + c] = w[t];
        wk[(DC + t) * D + c] = fmaf(sh.q[t][c], run, -x);
      } else {
        vo[t * a.dv + c - D] = w[t];
        vo[(DC + t) * a.dv + c - D] = x;
      }
    }
    if (is_k) {
#pragma unroll
      for (int t = DC - 1; t >= 0; --t) {
        wk[(2 * DC + t) * D + c] = sh.k[t][c] * (HEAD ? sh.g[t][DC - 1] : tail);
        if (!HEAD) tail *= sh.g[t][c];
      }
      wk[3 * DC * D + c] = decay;
    }
  }
}

__device__ __forceinline__ void dc_cp16(uint32_t dst, const float* src, bool ok) {      // zeros where !ok
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

#define DC_STAGES(D) ((D) == 64 ? 3 : 2)      // heads of 128: two, so that four blocks share a multiprocessor
#define DC_STAGE(D, COLS) (DC_WORDS(D) + 2 * DC * (COLS))      // floats of a chunk in shared memory

// The sequence of a block: the blockIdx.z-th longest, so that the blocks of the longest run, which the kernel waits for, are placed
// first, a multiprocessor each, and the others beside them.  Runs of 333, 769 and 1,777 tokens with 16 heads of 128 in the batch's order,
// the longest last: its blocks lay two and three to a multiprocessor and took 371 us, 184 by themselves.
// Beyond 64 sequences in the batch's order: the chip is full either way.
__device__ __forceinline__ int dc_longest_first(const int* cu_q, int n_seqs, int* chosen) {
  if (n_seqs == 1 || n_seqs > 64) return blockIdx.z;
  for (int s = threadIdx.x; s < n_seqs; s += blockDim.x) {
    const int mine = cu_q[s + 1] - cu_q[s];
    int before = 0;
    for (int j = 0; j < n_seqs; ++j) {
      const int other = cu_q[j + 1] - cu_q[j];
      before += other > mine || (other == mine && j < s);
    }
    if (before == (int)blockIdx.z) *chosen = s;
  }
  __syncthreads();
  return *chosen;
}

// COLS columns of one head's state: CPT of them per group of 16 lanes, a lane holding rows 4 (lane + 16 j) .. + 3.  dv a
// multiple of 4 (16-byte copies of COLS columns).
template <int D, int COLS, int CPT>
__global__ void __launch_bounds__(COLS / CPT * 16, 2)
dc_scan_kernel(DeltaChunkArgs a) {
  pdl_wait();
  constexpr int NTH = COLS / CPT * 16, NJ = D / 64, R = D / 16;
  constexpr size_t STAGE = DC_STAGE(D, COLS);
  static_assert(D % 64 == 0 && COLS % 4 == 0 && COLS % CPT == 0 && NTH % 32 == 0, "sizes of a block");
  extern __shared__ __align__(16) float dc_smem[];
  // behind the chunks, not a variable of its own: 16 static bytes put every row of the chunks across one more 128-byte line of shared memory
  // (the mixer of two runs of 1,777 tokens, heads of 128: 601 us against 549)
  int* chosen = (int*)(dc_smem + DC_STAGES(D) * STAGE + COLS * DC);
  const int seq = dc_longest_first(a.cu_q, a.n_seqs, chosen), h = blockIdx.y, c0 = blockIdx.x * COLS;
  const int tid = threadIdx.x, rl = tid & 15, col = (tid >> 4) * CPT;
  const int q_begin = a.cu_q[seq], q_len = a.cu_q[seq + 1] - q_begin;
  if (q_len <= 0) return;
  const int dv = a.dv, chunks = (q_len + DC - 1) / DC;
  const size_t slot0 = (size_t)(q_begin / DC) + seq;
  float* S_g = a.state + ((size_t)a.slots[seq] * a.heads + h) * D * dv;
  float* xs = dc_smem + DC_STAGES(D) * STAGE + col * DC;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(dc_smem);

  auto issue = [&](int c) {
    if (c < chunks) {
      const size_t item = (slot0 + c) * a.heads + h;
      const uint32_t dst = base + (uint32_t)((c % DC_STAGES(D)) * STAGE * 4);
      const float* src = a.wq + item * DC_WORDS(D) + tid * 4;
#pragma unroll
      for (int i = 0; i < DC_WORDS(D); i += NTH * 4)
        if (i + NTH * 4 <= DC_WORDS(D) || i + tid * 4 < DC_WORDS(D)) dc_cp16(dst + (i + tid * 4) * 4, src + i, true);
      const float* vo = a.vo + item * 2 * DC * dv + c0;
#pragma unroll
      for (int i = 0; i < 2 * DC * (COLS / 4); i += NTH) {
        const int t = (i + tid) / (COLS / 4), e = (i + tid) % (COLS / 4) * 4;
        const bool ok = c0 + e < dv;
        if (i + NTH <= 2 * DC * (COLS / 4) || t < 2 * DC) dc_cp16(dst + (DC_WORDS(D) + t * COLS + e) * 4, ok ? vo + (size_t)t * dv + e : vo, ok);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < DC_STAGES(D) - 1; ++c) issue(c);

  float S[CPT][R];
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
    for (int r = 0; r < R; ++r)
      S[cc][r] = c0 + col + cc < dv ? S_g[(size_t)(4 * (rl + 16 * (r >> 2)) + (r & 3)) * dv + c0 + col + cc] : 0.f;

  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DC_STAGES(D) - 2) : "memory");
    __syncthreads();      // chunk c has arrived; everybody has left chunk c - 1, whose place the next copies take
    issue(c + DC_STAGES(D) - 1);
    const float* buf = dc_smem + (c % DC_STAGES(D)) * STAGE;
    const float* vs = buf + DC_WORDS(D);
    // wk S (half 0) or q' S (half 1): this lane's rows
    auto rows_of = [&](int half, float (&sum)[CPT][DC]) {
#pragma unroll
      for (int t = 0; t < DC; ++t) {
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) sum[cc][t] = 0.f;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float4 x = *(const float4*)(buf + (half * DC + t) * D + 4 * (rl + 16 * j));
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc)
            sum[cc][t] = fmaf(x.x, S[cc][4 * j], fmaf(x.y, S[cc][4 * j + 1], fmaf(x.z, S[cc][4 * j + 2], fmaf(x.w, S[cc][4 * j + 3], sum[cc][t]))));
        }
      }
    };
    // over the 16 lanes: a lane keeps one half of its sums and hands the other on, down to token rl's
    auto over_lanes = [&](float (&sum)[CPT][DC]) {
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
        for (int m = 8; m > 0; m >>= 1) {
          const bool up = rl & m;
#pragma unroll
          for (int i = 0; i < m; ++i) {
            const float keep = up ? sum[cc][m + i] : sum[cc][i], give = up ? sum[cc][i] : sum[cc][m + i];
            sum[cc][i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
          }
        }
    };
    float wks[CPT][DC], qs[CPT][DC];
    rows_of(0, wks);
    rows_of(1, qs);
    over_lanes(wks);
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc) xs[cc * DC + rl] = vs[rl * COLS + col + cc] - wks[cc][0];
    over_lanes(qs);
    if (c * DC + rl < q_len) {
      float* to = a.o + ((size_t)(q_begin + c * DC + rl) * a.heads + h) * dv + c0 + col;
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc)
        if (c0 + col + cc < dv) to[cc] = vs[(DC + rl) * COLS + col + cc] + qs[cc][0];
    }
    __syncwarp();
    float u[CPT][DC];
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
      for (int t = 0; t < DC; t += 4) {
        const float4 x = *(const float4*)(xs + cc * DC + t);
        u[cc][t] = x.x; u[cc][t + 1] = x.y; u[cc][t + 2] = x.z; u[cc][t + 3] = x.w;
      }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const float4 g = *(const float4*)(buf + 3 * DC * D + 4 * (rl + 16 * j));
      // the chunk's writes are summed before they join the state: one rounding of the larger number instead of sixteen
      float4 add[CPT];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) add[cc] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int t = 0; t < DC; ++t) {
        const float4 x = *(const float4*)(buf + (2 * DC + t) * D + 4 * (rl + 16 * j));
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          add[cc].x = fmaf(x.x, u[cc][t], add[cc].x); add[cc].y = fmaf(x.y, u[cc][t], add[cc].y);
          add[cc].z = fmaf(x.z, u[cc][t], add[cc].z); add[cc].w = fmaf(x.w, u[cc][t], add[cc].w);
        }
      }
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        S[cc][4 * j] = fmaf(S[cc][4 * j], g.x, add[cc].x); S[cc][4 * j + 1] = fmaf(S[cc][4 * j + 1], g.y, add[cc].y);
        S[cc][4 * j + 2] = fmaf(S[cc][4 * j + 2], g.z, add[cc].z); S[cc][4 * j + 3] = fmaf(S[cc][4 * j + 3], g.w, add[cc].w);
      }
    }
    __syncwarp();      // xs is written again in the next chunk
  }
  pdl_launch_dependents();
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (c0 + col + cc < dv) S_g[(size_t)(4 * (rl + 16 * (r >> 2)) + (r & 3)) * dv + c0 + col + cc] = S[cc][r];
}

// Columns a block and a thread.  The scan is bound by the pipe of shared memory: a 16-byte read of a warp takes it four clocks also where half
// of its lanes read the same, a shuffle about three.  More columns a thread read the chunk's rows fewer times, but the chain of one chunk gets
// longer; so heads of 64 take the narrow form as long as two of its blocks a multiprocessor hold all.  A column's sums have the same order in
// either form: they depend neither on it nor on the batch.  Measured, us, the scan, 16 heads of 64, narrow / wide: 2,048 tokens 106 / 167,
// 1,024 + 2,048 122 / 167, 4 x 2,048 233 / 207.  The whole mixer, with the copies' loops rolled and runs in the batch's order / now: heads of 64, 2,048
// tokens 264 / 194, 1,024 + 2,048 318 / 246, 4 x 1,500 430 / 386; heads of 128, 1,777 tokens 322 / 299, 2 x 1,777 576 / 549, 333 + 769 + 1,777
// 584 / 511, 3 x 1,000 475 / 455, 4 x 512 327 / 315.  32 lanes a column for many heads of 128 gained less than that and summed in another order.
template <int D, int COLS, int CPT>
static int dc_launch_form(const DeltaChunkArgs& a, cudaStream_t stream) {
  constexpr size_t smem = sizeof(float) * (DC_STAGES(D) * DC_STAGE(D, COLS) + COLS * DC + 4);
  auto kernel = dc_scan_kernel<D, COLS, CPT>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  // an ordinary launch: started early, while the kernel before still holds multiprocessors, the few long blocks of a
  // single sequence would be packed several to one and stay there
  kernel<<<dim3((a.dv + COLS - 1) / COLS, a.heads, a.n_seqs), dim3(COLS / CPT * 16), smem, stream>>>(a);
  return (int)cudaPeekAtLastError();
}
template <int D>
static int dc_launch(const DeltaChunkArgs& a, cudaStream_t stream) {
  if constexpr (D == 64)
    if ((long)((a.dv + 7) / 8) * a.heads * a.n_seqs <= 296) return dc_launch_form<D, 8, 2>(a, stream);
  return dc_launch_form<D, 16, D == 64 ? 4 : 2>(a, stream);
}
