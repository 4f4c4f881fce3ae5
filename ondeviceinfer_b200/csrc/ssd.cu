// A selective state-space mixer with a scalar decay per head (the recurrent form of the state-space duality):
// what lies between its input projection and its output projection.
//
// A token's row of the input projection is [ z: inner | x: inner | B: G N | C: G N | dt: heads ], inner = heads P.
//
//  conv        x, B and C together (inner + 2 G N channels) pass a causal convolution over time per channel,
//              taps w[c, 0..taps-1] (the last one is the current token's) and a bias, then SiLU; inputs before the
//              first token that a sequence brings come from its state (its last taps - 1 inputs, fp32, zero before
//              its start).  fp32 sums; the result stays fp32 for the recurrence.
//  conv_state  the state moved on by the tokens that the sequence brought.
//  scan        per sequence and head h (group g = h / (heads / G)), over the sequence's tokens in order:
//                dt = softplus(dt_raw + dt_bias[h]);  S <- exp(-exp(A_log[h]) dt) S + dt B_g x_h^T;  y = S^T C_g + D[h] x_h
//              with S [N, P] fp32 per (sequence, head), kept in the cache between steps.  A block owns 32 columns of S;
//              a column lives in the registers of 8 or 16 lanes, the read-out is a sum over those lanes; 16 tokens of B, C, x
//              and the decays are staged in shared memory at a time, the next 16 by asynchronous copies meanwhile.
//  gate_norm   v = y * silu(z); v is RMS-normed in `norm_groups` equal parts of a token's row (each part by its own
//              root mean square, eps inside the root), times a weight per lane, rounded once to T.
//
// Everything but the projection's own output is fp32 in both compute dtypes.
#include "run_chunks.cuh"
#include <type_traits>

#define SSD_MAX_TAPS 16
#define SSD_TCH 16          // tokens staged at a time
#define SSD_COLS 32         // most columns of S per block (a kernel form takes 32 or 8)

struct SsdArgs {
  const void* proj;       // [n_tokens, ld] in T
  const float* conv_w;    // [C, taps]
  const float* conv_b;    // [C]
  const float* dt_bias;   // [heads]
  const float* a_log;     // [heads]
  const float* d_skip;    // [heads]
  const float* norm_w;    // [inner]
  float* conv_state;      // [slots, taps - 1, C]; null when taps == 1
  float* state;           // [slots, heads, N, P]
  float* xbc;             // [n_tokens, C] scratch
  float* y;               // [n_tokens, inner] scratch
  float* chunks;          // scratch of the scan in chunks (ssd_chunk_floats in ops.py says how much); null: token by token
  void* out;              // [n_tokens, inner] in T
  const int* cu_q;        // [n_seqs + 1]
  const int* tok_seq;     // [n_tokens]
  const int* slots;       // [n_seqs]
  int n_tokens, n_seqs, ld, heads, P, N, G, taps, norm_groups;
  float eps;
};

__device__ __forceinline__ float ssd_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float ssd_silu(float x) { return x / (1.f + expf(-x)); }

template <typename T>
__device__ __forceinline__ float ssd_conv_input(const SsdArgs& a, int inner, int C, int q_begin, int slot, int idx, int c) {
  // input `idx` of the sequence's run in this step; negative indices reach into the convolution state
  if (idx >= 0) return to_f<T>(((const T*)a.proj)[(size_t)(q_begin + idx) * a.ld + inner + c]);
  return a.conv_state[((size_t)slot * (a.taps - 1) + (a.taps - 1 + idx)) * C + c];
}

template <typename T>
__global__ void __launch_bounds__(256)
ssd_conv_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int inner = a.heads * a.P, C = inner + 2 * a.G * a.N;
  const int t = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int seq = a.tok_seq[t];
  const int q_begin = a.cu_q[seq], slot = a.slots[seq];
  const int li = t - q_begin;
  float acc = a.conv_b[c];
  for (int j = 0; j < a.taps; ++j)
    acc = fmaf(a.conv_w[(size_t)c * a.taps + j], ssd_conv_input<T>(a, inner, C, q_begin, slot, li - (a.taps - 1) + j, c), acc);
  a.xbc[(size_t)t * C + c] = ssd_silu(acc);
}

// Four neighbouring elements as floats.
template <typename T> __device__ __forceinline__ float4 ssd_load4(const T* p);
template <> __device__ __forceinline__ float4 ssd_load4<float>(const float* p) { return *(const float4*)p; }
template <> __device__ __forceinline__ float4 ssd_load4<bf16>(const bf16* p) {
  const uint2 raw = *(const uint2*)p;
  const float2 lo = __bfloat1622float2(*(const __nv_bfloat162*)&raw.x), hi = __bfloat1622float2(*(const __nv_bfloat162*)&raw.y);
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// The convolution of runs of tokens with four taps: a thread takes four channels of SSD_CT neighbouring tokens and reads each
// input once, 8 or 16 bytes at a time, where the kernel above reads it once per tap and token, an element at a time (2,048 tokens
// of 2,304 channels: 13 us against 45; the bytes take 4).  Tokens that reach back before their run's start, or lie on both sides of a
// border between runs, go one by one.
#define SSD_CT 8
#define SSD_CONV4_LEAST (1L << 19)      // inputs in all from which that pays
template <typename T>
__global__ void __launch_bounds__(128)
ssd_conv4_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int inner = a.heads * a.P, C = inner + 2 * a.G * a.N;
  const int t0 = blockIdx.x * SSD_CT, c = (blockIdx.y * 128 + threadIdx.x) * 4;
  if (c >= C) return;
  const int nt = min(SSD_CT, a.n_tokens - t0);
  float w[4][4];                             // [channel][tap]
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float4 x = *(const float4*)(a.conv_w + (size_t)(c + e) * 4);
    w[e][0] = x.x; w[e][1] = x.y; w[e][2] = x.z; w[e][3] = x.w;
  }
  const float4 bias = *(const float4*)(a.conv_b + c);
  auto store = [&](int t, const float4 (&x)[4]) {      // x: the token's inputs, oldest first
    float4 y = bias;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      y.x = fmaf(w[0][j], x[j].x, y.x); y.y = fmaf(w[1][j], x[j].y, y.y); y.z = fmaf(w[2][j], x[j].z, y.z); y.w = fmaf(w[3][j], x[j].w, y.w);
    }
    *(float4*)(a.xbc + (size_t)t * C + c) = make_float4(ssd_silu(y.x), ssd_silu(y.y), ssd_silu(y.z), ssd_silu(y.w));
  };
  const int seq = a.tok_seq[t0];
  if (nt == SSD_CT && a.tok_seq[t0 + SSD_CT - 1] == seq && t0 - a.cu_q[seq] >= 3) {
    const T* in = (const T*)a.proj + (size_t)(t0 - 3) * a.ld + inner + c;
    float4 x[SSD_CT + 3];
#pragma unroll
    for (int i = 0; i < SSD_CT + 3; ++i) x[i] = ssd_load4<T>(in + (size_t)i * a.ld);
#pragma unroll
    for (int t = 0; t < SSD_CT; ++t) {
      const float4 of[4] = {x[t], x[t + 1], x[t + 2], x[t + 3]};
      store(t0 + t, of);
    }
    return;
  }
  for (int t = t0; t < t0 + nt; ++t) {
    const int own = a.tok_seq[t], q_begin = a.cu_q[own], slot = a.slots[own];
    float4 of[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int idx = t - q_begin - 3 + j;
      of[j] = idx >= 0 ? ssd_load4<T>((const T*)a.proj + (size_t)(q_begin + idx) * a.ld + inner + c)
                       : *(const float4*)(a.conv_state + ((size_t)slot * 3 + 3 + idx) * C + c);
    }
    store(t, of);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
ssd_conv_state_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int inner = a.heads * a.P, C = inner + 2 * a.G * a.N;
  const int seq = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int q_begin = a.cu_q[seq], q_len = a.cu_q[seq + 1] - q_begin, slot = a.slots[seq];
  const int keep = a.taps - 1;
  float next[SSD_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < SSD_MAX_TAPS; ++j)
    if (j < keep) next[j] = ssd_conv_input<T>(a, inner, C, q_begin, slot, q_len - keep + j, c);
#pragma unroll
  for (int j = 0; j < SSD_MAX_TAPS; ++j)
    if (j < keep) a.conv_state[((size_t)slot * keep + j) * C + c] = next[j];
}

__device__ __forceinline__ void ssd_cp4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ssd_cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ssd_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void ssd_cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// LANES: lanes that share a column of S (8 or 16); NPT: rows of S per lane (N <= LANES NPT).  VEC (N a multiple of 4,
// 16-byte aligned rows of xbc): a lane owns rows 4 (ns + LANES j) .. + 3 of its column and reads B and C four at a time;
// else rows ns + LANES k, one at a time.
// Two staging buffers: while the block works through one chunk of SSD_TCH tokens, the asynchronous copies of the next
// chunk's B, C and x (and the loads of its step sizes) are in flight; one barrier per chunk.
// COLS: columns of S per block (COLS * 8 threads): fewer columns make more blocks, which is what a step of one long
// sequence needs, since each warp's time is the chain of its tokens.
template <typename T, int NPT, bool VEC, int COLS, int LANES>
__global__ void __launch_bounds__(COLS * LANES)
ssd_scan_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float ssd_smem[];
  const int N = a.N, P = a.P, inner = a.heads * P, C = inner + 2 * a.G * N;
  const int stage = SSD_TCH * (2 * N + COLS) + 2 * SSD_TCH;      // floats of one buffer
  const int tid = threadIdx.x, ns = tid % LANES, pc = tid / LANES;
  const int h = blockIdx.y, seq = blockIdx.z, g = h / (a.heads / a.G);
  const int p0 = blockIdx.x * COLS, p = p0 + pc;
  const int q_begin = a.cu_q[seq], q_len = a.cu_q[seq + 1] - q_begin;
  if (q_len <= 0) return;
  const int slot = a.slots[seq];
  float* S = a.state + ((size_t)slot * a.heads + h) * N * P;
  auto row_of = [&](int k) { return VEC ? 4 * (ns + LANES * (k >> 2)) + (k & 3) : ns + LANES * k; };
  float s[NPT];
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const int n = row_of(k);
    s[k] = (n < N && p < P) ? S[(size_t)n * P + p] : 0.f;
  }
  const float neg_a = -expf(a.a_log[h]), dt_b = a.dt_bias[h], dskip = a.d_skip[h];
  const T* dt_col = (const T*)a.proj + 2 * inner + 2 * a.G * N + h;
  const int n_chunks = (q_len + SSD_TCH - 1) / SSD_TCH;

  // buffer layout: B [TCH][N], C [TCH][N], x [TCH][COLS], dt [TCH], decay [TCH]
  auto issue = [&](int c) {
    float* buf = ssd_smem + (size_t)(c & 1) * stage;
    const int base = c * SSD_TCH, nt = min(SSD_TCH, q_len - base);
    const float* rows = a.xbc + (size_t)(q_begin + base) * C;
    // a warp copies a token's B and C rows, token after token (no division in the loop)
    const int warp = tid >> 5, lane = tid & 31, n_warps = (COLS * LANES) >> 5;
    for (int tt = warp; tt < nt; tt += n_warps) {
      const float* src = rows + (size_t)tt * C + inner + (size_t)g * N;
      float* dB = buf + tt * N;
      float* dC = buf + SSD_TCH * N + tt * N;
      if (VEC) {
        for (int j = 4 * lane; j < N; j += 128) { ssd_cp16(dB + j, src + j); ssd_cp16(dC + j, src + (size_t)a.G * N + j); }
      } else {
        for (int n = lane; n < N; n += 32) { ssd_cp4(dB + n, src + n); ssd_cp4(dC + n, src + (size_t)a.G * N + n); }
      }
    }
    float* sX = buf + 2 * SSD_TCH * N;
    for (int i = tid; i < nt * COLS; i += blockDim.x) {
      const int tt = i / COLS, cc = i % COLS;
      if (p0 + cc < P) ssd_cp4(sX + i, rows + (size_t)tt * C + (size_t)h * P + p0 + cc);
      else sX[i] = 0.f;
    }
    ssd_cp_commit();
  };
  auto step_sizes = [&](int c, float raw) {      // by thread tid < tokens of chunk c
    float* buf = ssd_smem + (size_t)(c & 1) * stage + SSD_TCH * (2 * N + COLS);
    const float dt = ssd_softplus(raw + dt_b);
    buf[tid] = dt;
    buf[SSD_TCH + tid] = expf(neg_a * dt);
  };

  issue(0);
  if (tid < min(SSD_TCH, q_len)) step_sizes(0, to_f<T>(dt_col[(size_t)(q_begin + tid) * a.ld]));
  for (int c = 0; c < n_chunks; ++c) {
    ssd_cp_wait_all();
    __syncthreads();      // chunk c is in its buffer; everybody has left chunk c - 1, whose buffer takes chunk c + 1
    const int base = c * SSD_TCH, nt = min(SSD_TCH, q_len - base);
    const bool more = c + 1 < n_chunks;
    const int nt_next = more ? min(SSD_TCH, q_len - base - SSD_TCH) : 0;
    float raw_next = 0.f;
    if (more) {
      issue(c + 1);
      if (tid < nt_next) raw_next = to_f<T>(dt_col[(size_t)(q_begin + base + SSD_TCH + tid) * a.ld]);
    }
    const float* buf = ssd_smem + (size_t)(c & 1) * stage;
    const float* sB = buf;
    const float* sC = buf + SSD_TCH * N;
    const float* sX = buf + 2 * SSD_TCH * N;
    const float* sDt = sX + SSD_TCH * COLS;
    const float* sDa = sDt + SSD_TCH;
    // one token: the state's rows of this lane move on, the read-out is summed over the column's lanes
    auto token = [&](int tt, auto full_tag) {
      constexpr bool FULL = decltype(full_tag)::value;      // N == 8 NPT: no row of the lane lies beyond the state
      const float x = sX[tt * COLS + pc], dt = sDt[tt], da = sDa[tt];
      const float dx = dt * x;
      const float* B = sB + tt * N;
      const float* Cc = sC + tt * N;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      if (VEC) {
#pragma unroll
        for (int j = 0; j < NPT / 4; ++j) {
          const int n = 4 * (ns + LANES * j);
          if (FULL || n < N) {
            const float4 b = *(const float4*)(B + n), cv = *(const float4*)(Cc + n);
            s[4 * j] = fmaf(da, s[4 * j], dx * b.x);         acc[0] = fmaf(s[4 * j], cv.x, acc[0]);
            s[4 * j + 1] = fmaf(da, s[4 * j + 1], dx * b.y); acc[1] = fmaf(s[4 * j + 1], cv.y, acc[1]);
            s[4 * j + 2] = fmaf(da, s[4 * j + 2], dx * b.z); acc[2] = fmaf(s[4 * j + 2], cv.z, acc[2]);
            s[4 * j + 3] = fmaf(da, s[4 * j + 3], dx * b.w); acc[3] = fmaf(s[4 * j + 3], cv.w, acc[3]);
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < NPT; ++k) {
          const int n = ns + LANES * k;
          if (FULL || n < N) {
            s[k] = fmaf(da, s[k], dx * B[n]);
            acc[k & 3] = fmaf(s[k], Cc[n], acc[k & 3]);
          }
        }
      }
      float sum = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
      for (int o = 1; o < LANES; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (ns == 0 && p < P) a.y[(size_t)(q_begin + base + tt) * inner + (size_t)h * P + p] = fmaf(dskip, x, sum);
    };
    // four tokens at a time: the state goes through them in order, their four read-outs are summed over the column's
    // lanes side by side, so that the shuffles' latency is paid once per four tokens (full states, VEC form)
    auto tokens4 = [&](int t0) {
      float x[4], dx[4], da[4], acc[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        x[u] = sX[(t0 + u) * COLS + pc];
        dx[u] = sDt[t0 + u] * x[u];
        da[u] = sDa[t0 + u];
        acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < NPT / 4; ++j) {
        const int n = 4 * (ns + LANES * j);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 b = *(const float4*)(sB + (t0 + u) * N + n), cv = *(const float4*)(sC + (t0 + u) * N + n);
          s[4 * j] = fmaf(da[u], s[4 * j], dx[u] * b.x);         acc[u][0] = fmaf(s[4 * j], cv.x, acc[u][0]);
          s[4 * j + 1] = fmaf(da[u], s[4 * j + 1], dx[u] * b.y); acc[u][1] = fmaf(s[4 * j + 1], cv.y, acc[u][1]);
          s[4 * j + 2] = fmaf(da[u], s[4 * j + 2], dx[u] * b.z); acc[u][2] = fmaf(s[4 * j + 2], cv.z, acc[u][2]);
          s[4 * j + 3] = fmaf(da[u], s[4 * j + 3], dx[u] * b.w); acc[u][3] = fmaf(s[4 * j + 3], cv.w, acc[u][3]);
        }
      }
      float sum[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) sum[u] = (acc[u][0] + acc[u][1]) + (acc[u][2] + acc[u][3]);
#pragma unroll
      for (int o = 1; o < LANES; o <<= 1) {
#pragma unroll
        for (int u = 0; u < 4; ++u) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
      }
      if (ns == 0 && p < P) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          a.y[(size_t)(q_begin + base + t0 + u) * inner + (size_t)h * P + p] = fmaf(dskip, x[u], sum[u]);
      }
    };
    if (N == LANES * NPT) {
      int tt = 0;
      if (VEC) {
        for (; tt + 4 <= nt; tt += 4) tokens4(tt);
      }
      for (; tt < nt; ++tt) token(tt, std::true_type{});
    } else {
      for (int tt = 0; tt < nt; ++tt) token(tt, std::false_type{});
    }
    if (more && tid < nt_next) step_sizes(c + 1, raw_next);
  }
#pragma unroll
  for (int k = 0; k < NPT; ++k) {
    const int n = row_of(k);
    if (n < N && p < P) S[(size_t)n * P + p] = s[k];
  }
}

// The scan over runs of tokens, SSD_L tokens at a time.  With a_t = exp(-exp(A_log) dt_t), G_t = a_0 .. a_t and D_ts = a_(s+1)
// .. a_t (products; nothing is divided, no difference of exponents is taken), S the state before the chunk:
//     y_t = G_t C_t S + sum_(s<=t) (C_t . B_s) D_ts dt_s x_s + D x_t
//     S  <- G_last S + sum_s B_s (D_last,s dt_s x_s)^T
//  states   every chunk and head at once: E = sum_s B_s (D_last,s dt_s x_s)^T and G_last; in further blocks every chunk and
//           group: the products C_t . B_s, which the heads of a group share;
//  pass     per element of S: E of every chunk gives way to the state before it;
//  outputs  every chunk and head at once: y.
// The products of decays are rounded once (DecayProduct); all else is plain fp32 multiply-adds, as token by token, where a
// sequence's tokens were one chain of them.  The mixer between its products, 32 heads of 128 x 64, us (in chunks, token by token):
// 2,048 tokens 187, 564; 2 x 1,024 183, 350; 8 x 1,000 715, 961; 512 79, 152; 128 63, 60.  What bounds outputs (66 us of those 187)
// and states (54) is shared memory: three 16-byte reads per 32 multiply-adds of a thread.
#define SSD_L 64

// dt_t and a_t of the chunk's tokens into shared memory; tokens behind the run's end have dt 0, a 1
template <typename T>
__device__ __forceinline__ void ssd_chunk_steps(const SsdArgs& a, int h, size_t tok, int nt, float* dt_s, float* a_s) {
  const int t = threadIdx.x;
  if (t < SSD_L) {
    float dt = 0.f, da = 1.f;
    if (t < nt) {
      const T* raw = (const T*)a.proj + (tok + t) * a.ld + 2 * (size_t)a.heads * a.P + 2 * (size_t)a.G * a.N + h;
      dt = ssd_softplus(to_f<T>(*raw) + a.dt_bias[h]);
      da = expf(-expf(a.a_log[h]) * dt);
    }
    dt_s[t] = dt;
    a_s[t] = da;
  }
}

struct SsdScratch {
  float* E;               // [slots, heads, N, P]
  float* cb;              // [slots, G, L (s), L (t)]: C_t . B_s
  float* gamma;           // [slots, heads]
};
static __host__ __device__ __forceinline__ SsdScratch ssd_scratch(const SsdArgs& a) {
  const size_t slots = (size_t)a.n_tokens / SSD_L + a.n_seqs;
  SsdScratch s;
  s.E = a.chunks;
  s.cb = s.E + slots * a.heads * a.N * a.P;
  s.gamma = s.cb + slots * a.G * SSD_L * SSD_L;
  return s;
}

#define SSD_PAD (SSD_L + 4)

// 32 rows of a product's reduction (CAUSAL: row k only into the outputs m >= k0 + k): acc[i][j] += sum_k A[k][m(i)] B[k][n(j)],
// m = 4 mt + (0..3) and 32 + 4 mt + (0..3), n = 4 nt + (0..3); A rows of SSD_PAD, B rows of SSD_L words
template <bool CAUSAL = false>
__device__ __forceinline__ void ssd_mma32(float (&acc)[8][4], const float* A, const float* B, int mt, int nt, int k0 = 0) {
#pragma unroll 1
  for (int half = 0; half < 32; half += 16) {
    float part[8][4] = {};      // sums of sixteen products, then of those: fewer roundings of large numbers than one chain
#pragma unroll
    for (int k = half; k < half + 16; ++k) {
      const float4 a0 = *(const float4*)(A + k * SSD_PAD + 4 * mt), a1 = *(const float4*)(A + k * SSD_PAD + 32 + 4 * mt);
      const float4 b = *(const float4*)(B + k * SSD_L + 4 * nt);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (!CAUSAL || (i & 4) * 8 + 4 * mt + (i & 3) >= k0 + k) part[i][j] = fmaf(av[i], bv[j], part[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
  }
}

// 64 tokens x 32 lanes of rows `src` (pitch ld; tokens from nt on are zero) times w[t], turned over: dst[lane][t]
__device__ __forceinline__ void ssd_stage_turned(float* dst, int pitch, const float* src, size_t ld, int nt, const float* w) {
  for (int i = threadIdx.x; i < SSD_L * 8; i += blockDim.x) {
    const int t = i >> 3, k = (i & 7) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < nt) v = *(const float4*)(src + (size_t)t * ld + k);
    const float f = w != nullptr ? w[t] : 1.f;
    dst[k * pitch + t] = v.x * f; dst[(k + 1) * pitch + t] = v.y * f;
    dst[(k + 2) * pitch + t] = v.z * f; dst[(k + 3) * pitch + t] = v.w * f;
  }
}

// Blocks y < heads * ceil(P / 64) * (N / 64): 64 rows x 64 columns of a head's E; those behind: C B^T of a group.
template <typename T>
__global__ void __launch_bounds__(128)
ssd_states_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) float As[32 * SSD_PAD], Bs[32 * SSD_L];
  __shared__ float dt_s[SSD_L], a_s[SSD_L], w_s[SSD_L];
  __shared__ int found[3];
  int seq, first, nt;
  if (!run_chunk<SSD_L>(a.cu_q, a.n_seqs, blockIdx.x, found, seq, first, nt)) return;
  const SsdScratch out = ssd_scratch(a);
  const int inner = a.heads * a.P, C = inner + 2 * a.G * a.N, tid = threadIdx.x;
  const size_t tok = (size_t)a.cu_q[seq] + first;
  const float* rows = a.xbc + tok * C;
  const int mt = tid >> 4, nn = tid & 15;
  const int p_tiles = (a.P + SSD_L - 1) / SSD_L, n_tiles = a.N / SSD_L, state_blocks = a.heads * p_tiles * n_tiles;
  float acc[8][4] = {};
  if ((int)blockIdx.y >= state_blocks) {          // rows s, columns t, over the lanes of B and C
    const int g = blockIdx.y - state_blocks;
    const float* Bg = rows + inner + (size_t)g * a.N;
    for (int n0 = 0; n0 < a.N; n0 += 32) {
      __syncthreads();
      ssd_stage_turned(As, SSD_PAD, Bg + n0, C, nt, nullptr);
      ssd_stage_turned(Bs, SSD_L, Bg + (size_t)a.G * a.N + n0, C, nt, nullptr);
      __syncthreads();
      ssd_mma32(acc, As, Bs, mt, nn);
    }
    float* cb = out.cb + ((size_t)blockIdx.x * a.G + g) * SSD_L * SSD_L;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *(float4*)(cb + (size_t)((i & 4) * 8 + 4 * mt + (i & 3)) * SSD_L + 4 * nn) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    return;
  }
  const int h = blockIdx.y / (p_tiles * n_tiles), p0 = blockIdx.y / n_tiles % p_tiles * SSD_L, n0 = blockIdx.y % n_tiles * SSD_L;
  ssd_chunk_steps<T>(a, h, tok, nt, dt_s, a_s);
  __syncthreads();
  if (tid < 32) {                                 // D_last,s dt_s: a lane two tokens, the products of all behind them by shuffles
    const float a0 = a_s[2 * tid], a1 = a_s[2 * tid + 1];
    DecayProduct run, other;                      // of this lane's tokens and those behind them
    run.times(a0);
    run.times(a1);
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
      other.hi = __shfl_down_sync(0xffffffffu, run.hi, m);
      other.lo = __shfl_down_sync(0xffffffffu, run.lo, m);
      if (tid + m < 32) run.times(other);
    }
    if (tid == 0 && p0 == 0 && n0 == 0) out.gamma[(size_t)blockIdx.x * a.heads + h] = run.value();
    other.hi = __shfl_down_sync(0xffffffffu, run.hi, 1);
    other.lo = __shfl_down_sync(0xffffffffu, run.lo, 1);
    if (tid == 31) other = DecayProduct();
    DecayProduct last = other;
    last.times(dt_s[2 * tid + 1]);
    other.times(a1);
    other.times(dt_s[2 * tid]);
    w_s[2 * tid + 1] = last.value();
    w_s[2 * tid] = other.value();
  }
  const float* Bg = rows + inner + (size_t)(h / (a.heads / a.G)) * a.N + n0;
  const float* X = rows + (size_t)h * a.P + p0;
  for (int s0 = 0; s0 < SSD_L; s0 += 32) {        // rows n, columns p, over the tokens
    __syncthreads();
    for (int i = tid; i < 32 * 16; i += 128) {
      const int s = i >> 4, k = (i & 15) * 4;
      float4 b = make_float4(0.f, 0.f, 0.f, 0.f), x = b;
      if (s0 + s < nt) {
        const float w = w_s[s0 + s];
        b = *(const float4*)(Bg + (size_t)(s0 + s) * C + k);
        if (p0 + k < a.P) x = *(const float4*)(X + (size_t)(s0 + s) * C + k);
        x.x *= w; x.y *= w; x.z *= w; x.w *= w;
      }
      *(float4*)(As + s * SSD_PAD + k) = b;
      *(float4*)(Bs + s * SSD_L + k) = x;
    }
    __syncthreads();
    ssd_mma32(acc, As, Bs, mt, nn);
  }
  float* E = out.E + (((size_t)blockIdx.x * a.heads + h) * a.N + n0) * a.P + p0;
  if (p0 + 4 * nn < a.P) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *(float4*)(E + (size_t)((i & 4) * 8 + 4 * mt + (i & 3)) * a.P + 4 * nn) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  }
}

// Four elements of a head's state per thread, chunk after chunk; the loads of the next chunks run ahead.
__global__ void __launch_bounds__(128)
ssd_pass_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.z, h = blockIdx.y, e = (blockIdx.x * 128 + threadIdx.x) * 4;
  const int q_begin = a.cu_q[seq], q_len = a.cu_q[seq + 1] - q_begin, size = a.N * a.P;
  if (q_len <= 0 || e >= size) return;
  const SsdScratch sc = ssd_scratch(a);
  const int chunks = (q_len + SSD_L - 1) / SSD_L;
  const size_t slot0 = (size_t)(q_begin / SSD_L) + seq, step = (size_t)a.heads * size;
  float* E = sc.E + (slot0 * a.heads + h) * size + e;
  const float* gamma = sc.gamma + slot0 * a.heads + h;
  float4* S_g = (float4*)(a.state + ((size_t)a.slots[seq] * a.heads + h) * size + e);
  float4 S = *S_g;
  for (int c0 = 0; c0 < chunks; c0 += 8) {
    float4 x[8];
    float g[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < chunks) { x[i] = *(const float4*)(E + (c0 + i) * step); g[i] = gamma[(size_t)(c0 + i) * a.heads]; }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c0 + i < chunks) {
        *(float4*)(E + (c0 + i) * step) = S;
        S.x = fmaf(g[i], S.x, x[i].x); S.y = fmaf(g[i], S.y, x[i].y); S.z = fmaf(g[i], S.z, x[i].z); S.w = fmaf(g[i], S.w, x[i].w);
      }
  }
  *S_g = S;
}

template <typename T>
__global__ void __launch_bounds__(128)
ssd_outputs_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) float As[32 * SSD_PAD], Bs[32 * SSD_L];
  __shared__ __align__(16) float Ds[SSD_L * SSD_PAD];      // [s][t]: D_ts dt_s, 0 for t < s
  __shared__ float dt_s[SSD_L], a_s[SSD_L], g_s[SSD_L];
  __shared__ int found[3];
  int seq, first, nt;
  if (!run_chunk<SSD_L>(a.cu_q, a.n_seqs, blockIdx.x, found, seq, first, nt)) return;
  const SsdScratch sc = ssd_scratch(a);
  const int inner = a.heads * a.P, C = inner + 2 * a.G * a.N, tid = threadIdx.x;
  const int p_tiles = (a.P + SSD_L - 1) / SSD_L, h = blockIdx.y / p_tiles, p0 = blockIdx.y % p_tiles * SSD_L, g = h / (a.heads / a.G);
  const size_t tok = (size_t)a.cu_q[seq] + first;
  const float* rows = a.xbc + tok * C;
  const float* X = rows + (size_t)h * a.P + p0;
  ssd_chunk_steps<T>(a, h, tok, nt, dt_s, a_s);
  __syncthreads();
  if (tid < SSD_L) {                              // a thread a token s: its decays on the way to every later token
    DecayProduct d;
    d.hi = dt_s[tid];
#pragma unroll 16
    for (int t = 0; t < SSD_L; ++t) {
      if (t > tid) d.times(a_s[t]);
      Ds[tid * SSD_PAD + t] = t < tid ? 0.f : d.value();
    }
  } else if (tid == SSD_L) {
    DecayProduct run;
#pragma unroll 16
    for (int t = 0; t < SSD_L; ++t) { run.times(a_s[t]); g_s[t] = run.value(); }
  }
  const int mt = tid >> 4, nn = tid & 15;
  float acc[8][4] = {};
  const float* S = sc.E + ((size_t)blockIdx.x * a.heads + h) * a.N * a.P + p0;
  const float* Cg = rows + inner + (size_t)a.G * a.N + (size_t)g * a.N;
  for (int n0 = 0; n0 < a.N; n0 += 32) {          // rows t, columns p, over the lanes of the state
    __syncthreads();
    ssd_stage_turned(As, SSD_PAD, Cg + n0, C, nt, g_s);
    for (int i = tid; i < 32 * 16; i += 128) {
      const int n = i >> 4, k = (i & 15) * 4;
      *(float4*)(Bs + n * SSD_L + k) = p0 + k < a.P ? *(const float4*)(S + (size_t)(n0 + n) * a.P + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    ssd_mma32(acc, As, Bs, mt, nn);
  }
  const float* cb = sc.cb + ((size_t)blockIdx.x * a.G + g) * SSD_L * SSD_L;
  for (int s0 = 0; s0 < nt; s0 += 32) {           // over the chunk's tokens
    __syncthreads();
    bool odd = false;      // a value that is not finite: times the zeros of the earlier tokens' rows it would reach them
    for (int i = tid; i < 32 * 16; i += 128) {
      const int s = i >> 4, k = (i & 15) * 4;
      const float4 c = *(const float4*)(cb + (size_t)(s0 + s) * SSD_L + k), d = *(const float4*)(Ds + (s0 + s) * SSD_PAD + k);
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s0 + s < nt && p0 + k < a.P) x = *(const float4*)(X + (size_t)(s0 + s) * C + k);
      const float4 m = make_float4(c.x * d.x, c.y * d.y, c.z * d.z, c.w * d.w);
      odd = odd || !isfinite(((m.x + m.y) + (m.z + m.w)) * 0.f + ((x.x + x.y) + (x.z + x.w)) * 0.f);
      *(float4*)(As + s * SSD_PAD + k) = m;
      *(float4*)(Bs + s * SSD_L + k) = x;
    }
    if (__syncthreads_or(odd)) ssd_mma32<true>(acc, As, Bs, mt, nn, s0);
    else ssd_mma32(acc, As, Bs, mt, nn);
  }
  if (p0 + 4 * nn < a.P) {
    const float skip = a.d_skip[h];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = (i & 4) * 8 + 4 * mt + (i & 3);
      if (t >= nt) continue;
      const float4 x = *(const float4*)(X + (size_t)t * C + 4 * nn);
      *(float4*)(a.y + (tok + t) * inner + (size_t)h * a.P + p0 + 4 * nn) =
          make_float4(fmaf(skip, x.x, acc[i][0]), fmaf(skip, x.y, acc[i][1]), fmaf(skip, x.z, acc[i][2]), fmaf(skip, x.w, acc[i][3]));
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
ssd_gate_norm_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float scratch[33];
  const int inner = a.heads * a.P, part = inner / a.norm_groups;
  const int t = blockIdx.x, grp = blockIdx.y;
  const T* z = (const T*)a.proj + (size_t)t * a.ld + (size_t)grp * part;
  const float* y = a.y + (size_t)t * inner + (size_t)grp * part;
  float ss = 0.f;
  for (int i = threadIdx.x; i < part; i += blockDim.x) {
    const float v = y[i] * ssd_silu(to_f<T>(z[i]));
    ss = fmaf(v, v, ss);
  }
  ss = block_sum(ss, scratch);
  const float inv = 1.0f / sqrtf(ss / (float)part + a.eps);
  T* out = (T*)a.out + (size_t)t * inner + (size_t)grp * part;
  const float* w = a.norm_w + (size_t)grp * part;
  for (int i = threadIdx.x; i < part; i += blockDim.x) {
    const float v = y[i] * ssd_silu(to_f<T>(z[i]));
    out[i] = from_f<T>(v * inv * w[i]);
  }
}

// The same with a part's elements in registers, 4 NV a thread: read once, the logistic function taken once (2,048 tokens of 2,048:
// 9 us against 20).
template <typename T, int NV>
__global__ void __launch_bounds__(256)
ssd_gate_norm4_kernel(SsdArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float scratch[33];
  const int inner = a.heads * a.P, part = inner / a.norm_groups;
  const size_t at = (size_t)blockIdx.y * part;
  const T* z = (const T*)a.proj + (size_t)blockIdx.x * a.ld + at;
  const float* y = a.y + (size_t)blockIdx.x * inner + at;
  float4 v[NV];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (threadIdx.x + 256 * k) * 4;
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < part) {
      const float4 yv = *(const float4*)(y + i), zv = ssd_load4<T>(z + i);
      v[k] = make_float4(yv.x * ssd_silu(zv.x), yv.y * ssd_silu(zv.y), yv.z * ssd_silu(zv.z), yv.w * ssd_silu(zv.w));
      ss = fmaf(v[k].x, v[k].x, fmaf(v[k].y, v[k].y, fmaf(v[k].z, v[k].z, fmaf(v[k].w, v[k].w, ss))));
    }
  }
  ss = block_sum(ss, scratch);
  const float inv = 1.0f / sqrtf(ss / (float)part + a.eps);
  T* out = (T*)a.out + (size_t)blockIdx.x * inner + at;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = (threadIdx.x + 256 * k) * 4;
    if (i < part) {
      const float4 w = *(const float4*)(a.norm_w + at + i);
      const float o[4] = {v[k].x * inv * w.x, v[k].y * inv * w.y, v[k].z * inv * w.z, v[k].w * inv * w.w};
      if (sizeof(T) == 4) {
        *(float4*)((float*)out + i) = make_float4(o[0], o[1], o[2], o[3]);
      } else {
        uint2 r;
        *(__nv_bfloat162*)&r.x = __floats2bfloat162_rn(o[0], o[1]);
        *(__nv_bfloat162*)&r.y = __floats2bfloat162_rn(o[2], o[3]);
        *(uint2*)((bf16*)out + i) = r;
      }
    }
  }
}

template <typename T>
static int ssd_gate_norm(const SsdArgs& a, bool vec, cudaStream_t stream) {
  const int part = a.heads * a.P / a.norm_groups;
  const dim3 grid(a.n_tokens, a.norm_groups);
  if (vec && part % 4 == 0 && part <= 4096) {
    auto kernel = part <= 1024 ? ssd_gate_norm4_kernel<T, 1> : part <= 2048 ? ssd_gate_norm4_kernel<T, 2> : ssd_gate_norm4_kernel<T, 4>;
    return launch_pdl(kernel, grid, dim3(256), 0, stream, a);
  }
  return launch_pdl((ssd_gate_norm_kernel<T>), grid, dim3(256), 0, stream, a);
}

template <typename T>
static int ssd_launch(const SsdArgs& a, cudaStream_t stream) {
  const int inner = a.heads * a.P, C = inner + 2 * a.G * a.N;
  // rows and parts of rows in pieces of four elements
  const bool vec4 = inner % 4 == 0 && a.ld % 4 == 0 && (uintptr_t)a.proj % (4 * sizeof(T)) == 0 && (uintptr_t)a.out % (4 * sizeof(T)) == 0 &&
                    (((uintptr_t)a.y | (uintptr_t)a.norm_w | (uintptr_t)a.xbc | (uintptr_t)a.conv_w | (uintptr_t)a.conv_b | (uintptr_t)a.conv_state) & 15) == 0;
  // the pieces of eight tokens where there are enough of them: below, their longer way through a block is not made up for (one run of 16
  // tokens of 640 channels 14.8 us the mixer against 10.9, of 40 19.9 against 16.6; 100 tokens of 2,304 50 and 50)
  if (vec4 && C % 4 == 0 && a.taps == 4 && a.n_tokens >= 2 * SSD_CT * a.n_seqs && (long)a.n_tokens * C >= SSD_CONV4_LEAST)
    odi_rc = launch_pdl((ssd_conv4_kernel<T>), dim3((a.n_tokens + SSD_CT - 1) / SSD_CT, (C / 4 + 127) / 128), dim3(128), 0, stream, a);
  else
    odi_rc = launch_pdl((ssd_conv_kernel<T>), dim3(a.n_tokens, (C + 255) / 256), dim3(256), 0, stream, a);
  if (odi_rc == 0 && a.taps > 1)
    odi_rc = launch_pdl((ssd_conv_state_kernel<T>), dim3(a.n_seqs, (C + 255) / 256), dim3(256), 0, stream, a);
  if (a.chunks != nullptr) {
    const int p_tiles = (a.P + SSD_L - 1) / SSD_L;
    const unsigned slots = (unsigned)run_chunk_slots(a.n_tokens, a.n_seqs, SSD_L);
    if (odi_rc == 0) odi_rc = launch_pdl((ssd_states_kernel<T>), dim3(slots, a.heads * p_tiles * (a.N / SSD_L) + a.G), dim3(128), 0, stream, a);
    if (odi_rc == 0) odi_rc = launch_pdl(ssd_pass_kernel, dim3((a.N * a.P + 511) / 512, a.heads, a.n_seqs), dim3(128), 0, stream, a);
    if (odi_rc == 0) odi_rc = launch_pdl((ssd_outputs_kernel<T>), dim3(slots, a.heads * p_tiles), dim3(128), 0, stream, a);
    if (odi_rc == 0) odi_rc = ssd_gate_norm<T>(a, vec4, stream);
    return launch_status();
  }
  // Two forms: 32 columns a block when that already gives two blocks per multiprocessor (many sequences); else 8
  // columns, four times the blocks, since a warp's time is the chain of its sequence's tokens and a step of one long
  // sequence has nothing else to run beside it.  (Measured at 32 heads of 64 columns, 128 rows, 2,048 tokens: 32
  // columns 1,080 us, 8 columns 545 us, 8 columns over 16 lanes each 640 us.)
  const bool narrow = (long)((a.P + 31) / 32) * a.heads * a.n_seqs < 2 * 148;
  // Few blocks that live long start only when the kernel before has left: started early they are packed several to a
  // multiprocessor beside it and stay there (8 heads of 64 x 64, one run of 600 tokens: 129 to 271 us by what ran before).
  const bool spread = narrow && a.n_tokens >= 32 * (long)a.n_seqs;
  const int cols = narrow ? 8 : SSD_COLS;
  const dim3 grid((a.P + cols - 1) / cols, a.heads, a.n_seqs);
  const size_t smem = 2 * sizeof(float) * (SSD_TCH * (2 * (size_t)a.N + cols) + 2 * SSD_TCH);
  const int C_all = a.heads * a.P + 2 * a.G * a.N;
  const bool vec = a.N % 4 == 0 && C_all % 4 == 0 && (a.heads * a.P) % 4 == 0 && ((uintptr_t)a.xbc & 15) == 0;
  if (odi_rc == 0) {
#define ODI_SCAN_FORM(NPT, VEC, COLS, LANES) \
    do { if (smem > 48 * 1024) { \
           const cudaError_t e = cudaFuncSetAttribute(ssd_scan_kernel<T, NPT, VEC, COLS, LANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
           if (e != cudaSuccess) return (int)e; } \
         if (spread) { \
           ssd_scan_kernel<T, NPT, VEC, COLS, LANES><<<grid, dim3(COLS * LANES), smem, stream>>>(a); \
           odi_rc = (int)cudaPeekAtLastError(); \
         } else odi_rc = launch_pdl((ssd_scan_kernel<T, NPT, VEC, COLS, LANES>), grid, dim3(COLS * LANES), smem, stream, a); } while (0)
#define ODI_SCAN(NPT_WIDE, NPT_NARROW) \
    do { if (vec) { if (narrow) ODI_SCAN_FORM(NPT_NARROW, true, 8, 8); else ODI_SCAN_FORM(NPT_WIDE, true, 32, 8); } \
         else { if (narrow) ODI_SCAN_FORM(NPT_NARROW, false, 8, 8); else ODI_SCAN_FORM(NPT_WIDE, false, 32, 8); } } while (0)
    if (a.N <= 32) ODI_SCAN(4, 4); else if (a.N <= 64) ODI_SCAN(8, 8); else if (a.N <= 128) ODI_SCAN(16, 16); else ODI_SCAN(32, 32);
#undef ODI_SCAN
#undef ODI_SCAN_FORM
  }
  if (odi_rc == 0) odi_rc = ssd_gate_norm<T>(a, vec4, stream);
  return launch_status();
}

// Kernels launched by one call: 3 token by token, 5 in chunks; one more with a convolution state.
extern "C" int odi_ssd(const SsdArgs* args, int dtype, cudaStream_t stream) {
  const SsdArgs a = *args;
  if (a.n_tokens <= 0 || a.n_seqs <= 0) return 0;
  if (a.heads <= 0 || a.P <= 0 || a.N <= 0 || a.G <= 0 || a.heads % a.G != 0 || a.taps < 1 || a.norm_groups <= 0 ||
      (a.heads * a.P) % a.norm_groups != 0)
    return ODI_ERR_ARGUMENT;
  if (a.N > 256 || a.taps > SSD_MAX_TAPS || a.heads > 65535 || a.n_seqs > 65535 || a.norm_groups > 65535) return ODI_ERR_UNSUPPORTED;
  if (a.taps > 1 && a.conv_state == nullptr) return ODI_ERR_ARGUMENT;
  if (a.chunks != nullptr && (a.N % SSD_L != 0 || a.P % 4 != 0 || ((uintptr_t)a.chunks | (uintptr_t)a.xbc | (uintptr_t)a.y | (uintptr_t)a.state) % 16 != 0 ||
                              (long)a.heads * ((a.P + SSD_L - 1) / SSD_L) * (a.N / SSD_L) + a.G > 65535))
    return ODI_ERR_UNSUPPORTED;
  return dtype == 0 ? ssd_launch<float>(a, stream) : ssd_launch<bf16>(a, stream);
}
