// Grouped matrix product: many small products C_g = A_g W_g^T in one launch, each group with a weight matrix of its own, fp32
// accumulation in an order that no other row of the launch changes.  T = float (the true 32-bit path): on the CUDA cores, over
// k = 0..K-1 in that order, or for groups of a few rows a lane's k and then the lanes by a tree.  T = bf16 with aligned operands: on
// the tensor cores (grouped_mma_kernel says how its sums are grouped); else, and for products per head of many rows and few
// k, as float in tiles.
//
// Two ways to say which rows belong to which group:
//  * dense (tile table null): every group has the same M rows; group g reads columns [g * a_group_off, +K) of
//    A's rows 0..M-1 and writes columns [g * c_group_off, +N) of C's rows (a product per head);
//  * by table (routed experts): tile t covers `tile_rows[t]` rows from `tile_row0[t]` on, in an order sorted
//    by group, all of group `tile_group[t]`; `n_tiles[0]` tiles exist (blocks beyond it leave).  Row i of that
//    order reads row `row_index[i] / index_div` of A (row i itself if row_index is null) and writes row i of C.
//
// Epilogues: 0 store as T, 1 store as fp32, 2 gated and clamped (W_g holds N gate rows then N up rows;
// g = min(gate, limit), u = clamp(up, -limit, limit), C = g * sigmoid(alpha * g) * (u + up_shift) as T), 3 the exact
// (erf) GELU of the sum as T, 4 its tanh form, 5 the square of max(sum, 0) as T.
//
// Tile on the CUDA cores: TM rows x 64 features per block of 256 threads, K in slices of 16 or 32 through shared memory (fp32).
// TM = 64 (4 x 4 outputs a thread) or 16 (1 x 4), chosen by the caller from the rows a group has; for float groups
// of a few rows there is a form that streams the weights through registers only (grouped_gemv_kernel).
#include "common.cuh"

#define TN 64

__device__ __forceinline__ float grouped_act(float z, int epi) {
  if (epi == 3) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f));
  if (epi == 4) return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
  if (epi == 5) { const float r = fmaxf(z, 0.f); return r * r; }
  return z;
}

struct GroupedArgs {
  const void* A;
  const void* W;
  void* C;
  const int* row_index;
  const int* tile_group;
  const int* tile_row0;
  const int* tile_rows;
  const int* n_tiles;
  long long a_group_off, w_group_stride, c_group_off;
  int lda, ldw, ldc, M, N, K, groups, index_div, epi;
  float limit, alpha, up_shift;
};

// Eight consecutive elements of a row as floats (16-byte loads; the caller has checked the alignment).
template <typename T> __device__ __forceinline__ void load8(const T* p, float* out);
template <> __device__ __forceinline__ void load8<float>(const float* p, float* out) {
  const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
  out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w; out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
}
template <> __device__ __forceinline__ void load8<bf16>(const bf16* p, float* out) {
  const uint4 raw = *(const uint4*)p;
  const __nv_bfloat162* h = (const __nv_bfloat162*)&raw;
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); out[2 * i] = f.x; out[2 * i + 1] = f.y; }
}

// A k-major tile in shared memory, [TK][STR] floats with 8 more floats after every 8 k: the four 8-element
// pieces of a row's 32 k land in different banks when one warp stores them.
#define SIDX(k, i, STR) ((k) * (STR) + ((k) >> 3) * 8 + (i))

// VEC: K, the row strides and the group offsets are multiples of 8 elements and the bases 16-byte aligned:
// slices of 32 k, one 8-element piece per thread and tile; else slices of 16 k, element by element.
template <typename T, int TM, bool GATED, bool VEC>
__global__ void __launch_bounds__(256)
grouped_gemm_kernel(GroupedArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int RPT = TM / 16;
  constexpr int TK = VEC ? 32 : 16;
  constexpr int ASTR = TM + 4, WSTR = TN + 4;
  __shared__ __align__(16) float As[TK * ASTR + (TK / 8) * 8];
  __shared__ __align__(16) float Ws[GATED ? 2 : 1][TK * WSTR + (TK / 8) * 8];
  __shared__ int arow[TM];
  const int tid = threadIdx.x;
  int group, row0, rows;
  if (a.tile_group != nullptr) {
    const int t = blockIdx.x;
    if (t >= a.n_tiles[0]) return;
    group = a.tile_group[t]; row0 = a.tile_row0[t]; rows = a.tile_rows[t];
  } else {
    group = blockIdx.z; row0 = blockIdx.x * TM; rows = min(TM, a.M - row0);
  }
  const int n0 = blockIdx.y * TN;
  if (tid < TM) {
    int r = -1;
    if (tid < rows) r = a.row_index != nullptr ? a.row_index[row0 + tid] / a.index_div : row0 + tid;
    arow[tid] = r;
  }
  __syncthreads();
  const T* A = (const T*)a.A + (a.tile_group != nullptr ? 0 : (size_t)group * a.a_group_off);
  const T* W = (const T*)a.W + (size_t)group * a.w_group_stride;
  const int tx = tid & 15, ty = tid >> 4;
  float acc[GATED ? 2 : 1][RPT][4] = {};

  // VEC: the pieces of the next slice are requested while the current one is multiplied
  float va[8], vw[GATED ? 2 : 1][8];
  const int piece = tid & 3, vrow = tid >> 2;
  auto fetch = [&](int k0) {
    const int k = k0 + piece * 8;
    const int src = tid < TM * 4 ? arow[vrow] : -1;
    if (src >= 0 && k < a.K) load8<T>(A + (size_t)src * a.lda + k, va);
    else {
#pragma unroll
      for (int i = 0; i < 8; ++i) va[i] = 0.f;
    }
    const bool in = n0 + vrow < a.N && k < a.K;
#pragma unroll
    for (int s = 0; s < (GATED ? 2 : 1); ++s) {
      if (in) load8<T>(W + (size_t)(s * a.N + n0 + vrow) * a.ldw + k, vw[s]);
      else {
#pragma unroll
        for (int i = 0; i < 8; ++i) vw[s][i] = 0.f;
      }
    }
  };
  if (VEC) fetch(0);

  for (int k0 = 0; k0 < a.K; k0 += TK) {
    __syncthreads();
    if (VEC) {
      if (tid < TM * 4) {
#pragma unroll
        for (int i = 0; i < 8; ++i) As[SIDX(piece * 8 + i, vrow, ASTR)] = va[i];
      }
#pragma unroll
      for (int s = 0; s < (GATED ? 2 : 1); ++s) {
#pragma unroll
        for (int i = 0; i < 8; ++i) Ws[s][SIDX(piece * 8 + i, vrow, WSTR)] = vw[s][i];
      }
      if (k0 + TK < a.K) fetch(k0 + TK);
    } else {
      for (int i = tid; i < TM * TK; i += 256) {
        const int r = i / TK, k = i % TK;
        const int src = arow[r];
        As[SIDX(k, r, ASTR)] = (src >= 0 && k0 + k < a.K) ? to_f<T>(A[(size_t)src * a.lda + k0 + k]) : 0.f;
      }
      for (int i = tid; i < TN * TK; i += 256) {
        const int n = i / TK, k = i % TK;
        const bool in = n0 + n < a.N && k0 + k < a.K;
        Ws[0][SIDX(k, n, WSTR)] = in ? to_f<T>(W[(size_t)(n0 + n) * a.ldw + k0 + k]) : 0.f;
        if (GATED) Ws[1][SIDX(k, n, WSTR)] = in ? to_f<T>(W[(size_t)(a.N + n0 + n) * a.ldw + k0 + k]) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      float ar[RPT];
#pragma unroll
      for (int i = 0; i < RPT; ++i) ar[i] = As[SIDX(k, ty * RPT + i, ASTR)];
#pragma unroll
      for (int s = 0; s < (GATED ? 2 : 1); ++s) {
        const float4 wv = *(const float4*)&Ws[s][SIDX(k, tx * 4, WSTR)];
        const float wr[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[s][i][j] = fmaf(ar[i], wr[j], acc[s][i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = ty * RPT + i;
    if (r >= rows) continue;
    const size_t crow = (size_t)(row0 + r) * a.ldc + (a.tile_group != nullptr ? 0 : (size_t)group * a.c_group_off);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= a.N) continue;
      if (GATED) {
        const float g = fminf(acc[0][i][j], a.limit);
        const float u = fminf(fmaxf(acc[GATED ? 1 : 0][i][j], -a.limit), a.limit);
        ((T*)a.C)[crow + n] = from_f<T>(g / (1.f + expf(-a.alpha * g)) * (u + a.up_shift));
      } else if (a.epi == 1) {
        ((float*)a.C)[crow + n] = acc[0][i][j];
      } else {
        ((T*)a.C)[crow + n] = from_f<T>(grouped_act(acc[0][i][j], a.epi));
      }
    }
  }
}

// Few rows per group (single-token steps): no tile of the weights in shared memory.  A block takes up to 4 rows
// of one group and 64 features (32 in the gated form); the rows wait in shared memory as floats, each of the 8 warps takes 8 weight
// rows (for the gated form 4 features: their gate and up rows), a lane reads 8 consecutive k of each weight row
// per step (16-byte loads, eight in flight) and keeps one sum per weight row and input row; sums are reduced over
// the lanes at the end (a fixed tree: the result of a row does not depend on the other rows of the launch).
// Needs what VEC needs.
#define GV_ROWS 4
template <bool GATED>
__global__ void __launch_bounds__(256, 2)
grouped_gemv_kernel(GroupedArgs a) {
  typedef float T;
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float xs[];       // [GV_ROWS][K]
  __shared__ int arow[GV_ROWS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int group, row0, rows;
  if (a.tile_group != nullptr) {
    const int t = blockIdx.x;
    if (t >= a.n_tiles[0]) return;
    group = a.tile_group[t]; row0 = a.tile_row0[t]; rows = a.tile_rows[t];
  } else {
    group = blockIdx.z; row0 = blockIdx.x * GV_ROWS; rows = min(GV_ROWS, a.M - row0);
  }
  if (tid < GV_ROWS) {
    int r = -1;
    if (tid < rows) r = a.row_index != nullptr ? a.row_index[row0 + tid] / a.index_div : row0 + tid;
    arow[tid] = r;
  }
  __syncthreads();
  const T* A = (const T*)a.A + (a.tile_group != nullptr ? 0 : (size_t)group * a.a_group_off);
  const T* W = (const T*)a.W + (size_t)group * a.w_group_stride;
  for (int i = tid * 8; i < GV_ROWS * a.K; i += 256 * 8) {
    const int r = i / a.K, k = i % a.K;
    float v[8];
    if (arow[r] >= 0) load8<T>(A + (size_t)arow[r] * a.lda + k, v);
    else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) xs[i + j] = v[j];
  }
  __syncthreads();
  // weight row j of this warp: plain form feature n0 + warp * 8 + j; gated form feature n0 + warp * 4 + j / 2,
  // its gate row (j even) or up row (j odd)
  const int n0 = blockIdx.y * (GATED ? 32 : 64);      // 8 warps x 8 weight rows: 64 features, or 32 gated ones
  const T* wrow[8];
  bool wlive[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int n = GATED ? n0 + warp * 4 + (j >> 1) : n0 + warp * 8 + j;
    wlive[j] = n < a.N;
    wrow[j] = W + (size_t)((GATED && (j & 1)) ? a.N + n : n) * a.ldw;
  }
  float acc[8][GV_ROWS] = {};
  for (int k = lane * 8; k < a.K; k += 256) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {       // four weight rows at a time: fewer registers, two blocks per SM
      float w[4][8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (wlive[half * 4 + j]) load8<T>(wrow[half * 4 + j] + k, w[j]);
        else {
#pragma unroll
          for (int e = 0; e < 8; ++e) w[j][e] = 0.f;
        }
      }
#pragma unroll
      for (int r = 0; r < GV_ROWS; ++r) {
        const float4 x0 = *(const float4*)&xs[r * a.K + k], x1 = *(const float4*)&xs[r * a.K + k + 4];
        const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[half * 4 + j][r] = fmaf(w[j][e], x[e], acc[half * 4 + j][r]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int r = 0; r < GV_ROWS; ++r) acc[j][r] = warp_sum(acc[j][r]);
  if (lane != 0) return;
#pragma unroll
  for (int r = 0; r < GV_ROWS; ++r) {
    if (r >= rows) continue;
    const size_t crow = (size_t)(row0 + r) * a.ldc + (a.tile_group != nullptr ? 0 : (size_t)group * a.c_group_off);
    if (GATED) {
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const int n = n0 + warp * 4 + f;
        if (n >= a.N) continue;
        const float g = fminf(acc[2 * f][r], a.limit);
        const float u = fminf(fmaxf(acc[2 * f + 1][r], -a.limit), a.limit);
        ((T*)a.C)[crow + n] = from_f<T>(g / (1.f + expf(-a.alpha * g)) * (u + a.up_shift));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int n = n0 + warp * 8 + j;
        if (n >= a.N) continue;
        if (a.epi == 1) ((float*)a.C)[crow + n] = acc[j][r];
        else ((T*)a.C)[crow + n] = from_f<T>(grouped_act(acc[j][r], a.epi));
      }
    }
  }
}

// bf16 on the tensor cores (mma.sync m16n8k16, fp32 sums): the weights are the 16-row operand, 8 NT input rows of a group the
// 8-column ones, so a group's weights pass once over a tile of its rows (a table's larger tile: once per 8 NT rows of it).  What
// bounds it is the stream of weights, so nothing stands between it and the tensor cores: a lane loads 16 bytes (8 neighbouring
// k) of its weight rows straight into registers, and of its input rows likewise; the k of an mma may come in any order as long as
// both operands agree, so those 8 are the lane's k of two mma.  A block owns 16 features (gated: and their 16 up rows) and all
// k: its four warps take pieces of 128 k in turn, all of a piece's loads on their way at once (about 100 KB a multiprocessor), the
// first weights before the input rows are looked up; the warps' sums meet in shared memory.  The tensor core cuts off what its
// sums cannot hold, so 16 k (gated: 8) are summed from zero there, the sums of a piece's 128 k pairwise and then to the rest by
// rounded additions, in an order that depends on neither the other rows nor NT.  Norm of the error of a sum against 64 bits, K = 64 / 256 /
// 1,024 / 4,096: 4.4e-8 / 5.7e-8 / 6.9e-8 / 8.5e-8; the CUDA cores' forms before: up to four rows a group 4.0e-8 / 5.5e-8 / 6.9e-8 / 9.5e-8, more
// rows 5.2e-8 / 1.1e-7 / 2.5e-7 / 6.1e-7.
// Measured, bf16, four of 32 experts of 2,048 x 1,024 a token, L2 flushed, up / gated up / down in us, against the forms before (lists
// of items walked by warps on the CUDA cores up to 4 rows an expert, else tiles of 16 rows there): 1 token 8 / 11 / 7 and 9 / 14 / 9, 8
// tokens 20 / 34 / 18 and 34 / 54 / 34 (the weights alone 13 / 26 / 13), 32 tokens 26 / 50 / 27 and 79 / 122 / 124, 56 tokens 30 / 56 / 30
// and 221 / 400 / 186, 250 tokens 70 / 123 / 72 and 467 / 810 / 434.  Tiles of 32 and 64 rows were no faster (250 tokens: 72 and 107).
// The gated form holds two accumulators, so eight sums of 16 k at once do not fit its registers; one after the other (32 k at a time)
// they were 7.2e-8 off at K = 2,048, met pairwise from sums of 8 k 2.7e-8 (products that cancel, where the CUDA cores gave 4.1e-8),
// and no slower (8 tokens 39 us against 42, 56 tokens 58 against 62, another run).
__device__ __forceinline__ void mma16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same product over the 32 k that four lanes hold, 8 each: four sums of 8 k (m16n8k8), met pairwise; with few registers.
__device__ __forceinline__ void mma_piece(float (&s)[4], const uint4& w0, const uint4& w1, const uint4& x) {
  auto quarter = [](float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(b), "f"(0.f));
  };
  float p[4], q[4];
  quarter(s, w0.x, w1.x, x.x);
  quarter(p, w0.y, w1.y, x.y);
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] += p[e];
  quarter(p, w0.z, w1.z, x.z);
  quarter(q, w0.w, w1.w, x.w);
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] += p[e] + q[e];
}
template <bool GATED, int NT>
__global__ void __launch_bounds__(128, GATED ? (NT == 1 ? 4 : 3) : (NT == 1 ? 6 : 5))      // six blocks a multiprocessor: 80 registers (56 tokens: 28 us, with 147 35)
grouped_mma_kernel(GroupedArgs a, int tm, int tiles) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int MT = GATED ? 2 : 1, ROWS = 8 * NT, PITCH = ROWS + 1, U = 4, PIECE = 32 * U;
  __shared__ float red[4][MT * 16][PITCH];
  __shared__ int arow[ROWS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const bool table = a.tile_group != nullptr;
  int group, tile_row0, tile_rows;
  if (table) {
    const int t = blockIdx.x % tiles;
    if (t >= a.n_tiles[0]) return;
    group = a.tile_group[t]; tile_row0 = a.tile_row0[t]; tile_rows = a.tile_rows[t];
  } else {
    group = blockIdx.z; tile_row0 = blockIdx.x % tiles * tm; tile_rows = min(tm, a.M - tile_row0);
  }
  const int n0 = blockIdx.x / tiles * 16;
  const bf16* A = (const bf16*)a.A + (table ? 0 : (size_t)group * a.a_group_off) + 8 * tq;
  const bf16* W = (const bf16*)a.W + (size_t)group * a.w_group_stride + 8 * tq;
  const bf16* wrow[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int n = n0 + 8 * i + gq;
      wrow[m][i] = n < a.N ? W + (size_t)(m ? a.N + n : n) * a.ldw : nullptr;
    }
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 w[U][MT][2];
  auto load_w = [&](int kc) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = kc + 32 * u;
      const bool in = k + 8 * tq < a.K;      // K is a multiple of 8: a lane's 8 are all inside or all outside
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          w[u][m][i] = zero;
          if (in && wrow[m][i] != nullptr) {
            uint4& r = w[u][m][i];
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(wrow[m][i] + k));
          }
        }
    }
  };
  for (int done = 0; done < tile_rows; done += ROWS) {
    const int row0 = tile_row0 + done, rows = min(ROWS, tile_rows - done);
    load_w(warp * PIECE);                    // on their way while the input rows are looked up
    if (tid < ROWS) arow[tid] = tid < rows ? (a.row_index != nullptr ? a.row_index[row0 + tid] / a.index_div : row0 + tid) : -1;
    __syncthreads();
    const bf16* xrow[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) xrow[j] = arow[8 * j + gq] >= 0 ? A + (size_t)arow[8 * j + gq] * a.lda : nullptr;
    float acc[MT][NT][4] = {};
    for (int kc = warp * PIECE; kc < a.K; kc += 4 * PIECE) {
      uint4 x[U][NT];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j)
          x[u][j] = xrow[j] != nullptr && kc + 32 * u + 8 * tq < a.K ? *(const uint4*)(xrow[j] + kc + 32 * u) : zero;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          if (GATED) {
            float s[2][4], t[4];
            static_assert(U == 4, "two pairs of sums");
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              mma_piece(s[h], w[2 * h][m][0], w[2 * h][m][1], x[2 * h][j]);
              mma_piece(t, w[2 * h + 1][m][0], w[2 * h + 1][m][1], x[2 * h + 1][j]);
#pragma unroll
              for (int e = 0; e < 4; ++e) s[h][e] += t[e];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[m][j][e] += s[0][e] + s[1][e];
            continue;
          }
          float c[2 * U][4] = {};
#pragma unroll
          for (int u = 0; u < U; ++u) {
            mma16(c[2 * u], w[u][m][0].x, w[u][m][1].x, w[u][m][0].y, w[u][m][1].y, x[u][j].x, x[u][j].y);
            mma16(c[2 * u + 1], w[u][m][0].z, w[u][m][1].z, w[u][m][0].w, w[u][m][1].w, x[u][j].z, x[u][j].w);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            acc[m][j][e] += ((c[0][e] + c[1][e]) + (c[2][e] + c[3][e])) + ((c[4][e] + c[5][e]) + (c[6][e] + c[7][e]));
        }
      load_w(kc + 4 * PIECE);
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) red[warp][16 * m + gq + 8 * (e >> 1)][8 * j + 2 * tq + (e & 1)] = acc[m][j][e];
    __syncthreads();
    const size_t c0 = table ? 0 : (size_t)group * a.c_group_off;
    auto sum = [&](int f, int r) { return (red[0][f][r] + red[1][f][r]) + (red[2][f][r] + red[3][f][r]); };
    for (int i = tid; i < 16 * rows; i += 128) {
      const int f = i & 15, r = i >> 4;
      if (n0 + f >= a.N) continue;
      const size_t at = (size_t)(row0 + r) * a.ldc + c0 + n0 + f;
      const float v = sum(f, r);
      if (GATED) {
        const float g = fminf(v, a.limit), up = fminf(fmaxf(sum(16 * (MT - 1) + f, r), -a.limit), a.limit);
        ((bf16*)a.C)[at] = from_f<bf16>(g / (1.f + expf(-a.alpha * g)) * (up + a.up_shift));
      } else if (a.epi == 1) {
        ((float*)a.C)[at] = v;
      } else {
        ((bf16*)a.C)[at] = from_f<bf16>(grouped_act(v, a.epi));
      }
    }
    __syncthreads();                         // the next rows' sums take the place of these
  }
}

static int launch_mma(const GroupedArgs& a, int max_tiles, int tm, cudaStream_t stream) {
  const bool table = a.tile_group != nullptr;
  if (table ? max_tiles <= 0 : a.M <= 0) return 0;
  const int tiles = table ? max_tiles : (a.M + tm - 1) / tm;
  const long blocks = (long)tiles * ((a.N + 15) / 16);
  if (blocks > 0x7fffffffL || (!table && a.groups > 65535)) return ODI_ERR_UNSUPPORTED;
  const dim3 grid((unsigned)blocks, 1, table ? 1 : a.groups);
  auto kernel = a.epi == 2 ? (tm <= 8 ? grouped_mma_kernel<true, 1> : grouped_mma_kernel<true, 2>)
                           : (tm <= 8 ? grouped_mma_kernel<false, 1> : grouped_mma_kernel<false, 2>);
  odi_rc = launch_pdl(kernel, grid, dim3(128), 0, stream, a, tm, tiles);
  return launch_status();
}

// max_tiles: with a tile table, the most tiles the table can hold (the grid's width).  tm: rows of a tile (a table must have been
// built for the same).  bf16 with aligned operands: 4, 8 or 16 rows on the tensor cores, 64 on the CUDA cores (a product per head of
// many rows and few k: grouped_heads_tile in ops.py says where).  Else 16 (8 with a table: the same form) or 64, or in float32 with
// aligned operands 4, the form for few rows (odi_grouped_gemm_takes_few_rows says whether it can run).
static bool vector_loads(const GroupedArgs& a) {
  return a.K % 8 == 0 && a.lda % 8 == 0 && a.ldw % 8 == 0 && a.a_group_off % 8 == 0 && a.w_group_stride % 8 == 0 &&
         (uintptr_t)a.A % 16 == 0 && (uintptr_t)a.W % 16 == 0;
}

extern "C" int odi_grouped_gemm_takes_few_rows(const GroupedArgs* args) {
  return vector_loads(*args) && (size_t)GV_ROWS * args->K * sizeof(float) <= 200 * 1024;
}

extern "C" int odi_grouped_gemm_takes_tensor(const GroupedArgs* args) { return vector_loads(*args); }

extern "C" int odi_grouped_gemm(const GroupedArgs* args, int max_tiles, int tm, int dtype, cudaStream_t stream) {
  const GroupedArgs a = *args;
  if (a.N <= 0 || a.groups <= 0) return 0;
  if (a.K <= 0 || (tm != GV_ROWS && tm != 8 && tm != 16 && tm != 64) || a.epi < 0 || a.epi > 5) return ODI_ERR_ARGUMENT;
  const bool vec = vector_loads(a);
  if (dtype == 1 && vec && tm != 64) return launch_mma(a, max_tiles, tm, stream);
  if (tm == 8 && a.tile_group == nullptr) return ODI_ERR_UNSUPPORTED;      // a table's tiles of 8 rows fit the form for 16
  if (tm == GV_ROWS) {
    if (dtype != 0 || !odi_grouped_gemm_takes_few_rows(args)) return ODI_ERR_UNSUPPORTED;      // bf16 operands that allow it have left above
    dim3 grid;
    const int per_block = a.epi == 2 ? 32 : 64;
    if (a.tile_group != nullptr) {
      if (max_tiles <= 0) return 0;
      grid = dim3(max_tiles, (a.N + per_block - 1) / per_block, 1);
    } else {
      if (a.M <= 0) return 0;
      grid = dim3((a.M + GV_ROWS - 1) / GV_ROWS, (a.N + per_block - 1) / per_block, a.groups);
      if (grid.z > 65535) return ODI_ERR_UNSUPPORTED;
    }
    if (grid.y > 65535) return ODI_ERR_UNSUPPORTED;
    const size_t smem = (size_t)GV_ROWS * a.K * sizeof(float);
    auto kernel = a.epi == 2 ? grouped_gemv_kernel<true> : grouped_gemv_kernel<false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    odi_rc = launch_pdl(kernel, grid, dim3(256), smem, stream, a);
    return launch_status();
  }
  dim3 grid;
  if (a.tile_group != nullptr) {
    if (max_tiles <= 0) return 0;
    grid = dim3(max_tiles, (a.N + TN - 1) / TN, 1);
  } else {
    if (a.M <= 0) return 0;
    grid = dim3((a.M + tm - 1) / tm, (a.N + TN - 1) / TN, a.groups);
    if (grid.z > 65535) return ODI_ERR_UNSUPPORTED;
  }
  if (grid.y > 65535) return ODI_ERR_UNSUPPORTED;
#define ODI_GG(T, TM, G, VEC) odi_rc = launch_pdl((grouped_gemm_kernel<T, TM, G, VEC>), grid, dim3(256), 0, stream, a)
#define ODI_GG_FORMS(T, VEC) \
  do { if (tm == 64) { if (gated) ODI_GG(T, 64, true, VEC); else ODI_GG(T, 64, false, VEC); } \
       else { if (gated) ODI_GG(T, 16, true, VEC); else ODI_GG(T, 16, false, VEC); } } while (0)
  const bool gated = a.epi == 2;
  if (dtype == 1 && vec) { if (gated) ODI_GG(bf16, 64, true, true); else ODI_GG(bf16, 64, false, true); }      // tiles of fewer rows: above
  else if (dtype == 1) ODI_GG_FORMS(bf16, false);
  else if (vec) ODI_GG_FORMS(float, true);
  else ODI_GG_FORMS(float, false);
#undef ODI_GG_FORMS
#undef ODI_GG
  return launch_status();
}
