// Runs of tokens cut into chunks of L: chunk c of sequence s lies at slot cu_q[s] / L + s + c, so that no two chunks share a
// slot and no sum over the sequences is needed; run_chunk_slots() slots hold them all.
#pragma once
#include "common.cuh"

static inline size_t run_chunk_slots(int n_tokens, int n_seqs, int L) { return (size_t)n_tokens / L + n_seqs; }

// Which chunk slot `b` holds: (sequence, first token of the chunk within its run, its tokens), by all threads of a block;
// false for a slot that holds none.  `found`: three ints of shared memory.
template <int L>
__device__ __forceinline__ bool run_chunk(const int* cu_q, int n_seqs, int b, int* found, int& seq, int& first, int& nt) {
  if (threadIdx.x == 0) found[0] = -1;
  __syncthreads();
  for (int s = threadIdx.x; s < n_seqs; s += blockDim.x) {
    const int begin = cu_q[s], len = cu_q[s + 1] - begin, lo = begin / L + s;
    if (b >= lo && b < lo + (len + L - 1) / L) { found[1] = (b - lo) * L; found[2] = min(L, len - (b - lo) * L); found[0] = s; }
  }
  __syncthreads();
  seq = found[0]; first = found[1]; nt = found[2];
  return seq >= 0;
}

// A product of decays carried as two floats and rounded once at the end: in the sums over a state's rows the errors of a chunk's
// decays, which all rows share, do not even out as those of rows that round by themselves do.
struct DecayProduct {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float a) {
    const float p = __fmul_rn(hi, a);
    lo = fmaf(lo, a, fmaf(hi, a, -p));
    hi = p;
  }
  __device__ __forceinline__ void times(const DecayProduct& o) {
    const float p = __fmul_rn(hi, o.hi);
    lo = fmaf(hi, o.lo, fmaf(lo, o.hi, fmaf(hi, o.hi, -p)));
    hi = p;
  }
  __device__ __forceinline__ float value() const { return hi + lo; }
};
