// The chunked matrix memory's scratch, which its kernels share, and the two products on the tensor cores.
#pragma once
#include "recurrent.cuh"

constexpr int CH = CHUNK_TOKENS;

// The scratch: per (chunk, head) the gates of its tokens, then per (chunk, head) what the chunk adds, replaced by S_0 and n_0.
struct Area {
  double* f;      // [chunks][heads][64] F_t
  float* i;       // [chunks][heads][64] i_t
  float* m;       // [chunks][heads][64] m_t
  float* m0;      // [chunks][heads][4]  m_0, m behind the chunk, F behind it (as float64 in two words)
  float* s;       // [chunks][heads][size]: S [dk][dvp], n [dk] (padded to a multiple of four)
  int dvp;
  size_t size;
  __host__ __device__ static size_t piece(int dk, int dvp) { return (size_t)dk * dvp + (dk + 3) / 4 * 4; }
  __host__ __device__ static size_t floats(int chunks, int heads, int dk, int dvp) { return (size_t)chunks * heads * (4 * CH + 4 + piece(dk, dvp)); }
  __host__ __device__ Area(float* scratch, int chunks, int heads, int dk, int dvp_) {
    const size_t n = (size_t)chunks * heads;
    f = (double*)scratch;
    i = scratch + n * 2 * CH;
    m = i + n * CH;
    m0 = m + n * CH;
    s = m0 + n * 4;
    dvp = dvp_;
    size = piece(dk, dvp_);
  }
};

int co_memory_sum_tc(const MemoryIn& P, int B, int base, int count, const Area& A, int* status, cudaStream_t stream);
int co_memory_out_tc(const MemoryIn& P, const HeadOut& E, int B, int base, int count, const Area& A, int* status, cudaStream_t stream);
