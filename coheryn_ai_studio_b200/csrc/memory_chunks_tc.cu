// The two products of the chunked matrix memory (memory_chunks.cu) on the 5th-generation tensor cores, to float32's accuracy: every
// float32 operand is the sum of three bfloat16 terms (tc_common.cuh, split3), and the six products of terms i + j <= 2 are formed (as in
// gemm_f32_tc.cu).  Error of the outputs against float64 (2-norm, relative) 1.3e-7 to 1.5e-7 from 64 to 256 key channels, by float32
// multiply-adds 2.0e-7 to 3.3e-7; of the state 1.2e-7 to 1.6e-7 and 1.5e-7 to 1.7e-7.
//
//   memory_sum_tc_kernel   a CTA per (chunk, head, 128 key channels): what the chunk adds to S and n;
//   memory_out_tc_kernel   a CTA per (chunk, head): scores, outputs, and the norm, weight and gate behind them.
//
// The value channels sit on the 128 lanes (HALVES = 2 times for more than 128 of them), so S_0 and v, whose rows hold them next to one
// another, are read from memory lane by lane, 128 bytes a warp, split in registers and written to TENSOR MEMORY as the operand A, 64
// values of k at a time, while the tensor cores work on the 64 before; nothing of them passes through shared memory.  The other operand's
// terms (q, the weighted scores, the weighted keys) stand in shared memory in the 128-byte swizzle.  The scores k q^T are formed the
// same way with the keys of the chunk on 64 of the lanes.  The tensor cores' accumulator, which cuts instead of rounding, holds 64 values
// of k at most: the sums over more key channels are added up by the threads, with ordinary float32 additions.
//
// What bounds it: the chain of a CTA.  A chunk's 60 MMAs take 5 us of it; the rest is the splits (a dozen integer and float32 operations
// a value), the weights of the scores, and the norm and gate of the rows, one after another.  With more than 128 value channels a CTA has
// an SM's tensor memory to itself; with fewer it takes half of it and two CTAs share an SM (with one, steps of many chunks of narrow
// heads were slower than by multiply-adds: 8 heads of 64 x 128, three requests of 1,024 tokens 120 us by multiply-adds, 144, and 120 now).  A warp passes
// each piece of code a few times only, so the loops are kept small (unrolled further they wait for instructions: 87 us for the outputs).
// Measured on a B200, all four kernels with L2 flushed, by multiply-adds and now: 8 heads of 128 x 256, one request of 2,048 tokens 167 and
// 135 us, 7 of them the gates' divisions; 8 heads of 128 x 128, 32 requests of 128 222 and 176; the worst, 2 heads of 32 x 128 and 128
// requests of 80, 108 and 128.
//
// Every wait is for the CTA's own products and is bounded: on expiry the kernel records an error code and winds down.
#include "tc_common.cuh"
#include "memory_chunks.cuh"

namespace {

constexpr int TERM_COLS = 32;                    // a term of 64 values of k in tensor memory
constexpr int A_COLS = 3 * TERM_COLS;
constexpr int TILE = CH * 128;                   // bytes of a term's 64 tokens by 64 values in shared memory
// Pairs of terms (A's, B's), the small products first.
__device__ constexpr int PAIR_A[6] = {2, 1, 0, 1, 0, 0}, PAIR_B[6] = {0, 1, 2, 0, 1, 0};

__device__ __forceinline__ void cp4(float* to, const float* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void cp16(float* to, const float* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Sixty-four values of this thread's lane, `stride` floats apart, into three terms; from `limit` on they are zero.
__device__ __forceinline__ void split_lane(unsigned (&t0)[32], unsigned (&t1)[32], unsigned (&t2)[32], const float* from, long stride, int limit) {
#pragma unroll
  for (int k0 = 0; k0 < 64; k0 += 32) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = k0 + j < limit ? from[(k0 + j) * stride] : 0.f;      // (32 loads in flight)
#pragma unroll
    for (int j = 0; j < 16; ++j) split3(v[2 * j], v[2 * j + 1], t0[k0 / 2 + j], t1[k0 / 2 + j], t2[k0 / 2 + j]);
  }
}
__device__ __forceinline__ void put_terms(unsigned to, const unsigned (&t0)[32], const unsigned (&t1)[32], const unsigned (&t2)[32]) {
  tmem_st32(to, t0);
  tmem_st32(to + TERM_COLS, t1);
  tmem_st32(to + 2 * TERM_COLS, t2);
  tmem_wait_st();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
// Eight neighbouring values of a row from global memory, zero from the `n`-th on.
__device__ __forceinline__ void load8(float (&x)[8], const float* p, int n, bool vec) {
  if (vec && n >= 8) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = j < n ? p[j] : 0.f;
  }
}
// Eight neighbouring values as one 16-byte piece per term: piece c of row r of a tile of 128-byte rows, `step` bytes between the terms.
__device__ __forceinline__ void put_piece(unsigned char* tile, int step, int r, int c, const float (&v)[8]) {
  uint4 t[3];
  split3(v[0], v[1], t[0].x, t[1].x, t[2].x);
  split3(v[2], v[3], t[0].y, t[1].y, t[2].y);
  split3(v[4], v[5], t[0].z, t[1].z, t[2].z);
  split3(v[6], v[7], t[0].w, t[1].w, t[2].w);
#pragma unroll
  for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(tile + j * step + r * 128 + ((c ^ (r & 7)) << 4)) = t[j];
}
// ... and their sum again (exact).
__device__ __forceinline__ void get_piece(const unsigned char* tile, int step, int r, int c, float (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
#pragma unroll
  for (int j = 2; j >= 0; --j) {
    const uint4 t = *reinterpret_cast<const uint4*>(tile + j * step + r * 128 + ((c ^ (r & 7)) << 4));
    const unsigned w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { v[2 * i] += __uint_as_float(w[i] << 16); v[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u); }
  }
}
template <int THREADS>
__device__ __forceinline__ void workers_meet() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }

struct Bars { unsigned long long a_full, done; unsigned tmem; };

// One thread sets up the barriers, one warp the columns; everybody meets.
__device__ __forceinline__ unsigned begin(Bars& B, int workers, int columns) {
  if (threadIdx.x == 0) {
    mbar_init(&B.a_full, workers);
    mbar_init(&B.done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&B.tmem)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return B.tmem;
}
__device__ __forceinline__ void end(unsigned tmem, int columns) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
  }
}

// grid (chunks, heads, ceil(dk / 128)), 4 HALVES + 1 warps.
template <int HALVES>
__global__ void __launch_bounds__(32 * (4 * HALVES + 1)) memory_sum_tc_kernel(MemoryIn P, int B, int base, Area A, int* status) {
  constexpr int WORKERS = 4 * HALVES, THREADS = 32 * WORKERS, TERM = 2 * TILE;      // a term of the keys: two tiles of 64 channels
  constexpr int A_AT = 128 * HALVES, COLUMNS = HALVES == 1 ? 256 : 512;
  extern __shared__ unsigned char smem_raw[];
  __shared__ Bars bars;
  __shared__ float ws[CH];
  unsigned char* ks = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);      // [3][2][64 tokens][64 channels]
  co_pdl_wait();
  const unsigned tmem = begin(bars, WORKERS, COLUMNS);
  const int h = blockIdx.y, dk = P.dk, dv = P.dv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) { end(tmem, COLUMNS); return; }
  const int d0 = blockIdx.z * 128, row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const size_t at = (size_t)blockIdx.x * P.heads + h;
  if (tid < CH) {
    const double last = *reinterpret_cast<const double*>(A.m0 + at * 4 + 2);
    ws[tid] = tid < nt ? expf((float)(last - A.f[at * CH + tid] + (double)A.i[at * CH + tid] - (double)A.m0[at * 4 + 1])) : 0.f;
  }
  __syncthreads();
  if (warp == WORKERS) {
    if (lane == 0) {
      if (!mbar_wait(&bars.a_full, 0)) atomicExch(status, 12);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      constexpr unsigned idesc = umma_idesc_b_mn(128, 128);
      for (int half = 0; half < HALVES; ++half)
#pragma unroll
        for (int p = 0; p < 6; ++p) {
          const unsigned long long db = umma_desc_offsets(ks + PAIR_B[p] * TERM, TILE, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_a_tmem(tmem + 128 * half, tmem + A_AT + half * A_COLS + PAIR_A[p] * TERM_COLS + 8 * k, db + (unsigned long long)(128 * k), idesc, (p | k) != 0);
        }
      umma_commit(&bars.done);
    }
  } else {
    const int quarter = warp & 3, half = warp >> 2, c = half * 128 + quarter * 32 + lane;
    unsigned t0[32], t1[32], t2[32];
    const float* v = P.v + (size_t)row0 * P.ld + (size_t)h * dv + c;
    split_lane(t0, t1, t2, v, P.ld, c < dv ? nt : 0);
    put_terms(tmem + ((unsigned)(quarter * 32) << 16) + A_AT + half * A_COLS, t0, t1, t2);
    const bool vec = P.ld % 4 == 0 && dk % 4 == 0 && ((uintptr_t)P.k & 15) == 0;
#pragma unroll 4
    for (int e = tid; e < CH * 16; e += THREADS) {
      const int t = e >> 4, d = 8 * (e & 15);
      float x[8];
      load8(x, P.k + (size_t)(row0 + t) * P.ld + (size_t)h * dk + d0 + d, t < nt ? dk - d0 - d : 0, vec);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] *= ws[t];
      put_piece(ks + (d >> 6) * TILE, TERM, t, (d & 63) >> 3, x);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.a_full);
    workers_meet<THREADS>();
    float* out = A.s + at * A.size;
    if (tid < 128 && d0 + tid < dk) {               // n: a channel a thread, over the tokens
      const unsigned char* from = ks + (tid >> 6) * TILE + 2 * (tid & 7);
      float n = 0.f;
#pragma unroll 8
      for (int t = 0; t < CH; ++t) {
        const unsigned char* x = from + t * 128 + ((((tid >> 3) & 7) ^ (t & 7)) << 4);
        float w[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) w[j] = __uint_as_float((unsigned)*reinterpret_cast<const unsigned short*>(x + j * TERM) << 16);
        n += w[2] + w[1] + w[0];
      }
      out[(size_t)dk * A.dvp + d0 + tid] = n;
    }
    __syncwarp();
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&bars.done, 0));
    if (!ok && lane == 0) atomicExch(status, 13);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    out += (size_t)d0 * A.dvp + c;
    for (int j0 = 0; j0 < 128 && d0 + j0 < dk && ok; j0 += 32) {
      unsigned r[32];
      tmem_ld32(tmem + ((unsigned)(quarter * 32) << 16) + 128 * half + j0, r);
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (d0 + j0 + j < dk && c < A.dvp) out[(size_t)(j0 + j) * A.dvp] = __uint_as_float(r[j]);
    }
  }
  end(tmem, COLUMNS);
}

// Shared memory of the output kernel, two areas.  First the keys' terms per 64 key channels; when the scores are formed, the scores and,
// behind them, with up to 128 value channels the weighted scores' terms and at the end the gates over both (two CTAs fit an SM up to 128
// key channels), with more the gates.  Second q's terms and, with more than 128 value channels, the weighted scores' terms; at the end the
// finished rows.  (The keys are an operand of 128 rows: what lies behind a tile's 64 is read too, for lanes that nobody reads.)
constexpr int SCORES = CH * (CH + 4) * 4;
static_assert(SCORES % 1024 == 0, "what lies behind the scores is a tile");
__host__ __device__ inline int q_tiles(int dk) { return (dk + 63) / 64; }
inline size_t larger(size_t a, size_t b) { return ((a > b ? a : b) + 1023) / 1024 * 1024; }
size_t out_tc_keys(int dk, int dv, int dvp) {
  const size_t keys = (size_t)q_tiles(dk) * 3 * TILE, gates = (size_t)CH * dvp * 4;
  return dv <= 128 ? larger(keys, larger(SCORES + 3 * TILE, gates)) : larger(keys, SCORES + gates);
}
size_t out_tc_smem(int dk, int dv, int dvp) {
  return 1024 + out_tc_keys(dk, dv, dvp) + larger((size_t)(q_tiles(dk) + (dv <= 128 ? 0 : 1)) * 3 * TILE, (size_t)CH * (dvp + 4) * 4);
}

// Sixteen columns of this thread's lane are added to sixteen others.
__device__ __forceinline__ void columns_add(unsigned to, unsigned from) {
  unsigned x[16], y[16];
  tmem_ld16(to, x);
  tmem_ld16(from, y);
#pragma unroll
  for (int j = 0; j < 16; ++j) x[j] = __float_as_uint(__uint_as_float(x[j]) + __uint_as_float(y[j]));
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      :: "r"(to), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(x[8]), "r"(x[9]), "r"(x[10]), "r"(x[11]),
         "r"(x[12]), "r"(x[13]), "r"(x[14]), "r"(x[15]) : "memory");
  tmem_wait_st();
}

// Norm, weight and gate of the finished rows [64][pitch] of a head (head_out_chunk with four rows of a warp side by side, their gates
// and the head's weight in shared memory).  The code is small on purpose: each warp passes it once.
template <class To>
__device__ __forceinline__ void rows_out(const HeadOut& E, To* out, const float* os, int pitch, const float* gates, int ldg, const float* weight, int dv, int nt, int row0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const bool swish = E.gate_act == 1;
#pragma unroll 1
  for (int i = 4 * warp; i < nt; i += 4 * warps) {
    float inv[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int c = lane; c < dv; c += 32)
#pragma unroll
      for (int u = 0; u < 4; ++u) { const float x = os[(i + u) * pitch + c]; inv[u] = fmaf(x, x, inv[u]); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < 4; ++u) inv[u] += __shfl_xor_sync(0xffffffffu, inv[u], o);
    float mine = lane & 2 ? (lane & 1 ? inv[3] : inv[2]) : (lane & 1 ? inv[1] : inv[0]);      // one division and root for the four
    mine = 1.0f / sqrtf(mine / (float)dv + E.eps);
#pragma unroll
    for (int u = 0; u < 4; ++u) inv[u] = __shfl_sync(0xffffffffu, mine, u);
    To* to = out + (size_t)(row0 + i) * E.ldo;
#pragma unroll 2
    for (int c = lane; c < dv; c += 32) {
      const float w = weight[c];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float z = gates[(i + u) * ldg + c], g = swish ? z * rc_sigmoid(z) : rc_sigmoid(z);
        if (i + u < nt) to[(size_t)u * E.ldo + c] = (To)(os[(i + u) * pitch + c] * inv[u] * w * g * E.out_scale);
      }
    }
  }
}

// grid (chunks, heads), 4 HALVES + 1 warps.
template <int HALVES>
__global__ void __launch_bounds__(32 * (4 * HALVES + 1), 3 - HALVES) memory_out_tc_kernel(MemoryIn P, HeadOut E, int B, int base, Area A, int key_bytes, int* status) {
  constexpr int WORKERS = 4 * HALVES, THREADS = 32 * WORKERS;
  // D_P: the scores, 64 columns per block of 64 key channels, until they are taken out in front of the products with S_0.
  // D_S: the sum of S_0's blocks; D_V: the products with one block from the second on, then with the values.
  constexpr int D_P = 0, D_V = 0, D_S = 64 * HALVES, A_AT = 2 * 64 * HALVES, COLUMNS = HALVES == 1 ? 256 : 512;
  static_assert(A_AT + HALVES * A_COLS <= COLUMNS, "tensor memory");
  extern __shared__ unsigned char smem_raw[];
  __shared__ Bars bars;
  __shared__ double down[CH], up[CH];        // F_t - m_t, i_s - F_s
  __shared__ float ms[CH], as[CH], dens[CH], sums[4][CH], weight[256];
  unsigned char* ks = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);      // the keys' tiles [block][3], then:
  float* scores = (float*)ks;                               // [s][CH + 1]
  unsigned char* first = ks + key_bytes;                    // q's tiles [block][3], later the finished rows
  const int dk = P.dk, dv = P.dv, dvp = A.dvp, blocks = q_tiles(dk);
  unsigned char* ps = HALVES == 1 ? ks + SCORES : first + blocks * 3 * TILE;
  float* gates = (float*)(HALVES == 1 ? ks : ks + SCORES);  // [token][dvp]
  const unsigned tmem = begin(bars, WORKERS, COLUMNS);
  co_pdl_wait();
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) { end(tmem, COLUMNS); return; }
  const int row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const size_t at = (size_t)blockIdx.x * P.heads + h;
  if (tid < CH) {
    const double f = A.f[at * CH + tid];
    const float m = A.m[at * CH + tid];
    down[tid] = f - (double)m;
    up[tid] = (double)A.i[at * CH + tid] - f;
    ms[tid] = m;
    as[tid] = expf((float)(f + (double)A.m0[at * 4] - (double)m));
  }
  for (int i = tid; i < dv; i += blockDim.x) weight[i] = co_load_any(E.weight, E.weight_dtype, (size_t)h * E.weight_stride + i);
  // q and k in pieces of eight channels, k first; two pieces of a thread are on their way while two are split
  const bool vec = P.ld % 4 == 0 && dk % 4 == 0 && (((uintptr_t)P.q | (uintptr_t)P.k) & 15) == 0;
  const int pieces = 8 * blocks;
  const float q_scale = 1.0f / sqrtf((float)dk);
  float next[2][8];
  auto load = [&](int e) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int f = e + u * THREADS, keys = f < pieces * CH, g = keys ? f : f - pieces * CH, t = g / pieces, piece = g - t * pieces;
      load8(next[u], (keys ? P.k : P.q) + (size_t)(row0 + t) * P.ld + (size_t)h * dk + 8 * piece, t < nt ? dk - 8 * piece : 0, vec);
    }
  };
  if (warp < WORKERS) load(tid);
  __syncthreads();
  if (warp == WORKERS) {
    if (lane == 0) {
      constexpr unsigned idesc = umma_idesc(128, CH);
      bool ok = true;
      // step 0: the scores; then S_0's part, 64 channels at a time; then the values' part
      for (int b = 0; b < blocks + 2; ++b) {
        ok = ok && mbar_wait(&bars.a_full, b & 1);
        if (!ok) { atomicExch(status, 12); break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (b == 0) {
          for (int block = 0; block < blocks; ++block)
#pragma unroll
            for (int p = 0; p < 6; ++p) {
              const unsigned long long da = umma_desc(ks + (block * 3 + PAIR_A[p]) * TILE), db = umma_desc(first + (block * 3 + PAIR_B[p]) * TILE);
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_bf16(tmem + D_P + 64 * block, da + 2 * k, db + 2 * k, idesc, (p | k) != 0);
            }
        } else {
          const bool values = b == blocks + 1;
          const unsigned char* tile = values ? ps : first + (b - 1) * 3 * TILE;
          for (int half = 0; half < HALVES; ++half)
#pragma unroll
            for (int p = 0; p < 6; ++p) {
              const unsigned long long db = umma_desc(tile + PAIR_B[p] * TILE);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_bf16_a_tmem(tmem + (b == 1 ? D_S : D_V) + 64 * half, tmem + A_AT + half * A_COLS + PAIR_A[p] * TERM_COLS + 8 * k, db + 2 * k, idesc,
                                 (p | k) != 0);
            }
        }
        umma_commit(&bars.done);
      }
    }
  } else {
    const int quarter = warp & 3, half = warp >> 2, c = half * 128 + quarter * 32 + lane;
    const unsigned lanes = tmem + ((unsigned)(quarter * 32) << 16), terms = lanes + A_AT + half * A_COLS;
#pragma unroll 1
    for (int e = tid; e < 2 * pieces * CH; e += 2 * THREADS) {
      float x[2][8];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i >> 3][i & 7] = next[i >> 3][i & 7];
      if (e + 2 * THREADS < 2 * pieces * CH) load(e + 2 * THREADS);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int f = e + u * THREADS, keys = f < pieces * CH, g = keys ? f : f - pieces * CH, t = g / pieces, piece = g - t * pieces;
        const float by = keys ? 1.f : q_scale;
#pragma unroll
        for (int j = 0; j < 8; ++j) x[u][j] *= by;
        put_piece((keys ? ks : first) + (piece >> 3) * 3 * TILE, TILE, t, piece & 7, x[u]);
      }
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.a_full);
    auto fetch_gates = [&]() {
      const float* from = E.gate + (size_t)row0 * E.ldg + (size_t)h * dv;
      const bool vec = dv % 4 == 0 && E.ldg % 4 == 0 && ((uintptr_t)E.gate & 15) == 0;
      const int per = vec ? dv / 4 : dv;
#pragma unroll 1
      for (int t = warp; t < nt; t += WORKERS)
#pragma unroll 1
        for (int e = lane; e < per; e += 32) {
          if (vec) cp16(gates + t * dvp + 4 * e, from + (size_t)t * E.ldg + 4 * e);
          else cp4(gates + t * dvp + e, from + (size_t)t * E.ldg + e);
        }
      cp_commit();
    };
    bool ok = true;
    // The blocks of A, one copy of the code for all: S_0's rows, then the values.
#pragma unroll 1
    for (int b = 1; b <= blocks + 1; ++b) {
      const bool values = b == blocks + 1;
      const int d0 = 64 * (b - 1);
      if (values && quarter < 2) {
        // The weighted scores: lane s of the first two quarters, half of the tokens t for each half of the warps.
        const int s = quarter * 32 + lane;
        const double mine = up[s];
        float* score = scores + s * (CH + 1);
#pragma unroll 1
        for (int t = half * (CH / HALVES); t < (half + 1) * (CH / HALVES); t += 4) {
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            float x[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              x[i] = s <= t + j + i && t + j + i < nt ? score[t + j + i] * expf((float)(down[t + j + i] + mine)) : 0.f;
              score[t + j + i] = x[i];
            }
            unsigned y[3];
            split3(x[0], x[1], y[0], y[1], y[2]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              unsigned char* to = ps + (t + j + i) * 128 + (((s >> 3) ^ ((t + j + i) & 7)) << 4) + 2 * (s & 7);
#pragma unroll
              for (int k = 0; k < 3; ++k) *reinterpret_cast<unsigned short*>(to + k * TILE) = (unsigned short)(y[k] >> (16 * i));
            }
          }
        }
        fence_proxy_async();
      }
      unsigned t0[32], t1[32], t2[32];
      split_lane(t0, t1, t2, values ? P.v + (size_t)row0 * P.ld + (size_t)h * dv + c : A.s + at * A.size + (size_t)d0 * dvp + c,
                 values ? P.ld : (long)dvp, c >= (values ? dv : dvp) ? 0 : values ? nt : dk - d0);
      // the products with the block before have been formed when its columns are written
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.done, (b - 1) & 1)) && ok;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (b == 1) {       // the scores, added over the blocks, go to where the keys were
        if (quarter < 2)
#pragma unroll 1
          for (int t = half * (CH / HALVES); t < (half + 1) * (CH / HALVES); t += 16) {
            float* score = scores + (quarter * 32 + lane) * (CH + 1) + t;
            unsigned x[16];
            tmem_ld16(lanes + D_P + t, x);
#pragma unroll
            for (int j = 0; j < 16; ++j) score[j] = __uint_as_float(x[j]);
#pragma unroll 1
            for (int block = 1; block < blocks; ++block) {
              tmem_ld16(lanes + D_P + 64 * block + t, x);
#pragma unroll
              for (int j = 0; j < 16; ++j) score[j] += __uint_as_float(x[j]);
            }
          }
      } else if (b > 2)   // the block before is added to the sum
#pragma unroll 1
        for (int j = 64 * half; j < 64 * half + 64; j += 16) columns_add(lanes + D_S + j, lanes + D_V + j);
      put_terms(terms, t0, t1, t2);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.a_full);
      if (HALVES == 2 && b == 1) fetch_gates();      // the keys' tiles have been read: there is room
    }
    workers_meet<THREADS>();       // the scores stand
    // n_t . q_t, and with it the denominators
    {
      constexpr int PARTS = THREADS / CH;
      const int t = tid & (CH - 1), part = tid / CH;
      const float* n0 = A.s + at * A.size + (size_t)dk * dvp;
      float x = 0.f, y = 0.f;
#pragma unroll 2
      for (int piece = part; piece < 8 * blocks; piece += PARTS) {
        float q[8];
        get_piece(first + (piece >> 3) * 3 * TILE, TILE, t, piece & 7, q);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (8 * piece + j < dk) x = fmaf(q[j], n0[8 * piece + j], x);
      }
      for (int i = part; i < CH; i += PARTS) y += scores[i * (CH + 1) + t];
      sums[part][t] = fmaf(as[t], x, y);
      workers_meet<THREADS>();
      if (tid < CH) {
        float n = 0.f;
#pragma unroll
        for (int i = 0; i < PARTS; ++i) n += sums[i][tid];
        dens[tid] = 1.0f / (fmaxf(fabsf(n), expf(-ms[tid])) + 1e-6f);
      }
    }
    ok = __all_sync(0xffffffffu, mbar_wait(&bars.done, (blocks + 1) & 1)) && ok;
    if (!ok && lane == 0) atomicExch(status, 13);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    workers_meet<THREADS>();       // the denominators stand, nobody reads the tiles and scores any more
    if (HALVES == 1) fetch_gates();
    float* rows = (float*)first;
#pragma unroll 1
    for (int j0 = 0; j0 < CH; j0 += 16) {
      unsigned x[16], y[16];
      tmem_ld16(lanes + D_S + 64 * half + j0, x);
      tmem_ld16(lanes + D_V + 64 * half + j0, y);
      if (c < dvp)
#pragma unroll
        for (int j = 0; j < 16; ++j)
          rows[(j0 + j) * (dvp + 4) + c] = fmaf(as[j0 + j], __uint_as_float(x[j]), __uint_as_float(y[j])) * dens[j0 + j];
    }
    cp_wait<0>();
  }
  __syncthreads();
  if (E.out_dtype == CO_BF16) rows_out(E, (__nv_bfloat16*)E.out + (size_t)h * dv, (float*)first, dvp + 4, gates, dvp, weight, dv, nt, row0);
  else rows_out(E, (float*)E.out + (size_t)h * dv, (float*)first, dvp + 4, gates, dvp, weight, dv, nt, row0);
  end(tmem, COLUMNS);
}

}  // namespace

int co_memory_sum_tc(const MemoryIn& P, int B, int base, int count, const Area& A, int* status, cudaStream_t stream) {
  constexpr int smem = 1024 + 6 * TILE;
  auto kernel = P.dv <= 128 ? memory_sum_tc_kernel<1> : memory_sum_tc_kernel<2>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  co_launch(kernel, dim3(count, P.heads, (P.dk + 127) / 128), dim3(P.dv <= 128 ? 160 : 288), (size_t)smem, stream, P, B, base, A, status);
  CO_CHECK_LAUNCH("memory_sum_tc");
  return 0;
}
int co_memory_out_tc(const MemoryIn& P, const HeadOut& E, int B, int base, int count, const Area& A, int* status, cudaStream_t stream) {
  const size_t smem = out_tc_smem(P.dk, P.dv, A.dvp);
  auto kernel = P.dv <= 128 ? memory_out_tc_kernel<1> : memory_out_tc_kernel<2>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  co_launch(kernel, dim3(count, P.heads), dim3(P.dv <= 128 ? 160 : 288), smem, stream, P, E, B, base, A, (int)out_tc_keys(P.dk, P.dv, A.dvp), status);
  CO_CHECK_LAUNCH("memory_out_tc");
  return 0;
}
