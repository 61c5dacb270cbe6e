// out[M, N] = x[M, K] . W[N, K]^T (+ bias) of float32 operands to float32's accuracy on the 5th-generation tensor cores.
//
// Every float32 value from 2^-110 up is the exact sum of three bfloat16 ones, v = v0 + v1 + v2 (each the rest's nearest: 8 + 8 + 8 bits),
// and a product of two bfloat16 values is exact in the accumulator.  Of the nine products of terms the six with i + j <= 2 are formed; of
// the three left out two are below 2^-25 of |x w| each and one below 2^-33: together what rounding one product may cost.  The accumulator
// in tensor memory only ever holds 64 values of k, the small products first and x0 w0 last, and is then added to sums in registers with
// ordinary float32 additions: its own rounding (which truncates) touches the large products four times per 64 values, and a sum of K
// values has K / 64 roundings in place of the FMA chain's K.  Measured against float64: below.
//
// The operands swap places as in gemm_tc_few.cu: 128 output features sit on the lanes, BT tokens on the columns.  The tokens'
// three terms are written once by a small kernel and come by TMA; W is read once from memory in float32 and split on its way:
//
//   warp 0       producer: W boxes of 128 x 32 floats (a ring of three stages of 64 k, fetched before the wait for the kernel that makes x's terms),
//                x terms (two stages; from 96 tokens on a term is fetched again as soon as its last product is formed)
//   warp 1       issues 24 tcgen05.mma per stage: A = W's terms in TENSOR MEMORY, B = x's terms in shared memory
//   warps 2-5    split: a thread reads its feature's 64 values, writes 3 x 32 columns of bfloat16 pairs to tensor memory
//   warps 6-13   add a stage's accumulator (two of them in tensor memory) to their sums, and the epilogue
//
// What bounds it: the chain of a CTA's stages (W's tile, its split, the products, the sums) with one CTA per SM.  The profiler's counters:
// 313 x 17920 x 1536 keeps the tensor pipe 55 % busy, the integer pipe of the split 25 % and DRAM 27 %; one row by 17920 x 1536 DRAM 39 %
// and the integer pipe 30 %.  (With W's terms in shared memory as well that would move 480 KB a stage in place of 248.)  Measured on a B200
// (alone, L2 flushed, with the two small kernels; before: the CUDA cores, gemm_simt.cu): 313 x 17920 x 1536 417 -> 105 us, 313 x 1536 x 8960
// 216 -> 73, 313 x 1536 x 1536 77 -> 24, 2048 x 17920 x 1536 2,518 -> 632, one row by 17920 x 1536 84 -> 40.  Error against float64
// (2-norm, relative): 0.8e-7 to 1.2e-7 where the FMA chain has 2.8e-7 to 5.0e-7.
//
// A row's result does not depend on the other rows: K is cut into slices by the weight's shape alone, a slice's sum goes to a
// workspace (where there is more than one) and the slices are added in order.  Two kinds of results are formed again from the operands
// themselves, by float32 multiply-adds: one that is not finite (an infinity has no finite rest, so the terms' products would make it a
// NaN), and one so small that the bits which the split of operands under 2^-110 cuts off may count in it.  For the second the largest
// magnitude of the row and of the feature are kept: with operands of ordinary size beside the small ones nothing is formed again (an
// activation of 1e-34 leaves its row's results alone: 313 x 1536 x 8960 with one in every row 71 us, with none 69 to 73).  Where all of
// x is that small they are all formed again, in 3.8 ms.  Results in float32's subnormal range are good to a unit of 2^-149 per value of k.
// Every wait is bounded: on expiry the kernel records an error code and winds down.
#include "tc_common.cuh"

namespace {

constexpr int F_ROWS = 128;                      // features per tile
constexpr int W_STAGES = 3, X_STAGES = 2;
constexpr int W_BYTES = F_ROWS * BK * 4;         // two boxes of 128 rows x 128 bytes
constexpr int TERM_COLS = BK / 2;                // a term's columns in tensor memory: two k each

template <int BT>
struct F32Tile {
  static constexpr int X_TERM = BT * BK * 2, X_BYTES = 3 * X_TERM;
  static constexpr int SMEM = W_STAGES * W_BYTES + X_STAGES * X_BYTES + 1024 /* alignment */ + 256 /* barriers */;
  static constexpr int A_AT = 2 * BT, COLS_USED = A_AT + 2 * 3 * TERM_COLS;
  static constexpr int COLS = COLS_USED <= 256 ? 256 : 512;
  static constexpr bool BY_TERM = BT > 64;      // whether x's terms come and go one by one
  static constexpr int HALVES = BT >= 32 ? 2 : 1, PART = BT / HALVES;       // columns of an adding warp
  static_assert(COLS_USED <= 512 && PART % 16 == 0, "tensor memory");
};

// What the epilogue has to know of an operand's row: its largest magnitude, and whether the terms are short of some value's bits.
struct RowInfo { float largest; unsigned cut; };

// The three terms of x as [3][M][pitch] bfloat16, pitch = K rounded up to eight, and each row's RowInfo.  A CTA takes a row at a
// time, a thread eight values.
// Its successor, the product, fetches W before it waits for this kernel.  W may be the result of a kernel before this one, so that
// this kernel lets the product start only when what came before it is complete.
template <bool VEC>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, long ldx, int M, int K, int pitch, uint4* __restrict__ terms,
                                                         RowInfo* __restrict__ info) {
  __shared__ unsigned largest_of[8], cut_of[8];
  co_pdl_wait();
  co_pdl_launch_dependents();
  const int chunks = pitch / 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long n = (long)M * chunks;
  for (int m = blockIdx.x; m < M; m += gridDim.x) {
    unsigned largest = 0, cut = 0;
    for (int c = threadIdx.x; c < chunks; c += 256) {
      const int k = 8 * c;
      const float* p = x + m * ldx + k;
      float v[8];
      if (VEC && k + 8 <= K) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = k + j < K ? p[j] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) largest = max(largest, __float_as_uint(v[j]) & 0x7fffffffu);
      uint4 t[3];
      split3(v[0], v[1], t[0].x, t[1].x, t[2].x, cut);
      split3(v[2], v[3], t[0].y, t[1].y, t[2].y, cut);
      split3(v[4], v[5], t[0].z, t[1].z, t[2].z, cut);
      split3(v[6], v[7], t[0].w, t[1].w, t[2].w, cut);
#pragma unroll
      for (int j = 0; j < 3; ++j) terms[j * n + (long)m * chunks + c] = t[j];
    }
    largest = __reduce_max_sync(0xffffffffu, largest);
    cut = __reduce_or_sync(0xffffffffu, cut);
    if (lane == 0) { largest_of[warp] = largest; cut_of[warp] = cut; }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int w = 1; w < 8; ++w) { largest = max(largest, largest_of[w]); cut |= cut_of[w]; }
      info[m] = {__uint_as_float(largest), cut & 0xffffu};
    }
    __syncthreads();
  }
}

// A warp forms the products of the lanes in `bad` (lane l: feature n_first + l) with one row of x over [k0, k1) anew.
__device__ __noinline__ float sum_again(unsigned bad, const float* __restrict__ x, const float* __restrict__ w, int n_first, int K, int k0, int k1) {
  const int lane = threadIdx.x & 31;
  float mine = 0.f;
  while (bad) {
    const int l = __ffs(bad) - 1;
    bad &= bad - 1;
    const float* row = w + (size_t)(n_first + l) * K;
    float s = 0.f;
    for (int k = k0 + lane; k < k1; k += 32) s = fmaf(x[k], row[k], s);
    s = co_warp_sum(s);
    if (lane == l) mine = s;
  }
  return mine;
}

struct F32Args {
  const float* x; const float* w; const void* bias; float* out; float* apart;      // apart: [slice][M][N] (absent: one slice)
  int bias_dtype, M, N, K, per_slice;      // stages of 64 k per slice
  long ldx, ldo;
  const RowInfo* info;                     // of x's rows
  int* status;
};

// (Its successor starts at its end: launched ahead, the block of 512 tokens of 1536 x 8960 took 324 us in place of 316.)
template <int BT>
__global__ void __launch_bounds__(448, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const F32Args P) {
  using S = F32Tile<BT>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ RowInfo w_info[F_ROWS];                    // of W's rows, as far as this CTA's k go
  unsigned char* ws = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* xs = ws + W_STAGES * W_BYTES;
  unsigned long long* w_full = (unsigned long long*)(xs + X_STAGES * S::X_BYTES);
  unsigned long long* w_free = w_full + W_STAGES;
  unsigned long long* x_full = w_free + W_STAGES;       // [stage][term]
  unsigned long long* x_free = x_full + 2 * 3;          // [stage][term]; of term 0: all products are formed, W's terms are free and the sums stand
  unsigned long long* a_full = x_free + 2 * 3;          // W's terms stand in tensor memory
  unsigned long long* acc_free = a_full + 2;            // the sums have been read
  unsigned* tmem_slot = (unsigned*)(acc_free + 2);
  static_assert((2 * W_STAGES + 16) * 8 + 4 <= 256, "barriers fit their slot");
  constexpr int INFO_THREADS = 128 + 128 * S::HALVES;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * F_ROWS, m0 = blockIdx.y * BT;
  const int first = blockIdx.z * P.per_slice;
  const int stages = min(P.per_slice, (P.K + BK - 1) / BK - first);

  if (threadIdx.x == 0) {
    for (int s = 0; s < W_STAGES; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_free[s], 4); }
    for (int s = 0; s < 6; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_free[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&a_full[s], 4); mbar_init(&acc_free[s], 4 * S::HALVES); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(S::COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      auto fetch_w = [&](int kt) {
        const int s = kt % W_STAGES;
        unsigned char* to = ws + s * W_BYTES;
        mbar_expect_tx(&w_full[s], W_BYTES);      // (the map counts in halves of a float)
        tma_load_2d(to, &map_w, (first + kt) * 2 * BK, n0, &w_full[s]);
        tma_load_2d(to + W_BYTES / 2, &map_w, (first + kt) * 2 * BK + BK, n0, &w_full[s]);
      };
      for (int kt = 0; kt < W_STAGES && kt < stages; ++kt) fetch_w(kt);
      co_pdl_wait();
      for (int kt = 0; kt < stages; ++kt) {
        const int b = kt & 1;
        bool ok = true;
        for (int t = 2; t >= 0 && ok; --t) {      // in the order in which the products let go of them
          const int at = 3 * b + (S::BY_TERM ? t : 0);
          if (S::BY_TERM || t == 2) {
            ok = kt < 2 || mbar_wait(&x_free[at], ((kt >> 1) - 1) & 1);
            if (!ok) break;
            mbar_expect_tx(&x_full[at], S::BY_TERM ? S::X_TERM : S::X_BYTES);
          }
          tma_load_3d(xs + b * S::X_BYTES + t * S::X_TERM, &map_x, (first + kt) * BK, m0, t, &x_full[at]);
        }
        if (!ok) { atomicExch(P.status, 11); break; }
        const int next = kt + W_STAGES - 1;       // freed when stage kt - 1 was split
        if (kt >= 1 && next < stages) {
          if (!mbar_wait(&w_free[next % W_STAGES], (next / W_STAGES - 1) & 1)) { atomicExch(P.status, 11); break; }
          fetch_w(next);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr unsigned idesc = umma_idesc(F_ROWS, BT);
      for (int kt = 0; kt < stages; ++kt) {
        const int b = kt & 1;
        bool ok = mbar_wait(&a_full[b], (kt >> 1) & 1) && (kt < 2 || mbar_wait(&acc_free[b], ((kt >> 1) - 1) & 1));
        const unsigned acc = tmem + b * BT, terms = tmem + S::A_AT + b * 3 * TERM_COLS;
        const unsigned char* x = xs + b * S::X_BYTES;
        // small products before large ones as far as x2 and x1 can be let go early: what fetches them again takes as long as a stage's products
        constexpr int XT[6] = {2, 1, 1, 0, 0, 0}, WT[6] = {0, 1, 0, 2, 1, 0};
#pragma unroll
        for (int p = 0; p < 6; ++p) {
          if (p == 0 || (S::BY_TERM && XT[p] != XT[p - 1])) {
            ok = ok && mbar_wait(&x_full[3 * b + (S::BY_TERM ? XT[p] : 0)], (kt >> 1) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          const unsigned long long db = umma_desc(x + XT[p] * S::X_TERM);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_a_tmem(acc, terms + WT[p] * TERM_COLS + k * (UMMA_K / 2), db + 2 * k, idesc, (p | k) != 0);
          if (p == 5 || (S::BY_TERM && XT[p] != XT[p + 1])) umma_commit(&x_free[3 * b + XT[p]]);
        }
        if (!ok) { atomicExch(P.status, 12); break; }
      }
    }
  } else if (warp < 6) {
    const int quarter = warp & 3, row = quarter * 32 + lane;
    unsigned cut = 0;
    float largest = 0.f;
    for (int kt = 0; kt < stages; ++kt) {
      const int s = kt % W_STAGES, b = kt & 1;
      bool ok = mbar_wait(&w_full[s], (kt / W_STAGES) & 1);
      const unsigned char* from = ws + s * W_BYTES + row * 128;
      unsigned t0[32], t1[32], t2[32];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(from + h * (W_BYTES / 2) + ((c ^ (row & 7)) << 4));
          const int at = h * 16 + 2 * c;
          split3(v.x, v.y, t0[at], t1[at], t2[at], cut);
          split3(v.z, v.w, t0[at + 1], t1[at + 1], t2[at + 1], cut);
          largest = fmaxf(fmaxf(largest, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
        }
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_free[s]);
      if (kt >= 2) ok = ok && mbar_wait(&x_free[3 * b], ((kt >> 1) - 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { if (lane == 0) atomicExch(P.status, 14); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned to = tmem + ((unsigned)(quarter * 32) << 16) + S::A_AT + b * 3 * TERM_COLS;
      tmem_st32(to, t0);
      tmem_st32(to + TERM_COLS, t1);
      tmem_st32(to + 2 * TERM_COLS, t2);
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[b]);
    }
    w_info[row] = {largest, cut & 0xffffu};
    asm volatile("bar.arrive 1, %0;" ::"n"(INFO_THREADS) : "memory");
  } else if (warp < 6 + 4 * S::HALVES) {
    const int quarter = warp & 3, half = (warp - 6) >> 2;
    const int n_first = n0 + quarter * 32, n = n_first + lane, c0 = half * S::PART;
    float sum[S::PART];
#pragma unroll
    for (int j = 0; j < S::PART; ++j) sum[j] = 0.f;
    bool ok = true;
    co_pdl_wait();      // whether a row of x in this warp's columns was cut (and before the results are written: the predecessor may read there)
    unsigned x_cut = 0, x_largest = 0;
    for (int j = lane; j < S::PART && m0 + c0 + j < P.M; j += 32) {
      const RowInfo x = P.info[m0 + c0 + j];
      x_cut |= x.cut;
      x_largest = max(x_largest, __float_as_uint(x.largest));
    }
    x_cut = __any_sync(0xffffffffu, x_cut != 0);
    x_largest = __reduce_max_sync(0xffffffffu, x_largest);
    for (int kt = 0; kt < stages; ++kt) {
      const int b = kt & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&x_free[3 * b], (kt >> 1) & 1));
      if (!ok) { if (lane == 0) atomicExch(P.status, 13); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned from = tmem + ((unsigned)(quarter * 32) << 16) + b * BT + c0;
#pragma unroll
      for (int c = 0; c < S::PART; c += 16) {
        unsigned r[16];
        tmem_ld16(from + c, r);
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(r[j]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_free[b]);
    }
    asm volatile("bar.sync 1, %0;" ::"n"(INFO_THREADS) : "memory");      // W's rows have been looked at
    if (ok) {
      const int k0 = first * BK, k1 = min(P.K, (first + stages) * BK);
      const float bias = n < P.N && P.bias && !P.apart ? co_load_any(P.bias, P.bias_dtype, n) : 0.f;
      float* to = P.apart ? P.apart + ((size_t)blockIdx.z * P.M) * P.N + n : P.out + n;
      const long ld = P.apart ? P.N : P.ldo;
      // (few instructions per column: code that runs once comes from memory, and at ten times the length it took as long as the products)
      const int rows = min(S::PART, P.M - m0 - c0);
      float* at = to + (long)(m0 + c0) * ld;
      unsigned largest = 0, smallest = 0x7fffffffu;
#pragma unroll
      for (int j = 0; j < S::PART; ++j) {
        const unsigned size = __float_as_uint(sum[j]) & 0x7fffffffu;
        largest = max(largest, size);
        if (j < rows) smallest = min(smallest, size);
        if (j < rows && n < P.N) at[j * ld] = sum[j] + bias;
      }
      // less than 2^-133 of every value that was cut, times the other operand: a result of 2^25 times that is right to its last bit
      const RowInfo w = w_info[quarter * 32 + lane];
      const float unit = (float)(k1 - k0) * 0x1p-108f;
      const float most = unit * ((x_cut ? w.largest : 0.f) + (w.cut ? __uint_as_float(x_largest) : 0.f));
      if (__any_sync(0xffffffffu, n < P.N && (largest >= 0x7f800000u || __uint_as_float(smallest) < most))) {
        unsigned again[(S::PART + 31) / 32] = {};
#pragma unroll
        for (int j = 0; j < S::PART; ++j)
          if (j < rows) {
            const RowInfo x = P.info[m0 + c0 + j];
            const float least = unit * ((x.cut ? w.largest : 0.f) + (w.cut ? x.largest : 0.f)), size = fabsf(sum[j]);
            if (n < P.N && (!(size < INFINITY) || size < least)) again[j / 32] |= 1u << (j % 32);
          }
#pragma unroll 1
        for (int j = 0; j < rows; ++j) {
          unsigned word = again[0];
#pragma unroll
          for (int i = 1; i < (S::PART + 31) / 32; ++i) word = j / 32 == i ? again[i] : word;
          const unsigned bad = __ballot_sync(0xffffffffu, word >> (j % 32) & 1);
          if (!bad) continue;
          const float y = sum_again(bad, P.x + (m0 + c0 + j) * P.ldx, P.w, n_first, P.K, k0, k1);
          if (bad >> lane & 1) at[j * ld] = y + bias;
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(S::COLS) : "memory");
  }
}

// The slices' sums, added in order, with what the product's own epilogue does; a thread takes four columns where N allows.
template <int V>
__global__ void __launch_bounds__(256)
add_slices_kernel(const float* __restrict__ apart, int slices, const void* __restrict__ bias, int bias_dtype, float* __restrict__ out,
                  int M, int N, long ldo, int act) {
  co_pdl_launch_dependents();
  co_pdl_wait();
  const size_t size = (size_t)M * N, e = ((size_t)blockIdx.x * 256 + threadIdx.x) * V;
  if (e >= size) return;
  float v[V];
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = 0.f;
#pragma unroll 4
  for (int s = 0; s < slices; ++s) {
    float t[V];
    if (V == 4) *reinterpret_cast<float4*>(t) = *reinterpret_cast<const float4*>(apart + s * size + e);
    else t[0] = apart[s * size + e];
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] += t[i];
  }
  const size_t m = e / N;
  const int n = (int)(e - m * N);
#pragma unroll
  for (int i = 0; i < V; ++i) {
    float y = v[i];
    if (bias) y += co_load_any(bias, bias_dtype, n + i);
    out[m * ldo + n + i] = act ? co_gelu(y) : y;
  }
}

// Slices of K: about one CTA per SM at few rows, at least four stages each; a function of the weight's shape alone.  Measured on a B200 (us
// at 1, 313 and 2,048 rows, back to back): 1536 x 8960 for 100, 148 (here), 220 and 296 CTAs 28 / 78 / 399, 22 / 64 / 404, 29 / 74 / 486 and
// 26 / 84 / 541; 1024 x 1024 with at least two, four (here) and eight stages 8.4 / 15 / 84, 9.9 / 17 / 50 and 14 / 23 / 47.
int slices_of(int N, int K) {
  const int tiles = (N + F_ROWS - 1) / F_ROWS, k_tiles = (K + BK - 1) / BK;
  int s = (148 + tiles / 2) / tiles;
  if (s > k_tiles / 4) s = k_tiles / 4;
  if (s < 2) return 1;
  const int per = (k_tiles + s - 1) / s;
  return (k_tiles + per - 1) / per;
}
int pitch_of(int K) { return (K + 7) / 8 * 8; }
constexpr int BT_MOST = 160;
// Rows that are worked on at a time: their terms (6 bytes a value) and, where there are any, their slices' sums take 128 MB at most (the
// slices' sums then about stay in L2, where the adding kernel finds them), one tile of rows at least.  Measured on a B200 with 32, 64 and
// 128 MB: 2048 x 4096 x 4096 (five slices) 751, 530 and 453 us, 2048 x 1536 x 8960 (twelve) 454, 404 and 400.
int rows_at_once(int M, int N, int K, int act) {
  const int slices = slices_of(N, K);
  const double each = 6.0 * pitch_of(K) + 8.0 + (slices > 1 || act ? 4.0 * slices * N : 0.0);
  const double rows = floor((double)(128 << 20) / each / BT_MOST) * BT_MOST;
  return rows < BT_MOST ? (M < BT_MOST ? M : BT_MOST) : (rows < M ? (int)rows : M);
}
long terms_floats(long rows, int K) { return (3 * rows * pitch_of(K) / 2 + 2 * rows + 63) / 64 * 64; }      // and the rows' RowInfo

template <int BT>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const F32Args& P, int slices, cudaStream_t stream) {
  auto kernel = gemm_f32_tc_kernel<BT>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Tile<BT>::SMEM);
  if (e != cudaSuccess) CO_FAIL("gemm_f32_tc: %d bytes of shared memory: %s", F32Tile<BT>::SMEM, cudaGetErrorString(e));
  e = co_launch(kernel, dim3((P.N + F_ROWS - 1) / F_ROWS, (P.M + BT - 1) / BT, slices), dim3(448), F32Tile<BT>::SMEM, stream, mw, mx, P);
  if (e != cudaSuccess) CO_FAIL("gemm_f32_tc: launch failed: %s", cudaGetErrorString(e));
  CO_CHECK_LAUNCH("gemm_f32_tc");
  return 0;
}
}  // namespace

// Whether the kernel takes a weight of this shape: rows of 16-byte multiples, a tile of 128 features and a few stages of 64 k.
CO_EXPORT int coheryn_gemm_f32_tc_takes(int N, int K) { return N >= 128 && K >= 256 && K % 4 == 0; }
// Whether it is the faster one for this weight, whatever the rows (a function of the shape alone, so that all rows of a product go the
// same way).  Its two or three launches and its start lie against one or two launches of the FMA kernel.  Measured on a B200 from 1 to 1,500
// rows, back to back, this one's us and the FMA kernel's: 128 x 256 one row 8.4 and 8.4, 313 rows 14 and 9.1; 256 x 448 9 to 11 against 14 up
// to 64 rows, then 18 against 14 at 313; 1024 x 256 12 and 9.1 at 128 rows, 16 and 36 at 1,500; 4096 x 256 8.4 and 8.7 at one row, 12 and 24
// at 128; 128 x 512 9.7 and 15 at one row, 16 and 16 at 700, 192 x 512 the same; from there on it is ahead everywhere.
CO_EXPORT int coheryn_gemm_f32_tc_pays(int N, int K) { return coheryn_gemm_f32_tc_takes(N, K) && (K >= 512 || N >= 4096); }

// Floats of workspace (16-byte aligned) that a product with this activation needs.
CO_EXPORT long coheryn_gemm_f32_tc_workspace_floats(int M, int N, int K, int act) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int rows = rows_at_once(M, N, K, act), slices = slices_of(N, K);
  return terms_floats(rows, K) + (slices > 1 || act ? (long)slices * rows * N : 0);
}

// x: [M, K] with row stride ldx; w: [N, K] contiguous, 16-byte aligned; out: [M, N] with row stride ldo; all float32.
// act 0: the (biased) product; CO_ACT_GELU: its exact GELU.  status: device word that receives 11..14 if a bounded wait ran out.
CO_EXPORT int coheryn_gemm_f32_tc(const float* x, const float* w, const void* bias, int bias_dtype, float* out, int M, int N, int K,
                                  long ldx, long ldo, int act, int* status, float* workspace, long floats, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (!coheryn_gemm_f32_tc_takes(N, K)) CO_FAIL("gemm_f32_tc: a weight of %d x %d is not taken", N, K);
  if (act != 0 && act != CO_ACT_GELU) CO_FAIL("gemm_f32_tc: unknown activation %d", act);
  if (((uintptr_t)w & 15) || ((uintptr_t)workspace & 15)) CO_FAIL("gemm_f32_tc: the weight and the workspace must be 16-byte aligned");
  if (!workspace || floats < coheryn_gemm_f32_tc_workspace_floats(M, N, K, act)) CO_FAIL("gemm_f32_tc: the workspace of %ld floats is too small", floats);
  const int slices = slices_of(N, K), pitch = pitch_of(K), most = rows_at_once(M, N, K, act);
  const bool apart = slices > 1 || act != 0;      // what follows the sums is the adding kernel's
  CUtensorMap mw, mx;
  if (!make_map(&mw, w, N, 2L * K, 2L * K, F_ROWS)) CO_FAIL("gemm_f32_tc: cuTensorMapEncodeTiled failed (N=%d K=%d)", N, K);
  for (int m = 0; m < M; m += most, x += (size_t)most * ldx, out += (size_t)most * ldo) {
    const int rows = M - m < most ? M - m : most;
    // tiles of tokens as even as tiles of at most 160 allow
    const int tiles = (rows + BT_MOST - 1) / BT_MOST, each = (rows + tiles - 1) / tiles;
    const int bt = each <= 16 ? 16 : each <= 32 ? 32 : (each + 31) / 32 * 32;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 3}, strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)pitch * 2 * rows};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)bt, 1};
    if (!make_map_nd(&mx, workspace, 3, dims, strides, box)) CO_FAIL("gemm_f32_tc: cuTensorMapEncodeTiled failed (M=%d K=%d)", rows, K);
    const long chunks = (long)rows * (pitch / 8);
    RowInfo* info = reinterpret_cast<RowInfo*>((uint4*)workspace + 3 * chunks);
    const bool vec = ldx % 4 == 0 && !((uintptr_t)x & 15);
    co_launch(vec ? split_rows_kernel<true> : split_rows_kernel<false>, dim3(rows < 148 * 8 ? rows : 148 * 8), dim3(256), 0, stream, x, ldx, rows, K, pitch,
              (uint4*)workspace, info);
    CO_CHECK_LAUNCH("split_rows");
    const F32Args P = {x, w, bias, out, apart ? workspace + terms_floats(most, K) : nullptr, bias_dtype, rows, N, K,
                       ((K + BK - 1) / BK + slices - 1) / slices, ldx, ldo, info, status};
    const int rc = bt == 16 ? launch<16>(mw, mx, P, slices, stream) : bt == 32 ? launch<32>(mw, mx, P, slices, stream)
                 : bt == 64 ? launch<64>(mw, mx, P, slices, stream) : bt == 96 ? launch<96>(mw, mx, P, slices, stream)
                 : bt == 128 ? launch<128>(mw, mx, P, slices, stream) : launch<160>(mw, mx, P, slices, stream);
    if (rc) return rc;
    if (apart) {
      const bool four = N % 4 == 0;
      const size_t n = (size_t)rows * N / (four ? 4 : 1);
      co_launch(four ? add_slices_kernel<4> : add_slices_kernel<1>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, P.apart, slices, bias,
                bias_dtype, out, rows, N, ldo, act);
      CO_CHECK_LAUNCH("add_slices");
    }
  }
  return 0;
}
