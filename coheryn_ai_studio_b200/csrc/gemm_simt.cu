// out[M, N] = x[M, K] . W[N, K]^T (+ bias[N]) with float32 FMA accumulation on the CUDA
// cores: the matrix product of the true 32-bit path where a weight is small, unaligned or of
// another type (else gemm_f32_tc.cu), and the any-shape reference for the tensor-core kernels.
//
// An output element is the sum, in ascending order, of the sums over stretches of values of k, each of them accumulated in
// ascending order from zero.  The length of a stretch follows from the weight's shape; neither the tile of a launch nor
// whether the stretches are shared out over CTAs changes the order, so a row's result does not depend on the other rows of
// the batch.
//
// What bounds it: the FMA pipes (148 SMs x 128 a cycle).  A thread holds 8 x 8 outputs, so that a step of k costs it four
// 16-byte loads from shared memory for 64 multiply-adds, issued as pairs (fma.rn.f32x2: the same roundings, half the
// instructions); the tiles of the next 16 values of k are fetched into registers while the present ones are used.
// Measured on a B200 (float32, alone, L2 flushed; before: 64 x 64 tiles, 4 x 4 per thread, one buffer): 313 x 17920 x 1536
// 697 -> 417 us (41 TFLOP/s of 74), 2048 rows 3,593 -> 2,336 us, 313 x 1536 x 8960 830 -> 210 us, one row by 17920 x 1536
// 183 -> 84 us, one row by 1536 x 8960 955 -> 44 us; warm, 64 x 256 x 128 10.9 -> 5.9 us.
#include "common.cuh"

namespace {

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long both(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 halves(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// Four neighbouring values of a row from k on, zero from K on.
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T* row, int k, int K) {
  if (VEC) {
    if (k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (sizeof(T) == 4) return *reinterpret_cast<const float4*>(row + k);
    const uint2 u = *reinterpret_cast<const uint2*>(row + k);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
    return make_float4(__bfloat162float(a.x), __bfloat162float(a.y), __bfloat162float(b.x), __bfloat162float(b.y));
  }
  return make_float4(k < K ? co_to_float(row[k]) : 0.f, k + 1 < K ? co_to_float(row[k + 1]) : 0.f,
                     k + 2 < K ? co_to_float(row[k + 2]) : 0.f, k + 3 < K ? co_to_float(row[k + 3]) : 0.f);
}

template <typename TO>
__device__ __forceinline__ void store_out(TO* out, size_t at, float v, const void* bias, int bias_dtype, int n, int act) {
  if (bias) v += co_load_any(bias, bias_dtype, n);
  if (act) v = co_gelu(v);
  out[at] = co_from_float<TO>(v);
}

// BM x BN outputs per CTA, TM x TN per thread (rows and columns in groups of four, the groups apart).  `apart` (when the
// stretches of k are shared out): [stretch][M][N], blockIdx.z's own sum; else out.  MULTI: a CTA takes several stretches and
// holds their sum beside the present one's, which costs a third CTA per SM (62 % of the FMA pipes' cycles in use, waiting for
// shared memory with two warps per scheduler).
template <typename TX, typename TW, typename TO, int BM, int BN, int BK, int TM, int TN, bool VEC, bool MULTI>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MULTI ? 2 : 3)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, const void* __restrict__ bias, int bias_dtype, TO* __restrict__ out,
                 float* __restrict__ apart, int M, int N, int K, long ldx, long ldo, int act, int stretch, int n_split,
                 int k_split) {
  constexpr int THREADS = (BM / TM) * (BN / TN), PM = BM + 4, PN = BN + 4, XV = BM * BK / 4;
  constexpr int XL = (XV + THREADS - 1) / THREADS, WL = BN * BK / 4 / THREADS;      // 16-byte vectors of a tile per thread
  static_assert(WL * THREADS * 4 == BN * BK && TM % 4 == 0 && TN % 4 == 0, "whole vectors per thread");
  __shared__ __align__(16) float xs[2][BK][PM];
  __shared__ __align__(16) float ws[2][BK][PN];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / (BN / TN)) * 4, tn = (tid % (BN / TN)) * 4;
  // (a block-diagonal weight: a tile on one side of n_split reads its own columns of x alone)
  const int k_from = apart ? blockIdx.z * stretch : (n_split > 0 && n0 >= n_split ? k_split : 0);
  const int k_to = apart ? min(K, k_from + stretch) : (n0 + BN <= n_split ? k_split : K);
  float4 xr[XL], wr[WL];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < XL; ++e) {
      const int idx = tid + e * THREADS, r = idx / (BK / 4), c = 4 * (idx % (BK / 4));
      if (XV % THREADS && idx >= XV) break;
      xr[e] = m0 + r < M ? load4<TX, VEC>(x + (size_t)(m0 + r) * ldx, k0 + c, k_to) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int e = 0; e < WL; ++e) {
      const int idx = tid + e * THREADS, r = idx / (BK / 4), c = 4 * (idx % (BK / 4));
      wr[e] = n0 + r < N ? load4<TW, VEC>(w + (size_t)(n0 + r) * K, k0 + c, k_to) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto keep = [&](int b) {
#pragma unroll
    for (int e = 0; e < XL; ++e) {
      const int idx = tid + e * THREADS, r = idx / (BK / 4), c = 4 * (idx % (BK / 4));
      if (XV % THREADS && idx >= XV) break;
      xs[b][c][r] = xr[e].x; xs[b][c + 1][r] = xr[e].y; xs[b][c + 2][r] = xr[e].z; xs[b][c + 3][r] = xr[e].w;
    }
#pragma unroll
    for (int e = 0; e < WL; ++e) {
      const int idx = tid + e * THREADS, r = idx / (BK / 4), c = 4 * (idx % (BK / 4));
      ws[b][c][r] = wr[e].x; ws[b][c + 1][r] = wr[e].y; ws[b][c + 2][r] = wr[e].z; ws[b][c + 3][r] = wr[e].w;
    }
  };
  unsigned long long acc[TM][TN / 2];
  float total[MULTI ? TM : 1][MULTI ? TN : 1];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      if (MULTI) total[i][j] = 0.f;
      acc[i][j / 2] = 0ull;
    }
  fetch(k_from);
  keep(0);
  __syncthreads();
  int b = 0;
  for (int k0 = k_from; k0 < k_to; k0 += BK, b ^= 1) {
    if (k0 + BK < k_to) fetch(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
      unsigned long long v[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 t = *reinterpret_cast<const float4*>(&xs[b][kk][tm + (i / 4) * (BM / (TM / 4))]);
        a[i] = t.x; a[i + 1] = t.y; a[i + 2] = t.z; a[i + 3] = t.w;
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&ws[b][kk][tn + (j / 4) * (BN / (TN / 4))]);
        v[j / 2] = t.x; v[j / 2 + 1] = t.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const unsigned long long aa = both(a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, v[j]);
      }
    }
    if (MULTI && ((k0 + BK) % stretch == 0 || k0 + BK >= k_to)) {      // the end of a stretch
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; j += 2) {
          const float2 t = halves(acc[i][j / 2]);
          total[i][j] += t.x; total[i][j + 1] += t.y;
          acc[i][j / 2] = 0ull;
        }
    }
    if (k0 + BK < k_to) {
      keep(b ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + tm + (i / 4) * (BM / (TM / 4)) + (i & 3);
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tn + (j / 4) * (BN / (TN / 4)) + (j & 3);
      if (gn >= N) continue;
      const float2 t = halves(acc[i][j / 2]);
      const float v = MULTI ? total[i][j] : 0.f + ((j & 1) ? t.y : t.x);
      if (apart) apart[((size_t)blockIdx.z * M + gm) * N + gn] = v;
      else store_out(out, (size_t)gm * ldo + gn, v, bias, bias_dtype, gn, act);
    }
  }
}

// The sums of the stretches of k, added in order, with what the product's own epilogue does.
template <typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_add_kernel(const float* __restrict__ apart, int stretches, const void* __restrict__ bias, int bias_dtype, TO* __restrict__ out,
                     int M, int N, long ldo, int act) {
  const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x, size = (size_t)M * N;
  if (e >= size) return;
  float v = 0.f;
#pragma unroll 4
  for (int s = 0; s < stretches; ++s) v += apart[s * size + e];
  const size_t m = e / N;
  const int n = (int)(e - m * N);
  store_out(out, m * ldo + n, v, bias, bias_dtype, n, act);
}

// Values of k per stretch: a wide weight makes tiles enough for the chip by itself and keeps long stretches (one CTA then
// needs no second set of sums up to k = 2048); a narrow one is cut finely, so that few rows still fill the chip.
int stretch_of(int N) { return N >= 4096 ? 2048 : 512; }

// Tiles: 64 x 128 (128 threads; 128 x 128 would leave more of the last tile idle), or 16 x 64 with 64 values of k at a time (16 KB of
// the weight per CTA), for a decode step, which is bound by the weight's stream, and where a product is so small that the large
// tiles leave most SMs idle and each CTA's chain of k is what takes the time: up to about three small tiles per SM, a few more
// when the sums are short.  Measured on a B200 with the large tiles and with the small ones: 17 x 3584 x 512 (112 small tiles) 38.0 and
// 16.7 us, 65 x 1536 x 1536 (360) 42 and 36, 130 x 3584 x 512 (504) 42 and 41, 130 x 1536 x 1536 (648) 42 and 63, 2048 x 64 x 64 (128)
// 10.7 and 4.4, 2048 x 256 x 128 (512) 15.9 and 12.3.  Sums of at most 32 values take 16 of k at a time (64 x 16 x 16: 4.1 and 3.1 us).
struct Plan { bool few; int rows, columns, apart; };      // tile; into how many CTAs the stretches of k go
Plan plan_of(int M, int N, int K) {
  const int n = (K + stretch_of(N) - 1) / stretch_of(N);
  const long small = (long)((N + 63) / 64) * ((M + 15) / 16) * n;
  Plan p;
  p.few = M <= 16 || small <= (K <= 128 ? 592 : 480);
  p.rows = p.few ? 16 : 64;
  p.columns = p.few ? 64 : 128;
  // one CTA each when the tiles alone would leave SMs idle, else one CTA for all
  const long tiles = (long)((N + p.columns - 1) / p.columns) * ((M + p.rows - 1) / p.rows);
  p.apart = n > 1 && tiles < 2 * 148 ? n : 1;
  return p;
}

// The sums of the stretches wait in a workspace of [stretch][row][column]: 64 MB at most (it stays in L2, where the adding kernel
// finds it), so a product of many rows by a long k goes in blocks of that many rows, one after the other; one row tile at least,
// whose sums are an eighth of the weight's own (float32) bytes.  640 x 3584 x 18944 (37 stretches) would take 339 MB at once.
int rows_at_once(int apart, int N) {
  const long rows = (1L << 24) / ((long)apart * N) / 64 * 64;
  return rows < 64 ? 64 : (int)(rows < (1L << 30) ? rows : 1L << 30);
}
long workspace_floats(int M, int N, int apart) {
  if (apart <= 1) return 0;
  const int rows = rows_at_once(apart, N);
  return (long)apart * (M < rows ? M : rows) * N;
}

template <typename TX, typename TW, typename TO>
int run(const TX* x, const TW* w, const void* bias, int bias_dtype, TO* out, int M, int N, int K, long ldx, long ldo, int act,
        float* workspace, long floats, int n_split, int k_split, cudaStream_t stream) {
  const bool vec = K % 4 == 0 && k_split % 4 == 0 && ldx % 4 == 0 && (uintptr_t)x % (4 * sizeof(TX)) == 0 && (uintptr_t)w % (4 * sizeof(TW)) == 0;
  const Plan p = plan_of(M, N, K);
  int n = p.apart;
  if (n > 1 || K > stretch_of(N)) n_split = 0;       // the stretches are those of a full row
  if (n > 1 && (!workspace || floats < workspace_floats(M, N, n))) n = 1;
  float* apart = n > 1 ? workspace : nullptr;
  const int stretch = stretch_of(N), most = n > 1 ? rows_at_once(n, N) : M;
  for (int m = 0; m < M; m += most, x += (size_t)most * ldx, out += (size_t)most * ldo) {
    const int rows = M - m < most ? M - m : most;
    const dim3 grid((N + p.columns - 1) / p.columns, (rows + p.rows - 1) / p.rows, n);
#define GO(BM, BN, BK, T, VEC, MULTI)                                                                                       \
  gemm_simt_kernel<TX, TW, TO, BM, BN, BK, T, T, VEC, MULTI><<<grid, (BM / T) * (BN / T), 0, stream>>>(                     \
      x, w, bias, bias_dtype, out, apart, rows, N, K, ldx, ldo, act, stretch, n_split, k_split)
#define BY_TILE(VEC, MULTI) if (p.few) GO(16, 64, 64, 4, VEC, MULTI); else GO(64, 128, 16, 8, VEC, MULTI)
    if (p.few && K <= 32) { if (vec) GO(16, 64, 16, 4, true, false); else GO(16, 64, 16, 4, false, false); }
    else if (n == 1 && K > stretch) { if (vec) { BY_TILE(true, true); } else { BY_TILE(false, true); } }
    else { if (vec) { BY_TILE(true, false); } else { BY_TILE(false, false); } }
#undef BY_TILE
#undef GO
    CO_CHECK_LAUNCH("gemm_simt");
    if (n > 1) {
      const size_t size = (size_t)rows * N;
      gemm_simt_add_kernel<TO><<<(unsigned)((size + 255) / 256), 256, 0, stream>>>(apart, n, bias, bias_dtype, out, rows, N, ldo, act);
      CO_CHECK_LAUNCH("gemm_simt_add");
    }
  }
  return 0;
}
}  // namespace

// The floats of workspace with which a product of this shape shares its stretches of k out over CTAs (0: it does not).
CO_EXPORT long coheryn_gemm_simt_workspace_floats(int M, int N, int K) {
  return M > 0 && N > 0 && K > 0 ? workspace_floats(M, N, plan_of(M, N, K).apart) : 0;
}

// How a product of this shape is laid out: rows and columns of a tile, CTAs that its stretches of k go to.
CO_EXPORT void coheryn_gemm_simt_plan(int M, int N, int K, int* rows, int* columns, int* apart) {
  const Plan p = plan_of(M, N, K);
  *rows = p.rows; *columns = p.columns; *apart = p.apart;
}

// x: [M, K] with row stride ldx; w: [N, K] contiguous; out: [M, N] with row stride ldo.
// act 0: the (biased) product; CO_ACT_GELU: its exact GELU.  workspace may be absent: one CTA then takes all of k.
// n_split > 0: w is block-diagonal, its first n_split rows are zero from k_split on and the others zero up to there; tiles on
// one side then leave the zeros out.
CO_EXPORT int coheryn_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, const void* bias,
                                int bias_dtype, void* out, int out_dtype, int M, int N, int K, long ldx,
                                long ldo, int act, float* workspace, long floats, int n_split, int k_split, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) CO_FAIL("gemm_simt: K must be positive");
  if (act != 0 && act != CO_ACT_GELU) CO_FAIL("gemm_simt: unknown activation %d", act);
  if (n_split < 0 || n_split > N || (n_split && (k_split <= 0 || k_split >= K))) CO_FAIL("gemm_simt: blocks of %d rows and %d columns", n_split, k_split);
#define RUN(TX, TW, TO) return run((const TX*)x, (const TW*)w, bias, bias_dtype, (TO*)out, M, N, K, ldx, ldo, act, workspace, floats, n_split, k_split, stream)
  if (x_dtype == CO_F32 && w_dtype == CO_F32 && out_dtype == CO_F32) RUN(float, float, float);
  if (x_dtype == CO_BF16 && w_dtype == CO_BF16 && out_dtype == CO_BF16) RUN(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
  if (x_dtype == CO_BF16 && w_dtype == CO_BF16 && out_dtype == CO_F32) RUN(__nv_bfloat16, __nv_bfloat16, float);
  if (x_dtype == CO_F32 && w_dtype == CO_BF16 && out_dtype == CO_F32) RUN(float, __nv_bfloat16, float);   // a float32 intermediate times a stored weight
#undef RUN
  CO_FAIL("gemm_simt: unsupported dtypes x=%d w=%d out=%d", x_dtype, w_dtype, out_dtype);
}
