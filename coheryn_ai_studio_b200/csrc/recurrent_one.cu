// The gated delta rule and the matrix memory for steps in which every request brings one token (decoding).
//
// What bounds such a step is the state, read and written once: 50 MB for 32 requests of 12 heads of 128 x 128.  The scans of recurrent.cu
// give neighbouring lanes the key channels of a column, which suits a chain of many tokens and reads a row's 512 bytes in pieces of 16
// from as many warps.  Here a warp takes whole rows of S: lane l holds the columns 4 l to 4 l + 3 (of every 128) of its warp's DK / SPLIT
// rows, so that loads and stores are 512 consecutive bytes, and the columns' sums are added across the warps through shared memory.
// Every product and sum is formed in the order of the scans (a part of the key channels by even and odd channels, the parts in the
// scans' tree), so a sequence has the same bits whichever kernel a step takes.  Measured on a B200 (32 requests, 12 heads of 128 x 128):
// 31.6 -> 19.6 us (delta rule); 8 heads of 128 x 256: 36.7 -> 22.5 us (matrix memory); one request of 12 heads: 11.4 -> 9.1.
#include "recurrent.cuh"

namespace {

// The sum over the parts in the order of the scans' shuffles: distance SPLIT / 2, .., 1.
template <int SPLIT>
__device__ __forceinline__ float parts_sum(const float* red, int pitch, int col) {
  float x[SPLIT];
#pragma unroll
  for (int p = 0; p < SPLIT; ++p) x[p] = red[p * pitch + col];
#pragma unroll
  for (int o = SPLIT / 2; o > 0; o >>= 1)
#pragma unroll
    for (int p = 0; p < o; ++p) x[p] += x[p + o];
  return x[0];
}

// A warp's rows of S: ROWS of them from d0 on, TILES times 128 columns.
template <int ROWS, int TILES>
__device__ __forceinline__ void rows_load(float4 (&S)[TILES][ROWS], const float* st, int d0, int dk, int dv) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int z = 0; z < TILES; ++z)
#pragma unroll
    for (int d = 0; d < ROWS; ++d)
      S[z][d] = d0 + d < dk && 128 * z + 4 * lane < dv ? *reinterpret_cast<const float4*>(st + (size_t)(d0 + d) * dv + 128 * z + 4 * lane)
                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
}
template <int ROWS, int TILES>
__device__ __forceinline__ void rows_store(const float4 (&S)[TILES][ROWS], float* st, int d0, int dk, int dv) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int z = 0; z < TILES; ++z)
#pragma unroll
    for (int d = 0; d < ROWS; ++d)
      if (d0 + d < dk && 128 * z + 4 * lane < dv) *reinterpret_cast<float4*>(st + (size_t)(d0 + d) * dv + 128 * z + 4 * lane) = S[z][d];
}
__device__ __forceinline__ void mad(float4& sum, const float4& s, float k) {
  sum.x = fmaf(s.x, k, sum.x); sum.y = fmaf(s.y, k, sum.y); sum.z = fmaf(s.z, k, sum.z); sum.w = fmaf(s.w, k, sum.w);
}
__device__ __forceinline__ float4 both(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// grid (requests, heads), SPLIT warps.
template <int DK, int SPLIT, int TILES>
__global__ void __launch_bounds__(32 * SPLIT, DK / SPLIT * TILES <= 8 ? 2 : 1) delta_one_kernel(DeltaIn P, HeadOut E) {
  constexpr int ROWS = DK / SPLIT, COLS = 128 * TILES, THREADS = 32 * SPLIT;
  __shared__ __align__(16) float qs[DK], ks[DK], gs[DK], red[SPLIT][COLS], us[COLS], os[COLS];
  co_pdl_launch_dependents();
  co_pdl_wait();
  const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d0 = warp * ROWS;
  const int dk = P.dk, dv = P.dv, start = P.cu_q[r], len = P.cu_q[r + 1] - start;
  if (len <= 0) return;
  const int g = h / (P.heads / P.kv_heads);
  float* state = P.state + (size_t)P.state_slots[r] * P.state_stride + (size_t)h * dk * dv;
  float4 S[TILES][ROWS];
  rows_load<ROWS, TILES>(S, state, d0, dk, dv);
  const float rate = expf(co_load_any(P.rate_log, P.rate_log_dtype, h));
  const float q_scale = 1.0f / sqrtf((float)dk);
  for (int i = 0; i < len; ++i) {
    const size_t row = (size_t)(start + i);
    for (int d = tid; d < DK; d += THREADS) {
      float qv = 0.f, kv = 0.f, gv = 1.f;
      if (d < dk) {
        qv = P.q[row * P.ld_qkv + (size_t)g * dk + d];
        kv = P.k[row * P.ld_qkv + (size_t)g * dk + d];
        const size_t sc = P.decay_channels == 1 ? (size_t)h : (size_t)h * dk + d;
        const float z = P.step[row * P.ld_step + sc] + co_load_any(P.step_bias, P.step_bias_dtype, sc);
        gv = expf(-rate * rc_softplus(z));
      }
      qs[d] = qv; ks[d] = kv; gs[d] = gv;
    }
    const float beta = rc_sigmoid(P.beta[row * P.ld_beta + h]);
    float v[(COLS + THREADS - 1) / THREADS];
#pragma unroll
    for (int j = 0; j < (COLS + THREADS - 1) / THREADS; ++j) {
      const int c = tid + j * THREADS;
      v[j] = c < dv ? P.v[row * P.ld_qkv + (size_t)h * dv + c] : 0.f;
    }
    __syncthreads();
    if (warp < 2) {           // q and k become unit vectors (q also divided by sqrt(dk))
      float* x = warp ? ks : qs;
      float ss = 0.f;
      for (int d = lane; d < DK; d += 32) ss = fmaf(x[d], x[d], ss);
      ss = co_warp_sum(ss);
      const float inv = (warp ? 1.0f : q_scale) / sqrtf(ss + 1e-6f);
      for (int d = lane; d < DK; d += 32) x[d] *= inv;
    }
    __syncthreads();
#pragma unroll
    for (int z = 0; z < TILES; ++z) {
      float4 even = make_float4(0.f, 0.f, 0.f, 0.f), odd = even;
#pragma unroll
      for (int d = 0; d < ROWS; ++d) {
        const float gg = gs[d0 + d];
        S[z][d].x *= gg; S[z][d].y *= gg; S[z][d].z *= gg; S[z][d].w *= gg;
        mad(d & 1 ? odd : even, S[z][d], ks[d0 + d]);
      }
      *reinterpret_cast<float4*>(&red[warp][128 * z + 4 * lane]) = both(even, odd);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < (COLS + THREADS - 1) / THREADS; ++j) {
      const int c = tid + j * THREADS;
      if (c < COLS) us[c] = beta * (v[j] - parts_sum<SPLIT>(red[0], COLS, c));
    }
    __syncthreads();
#pragma unroll
    for (int z = 0; z < TILES; ++z) {
      const float4 u = *reinterpret_cast<const float4*>(&us[128 * z + 4 * lane]);
      float4 even = make_float4(0.f, 0.f, 0.f, 0.f), odd = even;
#pragma unroll
      for (int d = 0; d < ROWS; ++d) {
        mad(S[z][d], u, ks[d0 + d]);
        mad(d & 1 ? odd : even, S[z][d], qs[d0 + d]);
      }
      *reinterpret_cast<float4*>(&red[warp][128 * z + 4 * lane]) = both(even, odd);
    }
    if (i + 1 == len) rows_store<ROWS, TILES>(S, state, d0, dk, dv);
    __syncthreads();
    for (int c = tid; c < COLS; c += THREADS) os[c] = parts_sum<SPLIT>(red[0], COLS, c);
    __syncthreads();
    head_out_chunk(E, os, COLS, dv, 1, start + i, h);
  }
}

// grid (requests, heads), SPLIT warps.
template <int DK, int SPLIT, int TILES>
__global__ void __launch_bounds__(32 * SPLIT, DK / SPLIT * TILES <= 8 ? 2 : 1) memory_one_kernel(MemoryIn P, HeadOut E) {
  constexpr int ROWS = DK / SPLIT, COLS = 128 * TILES, THREADS = 32 * SPLIT, NJ = (DK + 31) / 32;
  __shared__ __align__(16) float qs[DK], ks[DK], red[SPLIT][COLS], os[COLS], factors[3];      // a, b, the denominator
  co_pdl_launch_dependents();
  co_pdl_wait();
  const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d0 = warp * ROWS;
  const int dk = P.dk, dv = P.dv, start = P.cu_q[r], len = P.cu_q[r + 1] - start;
  if (len <= 0) return;
  float* slot = P.state + (size_t)P.state_slots[r] * P.state_stride;
  float* state = slot + (size_t)h * dk * dv;
  float* n_state = slot + (size_t)P.heads * dk * dv + (size_t)h * dk;
  float* m_state = slot + (size_t)P.heads * dk * dv + (size_t)P.heads * dk + h;
  float4 S[TILES][ROWS];
  rows_load<ROWS, TILES>(S, state, d0, dk, dv);
  float n[NJ], m = 0.f;      // warp 0: lane holds n[lane + 32 j]
  if (warp == 0) {
#pragma unroll
    for (int j = 0; j < NJ; ++j) n[j] = lane + 32 * j < dk ? n_state[lane + 32 * j] : 0.f;
    m = *m_state;
  }
  const float q_scale = 1.0f / sqrtf((float)dk);
  const float bi = co_load_any(P.bias_i, P.bias_dtype, h), bf = co_load_any(P.bias_f, P.bias_dtype, h);
  for (int i = 0; i < len; ++i) {
    const size_t row = (size_t)(start + i);
    for (int d = tid; d < DK; d += THREADS) {
      qs[d] = d < dk ? P.q[row * P.ld + (size_t)h * dk + d] * q_scale : 0.f;
      ks[d] = d < dk ? P.k[row * P.ld + (size_t)h * dk + d] : 0.f;
    }
    float4 v[TILES];
#pragma unroll
    for (int z = 0; z < TILES; ++z) {
      const float* from = P.v + row * P.ld + (size_t)h * dv + 128 * z + 4 * lane;
      v[z] = 128 * z + 4 * lane < dv ? make_float4(from[0], from[1], from[2], from[3]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    if (warp == 0) {
      const float in = P.cap * tanhf((P.gi[row * P.ld_gate + h] + bi) / P.cap);
      const float z = P.cap * tanhf((P.gf[row * P.ld_gate + h] + bf) / P.cap);
      const float f = -rc_softplus(-z);          // log sigmoid
      const float m_new = fmaxf(f + m, in);
      const float a = expf(f + m - m_new), b = expf(in - m_new);
      m = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int d = lane + 32 * j;
        if (d < DK) {
          n[j] = fmaf(b, ks[d], a * n[j]);
          sum = fmaf(n[j], qs[d], sum);
        }
      }
      sum = co_warp_sum(sum);
      if (lane == 0) { factors[0] = a; factors[1] = b; factors[2] = fmaxf(fabsf(sum), expf(-m)) + 1e-6f; }
    }
    __syncthreads();
    const float a = factors[0], b = factors[1];
#pragma unroll
    for (int z = 0; z < TILES; ++z) {
      const float4 bv = make_float4(b * v[z].x, b * v[z].y, b * v[z].z, b * v[z].w);
      float4 even = make_float4(0.f, 0.f, 0.f, 0.f), odd = even;
#pragma unroll
      for (int d = 0; d < ROWS; ++d) {
        const float k = ks[d0 + d];
        S[z][d].x = fmaf(bv.x, k, a * S[z][d].x); S[z][d].y = fmaf(bv.y, k, a * S[z][d].y);
        S[z][d].z = fmaf(bv.z, k, a * S[z][d].z); S[z][d].w = fmaf(bv.w, k, a * S[z][d].w);
        mad(d & 1 ? odd : even, S[z][d], qs[d0 + d]);
      }
      *reinterpret_cast<float4*>(&red[warp][128 * z + 4 * lane]) = both(even, odd);
    }
    if (i + 1 == len) rows_store<ROWS, TILES>(S, state, d0, dk, dv);
    __syncthreads();
    for (int c = tid; c < COLS; c += THREADS) os[c] = parts_sum<SPLIT>(red[0], COLS, c) / factors[2];
    __syncthreads();
    head_out_chunk(E, os, COLS, dv, 1, start + i, h);
  }
  if (warp == 0) {
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      if (lane + 32 * j < dk) n_state[lane + 32 * j] = n[j];
    if (lane == 0) *m_state = m;
  }
}

}  // namespace

// Whether the rows of S can be moved in vectors of four columns and a warp's rows fit its registers.
bool co_one_token_takes(int dk, int dv, const float* state, long stride) {
  return dv % 4 == 0 && stride % 4 == 0 && ((uintptr_t)state & 15) == 0 && (dk <= 128 || dv <= 128);
}

#define BY_TILES(KERNEL, D)                                                                                                                 \
  {                                                                                                                                        \
    constexpr int SP = scan_split(D);                                                                                                      \
    if (P.dv <= 128) co_launch(KERNEL<D, SP, 1>, dim3(B, P.heads), dim3(32 * SP), 0, stream, P, E);                                         \
    else co_launch(KERNEL<(D > 128 ? 128 : D), scan_split(D > 128 ? 128 : D), 2>, dim3(B, P.heads), dim3(32 * SP), 0, stream, P, E);        \
  }
int co_delta_one(const DeltaIn& P, const HeadOut& E, int B, cudaStream_t stream) {
  const int dk = P.dk;
#define LAUNCH(D) BY_TILES(delta_one_kernel, D)
  CO_SCAN_CASES(LAUNCH)
#undef LAUNCH
  CO_CHECK_LAUNCH("delta_one");
  return 0;
}
int co_memory_one(const MemoryIn& P, const HeadOut& E, int B, cudaStream_t stream) {
  const int dk = P.dk;
#define LAUNCH(D) BY_TILES(memory_one_kernel, D)
  CO_SCAN_CASES(LAUNCH)
#undef LAUNCH
  CO_CHECK_LAUNCH("memory_one");
  return 0;
}
