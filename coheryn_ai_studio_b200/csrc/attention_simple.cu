// Causal (optionally windowed) grouped-query attention over cache pages, float32
// arithmetic throughout.  It is the attention of the true 32-bit path and the any-shape
// reference of the bfloat16 tensor-core kernels.  A block takes a token and several query
// heads of a group (attention_group_kernel) or, for shapes that allow no vector loads, one
// head (attention_simple_kernel).
//
// For token t of request r at position p the keys are positions first..p of r's cache,
// first = max(0, p - window + 1) with a window, else 0; the cache already holds the
// keys that this step wrote.  The block's W warps (eight, or four for one head) each run an
// online softmax over the keys k = first + warp, first + warp + W, ...; their (max, sum,
// accumulator) triples are merged in warp order.  The result therefore depends only on (p, first), never on
// how the step was cut or batched.
//
// What bounds it: with a block per (token, query head), the reads of the same keys and values by every head of a group (1 KB a key and
// head), and a warp's chain per key (page number, loads, five shuffles, the exponentials).  Where head sizes and addresses allow
// 16-byte (bfloat16: 8-byte) loads, a block takes up to eight heads of a group, and each of eight warps (keys k = first + warp,
// first + warp + 8, ...) two of its keys at a time, whose chains run side by side; the maximum moves once for the two, and the page
// numbers are asked for a turn ahead.  A head's operations and their order do not depend on how many heads share a block.  Other
// shapes go key by key and head by head.  Measured on a B200 (float32, 12 heads of 128 over 2): 313 tokens 139 -> 76 us, 640 tokens 493 -> 218,
// one token over 1,000 keys 178 -> 47, 28 heads over 4 274 -> 140; four keys at a time: 94, 297 and 37 (157 registers, one block per SM).
//
// Options of other attention designs: values of another head size than keys (`hdv`); a score that
// loses slopes[h] * (p - key position) (a bias that grows with distance, one slope per query head);
// an output multiplied by a constant.
#include "common.cuh"

namespace {
constexpr int WARPS = 4;
constexpr int MAX_PER_LANE = 8;  // head sizes up to 256

// The warps' (maximum, sum, sums) merged in warp order into a row of the output.
template <typename T, int N>
__device__ __forceinline__ void merge_and_write(T* orow, const float* merge_acc, const float* merge_m, const float* merge_l, int hdv, float out_scale) {
  float M = -INFINITY;
#pragma unroll
  for (int w = 0; w < N; ++w) M = fmaxf(M, merge_m[w]);
  float L = 0.f;
  float f[N];
#pragma unroll
  for (int w = 0; w < N; ++w) {
    f[w] = merge_m[w] == -INFINITY ? 0.f : expf(merge_m[w] - M);
    L += merge_l[w] * f[w];
  }
  const float inv = 1.0f / L;
  for (int d = threadIdx.x; d < hdv; d += blockDim.x) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < N; ++w) o += merge_acc[w * hdv + d] * f[w];
    orow[d] = co_from_float<T>(o * inv * out_scale);
  }
}

template <typename T>
__global__ void __launch_bounds__(WARPS * 32)
attention_simple_kernel(const T* __restrict__ q, long q_stride, T* __restrict__ out, long out_stride,
                        const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                        const int* __restrict__ block_tables, int max_blocks,
                        const int* __restrict__ token_req, const int* __restrict__ positions, int nh,
                        int nkv, int hd, int hdv, int page_size, int window, float scale,
                        const float* __restrict__ slopes, float out_scale) {
  extern __shared__ float smem[];
  float* qs = smem;                         // [hd]
  float* merge_acc = smem + hd;             // [WARPS][hdv]
  __shared__ float merge_m[WARPS], merge_l[WARPS];

  const int t = blockIdx.x, h = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int req = token_req[t];
  const int pos = positions[t];
  const int first = window > 0 ? max(0, pos - window + 1) : 0;
  const int kvh = h / (nh / nkv);
  const int* table = block_tables + (size_t)req * max_blocks;

  const T* qrow = q + (size_t)t * q_stride + (size_t)h * hd;
  for (int d = threadIdx.x; d < hd; d += blockDim.x) qs[d] = co_to_float(qrow[d]);
  __syncthreads();

  const float slope = slopes ? slopes[h] : 0.f;
  float m = -INFINITY, l = 0.f;
  float acc[MAX_PER_LANE];
#pragma unroll
  for (int i = 0; i < MAX_PER_LANE; ++i) acc[i] = 0.f;

  for (int kp = first + warp; kp <= pos; kp += WARPS) {
    const int page = table[kp / page_size];
    const size_t row = ((size_t)page * nkv + kvh) * page_size + (kp % page_size);
    const T* kr = k_cache + row * hd;
    const T* vr = v_cache + row * hdv;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
      const int d = lane + 32 * i;
      if (d < hd) dot = fmaf(qs[d], co_to_float(kr[d]), dot);
    }
    dot = co_warp_sum(dot);
    const float s = dot * scale - slope * (float)(pos - kp);
    const float m_new = fmaxf(m, s);
    const float corr = expf(m - m_new);  // exp(-inf) = 0 on the first key
    const float p = expf(s - m_new);
    l = l * corr + p;
#pragma unroll
    for (int i = 0; i < MAX_PER_LANE; ++i) {
      const int d = lane + 32 * i;
      if (d < hdv) acc[i] = acc[i] * corr + p * co_to_float(vr[d]);
    }
    m = m_new;
  }
  if (lane == 0) { merge_m[warp] = m; merge_l[warp] = l; }
#pragma unroll
  for (int i = 0; i < MAX_PER_LANE; ++i) {
    const int d = lane + 32 * i;
    if (d < hdv) merge_acc[warp * hdv + d] = acc[i];
  }
  __syncthreads();
  merge_and_write<T, WARPS>(out + (size_t)t * out_stride + (size_t)h * hdv, merge_acc, merge_m, merge_l, hdv, out_scale);
}

// Four neighbouring values of a row.
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s)))); }
__device__ __forceinline__ float4 mad4(float f, float4 v, float4 a) {
  return make_float4(fmaf(f, v.x, a.x), fmaf(f, v.y, a.y), fmaf(f, v.z, a.z), fmaf(f, v.w, a.w));
}

// The same over the same keys, KEYS of a warp's at a time, for HEADS query heads of one kv head; a lane holds the channels 4 lane + 128 i of
// keys, values and outputs.  grid (tokens, heads / HEADS).
constexpr int KEYS = 2, GROUP_WARPS = 8;
template <typename T, int NV, int HEADS>
__global__ void __launch_bounds__(GROUP_WARPS * 32)
attention_group_kernel(const T* __restrict__ q, long q_stride, T* __restrict__ out, long out_stride,
                       const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                       const int* __restrict__ block_tables, int max_blocks,
                       const int* __restrict__ token_req, const int* __restrict__ positions, int nh,
                       int nkv, int hd, int hdv, int page_size, int window, float scale,
                       const float* __restrict__ slopes, float out_scale) {
  extern __shared__ __align__(16) float smem[];
  float* merge_acc = smem;                  // [HEADS][GROUP_WARPS][hdv]
  __shared__ float merge_m[HEADS][GROUP_WARPS], merge_l[HEADS][GROUP_WARPS];

  const int t = blockIdx.x, h0 = blockIdx.y * HEADS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pos = positions[t];
  const int first = window > 0 ? max(0, pos - window + 1) : 0;
  const int kvh = h0 / (nh / nkv);
  const int* table = block_tables + (size_t)token_req[t] * max_blocks;
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);

  float4 qs[HEADS][NV], acc[HEADS][NV];
  float slope[HEADS], m[HEADS], l[HEADS];
#pragma unroll
  for (int h = 0; h < HEADS; ++h) {
    const T* qrow = q + (size_t)t * q_stride + (size_t)(h0 + h) * hd;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int d = 4 * lane + 128 * i;
      qs[h][i] = d < hd ? make_float4(co_to_float(qrow[d]), co_to_float(qrow[d + 1]), co_to_float(qrow[d + 2]), co_to_float(qrow[d + 3])) : none;
      acc[h][i] = none;
    }
    slope[h] = slopes ? slopes[h0 + h] : 0.f;
    m[h] = -INFINITY;
    l[h] = 0.f;
  }
  int pages[KEYS];                          // of the keys of the next turn: asked for a turn ahead
  auto look_up = [&](int kp) {
#pragma unroll
    for (int u = 0; u < KEYS; ++u) pages[u] = kp + GROUP_WARPS * u <= pos ? table[(kp + GROUP_WARPS * u) / page_size] : 0;
  };
  look_up(first + warp);
  for (int kp = first + warp; kp <= pos; kp += GROUP_WARPS * KEYS) {
    float4 kk[KEYS][NV], vv[KEYS][NV];
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      const int key = kp + GROUP_WARPS * u;
      const size_t row = ((size_t)pages[u] * nkv + kvh) * page_size + (key % page_size);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int d = 4 * lane + 128 * i;
        kk[u][i] = key <= pos && d < hd ? load4(k_cache + row * hd + d) : none;
        vv[u][i] = key <= pos && d < hdv ? load4(v_cache + row * hdv + d) : none;
      }
    }
    look_up(kp + GROUP_WARPS * KEYS);
    float s[HEADS][KEYS];
#pragma unroll
    for (int h = 0; h < HEADS; ++h)
#pragma unroll
      for (int u = 0; u < KEYS; ++u) {
        s[h][u] = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) s[h][u] = dot4(qs[h][i], kk[u][i], s[h][u]);
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int h = 0; h < HEADS; ++h)
#pragma unroll
        for (int u = 0; u < KEYS; ++u) s[h][u] += __shfl_xor_sync(0xffffffffu, s[h][u], o);
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      float m_new = m[h];
#pragma unroll
      for (int u = 0; u < KEYS; ++u) {
        const int key = kp + GROUP_WARPS * u;
        s[h][u] = key <= pos ? s[h][u] * scale - slope[h] * (float)(pos - key) : -INFINITY;
        m_new = fmaxf(m_new, s[h][u]);
      }
      const float corr = expf(m[h] - m_new);  // exp(-inf) = 0 on the first keys
      l[h] *= corr;
#pragma unroll
      for (int i = 0; i < NV; ++i) acc[h][i] = make_float4(acc[h][i].x * corr, acc[h][i].y * corr, acc[h][i].z * corr, acc[h][i].w * corr);
#pragma unroll
      for (int u = 0; u < KEYS; ++u)
        if (kp + GROUP_WARPS * u <= pos) {
          const float p = expf(s[h][u] - m_new);
          l[h] += p;
#pragma unroll
          for (int i = 0; i < NV; ++i) acc[h][i] = mad4(p, vv[u][i], acc[h][i]);
        }
      m[h] = m_new;
    }
  }
#pragma unroll
  for (int h = 0; h < HEADS; ++h) {
    if (lane == 0) { merge_m[h][warp] = m[h]; merge_l[h][warp] = l[h]; }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int d = 4 * lane + 128 * i;
      if (d < hdv) *reinterpret_cast<float4*>(merge_acc + (h * GROUP_WARPS + warp) * hdv + d) = acc[h][i];
    }
  }
  __syncthreads();
  for (int h = 0; h < HEADS; ++h)
    merge_and_write<T, GROUP_WARPS>(out + (size_t)t * out_stride + (size_t)(h0 + h) * hdv, merge_acc + h * GROUP_WARPS * hdv, merge_m[h], merge_l[h], hdv, out_scale);
}
}  // namespace

CO_EXPORT int coheryn_attention_simple_ex(const void* q, long q_stride, void* out, long out_stride,
                                          const void* k_cache, const void* v_cache, int dtype,
                                          const int* block_tables, int max_blocks, const int* token_req,
                                          const int* positions, int T, int nh, int nkv, int hd, int hdv, int page_size,
                                          int window, float scale, const float* slopes, float out_scale,
                                          cudaStream_t stream) {
  if (T <= 0) return 0;
  if (hd > 32 * MAX_PER_LANE || hdv > 32 * MAX_PER_LANE || hd < 1 || hdv < 1)
    CO_FAIL("attention_simple: head sizes %d and %d must lie in 1..%d", hd, hdv, 32 * MAX_PER_LANE);
  if (nkv <= 0 || nh % nkv != 0) CO_FAIL("attention_simple: %d heads do not group over %d kv heads", nh, nkv);
  // query heads per block: the most, up to eight (with heads wider than 128: four), that divide a group and leave two blocks per SM: a
  // few decoded tokens want their heads side by side
  const int G = nh / nkv, most = hd <= 128 && hdv <= 128 ? 8 : 4;
  int heads = most;
  while (heads > 1 && (G % heads || (long)T * (nh / heads) < 2 * 148)) --heads;
#define ARGS(TY) (const TY*)q, q_stride, (TY*)out, out_stride, (const TY*)k_cache, (const TY*)v_cache, block_tables, max_blocks, token_req, \
                 positions, nh, nkv, hd, hdv, page_size, window, scale, slopes, out_scale
#define HEADS_CASE(TY, NV, N) \
  case N: attention_group_kernel<TY, NV, N><<<dim3(T, nh / N), GROUP_WARPS * 32, (size_t)N * GROUP_WARPS * hdv * sizeof(float), stream>>>(ARGS(TY)); break;
#define GO(TY)                                                                                                                  \
  if (hd % 4 == 0 && hdv % 4 == 0 && (uintptr_t)k_cache % (4 * sizeof(TY)) == 0 && (uintptr_t)v_cache % (4 * sizeof(TY)) == 0) { \
    if (most == 8) switch (heads) {                                                                                             \
      HEADS_CASE(TY, 1, 1) HEADS_CASE(TY, 1, 2) HEADS_CASE(TY, 1, 3) HEADS_CASE(TY, 1, 4)                                       \
      HEADS_CASE(TY, 1, 5) HEADS_CASE(TY, 1, 6) HEADS_CASE(TY, 1, 7) HEADS_CASE(TY, 1, 8)                                       \
    } else switch (heads) { HEADS_CASE(TY, 2, 1) HEADS_CASE(TY, 2, 2) HEADS_CASE(TY, 2, 3) HEADS_CASE(TY, 2, 4) }               \
  } else attention_simple_kernel<TY><<<dim3(T, nh), WARPS * 32, ((size_t)hd + (size_t)WARPS * hdv) * sizeof(float), stream>>>(ARGS(TY))
  if (dtype == CO_F32) { GO(float); }
  else if (dtype == CO_BF16) { GO(__nv_bfloat16); }
  else CO_FAIL("attention_simple: unknown dtype %d", dtype);
#undef GO
#undef HEADS_CASE
#undef ARGS
  CO_CHECK_LAUNCH("attention_simple");
  return 0;
}

CO_EXPORT int coheryn_attention_simple(const void* q, long q_stride, void* out, long out_stride,
                                       const void* k_cache, const void* v_cache, int dtype,
                                       const int* block_tables, int max_blocks, const int* token_req,
                                       const int* positions, int T, int nh, int nkv, int hd, int page_size,
                                       int window, float scale, cudaStream_t stream) {
  return coheryn_attention_simple_ex(q, q_stride, out, out_stride, k_cache, v_cache, dtype, block_tables, max_blocks,
                                     token_req, positions, T, nh, nkv, hd, hd, page_size, window, scale, nullptr, 1.0f,
                                     stream);
}
