// The stabilised matrix memory for runs of many tokens, in chunks of 64 (float32; the sums of log gates in float64).
//
// Inside a chunk let F_t be the sum of the log forget gates up to and with token t, i_t the log input gate, m_0 and S_0, n_0 the
// maximum and the (stabilised) state in front of it.  Then
//
//   m_t = max(F_t + m_0, max_{s <= t} F_t - F_s + i_s),     w_ts = exp(F_t - F_s + i_s - m_t),   a_t = exp(F_t + m_0 - m_t)
//   S_t = a_t S_0 + sum_{s <= t} w_ts k_s v_s^T,            n_t likewise with k_s alone
//   o_t = (a_t S_0^T q_t + sum_{s <= t} w_ts (q_t . k_s) v_s) / (max(|n_t . q_t|, exp(-m_t)) + 1e-6)
//
//   memory_gates_kernel   a CTA per (run, head): F, i, m of every token and m_0 of every chunk;
//   memory_sum_kernel     a CTA per (chunk, head, 64 key channels, 128 value channels): what the chunk adds to S and n;
//   memory_carry_kernel   over a run's chunks, element by element: the S_0 and n_0 of every chunk; the last ones are kept;
//   memory_out_kernel     a CTA per (chunk, head): the outputs and the norm, weight and gate behind them.
//
// Every exponent is a difference of float64 sums, so that a weight is as exact however far the gates have summed up.  The maxima
// m are kept in float32, so an exponent may exceed zero by the rounding of m (3e-5 at m = 1,000): S, n and exp(-m) all use the same
// rounded m, and what it is off by cancels between numerator and denominator.
//
// A value or key that is not finite makes the outputs of its whole chunk so, not only those from its token on: a zero weight times
// it is not zero.
//
// What bounds it: the scan token by token is a chain of dependent multiply-adds and shuffles on a CTA per (head, 64 value
// channels): 0.65 us per token with 32 of 148 SMs at work.  Here only the carry is a chain, of one multiply-add per chunk and
// element; the rest are products over all chunks at once.  Measured on a B200 (8 heads of 128 x 256, one request of 2,048
// tokens): 14 + 38 + 16 + 94 us in place of 1,350 us (1,850 with the kernels behind the scan launched ahead and waiting beside it).
//
// A run of fewer than CHUNK_FROM tokens is left to the scan (recurrent.cu), request by request: of the other requests only
// whether the step goes in chunks at all (recurrent.cu, coheryn_*_chunks_pay) can reach a row, not its order of additions.
#include "recurrent.cuh"

namespace {

constexpr int CH = CHUNK_TOKENS;
constexpr int TP = CH + 4;           // pitch of [channel][token] tiles

__device__ __forceinline__ void cp4(float* smem_dst, const float* src) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16(float* smem_dst, const float* src) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

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

// grid (runs, heads), GATE_WARPS warps.  A warp takes every GATE_WARPS-th chunk, two tokens per lane; what the chunks hand to one
// another is the running maximum alone, a chain of one step per chunk that one thread walks between the two passes (a warp per
// head that walked the chunks from beginning to end took 30 us for 32 of them).
constexpr int GATE_WARPS = 16;
__global__ void __launch_bounds__(32 * GATE_WARPS) memory_gates_kernel(MemoryIn P, int B, int base, int count, Area A) {
  co_pdl_launch_dependents();
  co_pdl_wait();
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Run R;
  if (!find_run(P.cu_q, B, blockIdx.x, true, R)) return;
  // the run's chunks among the `count` that are worked on, from `base` on
  const int from = max(0, base - R.first), to = min((R.len + CH - 1) / CH, base + count - R.first), first = R.first - base;
  if (from >= to) return;
  float* m_state = P.state + (size_t)P.state_slots[R.r] * P.state_stride + (size_t)P.heads * P.dk * P.dv + (size_t)P.heads * P.dk + h;
  const float bi = co_load_any(P.bias_i, P.bias_dtype, h), bf = co_load_any(P.bias_f, P.bias_dtype, h);
  // the largest i_s - F_s up to and with this lane's tokens
  auto best_of = [&](const double (&F)[2], const float (&li)[2], int nt, double (&best)[2]) {
    const double p0 = 2 * lane < nt ? (double)li[0] - F[0] : -1e300, p1 = fmax(p0, 2 * lane + 1 < nt ? (double)li[1] - F[1] : -1e300);
    double x = p1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x = fmax(x, y);
    }
    const double before = __shfl_up_sync(0xffffffffu, x, 1);
    best[0] = fmax(lane ? before : -1e300, p0);
    best[1] = x;
  };
  for (int c = from + warp; c < to; c += GATE_WARPS) {
    const int nt = min(CH, R.len - c * CH);
    float li[2];
    double F[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const size_t row = (size_t)(R.start + min(c * CH + 2 * lane + u, R.len - 1));
      li[u] = P.cap * tanhf((P.gi[row * P.ld_gate + h] + bi) / P.cap);
      const float z = P.cap * tanhf((P.gf[row * P.ld_gate + h] + bf) / P.cap);
      F[u] = 2 * lane + u < nt ? (double)-rc_softplus(-z) : 0.0;       // log sigmoid; tokens beyond the last add nothing
    }
    const double second = F[1];
    double x = F[0] + F[1];                         // sums up to and with this lane's tokens
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    F[0] = x - second;
    F[1] = x;
    double best[2];
    best_of(F, li, nt, best);
    const size_t at = (size_t)(first + c) * P.heads + h;
#pragma unroll
    for (int u = 0; u < 2; ++u) { A.f[at * CH + 2 * lane + u] = F[u]; A.i[at * CH + 2 * lane + u] = li[u]; }
    if (lane == 31) {
      *reinterpret_cast<double*>(A.m0 + at * 4) = best[1];
      *reinterpret_cast<double*>(A.m0 + at * 4 + 2) = F[1];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float m0 = *m_state;
    for (int c0 = from; c0 < to; c0 += 8) {
      double best[8], end[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + i < to) {
          const float* p = A.m0 + ((size_t)(first + c0 + i) * P.heads + h) * 4;
          best[i] = *reinterpret_cast<const double*>(p);
          end[i] = *reinterpret_cast<const double*>(p + 2);
        }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + i < to) {
          float* p = A.m0 + ((size_t)(first + c0 + i) * P.heads + h) * 4;
          const float m1 = (float)(end[i] + fmax((double)m0, best[i]));
          p[0] = m0; p[1] = m1;
          m0 = m1;
        }
    }
    *m_state = m0;
  }
  __syncthreads();
  for (int c = from + warp; c < to; c += GATE_WARPS) {
    const size_t at = (size_t)(first + c) * P.heads + h;
    const double F[2] = {A.f[at * CH + 2 * lane], A.f[at * CH + 2 * lane + 1]};
    const float li[2] = {A.i[at * CH + 2 * lane], A.i[at * CH + 2 * lane + 1]};
    const double m0 = (double)A.m0[at * 4];
    double best[2];
    best_of(F, li, min(CH, R.len - c * CH), best);
#pragma unroll
    for (int u = 0; u < 2; ++u) A.m[at * CH + 2 * lane + u] = (float)(F[u] + fmax(m0, best[u]));
  }
}

// acc rows 4 la + i and 32 + 4 la + i of a 64-row product, four neighbouring columns: acc[t][c] += left[k][t] right[k][c].
template <int TC>
__device__ __forceinline__ void mac(float (&acc)[8][TC], const float* left, const float* right) {
  float b[TC];
  if (TC == 4) { const float4 x = ld4(right); b[0] = x.x; b[1] = x.y; b[2 % TC] = x.z; b[3 % TC] = x.w; }
  else { const float2 x = *reinterpret_cast<const float2*>(right); b[0] = x.x; b[1] = x.y; }
  const float4 l = ld4(left), u = ld4(left + 32);
#pragma unroll
  for (int c = 0; c < TC; ++c) {
    acc[0][c] = fmaf(l.x, b[c], acc[0][c]); acc[1][c] = fmaf(l.y, b[c], acc[1][c]);
    acc[2][c] = fmaf(l.z, b[c], acc[2][c]); acc[3][c] = fmaf(l.w, b[c], acc[3][c]);
    acc[4][c] = fmaf(u.x, b[c], acc[4][c]); acc[5][c] = fmaf(u.y, b[c], acc[5][c]);
    acc[6][c] = fmaf(u.z, b[c], acc[6][c]); acc[7][c] = fmaf(u.w, b[c], acc[7][c]);
  }
}
template <int TC>
__device__ __forceinline__ void zero(float (&acc)[8][TC]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < TC; ++c) acc[i][c] = 0.f;
}
__device__ __forceinline__ int row_of(int i, int la) { return (i < 4 ? 0 : 32) + 4 * la + (i & 3); }

// grid (chunks, heads, ceil(dk / 64) * ceil(dvp / 128)), 256 threads.
__global__ void __launch_bounds__(256) memory_sum_kernel(MemoryIn P, int B, int base, Area A) {
  extern __shared__ __align__(16) float sm[];
  float* Ks = sm;                    // [64 tokens][64 channels], weighted
  float* Vs = Ks + CH * 64;          // [64 tokens][128]
  float* ws = Vs + CH * 128;         // [64] what a token weighs at the end of the chunk
  co_pdl_launch_dependents();
  co_pdl_wait();
  const int h = blockIdx.y, dk = P.dk, dv = P.dv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) return;
  const int nv = (A.dvp + 127) / 128, d0 = (blockIdx.z / nv) * 64, c0 = (blockIdx.z % nv) * 128;
  const int row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const size_t at = (size_t)blockIdx.x * P.heads + h;
  if (tid < CH) {
    const double end = *reinterpret_cast<const double*>(A.m0 + at * 4 + 2);
    ws[tid] = tid < nt ? expf((float)(end - A.f[at * CH + tid] + (double)A.i[at * CH + tid] - (double)A.m0[at * 4 + 1])) : 0.f;
  }
#pragma unroll 8
  for (int e = tid; e < CH * 128; e += 256) {
    const int t = e >> 7, c = c0 + (e & 127);
    Vs[e] = t < nt && c < dv ? P.v[(size_t)(row0 + t) * P.ld + (size_t)h * dv + c] : 0.f;
  }
  __syncthreads();
#pragma unroll 8
  for (int e = tid; e < CH * 64; e += 256) {
    const int t = e >> 6, d = d0 + (e & 63);
    Ks[e] = t < nt && d < dk ? P.k[(size_t)(row0 + t) * P.ld + (size_t)h * dk + d] * ws[t] : 0.f;
  }
  __syncthreads();
  const int la = lane >> 2, col = warp * 16 + 4 * (lane & 3);
  float acc[8][4];
  zero(acc);
#pragma unroll 8
  for (int s = 0; s < CH; ++s) mac<4>(acc, Ks + s * 64 + 4 * la, Vs + s * 128 + col);
  float* out = A.s + at * A.size;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int d = d0 + row_of(i, la);
    if (d < dk && c0 + col < A.dvp) st4(out + (size_t)d * A.dvp + c0 + col, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
  }
  if (c0 == 0 && tid < 64 && d0 + tid < dk) {
    float n = 0.f;
    for (int s = 0; s < CH; ++s) n += Ks[s * 64 + tid];
    out[(size_t)dk * A.dvp + d0 + tid] = n;
  }
}

// grid (ceil(size / 1024), heads, runs), 256 threads of four neighbouring elements each; the chunks ahead are requested eight at
// a time.
__global__ void __launch_bounds__(256) memory_carry_kernel(MemoryIn P, int B, int base, int count, Area A) {
  co_pdl_launch_dependents();
  co_pdl_wait();
  const int h = blockIdx.y, dk = P.dk, dv = P.dv;
  Run R;
  if (!find_run(P.cu_q, B, blockIdx.z, true, R)) return;
  const size_t e = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (e >= A.size) return;
  const int from = max(0, base - R.first), chunks = min((R.len + CH - 1) / CH, base + count - R.first) - from;      // of the run, among those worked on
  if (chunks <= 0) return;
  const int d = (int)(e / A.dvp), c = (int)(e % A.dvp);
  float* slot = P.state + (size_t)P.state_slots[R.r] * P.state_stride;
  float* st = d < dk ? slot + ((size_t)h * dk + d) * dv + c : slot + (size_t)P.heads * dk * dv + (size_t)h * dk + (e - (size_t)dk * A.dvp);
  const int left = d < dk ? dv - c : dk - (int)(e - (size_t)dk * A.dvp);      // entries of the state from here on
  float s[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = j < left ? st[j] : 0.f;
  const size_t step = (size_t)P.heads * A.size;
  float* p = A.s + ((size_t)(R.first - base + from) * P.heads + h) * A.size + e;
  const float* g = A.m0 + ((size_t)(R.first - base + from) * P.heads + h) * 4;
  constexpr int AHEAD = 8;
  for (int i0 = 0; i0 < chunks; i0 += AHEAD) {
    float4 x[AHEAD];
    float a[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (i0 + i < chunks) {
        x[i] = ld4(p + (i0 + i) * step);
        const float* q = g + (size_t)(i0 + i) * P.heads * 4;
        a[i] = expf((float)(*reinterpret_cast<const double*>(q + 2) + (double)q[0] - (double)q[1]));
      }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (i0 + i < chunks) {
        st4(p + (i0 + i) * step, make_float4(s[0], s[1], s[2], s[3]));
        s[0] = fmaf(a[i], s[0], x[i].x); s[1] = fmaf(a[i], s[1], x[i].y); s[2] = fmaf(a[i], s[2], x[i].z); s[3] = fmaf(a[i], s[3], x[i].w);
      }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < left) st[j] = s[j];
}

// grid (chunks, heads), 2 W threads: all value channels of a head in one tile of W.  smem: the tile's rows of S and v in slices
// of 16, two deep (before that, keys in slices of 64 channels), q, the weighted scores; the finished rows over the first two.
constexpr int SLICE = 16;
size_t out_smem(int W, int dk, int dvp) {
  const int dkp = (dk + SLICE - 1) / SLICE * SLICE;
  size_t first = (size_t)2 * SLICE * W, keys = (size_t)64 * TP, qs = (size_t)dkp * TP, rows = (size_t)CH * (dvp + 4);
  if (first < keys) first = keys;
  if (first + qs < rows) first = rows - qs;
  first = (first + 3) / 4 * 4;
  return sizeof(float) * (first + qs + (size_t)CH * TP + 8 * CH) ;
}

template <int W>
__global__ void __launch_bounds__(2 * W, 512 / W) memory_out_kernel(MemoryIn P, HeadOut E, int B, int base, Area A, int first_floats) {
  constexpr int THREADS = 2 * W;
  extern __shared__ __align__(16) float sm[];
  const int dk = P.dk, dv = P.dv, dvp = A.dvp, dkp = (dk + SLICE - 1) / SLICE * SLICE;
  float* area = sm;                       // slices, keys; at the end the finished rows [64][dvp + 4]
  float* Qt = sm + first_floats;          // [dkp][TP] q / sqrt(dk), transposed
  float* Pt = Qt + dkp * TP;              // [s][TP] w_ts (q_t . k_s), zero for s > t
  float* as = Pt + CH * TP;               // [64] a_t
  float* dens = as + CH;                  // [64]
  float* sums = dens + CH;                // [4][64]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, la = lane >> 2;
  co_pdl_launch_dependents();
  co_pdl_wait();
  const int h = blockIdx.y;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) return;
  const int row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const size_t at = (size_t)blockIdx.x * P.heads + h;
  const float q_scale = 1.0f / sqrtf((float)dk);
  const double* F = A.f + at * CH;
  const float* gi = A.i + at * CH;
  const float* gm = A.m + at * CH;
  // a warp takes eight tokens by four channels at a time: sectors of 32 bytes are read whole, and the transposed stores fall on
  // different banks
#pragma unroll 8
  for (int e = tid; e < dkp * CH; e += THREADS) {
    const int d = (e & 7) + 8 * (e / (8 * CH)), t = (e >> 3) % CH;
    Qt[d * TP + t] = t < nt && d < dk ? P.q[(size_t)(row0 + t) * P.ld + (size_t)h * dk + d] * q_scale : 0.f;
  }
  if (tid < CH) as[tid] = expf((float)(F[tid] + (double)A.m0[at * 4] - (double)gm[tid]));
  {
    float acc[8][2];
    zero(acc);
    const int col = warp * 8 + 2 * (lane & 3);      // the first eight warps
    for (int d0 = 0; d0 < dk; d0 += 64) {
      const int n = min(64, dk - d0);
      if (d0) __syncthreads();
#pragma unroll
      for (int e = tid; e < 64 * CH; e += THREADS) {
        const int d = (e & 7) + 8 * (e / (8 * CH)), t = (e >> 3) % CH;
        if (d < n) area[d * TP + t] = t < nt ? P.k[(size_t)(row0 + t) * P.ld + (size_t)h * dk + d0 + d] : 0.f;
      }
      __syncthreads();
      if (warp < 8) {
#pragma unroll 4
        for (int d = 0; d < n; ++d) mac<2>(acc, Qt + (d0 + d) * TP + 4 * la, area + d * TP + col);
      }
    }
    if (warp < 8) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int s = col + c;
        const double fs = (double)gi[s] - F[s];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int t = row_of(i, la);
          Pt[s * TP + t] = s <= t && t < nt ? acc[i][c] * expf((float)(F[t] + fs - (double)gm[t])) : 0.f;
        }
      }
    }
  }
  __syncthreads();
  auto stage = [&](int i) {               // slice i: rows of S_0, then of v
    float* to = area + (i & 1) * SLICE * W;
    const int k0 = i * SLICE;
    if (k0 < dkp) {
      const float* rows = A.s + at * A.size + (size_t)k0 * dvp;
      for (int e = tid; e < SLICE * W / 4; e += THREADS) {
        const int k = e / (W / 4), c = 4 * (e % (W / 4));
        if (c >= dvp) continue;
        if (k0 + k < dk) cp16(to + k * W + c, rows + (size_t)k * dvp + c);
        else st4(to + k * W + c, make_float4(0.f, 0.f, 0.f, 0.f));
      }
    } else {
      for (int e = tid; e < SLICE * W; e += THREADS) {
        const int k = e / W, c = e % W, t = k0 - dkp + k;
        if (c >= dvp) continue;
        if (t < nt && c < dv) cp4(to + e, P.v + (size_t)(row0 + t) * P.ld + (size_t)h * dv + c);
        else to[e] = 0.f;
      }
    }
    cp_commit();
  };
  stage(0);
  // n_t . q_t, and with it the denominators (meanwhile the first slice is on its way)
  if (tid < 256) {
    const int t = tid & 63, part = tid >> 6;
    const float* n0 = A.s + at * A.size + (size_t)dk * dvp;
    float x = 0.f, y = 0.f;
    for (int d = part; d < dk; d += 4) x = fmaf(Qt[d * TP + t], n0[d], x);
    for (int s = part; s < CH; s += 4) y += Pt[s * TP + t];
    sums[part * CH + t] = fmaf(as[t], x, y);
  }
  __syncthreads();
  if (tid < CH)
    dens[tid] = 1.0f / (fmaxf(fabsf((sums[tid] + sums[CH + tid]) + (sums[2 * CH + tid] + sums[3 * CH + tid])), expf(-gm[tid])) + 1e-6f);
  const int col = warp * 16 + 4 * (lane & 3);
  float acc[8][4];
  zero(acc);
  const int state_slices = dkp / SLICE, slices = state_slices + CH / SLICE;
  for (int i = 0; i < slices; ++i) {
    if (i + 1 < slices) { stage(i + 1); cp_wait<1>(); }
    else cp_wait<0>();
    __syncthreads();
    if (i == state_slices) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float a = as[row_of(r, la)];
        acc[r][0] *= a; acc[r][1] *= a; acc[r][2] *= a; acc[r][3] *= a;
      }
    }
    const float* left = (i < state_slices ? Qt + i * SLICE * TP : Pt + (i - state_slices) * SLICE * TP) + 4 * la;
    const float* right = area + (i & 1) * SLICE * W + col;
#pragma unroll
    for (int k = 0; k < SLICE; ++k) mac<4>(acc, left + k * TP, right + k * W);
    __syncthreads();
  }
  if (col < dvp) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = row_of(i, la);
      const float x = dens[t];
      st4(area + t * (dvp + 4) + col, make_float4(acc[i][0] * x, acc[i][1] * x, acc[i][2] * x, acc[i][3] * x));
    }
  }
  __syncthreads();
  head_out_chunk(E, area, dvp + 4, dv, nt, row0, h);
}

int padded(int dv) { return (dv + 15) / 16 * 16; }

}  // namespace

bool co_memory_chunks_take(int dk, int dv) { return dk >= 1 && dk <= 256 && dv >= 1 && dv <= 256; }

static int memory_chunks_at_once(int heads, int dk, int dv) { return chunks_at_once(Area::floats(1, heads, dk, padded(dv))); }

long co_memory_chunk_floats(int chunks, int heads, int dk, int dv) {
  const int at_once = memory_chunks_at_once(heads, dk, dv);
  return (long)Area::floats(chunks < at_once ? chunks : at_once, heads, dk, padded(dv));
}

int co_memory_chunks(const MemoryIn& P, const HeadOut& E, int B, int chunks, int runs, float* scratch, cudaStream_t stream) {
  const int dvp = padded(P.dv), at_once = memory_chunks_at_once(P.heads, P.dk, P.dv);
  const size_t sum_smem = sizeof(float) * (CH * 64 + CH * 128 + CH);
  cudaFuncSetAttribute(memory_sum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sum_smem);
  const int W = dvp <= 128 ? 128 : 256;
  const size_t smem = out_smem(W, P.dk, dvp);
  const int dkp = (P.dk + SLICE - 1) / SLICE * SLICE;
  const int first = (int)(smem / sizeof(float)) - (dkp * TP + CH * TP + 8 * CH);
  auto out = W == 128 ? memory_out_kernel<128> : memory_out_kernel<256>;
  cudaFuncSetAttribute(out, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  for (int base = 0; base < chunks; base += at_once) {
    const int count = chunks - base < at_once ? chunks - base : at_once;
    const Area A(scratch, count, P.heads, P.dk, dvp);
    co_launch(memory_gates_kernel, dim3(runs, P.heads), dim3(32 * GATE_WARPS), 0, stream, P, B, base, count, A);
    CO_CHECK_LAUNCH("memory_gates");
    co_launch(memory_sum_kernel, dim3(count, P.heads, ((P.dk + 63) / 64) * ((dvp + 127) / 128)), dim3(256), sum_smem, stream, P, B, base, A);
    CO_CHECK_LAUNCH("memory_sum");
    co_launch(memory_carry_kernel, dim3((unsigned)((A.size + 1023) / 1024), P.heads, runs), dim3(256), 0, stream, P, B, base, count, A);
    CO_CHECK_LAUNCH("memory_carry");
    co_launch(out, dim3(count, P.heads), dim3(2 * W), smem, stream, P, E, B, base, A, first);
    CO_CHECK_LAUNCH("memory_out");
  }
  return 0;
}
