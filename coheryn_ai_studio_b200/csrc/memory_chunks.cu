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
//   memory_sum_tc_kernel  (memory_chunks_tc.cu) what a chunk adds to S and n;
//   memory_carry_kernel   over a run's chunks, element by element: the S_0 and n_0 of every chunk; the last ones are kept;
//   memory_out_tc_kernel  (memory_chunks_tc.cu) the outputs and the norm, weight and gate behind them.
//
// Every exponent is a difference of float64 sums, rounded once, so that a weight is as exact however far the gates have summed up.  The maxima
// m are kept in float32, so an exponent may exceed zero by the rounding of m (3e-5 at m = 1,000): S, n and exp(-m) all use the same
// rounded m, and what it is off by cancels between numerator and denominator.
//
// A value, key, query or state that is not finite makes the outputs of its whole chunk so (of the head's value channels it reaches), not
// only those from its token on: a zero weight times it is not zero.  The products split every operand into three bfloat16 terms: one
// of 3.39e38 and more counts as not finite, and of one under 2^-110 up to 2^-133 is cut off, which the norm's eps hides.
//
// What bounds it: the scan token by token is a chain of dependent multiply-adds and shuffles on a CTA per (head, 64 value
// channels): 0.65 us per token with 32 of 148 SMs at work.  Here only the carry is a chain, of one multiply-add per chunk and
// element; the rest are products over all chunks at once.  Measured on a B200 (8 heads of 128 x 256, one request of 2,048
// tokens, L2 flushed): 135 us in place of 1,377 (by the profiler's clock, one kernel at a time from cold caches, 15 + 31 + 26 + 80).
//
// A run of fewer than CHUNK_FROM tokens is left to the scan (recurrent.cu), request by request: of the other requests only
// whether the step goes in chunks at all (recurrent.cu, coheryn_*_chunks_pay) can reach a row, not its order of additions.
#include "memory_chunks.cuh"

namespace {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// grid (runs, heads), GATE_WARPS warps.  A warp takes every GATE_WARPS-th chunk, two tokens per lane; what the chunks hand to one
// another is the running maximum alone, a chain of one step per chunk that one thread walks between the two passes (a warp per
// head that walked the chunks from beginning to end took 30 us for 32 of them).
constexpr int GATE_WARPS = 16;
__global__ void __launch_bounds__(32 * GATE_WARPS) memory_gates_kernel(MemoryIn P, int B, int base, int count, Area A) {
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

// grid (ceil(size / 1024), heads, runs), 256 threads of four neighbouring elements each; the chunks ahead are requested eight at
// a time.
__global__ void __launch_bounds__(256) memory_carry_kernel(MemoryIn P, int B, int base, int count, Area A) {
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

int padded(int dv) { return (dv + 15) / 16 * 16; }

}  // namespace

bool co_memory_chunks_take(int dk, int dv) { return dk >= 1 && dk <= 256 && dv >= 1 && dv <= 256; }

static int memory_chunks_at_once(int heads, int dk, int dv) { return chunks_at_once(Area::floats(1, heads, dk, padded(dv))); }

long co_memory_chunk_floats(int chunks, int heads, int dk, int dv) {
  const int at_once = memory_chunks_at_once(heads, dk, dv);
  return (long)Area::floats(chunks < at_once ? chunks : at_once, heads, dk, padded(dv));
}

int co_memory_chunks(const MemoryIn& P, const HeadOut& E, int B, int chunks, int runs, float* scratch, int* status, cudaStream_t stream) {
  const int dvp = padded(P.dv), at_once = memory_chunks_at_once(P.heads, P.dk, P.dv);
  for (int base = 0; base < chunks; base += at_once) {
    const int count = chunks - base < at_once ? chunks - base : at_once;
    const Area A(scratch, count, P.heads, P.dk, dvp);
    co_launch(memory_gates_kernel, dim3(runs, P.heads), dim3(32 * GATE_WARPS), 0, stream, P, B, base, count, A);
    CO_CHECK_LAUNCH("memory_gates");
    if (co_memory_sum_tc(P, B, base, count, A, status, stream)) return 1;
    co_launch(memory_carry_kernel, dim3((unsigned)((A.size + 1023) / 1024), P.heads, runs), dim3(256), 0, stream, P, B, base, count, A);
    CO_CHECK_LAUNCH("memory_carry");
    if (co_memory_out_tc(P, E, B, base, count, A, status, stream)) return 1;
  }
  return 0;
}
