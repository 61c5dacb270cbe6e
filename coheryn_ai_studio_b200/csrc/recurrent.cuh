// What the kernels of the recurrent mixers share: their inputs, and the norm per head with a weight and a gate behind them.
#pragma once
#include "common.cuh"

// ---------------------------------------------------------------------------------
// What both scans share: the output of a chunk of tokens (os [CT][dvp], one head) is divided by its root mean
// square over the value channels, multiplied by a weight and by the sigmoid of a gate's pre-activation, and
// written in the output's dtype.  A warp takes a token.
// ---------------------------------------------------------------------------------
struct HeadOut {
  void* out; int out_dtype; long ldo;          // [T, heads * dv]
  const void* weight; int weight_dtype;        // [dv] shared by the heads (weight_stride 0) or [heads * dv]
  int weight_stride;
  const float* gate; long ldg;                 // pre-activations [T, heads * dv]
  float eps, out_scale;
  // When the columns of a head are split over several CTAs (a long prompt of few requests that the scans take: more SMs at work),
  // no CTA sees a whole head: the scans then leave the unnormalised outputs in `raw` [T, heads * dv] and a second kernel applies
  // norm, weight and gate, in the same order of operations.  `nm_next`: where the matrix memory's n and m of each (request,
  // head) wait until every CTA of the head has read the old ones ([B][heads][dk + 1]).
  float* raw; long ldr;
  float* nm_next;
  int gate_act;                                // what the gate's pre-activation passes: 0 sigmoid, 1 SiLU
};

// ---------------------------------------------------------------------------------
// The inputs of the two scans (see recurrent.cu for the recurrences).
// ---------------------------------------------------------------------------------
struct DeltaIn {
  const float* q; const float* k; const float* v; long ld_qkv;   // after convolution and SiLU: [T, kv_heads*dk], .., [T, heads*dv]
  const float* beta; long ld_beta;                               // pre-activation of beta [T, heads]
  const float* step; long ld_step;                               // pre-activation of the step size [T, heads*dc] (bias not added)
  const void* step_bias; int step_bias_dtype;                    // [heads*dc]; dc = decay_channels
  const void* rate_log; int rate_log_dtype;                      // [heads]: decay = exp(-exp(rate_log) * softplus(step + bias))
  float* state; long state_stride;                               // per slot: S [heads, dk, dv]
  const int* cu_q; const int* state_slots;
  int heads, kv_heads, dk, dv;
  int decay_channels;                                            // dk: a decay per head and key channel; 1: one per head
};

struct MemoryIn {
  const float* q; const float* k; const float* v; long ld;       // projections [T, heads*dk], .., [T, heads*dv] (one row stride)
  const float* gi; const float* gf; long ld_gate;                // pre-activations of the input and forget gates [T, heads]
  const void* bias_i; const void* bias_f; int bias_dtype;        // [heads]
  float cap;                                                     // gates are capped: cap * tanh(z / cap)
  float* state; long state_stride;                               // per slot: S [heads, dk, dv], n [heads, dk], m [heads]
  const int* cu_q; const int* state_slots;
  int heads, dk, dv;
};

// In a step for which that is faster (coheryn_*_chunks_pay) runs of at least CHUNK_FROM tokens go chunk by chunk (delta_chunks.cu,
// memory_chunks.cu), shorter ones token by token (recurrent.cu), request by request.
constexpr int CHUNK_TOKENS = 64, CHUNK_FROM = 48;
// `chunks` and `runs`: how many chunks and how many such runs the step holds at most (CTAs beyond the last return at once);
// `scratch`: at least co_*_chunk_floats floats.
// The scratch of a step of many chunks is bounded: the kernels work on as many chunks at a time as 256 MB hold (`each` floats per
// chunk), one after the other; a run's state goes from one to the next through its slot, as it does from step to step.
constexpr int chunks_at_once(size_t each) { return each >= (1u << 26) ? 1 : (int)((1u << 26) / each); }
bool co_delta_chunks_take(int dk, int dv);
long co_delta_chunk_floats(int chunks, int heads, int dk, int dv);
int co_delta_chunks(const DeltaIn& P, const HeadOut& E, int B, int chunks, int runs, float* scratch, cudaStream_t stream);
bool co_memory_chunks_take(int dk, int dv);
long co_memory_chunk_floats(int chunks, int heads, int dk, int dv);
// `status`: device word that receives a code if a bounded wait for the tensor cores ran out.
int co_memory_chunks(const MemoryIn& P, const HeadOut& E, int B, int chunks, int runs, float* scratch, int* status, cudaStream_t stream);

// No co_pdl_launch_dependents() in the kernels of the scans and chunks and in the convolution in front of them: a successor that is
// launched ahead only sits beside them, and its early CTAs take SMs out of turn (several of them on one SM where another stands empty).
// Their successors start when they end.  Measured on a B200, whole mixers, launched ahead and not: delta rule, 16 heads of 64 x 64,
// runs of 9, 3, 263 and 217 tokens 163 and 131 us, 12 heads of 128 x 128, one run of 360 196 and 184, of 2,048 402 and 393; matrix
// memory, 8 heads of 128 x 256, runs of 400, 30 and 7 207 and 188.  Steps of a token per request (recurrent_one.cu) are too short for
// that and launch ahead.

// Lanes per group of columns and columns per group.  The more lanes share a column, the fewer steps a token costs
// each of them (the recurrence is a chain of dependent steps, and that chain is what bounds a long prompt): sixteen
// from 128 key channels on, eight from 64, four below.  Four columns per group (two for narrow heads); a head of more
// than 128 value channels takes twice as many so that the CTA stays within 512 threads.
constexpr int scan_split(int DK) { return DK >= 128 ? 16 : (DK >= 64 ? 8 : 4); }
// The key channels that the scans are built for, the smallest that hold `dk`.
#define CO_SCAN_CASES(LAUNCH)                                                                   \
  if (dk <= 16) { LAUNCH(16) } else if (dk <= 32) { LAUNCH(32) } else if (dk <= 48) { LAUNCH(48) } \
  else if (dk <= 64) { LAUNCH(64) } else if (dk <= 96) { LAUNCH(96) } else if (dk <= 128) { LAUNCH(128) } \
  else if (dk <= 192) { LAUNCH(192) } else { LAUNCH(256) }

// Steps in which every request brings one token (recurrent_one.cu): the same bits as the scans.
bool co_one_token_takes(int dk, int dv, const float* state, long stride);
int co_delta_one(const DeltaIn& P, const HeadOut& E, int B, cudaStream_t stream);
int co_memory_one(const MemoryIn& P, const HeadOut& E, int B, cudaStream_t stream);

namespace {

__device__ __forceinline__ float rc_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float rc_softplus(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ void rc_store(void* out, int dtype, size_t i, float v) {
  if (dtype == CO_BF16) ((__nv_bfloat16*)out)[i] = __float2bfloat16_rn(v);
  else ((float*)out)[i] = v;
}

__device__ __forceinline__ void head_out_chunk(const HeadOut& E, const float* os, int dvp, int dv, int nt, int row0, int h) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int i = warp; i < nt; i += warps) {
    float ss = 0.f;
    for (int c = lane; c < dv; c += 32) ss = fmaf(os[i * dvp + c], os[i * dvp + c], ss);
    ss = co_warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)dv + E.eps);
    const size_t row = (size_t)(row0 + i);
#pragma unroll 4
    for (int c = lane; c < dv; c += 32) {
      const float w = co_load_any(E.weight, E.weight_dtype, (size_t)h * E.weight_stride + c);
      const float z = E.gate[row * E.ldg + (size_t)h * dv + c];
      const float g = E.gate_act == 1 ? z * rc_sigmoid(z) : rc_sigmoid(z);
      rc_store(E.out, E.out_dtype, row * E.ldo + (size_t)h * dv + c, os[i * dvp + c] * inv * w * g * E.out_scale);
    }
  }
}

// The requests whose runs are cut into chunks, counted in the order of the step: the request of chunk `want` (of all
// requests) or, with `by_request`, the `want`-th such request.  Every warp finds it by itself.
struct Run {
  int r, start, len;      // request, first token of the step, tokens
  int chunk, first;       // chunk inside the run, ordinal of the run's first chunk
};
__device__ __forceinline__ bool find_run(const int* cu, int B, int want, bool by_request, Run& R) {
  const int lane = threadIdx.x & 31;
  int base = 0, chunks = 0;
  for (int r0 = 0; r0 < B; r0 += 32) {
    const int q = r0 + lane;
    const int a = q < B ? cu[q] : 0, n = q < B ? cu[q + 1] - a : 0;
    const int c = n >= CHUNK_FROM ? (n + CHUNK_TOKENS - 1) / CHUNK_TOKENS : 0;
    int x = c, y = c ? 1 : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int xo = __shfl_up_sync(0xffffffffu, x, o), yo = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) { x += xo; y += yo; }
    }
    const unsigned hit = __ballot_sync(0xffffffffu, base + (by_request ? y : x) > want);
    if (hit) {
      const int src = __ffs(hit) - 1;
      R.r = r0 + src;
      R.start = __shfl_sync(0xffffffffu, a, src);
      R.len = __shfl_sync(0xffffffffu, n, src);
      R.first = chunks + __shfl_sync(0xffffffffu, x - c, src);
      R.chunk = by_request ? 0 : want - R.first;
      return true;
    }
    const int tx = __shfl_sync(0xffffffffu, x, 31), ty = __shfl_sync(0xffffffffu, y, 31);
    chunks += tx;
    base += by_request ? ty : tx;
  }
  return false;
}

}  // namespace
