// A recurrent mixer (the gated delta rule or the matrix memory, csrc/recurrent.cu) in bfloat16 enqueued by ONE call from the host
// language: the product with the stacked projections, the short convolution and the second steps of low-rank projections (delta rule),
// the recurrence with the norm and gate behind it, the output product.
//
// What bounded it: done from Python a decode step's six or seven calls with the checks, slices and allocations between them take 110 us
// of host time, and the kernels of 32 requests 50 us.  The choice of kernels is that of ops.py (its thresholds come with the call) and
// of parts/recurrent.py's sequence; a product that ops.py would hand to a kernel this file does not call is answered with
// CO_MIXER_UNSUPPORTED before anything is launched, and the caller runs its own sequence.  Temporaries live in one scratch area that
// the caller provides for the call (its size is asked for with dry_run = 1).
#include "block_routes.h"

extern "C" {
long coheryn_gemm_simt_workspace_floats(int M, int N, int K);
int coheryn_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, const void* bias, int bias_dtype, void* out, int out_dtype, int M,
                      int N, int K, long ldx, long ldo, int act, float* workspace, long floats, int n_split, int k_split, cudaStream_t stream);
}

// Entry points of the recurrent mixers' library (a library of its own).
typedef int (*co_conv_fn)(const float* x, long ldx, float* y, long ldy, const void* taps, int taps_dtype, int n, int C, float* state,
                          long state_stride, const int* token_req, const int* cu_q, const int* state_slots, int T, int B, int update_state,
                          cudaStream_t stream);
typedef int (*co_delta_fn)(const float* q, const float* k, const float* v, long ld_qkv, const float* beta, long ld_beta, const float* step,
                           long ld_step, const void* step_bias, int step_bias_dtype, const void* rate_log, int rate_log_dtype, float* state,
                           long state_stride, const int* cu_q, const int* state_slots, int B, int heads, int kv_heads, int dk, int dv, void* out,
                           int out_dtype, long ldo, const void* weight, int weight_dtype, int weight_stride, const float* gate, long ldg,
                           float eps, float out_scale, int total_tokens, float* scratch, long scratch_floats, int decay_channels, int gate_act,
                           int chunks, int runs, int short_runs, cudaStream_t stream);
typedef int (*co_memory_fn)(const float* q, const float* k, const float* v, long ld, const float* gi, const float* gf, long ld_gate,
                            const void* bias_i, const void* bias_f, int bias_dtype, float cap, float* state, long state_stride,
                            const int* cu_q, const int* state_slots, int B, int heads, int dk, int dv, void* out, int out_dtype, long ldo,
                            const void* weight, int weight_dtype, int weight_stride, const float* gate, long ldg, float eps, float out_scale,
                            int total_tokens, float* scratch, long scratch_floats, int chunks, int runs, int short_runs, int* status,
                            cudaStream_t stream);
typedef long (*co_chunk_floats_fn)(int chunks, int heads, int dk, int dv);
typedef int (*co_chunks_pay_fn)(int heads, int dk, int dv, int B, int T, int longest, int chunks);

// What a mixer is made of: constant from the moment its weights are bound.
struct CoMixerLayer {
  const void *w_in, *w_second, *w_o;                  // w_second: the block-diagonal second steps [second_n][second_k] (null: none)
  const void *conv_w, *bias_a, *bias_b, *norm_w;      // delta rule: bias_a the step's bias, bias_b the rates; memory: of the input and forget gates
  co_conv_fn conv; co_delta_fn delta; co_memory_fn memory; co_chunk_floats_fn chunk_floats; co_chunks_pay_fn chunks_pay;
  float eps, out_scale, cap;
  int memory_kind;                                    // 1: matrix memory, 0: gated delta rule
  int width, columns, heads, kv_heads, dk, dv, taps, decay_channels, gate_act, in_chunks, chunk_from, chunk_tokens;
  int at_q, at_k, at_v, at_g, at_a, at_b;             // first columns of the projections (a, b: step or input gate, beta or forget gate;
                                                      // with w_second: a the first low-rank one, g behind it)
  int second_n, second_k, second_rows, second_columns;
  int conv_dtype, bias_a_dtype, bias_b_dtype, norm_dtype;
};
struct CoMixerStep {
  const int *token_req, *cu_q, *state_slots;
  int* tc_status;
  cudaStream_t stream;
  int T, B;
  const int* q_lens;                                  // on the host: tokens of every request (null: not counted)
};

#define CO_MIXER_UNSUPPORTED 3         // nothing was launched: run the operations one by one
#define CO_MIXER_RECURRENT_FAILED 2    // the message is the recurrent mixers' library's

namespace {

#define RUN(call)                      \
  do {                                 \
    if (launch) {                      \
      const int rc__ = (call);         \
      if (rc__) return rc__;           \
    }                                  \
  } while (0)
#define RUN_RECURRENT(call)                                \
  do {                                                     \
    if (launch && (call)) return CO_MIXER_RECURRENT_FAILED; \
  } while (0)

// y [M][N] (float32) = x w^T by the kernel that ops.linear chooses.
int product(const Router& R, Arena& A, bool launch, const CoMixerStep& S, const void* x, long ldx, const void* w, float* y, long ldy, int M, int N, int K) {
  int splits;
  switch (R.linear(M, N, K, ldx, x, w, false, &splits)) {
    case R_FEW:
      RUN(coheryn_gemm_bf16_tc_few(x, w, nullptr, CO_F32, y, CO_F32, M, N, K, ldx, ldy, 0, S.tc_status, nullptr, 0, 0, S.stream));
      return 0;
    case R_SMALL:
      RUN(coheryn_gemm_bf16_small(x, w, nullptr, CO_F32, y, CO_F32, M, N, K, ldx, ldy, 0, S.stream));
      return 0;
    case R_TC: {
      const long floats = coheryn_gemm_tc_workspace_floats(M, N, K);
      float* ws = floats ? (float*)A.take((size_t)floats * 4) : nullptr;
      RUN(coheryn_gemm_bf16_tc(x, w, nullptr, CO_F32, y, CO_F32, M, N, K, ldx, ldy, 0, S.tc_status, ws, floats, S.stream));
      return 0;
    }
    default:
      return CO_MIXER_UNSUPPORTED;
  }
}

// The runs of a step that go in chunks (ops.py, _chunked_runs): their chunks, how many they are, whether others are left.
struct Runs { int chunks, runs, rest; };
Runs chunked_runs(const CoMixerLayer& L, const CoMixerStep& S) {
  const Runs none{0, 0, 1};
  const int first = L.chunk_from, size = L.chunk_tokens;
  if (!L.in_chunks || S.T - S.B + 1 < first) return none;
  Runs r = none;
  int longest = 0;
  if (S.q_lens) {
    for (int i = 0; i < S.B; ++i)
      if (S.q_lens[i] >= first) {
        r.chunks += (S.q_lens[i] + size - 1) / size;
        ++r.runs;
        longest = S.q_lens[i] > longest ? S.q_lens[i] : longest;
      }
    if (!r.runs) return none;
    r.rest = r.runs < S.B;
  } else {
    r.runs = S.B < S.T / first ? S.B : S.T / first;
    longest = S.T - S.B + 1;
    r.chunks = S.T / size + r.runs;
  }
  return L.chunks_pay(L.heads, L.dk, L.dv, S.B, S.T, longest, r.chunks) ? r : none;
}

int mixer_pass(const CoMixerLayer& L, const CoMixerStep& S, const CoBlockTuning& tn, const void* x, long ldx, float* state, long state_stride,
               void* open, long ld_open, float* out, char* scratch, bool launch, long* scratch_bytes) {
  const int T = S.T, B = S.B, H = L.heads, dk = L.dk, dv = L.dv;
  const Router R{tn};
  Arena A{scratch, 0};
  float* proj = (float*)A.take((size_t)T * L.columns * 4);
  int rc = product(R, A, launch, S, x, ldx, L.w_in, proj, L.columns, T, L.columns, L.width);
  if (rc) return rc;
  void* o = open ? open : A.take((size_t)T * H * dv * 2);
  const long ldo = open ? ld_open : (long)H * dv;
  const Runs r = chunked_runs(L, S);
  // the scans' scratch: the chunks', or the unnormalised outputs (and what the scan prepares) of a long prompt of few requests
  const long extra = L.memory_kind ? (long)B * H * (dk + 1) : (long)T * (2 * L.kv_heads * dk + H * dk + H);
  const long floats = r.chunks ? L.chunk_floats(r.chunks, H, dk, dv) : dv <= 64 || (long)B * H > 74 || T < 64L * B ? 0 : (long)T * H * dv + extra;
  if (L.memory_kind) {
    float* area = floats ? (float*)A.take((size_t)floats * 4) : nullptr;
    RUN_RECURRENT(L.memory(proj + L.at_q, proj + L.at_k, proj + L.at_v, L.columns, proj + L.at_a, proj + L.at_b, L.columns, L.bias_a, L.bias_b,
                           L.bias_a_dtype, L.cap, state, state_stride, S.cu_q, S.state_slots, B, H, dk, dv, o, CO_BF16, ldo, L.norm_w, L.norm_dtype,
                           dv, proj + L.at_g, L.columns, L.eps, L.out_scale, T, area, floats, r.chunks, r.runs, r.rest, S.tc_status, S.stream));
  } else {
    const int G = L.kv_heads, C = 2 * G * dk + H * dv;
    float* qkv = (float*)A.take((size_t)T * C * 4);
    RUN_RECURRENT(L.conv(proj + L.at_q, L.columns, qkv, C, L.conv_w, L.conv_dtype, L.taps, C, state + (size_t)H * dk * dv, state_stride, S.token_req,
                         S.cu_q, S.state_slots, T, B, 1, S.stream));
    const float *steps = proj + L.at_a, *gate = proj + L.at_g;
    long ld_steps = L.columns, ldg = L.columns;
    if (L.w_second) {
      const long ws = coheryn_gemm_simt_workspace_floats(T, L.second_n, L.second_k);
      float* second = (float*)A.take((size_t)T * L.second_n * 4);
      float* area = ws ? (float*)A.take((size_t)ws * 4) : nullptr;
      RUN(coheryn_gemm_simt(proj + L.at_a, CO_F32, L.w_second, CO_BF16, nullptr, CO_F32, second, CO_F32, T, L.second_n, L.second_k, L.columns,
                            L.second_n, 0, area, ws, L.second_rows, L.second_columns, S.stream));
      steps = second;
      gate = second + H * L.decay_channels;
      ld_steps = ldg = L.second_n;
    }
    float* area = floats ? (float*)A.take((size_t)floats * 4) : nullptr;
    RUN_RECURRENT(L.delta(qkv, qkv + G * dk, qkv + 2 * G * dk, C, proj + L.at_b, L.columns, steps, ld_steps, L.bias_a, L.bias_a_dtype, L.bias_b,
                          L.bias_b_dtype, state, state_stride, S.cu_q, S.state_slots, B, H, G, dk, dv, o, CO_BF16, ldo, L.norm_w, L.norm_dtype, 0,
                          gate, ldg, L.eps, L.out_scale, T, area, floats, L.decay_channels, L.gate_act, r.chunks, r.runs, r.rest, S.stream));
  }
  if (out) {
    rc = product(R, A, launch, S, o, ldo, L.w_o, out, L.width, T, L.width, H * dv);
    if (rc) return rc;
  }
  *scratch_bytes = (long)A.off + 256;
  return 0;
}
#undef RUN
#undef RUN_RECURRENT
}  // namespace

// Runs (or, with dry_run, only plans) a mixer on x [T][width] (row stride ldx), continued from and left in `state` (row stride
// state_stride).  `open`: where the activations in front of the output product go (bfloat16 [T][heads * dv], row stride ld_open; null: into
// scratch); `out`: float32 [T][width] (null: the activations are all that is wanted).  Returns 0, 1 (an error of this library),
// CO_MIXER_RECURRENT_FAILED or CO_MIXER_UNSUPPORTED (nothing launched); *scratch_bytes receives what the call needs.
CO_EXPORT int coheryn_recurrent_mixer_bf16(const CoMixerLayer* layer, const CoMixerStep* step, const CoBlockTuning* tuning, const void* x, long ldx,
                                           float* state, long state_stride, void* open, long ld_open, float* out, void* scratch, long scratch_bytes,
                                           int dry_run, long* needed) {
  if (!layer || !step || !tuning || !needed) CO_FAIL("recurrent_mixer: a description is missing");
  if (step->T <= 0 || step->B <= 0 || (!open && !out)) return CO_MIXER_UNSUPPORTED;
  const int rc = mixer_pass(*layer, *step, *tuning, x, ldx, state, state_stride, open, ld_open, out, nullptr, false, needed);
  if (rc || dry_run) return rc;
  if (!scratch || scratch_bytes < *needed || ((uintptr_t)scratch & 255))
    CO_FAIL("recurrent_mixer: %ld bytes of scratch (256-byte aligned) are needed, %ld were given", *needed, scratch_bytes);
  if (!x || !state) CO_FAIL("recurrent_mixer: a buffer is missing");
  long again;
  return mixer_pass(*layer, *step, *tuning, x, ldx, state, state_stride, open, ld_open, out, (char*)scratch, true, &again);
}
