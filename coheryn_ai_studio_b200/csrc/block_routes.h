// What the files that enqueue whole layers from the host share: the choice of kernel for a product that ops.py makes (the
// thresholds come from there with every call), and the temporaries of a call in one area.
#pragma once
#include <cstdint>

#include "common.cuh"

extern "C" {
int coheryn_gemm_bf16_small(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int out_dtype, int M,
                            int N, int K, long ldx, long ldo, int epilogue, cudaStream_t stream);
long coheryn_gemm_tc_workspace_floats(int M, int N, int K);
int coheryn_gemm_bf16_tc(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int out_dtype, int M,
                         int N, int K, long ldx, long ldo, int epilogue, int* status, float* workspace,
                         long workspace_floats, cudaStream_t stream);
int coheryn_gemm_tc_few_splits(int N, int K);
int coheryn_gemm_bf16_tc_few(const void* x, const void* w, const void* bias, int bias_dtype, void* out, int out_dtype, int M,
                             int N, int K, long ldx, long ldo, int epilogue, int* status, float* workspace,
                             long workspace_floats, int defer, cudaStream_t stream);
}

// ops.py's thresholds, as they stand when the step is run.
struct CoBlockTuning {
  long small_weight_elements, few_large_weight, attn_oproj_merge_bytes;
  int few_m, few_defer_m, few_head_m, small_m, small_m_short, defer_min_k, defer_min_k_wide;
  int qkv_rope_m, qkv_parts_m, qkv_parts_few_from, attn_oproj_m;
};

namespace {

enum Route { R_NONE = 0, R_FEW, R_FEW_DEFER, R_SMALL, R_TC };

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

struct Router {
  const CoBlockTuning& t;
  bool operands_ok(int K, long ldx, const void* x, const void* w) const {
    return K % 8 == 0 && ldx % 8 == 0 && aligned16(x) && aligned16(w);
  }
  bool few_shape_ok(int M, int K, long ldx, const void* x, const void* w, int limit) const {
    return 0 < M && M <= limit && operands_ok(K, ldx, x, w);
  }
  bool few_ok(int M, int N, int K, long ldx, const void* x, const void* w) const {
    const int limit = (long)N * K >= t.few_large_weight ? t.few_head_m : t.few_m;
    return few_shape_ok(M, K, ldx, x, w, limit) && coheryn_gemm_tc_few_splits(N, K) == 1;
  }
  bool small_ok(int M, int N, int K, long ldx, const void* x, const void* w) const {
    return ((0 < M && M <= t.small_m) || (0 < M && M <= t.small_m_short && (long)N * K <= t.small_weight_elements)) &&
           operands_ok(K, ldx, x, w);
  }
  bool tc_ok(int M, int K, long ldx, const void* x, const void* w) const {
    return M > t.small_m && operands_ok(K, ldx, x, w);
  }
  // ops.linear: the route of y = x w^T and, for R_FEW_DEFER, the number of K slices.
  Route linear(int M, int N, int K, long ldx, const void* x, const void* w, bool partial_ok, int* splits) const {
    *splits = 1;
    if (partial_ok && M > 0 && K >= (M > t.small_m_short ? t.defer_min_k_wide : t.defer_min_k) &&
        few_shape_ok(M, K, ldx, x, w, t.few_defer_m)) {
      const int s = coheryn_gemm_tc_few_splits(N, K);
      if (s > 1) {
        *splits = s;
        return R_FEW_DEFER;
      }
    }
    if (few_ok(M, N, K, ldx, x, w)) return R_FEW;
    if (small_ok(M, N, K, ldx, x, w)) return R_SMALL;
    if (tc_ok(M, K, ldx, x, w)) return R_TC;
    return R_NONE;
  }
};

struct Arena {
  char* base;
  size_t off;
  void* workspace = nullptr;      // one area for the K slices of whichever many-rows product is running
  long workspace_floats = 0;
  void* take(size_t bytes) {
    off = (off + 255) & ~(size_t)255;
    void* p = base ? (void*)(base + off) : nullptr;
    off += bytes;
    return p;
  }
};

}  // namespace
