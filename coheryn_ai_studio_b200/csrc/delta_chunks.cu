// The gated delta rule for runs of many tokens, in chunks of 64 (float32 throughout).
//
// With g_t the decays of token t (per key channel), E_t their products from the chunk's first token on, S_0 the state in
// front of the chunk:
//
//   u_t = beta_t (v_t - (E_t k_t)^T S_0 - sum_{s < t} A_ts u_s),      A_ts = sum_d k_t k_s prod_{s < r <= t} g_r
//   o_t = (E_t q_t)^T S_0 + sum_{s <= t} B_ts u_s,                    B_ts likewise with q_t
//   S_C = diag(E_C) S_0 + sum_s (k_s prod_{s < r} g_r) u_s^T
//
// so U = T V - (T K~) S_0 with T = (I + diag(beta) strictly-lower(A))^-1 diag(beta) and K~ = E k.  Four kernels:
//
//   delta_chunk_kernel   a CTA per (chunk, head): A, B and the scaled q and k, into scratch;
//   delta_solve_kernel   a CTA per (chunk, head): T, W = T K~ and T V;
//   delta_state_kernel   a CTA per (request, head, 16 value channels): chunk after chunk U = T V - W S, S <- E_C S + K^ U;
//   delta_out_kernel     a CTA per (chunk, head): O = [Q~ | B] [S ; U] and the norm, weight and gate behind it.
//
// A value or key that is not finite makes the outputs of its whole chunk so, not only those from its token on (zeros of T and B
// times it); the state behind it is lost either way.
//
// All decays enter as products of the g between two tokens, over at most 16 tokens at a time and then over whole blocks of
// 16: no quotient and no exponent of a sum, so a decay of any strength is as exact as in the token-by-token scan.
//
// What bounds it: the scan token by token is a chain of dependent multiply-adds and shuffles, 0.55 us per token whatever the
// chip could do beside it.  Here the chain is two products of 64 x 128 x 16 per chunk; measured on a B200 (12 heads of 128 x
// 128, one request of 2,048 tokens) the four kernels take 264 us (70, 36, 100 and 58) in place of 1,150 us for the scan with its preparation.
//
// A run of fewer than CHUNK_FROM tokens is left to the scan (recurrent.cu), request by request: of the other requests only
// whether the step goes in chunks at all (recurrent.cu, coheryn_*_chunks_pay) can reach a row, not its order of additions.
#include "recurrent.cuh"

namespace {

constexpr int CH = CHUNK_TOKENS;     // tokens of a chunk
constexpr int BL = 16;               // tokens of a block inside it
constexpr int NP = CH + 4;           // pitch of the 64 x 64 matrices
constexpr int VS = 16;               // value channels per CTA of the state kernel
constexpr int THREADS = 256;

__device__ __forceinline__ void cp16(float* smem_dst, const float* src) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// Where the pieces of a (chunk, head) lie in the scratch.
template <int DK>
struct Piece {
  // K~ [64][DK] then W^T [DK][64], K^ [64][DK], [Q~^T ; B^T] [DK + 64][64], beta A [64][64], T V then U [64][dvp], S_0 [DK][dvp],
  // E_C [DK]
  float *wt, *kh, *qb, *n, *u, *s, *dec;
  __host__ __device__ static size_t floats(int dvp) { return (size_t)CH * DK * 3 + 2 * CH * CH + (size_t)(CH + DK) * dvp + DK; }
  __device__ Piece(float* scratch, size_t index, int dvp) {
    wt = scratch + index * floats(dvp);
    kh = wt + CH * DK;
    qb = kh + CH * DK;
    n = qb + (DK + CH) * CH;
    u = n + CH * CH;
    s = u + (size_t)CH * dvp;
    dec = s + (size_t)DK * dvp;
  }
};

// acc[0..3] rows la * 4 + i, acc[4..7] rows 32 + la * 4 + i of a 64-row product, TC neighbouring columns per thread:
// acc[t][c] += left[k][t] right[k][c].
template <int TC>
__device__ __forceinline__ void mac(float (&acc)[8][TC], const float* left, const float* right, bool low) {
  static_assert(TC == 2 || TC == 4, "");
  float b[TC];
  if (TC == 4) {
    const float4 x = ld4(right);
    b[0] = x.x; b[1] = x.y; b[2 % TC] = x.z; b[3 % TC] = x.w;
  } else {
    const float2 x = *reinterpret_cast<const float2*>(right);
    b[0] = x.x; b[1] = x.y;
  }
  if (low) {
    const float4 a = ld4(left);
#pragma unroll
    for (int c = 0; c < TC; ++c) {
      acc[0][c] = fmaf(a.x, b[c], acc[0][c]); acc[1][c] = fmaf(a.y, b[c], acc[1][c]);
      acc[2][c] = fmaf(a.z, b[c], acc[2][c]); acc[3][c] = fmaf(a.w, b[c], acc[3][c]);
    }
  }
  const float4 a = ld4(left + 32);
#pragma unroll
  for (int c = 0; c < TC; ++c) {
    acc[4][c] = fmaf(a.x, b[c], acc[4][c]); acc[5][c] = fmaf(a.y, b[c], acc[5][c]);
    acc[6][c] = fmaf(a.z, b[c], acc[6][c]); acc[7][c] = fmaf(a.w, b[c], acc[7][c]);
  }
}
template <int TC>
__device__ __forceinline__ void zero(float (&acc)[8][TC]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < TC; ++c) acc[i][c] = 0.f;
}
// Row of acc[i] of a thread whose lane group is la.
__device__ __forceinline__ int row_of(int i, int la) { return (i < 4 ? 0 : 32) + 4 * la + (i & 3); }

__device__ __forceinline__ void mac4(float (&acc)[4][4], const float4 a, const float4 b) {
  acc[0][0] = fmaf(a.x, b.x, acc[0][0]); acc[0][1] = fmaf(a.x, b.y, acc[0][1]); acc[0][2] = fmaf(a.x, b.z, acc[0][2]); acc[0][3] = fmaf(a.x, b.w, acc[0][3]);
  acc[1][0] = fmaf(a.y, b.x, acc[1][0]); acc[1][1] = fmaf(a.y, b.y, acc[1][1]); acc[1][2] = fmaf(a.y, b.z, acc[1][2]); acc[1][3] = fmaf(a.y, b.w, acc[1][3]);
  acc[2][0] = fmaf(a.z, b.x, acc[2][0]); acc[2][1] = fmaf(a.z, b.y, acc[2][1]); acc[2][2] = fmaf(a.z, b.z, acc[2][2]); acc[2][3] = fmaf(a.z, b.w, acc[2][3]);
  acc[3][0] = fmaf(a.w, b.x, acc[3][0]); acc[3][1] = fmaf(a.w, b.y, acc[3][1]); acc[3][2] = fmaf(a.w, b.z, acc[3][2]); acc[3][3] = fmaf(a.w, b.w, acc[3][3]);
}

// ---------------------------------------------------------------------------------
// A chunk of a head by itself: A, B and the scaled rows.  grid (chunks, heads).  A CTA keeps three tiles of 64 tokens by 64
// channels and takes 128 channels in two passes (everything here is by channel, except the norms of q and k, taken first, and
// the sums A and B, which go from pass to pass): three CTAs fit an SM.  With tiles of 128 channels two did, 384 CTAs were 1.3
// rounds of them and took 86 us (with the inverse and its products in the same kernel one CTA did, and took 163 us); every phase
// waits for shared memory, and warps are what hides that.  Measured on a B200 (2,048 tokens, 12 heads): 70 us.
// ---------------------------------------------------------------------------------
constexpr int CW = 64, CP = CW + 4;      // channels of a pass, pitch of its tiles
constexpr size_t CHUNK_SMEM = sizeof(float) * (3 * CH * CP + 4 * CW + 4 * CH + 2 * CH * 17);

template <int DK>
__global__ void __launch_bounds__(THREADS, 3) delta_chunk_kernel(DeltaIn P, int B, int base, float* __restrict__ scratch, int dvp) {
  constexpr int PASSES = DK / CW;
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                       // [64][CP] q, then q E
  float* Ks = Qs + CH * CP;             // [64][CP] k, then k E
  float* Gs = Ks + CH * CP;             // [64][CP] decays, then k times the decays behind it
  float* Dm = Gs + CH * CP;             // [4][CW] decay of a whole block
  float* betas = Dm + 4 * CW;           // [64]
  float* ones = betas + CH;             // [64] the decays of a head that has one for all its channels
  float* iqs = ones + CH;               // [64] what q and k are multiplied by
  float* iks = iqs + CH;
  float* As = iks + CH;                 // [64][17] the sums of A inside the blocks, of B
  float* Bs = As + CH * 17;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  co_pdl_wait();
  const int h = blockIdx.y, dk = P.dk;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) return;
  const int row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const int g = h / (P.heads / P.kv_heads);
  const float rate = expf(co_load_any(P.rate_log, P.rate_log_dtype, h));
  const bool per_head = P.decay_channels == 1;
  const Piece<DK> out(scratch, (size_t)blockIdx.x * P.heads + h, dvp);
  float* Nm = out.n;                    // [t][s] beta_t A_ts, written for s < t only
  float* Bt = out.qb + DK * CH;         // [s][t] B, transposed; zero for s > t

  // q and k become unit vectors (q also divided by sqrt(dk))
  const float q_scale = 1.0f / sqrtf((float)dk);
#pragma unroll 4
  for (int i = warp; i < CH; i += THREADS / 32) {
    float sq = 0.f, sk = 0.f;
    const size_t row = (size_t)(row0 + min(i, nt - 1)) * P.ld_qkv + (size_t)g * dk;
#pragma unroll
    for (int d = lane; d < DK; d += 32) {
      const float qv = d < dk ? P.q[row + d] : 0.f, kv = d < dk ? P.k[row + d] : 0.f;
      sq = fmaf(qv, qv, sq); sk = fmaf(kv, kv, sk);
    }
    sq = co_warp_sum(sq); sk = co_warp_sum(sk);
    if (lane == 0) { iqs[i] = q_scale / sqrtf(sq + 1e-6f); iks[i] = 1.0f / sqrtf(sk + 1e-6f); }
  }
  for (int e = tid; e < CH * CH; e += THREADS)
    if (e / CH > e % CH) Bt[e] = 0.f;
  if (tid < CH) {
    betas[tid] = tid < nt ? rc_sigmoid(P.beta[(size_t)(row0 + tid) * P.ld_beta + h]) : 0.f;
    if (per_head)
      ones[tid] = tid < nt ? expf(-rate * rc_softplus(P.step[(size_t)(row0 + tid) * P.ld_step + h] + co_load_any(P.step_bias, P.step_bias_dtype, h))) : 1.f;
  }
  __syncthreads();

  // between blocks i > j: a warp takes a pair of blocks, half of it the rows of k and half those of q, 4 x 4 a lane
  const int bi = warp < 1 ? 1 : (warp < 3 ? 2 : 3), bj = warp < 1 ? 0 : (warp < 3 ? warp - 1 : warp - 3);
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a) acc[a][0] = acc[a][1] = acc[a][2] = acc[a][3] = 0.f;

#pragma unroll 1
  for (int pass = 0; pass < PASSES; ++pass) {
    const int ch0 = pass * CW;
    if (pass) __syncthreads();          // the tiles of the pass before are stored
#pragma unroll 8
    for (int e = tid; e < CH * CW; e += THREADS) {
      const int i = e / CW, d = e % CW, ch = ch0 + d;
      float qv = 0.f, kv = 0.f, gv = 1.f;
      if (i < nt && ch < dk) {
        const size_t row = (size_t)(row0 + i);
        qv = P.q[row * P.ld_qkv + (size_t)g * dk + ch] * iqs[i];
        kv = P.k[row * P.ld_qkv + (size_t)g * dk + ch] * iks[i];
        if (!per_head) {
          const size_t sc = (size_t)h * dk + ch;
          gv = expf(-rate * rc_softplus(P.step[row * P.ld_step + sc] + co_load_any(P.step_bias, P.step_bias_dtype, sc)));
        }
      }
      Qs[i * CP + d] = qv; Ks[i * CP + d] = kv;
      Gs[i * CP + d] = per_head ? ones[i] : gv;
    }
    __syncthreads();
    // A and B inside the blocks of 16: eight lanes share a row, which walks back through its block with k_t and q_t decaying
    // token by token.  A warp takes a row of every block, then the row that makes all warps' walks equally long.
    {
      const int blk = lane >> 3, l8 = lane & 7;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        const int r = half ? 15 - warp : warp, t = BL * blk + r;
        float4 wk[2], wq[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) { wk[j] = ld4(Ks + t * CP + 32 * j + 4 * l8); wq[j] = ld4(Qs + t * CP + 32 * j + 4 * l8); }
        for (int s = r; s >= 0; --s) {
          const int row = BL * blk + s;
          float a = 0.f, b = 0.f;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (s < r) {
              const float4 gg = ld4(Gs + (row + 1) * CP + 32 * j + 4 * l8);
              wk[j].x *= gg.x; wk[j].y *= gg.y; wk[j].z *= gg.z; wk[j].w *= gg.w;
              wq[j].x *= gg.x; wq[j].y *= gg.y; wq[j].z *= gg.z; wq[j].w *= gg.w;
            }
            const float4 kk = ld4(Ks + row * CP + 32 * j + 4 * l8);
            a = fmaf(wk[j].x, kk.x, a); a = fmaf(wk[j].y, kk.y, a); a = fmaf(wk[j].z, kk.z, a); a = fmaf(wk[j].w, kk.w, a);
            b = fmaf(wq[j].x, kk.x, b); b = fmaf(wq[j].y, kk.y, b); b = fmaf(wq[j].z, kk.z, b); b = fmaf(wq[j].w, kk.w, b);
          }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
          if (l8 == 0) {
            if (pass) { a += As[t * 17 + s]; b += Bs[t * 17 + s]; }
            if (pass + 1 < PASSES) { As[t * 17 + s] = a; Bs[t * 17 + s] = b; }
            else {
              if (s < r) Nm[t * CH + row] = betas[t] * a;
              Bt[row * CH + t] = b;
            }
          }
        }
      }
    }
    __syncthreads();
    // Rows scaled inside their block: q and k by the decays up to and with their token, k also by those behind it.
    {
      const int d = tid % CW, blk = tid / CW, at = BL * blk * CP + d;
      float kr[BL], gr[BL];
#pragma unroll
      for (int r = 0; r < BL; ++r) { kr[r] = Ks[at + r * CP]; gr[r] = Gs[at + r * CP]; }
      float p = 1.f;
#pragma unroll
      for (int r = 0; r < BL; ++r) {
        p *= gr[r];
        Ks[at + r * CP] = kr[r] * p;
        Qs[at + r * CP] *= p;
      }
      Dm[blk * CW + d] = p;
      p = 1.f;
#pragma unroll
      for (int r = BL - 1; r >= 0; --r) { Gs[at + r * CP] = kr[r] * p; p *= gr[r]; }
    }
    __syncthreads();
    if (warp < 6) {
      const float* L = (lane < 16 ? Ks : Qs) + (BL * bi + ((lane >> 2) & 3)) * CP;      // rows +0, +4, +8, +12
      const float* Rt = Gs + (BL * bj + (lane & 3)) * CP;
      const float* d1 = Dm + (bj + 1) * CW;      // read where a block lies between the two
      const float* d2 = Dm + (bj + 2) * CW;
#pragma unroll 4
      for (int d = 0; d < CW; d += 4) {
        float4 x[4], y[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) { x[a] = ld4(L + 4 * a * CP + d); y[a] = ld4(Rt + 4 * a * CP + d); }
        if (bi - bj > 1) {
          float4 w = ld4(d1 + d);
          if (bi - bj > 2) { const float4 z = ld4(d2 + d); w.x *= z.x; w.y *= z.y; w.z *= z.z; w.w *= z.w; }
#pragma unroll
          for (int a = 0; a < 4; ++a) { y[a].x *= w.x; y[a].y *= w.y; y[a].z *= w.z; y[a].w *= w.w; }
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            acc[a][b] = fmaf(x[a].x, y[b].x, acc[a][b]); acc[a][b] = fmaf(x[a].y, y[b].y, acc[a][b]);
            acc[a][b] = fmaf(x[a].z, y[b].z, acc[a][b]); acc[a][b] = fmaf(x[a].w, y[b].w, acc[a][b]);
          }
      }
    }
    __syncthreads();
    // From the block to the chunk: q and k of block i by the decays of the blocks before it, the other k by those behind it.
    {
      const int d = tid % CW, blk = tid / CW, at = BL * blk * CP + d;
      float before = 1.f, behind = 1.f;
      for (int m = 0; m < blk; ++m) before *= Dm[m * CW + d];
      for (int m = blk + 1; m < 4; ++m) behind *= Dm[m * CW + d];
#pragma unroll
      for (int r = 0; r < BL; ++r) { Ks[at + r * CP] *= before; Qs[at + r * CP] *= before; Gs[at + r * CP] *= behind; }
    }
    __syncthreads();
#pragma unroll
    for (int e = tid; e < CH * CW / 4; e += THREADS) {
      const int t = e / (CW / 4), d = 4 * (e % (CW / 4));
      st4(out.kh + t * DK + ch0 + d, ld4(Gs + t * CP + d));
      st4(out.wt + t * DK + ch0 + d, ld4(Ks + t * CP + d));       // K~, which delta_solve_kernel replaces by W^T
    }
#pragma unroll
    for (int e = tid; e < CH * CW / 4; e += THREADS) {       // sixteen channels by two groups of four tokens per warp
      const int d = (e >> 1) % CW, t = 4 * ((e & 1) + 2 * (e / (2 * CW)));
      st4(out.qb + (ch0 + d) * CH + t, make_float4(Qs[t * CP + d], Qs[(t + 1) * CP + d], Qs[(t + 2) * CP + d], Qs[(t + 3) * CP + d]));
    }
    if (tid < CW) out.dec[ch0 + tid] = ((Dm[tid] * Dm[CW + tid]) * Dm[2 * CW + tid]) * Dm[3 * CW + tid];
  }
  if (warp < 6) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int t = BL * bi + ((lane >> 2) & 3) + 4 * a;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int s = BL * bj + (lane & 3) + 4 * b;
        if (lane < 16) Nm[t * CH + s] = betas[t] * acc[a][b];
        else Bt[s * CH + t] = acc[a][b];
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// T and its products with K~ and V.  grid (chunks, heads).
// ---------------------------------------------------------------------------------
template <int DK>
constexpr size_t solve_smem() { return sizeof(float) * (2 * CH * NP + CH * (DK + 4) + CH + 3 * BL * BL); }

template <int DK>
__global__ void __launch_bounds__(THREADS, 3) delta_solve_kernel(DeltaIn P, int B, int base, float* __restrict__ scratch, int dvp) {
  constexpr int DKP = DK + 4, TC = DK / 32;
  extern __shared__ __align__(16) float sm[];
  float* Nm = sm;                       // [t][s] beta_t A_ts, s < t
  float* Tt = Nm + CH * NP;             // [s][t] the inverse, transposed
  float* Ys = Tt + CH * NP;             // [64][DKP] K~, then tiles of v
  float* betas = Ys + CH * DKP;         // [64]
  float* Ms = betas + CH;               // [3][16][16]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  co_pdl_wait();
  const int h = blockIdx.y, dv = P.dv;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) return;
  const int row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const Piece<DK> out(scratch, (size_t)blockIdx.x * P.heads + h, dvp);
#pragma unroll
  for (int e = tid; e < CH * CH / 4; e += THREADS) {
    const int t = e / (CH / 4), s = 4 * (e % (CH / 4));
    float4 x = ld4(out.n + t * CH + s);
    x.x = s < t ? x.x : 0.f; x.y = s + 1 < t ? x.y : 0.f; x.z = s + 2 < t ? x.z : 0.f; x.w = s + 3 < t ? x.w : 0.f;
    st4(Nm + t * NP + s, x);
    st4(Tt + t * NP + s, make_float4(0.f, 0.f, 0.f, 0.f));
  }
#pragma unroll
  for (int e = tid; e < CH * DK / 4; e += THREADS) {
    const int t = e / (DK / 4), d = 4 * (e % (DK / 4));
    st4(Ys + t * DKP + d, ld4(out.wt + t * DK + d));
  }
  if (tid < CH) betas[tid] = tid < nt ? rc_sigmoid(P.beta[(size_t)(row0 + tid) * P.ld_beta + h]) : 0.f;
  __syncthreads();
  if (tid < CH) {
    // The inverses of the four 16 x 16 blocks on the diagonal: a lane takes a column.
    const int blk = tid >> 4, c = tid & 15;
    float x[BL];
#pragma unroll
    for (int r = 0; r < BL; ++r) x[r] = r == c ? 1.f : 0.f;
#pragma unroll
    for (int s = 0; s < BL; ++s)
#pragma unroll
      for (int r = s + 1; r < BL; ++r) x[r] = fmaf(-Nm[(BL * blk + r) * NP + BL * blk + s], x[s], x[r]);
#pragma unroll
    for (int r = 0; r < BL; r += 4) st4(Tt + (BL * blk + c) * NP + BL * blk + r, make_float4(x[r], x[r + 1], x[r + 2], x[r + 3]));
  }
  __syncthreads();
  // The inverse below its diagonal blocks, one distance after the other: T_ij = -T_ii sum_k N_ik T_kj.
#pragma unroll 1
  for (int dist = 1; dist < 4; ++dist) {
    const int a = tid >> 4, b = tid & 15;
    for (int i = dist; i < 4; ++i) {
      const int j = i - dist;
      float sum = 0.f;
      for (int x = BL * j; x < BL * i; x += 4) {
        const float4 n = ld4(Nm + (BL * i + a) * NP + x), t = ld4(Tt + (BL * j + b) * NP + x);
        sum = fmaf(n.x, t.x, sum); sum = fmaf(n.y, t.y, sum); sum = fmaf(n.z, t.z, sum); sum = fmaf(n.w, t.w, sum);
      }
      Ms[((i - dist) * BL + a) * BL + b] = sum;
    }
    __syncthreads();
    for (int i = dist; i < 4; ++i) {
      const int j = i - dist;
      float sum = 0.f;
#pragma unroll
      for (int x = 0; x < BL; ++x) sum = fmaf(Tt[(BL * i + x) * NP + BL * i + a], Ms[((i - dist) * BL + x) * BL + b], sum);
      Tt[(BL * j + b) * NP + BL * i + a] = -sum;
    }
    __syncthreads();
  }
  for (int e = tid; e < CH * CH; e += THREADS) Tt[(e / CH) * NP + e % CH] *= betas[e / CH];
  __syncthreads();

  const int la = lane >> 2, col = warp * 4 * TC + (lane & 3) * TC;
  float acc[8][TC];
  zero(acc);
#pragma unroll 4
  for (int s = 0; s < CH; ++s) mac<TC>(acc, Tt + s * NP + 4 * la, Ys + s * DKP + col, s < 32);
#pragma unroll
  for (int c = 0; c < TC; ++c) {
    st4(out.wt + (col + c) * CH + 4 * la, make_float4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]));
    st4(out.wt + (col + c) * CH + 32 + 4 * la, make_float4(acc[4][c], acc[5][c], acc[6][c], acc[7][c]));
  }
  for (int c0 = 0; c0 < dvp; c0 += DK) {
    __syncthreads();
#pragma unroll 8
    for (int e = tid; e < CH * DK; e += THREADS) {
      const int i = e / DK, c = e % DK;
      Ys[i * DKP + c] = i < nt && c0 + c < dv ? P.v[(size_t)(row0 + i) * P.ld_qkv + (size_t)h * dv + c0 + c] : 0.f;
    }
    __syncthreads();
    zero(acc);
#pragma unroll 4
    for (int s = 0; s < CH; ++s) mac<TC>(acc, Tt + s * NP + 4 * la, Ys + s * DKP + col, s < 32);
    if (c0 + col < dvp) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float* u = out.u + (size_t)row_of(i, la) * dvp + c0 + col;
#pragma unroll
        for (int c = 0; c < TC; c += 2) *reinterpret_cast<float2*>(u + c) = make_float2(acc[i][c], acc[i][c + 1]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// The chain over the chunks.  grid (ceil(dv / 16), heads, requests with chunks).  The products of 64 (or 128) rows by 16
// columns give each of sixteen warps 32 rows and a part of the sum (a slice of key channels, of tokens), 4 x 4 accumulators per
// thread; the parts are added through shared memory in a fixed order.
// ---------------------------------------------------------------------------------
template <int DK>
constexpr size_t state_smem() { return sizeof(float) * (2 * (2 * CH * DK + CH * VS + DK) + DK * VS + CH * VS + 8 * CH * VS); }
constexpr int STATE_THREADS = 512;
// Where a row of the parts lies: neighbouring groups of four rows swap odd and even, so that the eight lanes that store a
// 16-byte piece each of two such groups fall on all banks.
__device__ __forceinline__ int slot_of(int row) { return row ^ ((row >> 2) & 1); }

template <int DK>
__global__ void __launch_bounds__(STATE_THREADS, 1) delta_state_kernel(DeltaIn P, int B, int base, int count, float* __restrict__ scratch, int dvp) {
  constexpr int STAGE = 2 * CH * DK + CH * VS + DK;
  constexpr int DG = DK / 32, KG = 16 / DG;     // the update: warps over groups of 32 key channels, and over tokens
  extern __shared__ __align__(16) float sm[];
  float* S = sm + 2 * STAGE;                    // [DK][16]
  float* U = S + DK * VS;                       // [64][16]
  float* part = U + CH * VS;                    // [8][64][16], then [KG][DK][16]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  co_pdl_wait();
  const int h = blockIdx.y, c0 = blockIdx.x * VS, dk = P.dk, dv = P.dv;
  Run R;
  if (!find_run(P.cu_q, B, blockIdx.z, true, R)) return;
  // the run's chunks among the `count` that are worked on, from `base` on
  const int from = max(0, base - R.first), to = min((R.len + CH - 1) / CH, base + count - R.first);
  if (from >= to) return;
  float* state = P.state + (size_t)P.state_slots[R.r] * P.state_stride + (size_t)h * dk * dv;
  auto stage = [&](int c) {
    const Piece<DK> in(scratch, (size_t)(R.first + c - base) * P.heads + h, dvp);
    float* to = sm + (c & 1) * STAGE;
#pragma unroll 4
    for (int e = tid; e < 2 * CH * DK / 4; e += STATE_THREADS) cp16(to + 4 * e, in.wt + 4 * e);      // W^T and K^ are neighbours
    if (tid < CH * VS / 4) { const int t = tid >> 2, c4 = 4 * (tid & 3); cp16(to + 2 * CH * DK + t * VS + c4, in.u + (size_t)t * dvp + c0 + c4); }
    if (tid < DK / 4) cp16(to + 2 * CH * DK + CH * VS + 4 * tid, in.dec + 4 * tid);
    cp_commit();
  };
  stage(from);
  for (int e = tid; e < DK * VS; e += STATE_THREADS) {
    const int d = e / VS, c = c0 + e % VS;
    S[e] = d < dk && c < dv ? state[(size_t)d * dv + c] : 0.f;
  }
  const int la = lane >> 2, lb = 4 * (lane & 3);
  for (int c = from; c < to; ++c) {
    if (c + 1 < to) { stage(c + 1); cp_wait<1>(); }
    else cp_wait<0>();
    __syncthreads();
    const float* wt = sm + (c & 1) * STAGE;
    const float* kh = wt + CH * DK;
    const float* uv = kh + CH * DK;
    const float* dec = uv + CH * VS;
    const Piece<DK> out(scratch, (size_t)(R.first + c - base) * P.heads + h, dvp);
    for (int e = tid; e < DK * VS / 4; e += STATE_THREADS) st4(out.s + (size_t)(e >> 2) * dvp + c0 + 4 * (e & 3), ld4(S + 4 * e));
    {
      const int t = 32 * (warp & 1) + 4 * la, slice = warp >> 1;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
      for (int i = 0; i < DK / 8; ++i) {
        const int d = slice * (DK / 8) + i;
        mac4(acc, ld4(wt + d * CH + t), ld4(S + d * VS + lb));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) st4(part + (slice * CH + slot_of(t + i)) * VS + lb, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
    }
    __syncthreads();
    if (tid < CH * VS / 4) {
      const int t = tid >> 2, c4 = 4 * (tid & 3);
      float4 w = ld4(part + slot_of(t) * VS + c4);
#pragma unroll
      for (int p = 1; p < 8; ++p) {
        const float4 x = ld4(part + (p * CH + slot_of(t)) * VS + c4);
        w.x += x.x; w.y += x.y; w.z += x.z; w.w += x.w;
      }
      float4 u = ld4(uv + t * VS + c4);
      u.x -= w.x; u.y -= w.y; u.z -= w.z; u.w -= w.w;
      st4(U + t * VS + c4, u);
      st4(out.u + (size_t)t * dvp + c0 + c4, u);
    }
    __syncthreads();
    {
      const int d = 32 * (warp % DG) + 4 * la, kg = warp / DG;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
      for (int i = 0; i < CH / KG; ++i) {
        const int t = kg * (CH / KG) + i;
        mac4(acc, ld4(kh + t * DK + d), ld4(U + t * VS + lb));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) st4(part + (kg * DK + slot_of(d + i)) * VS + lb, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
    }
    __syncthreads();
    for (int e = tid; e < DK * VS / 4; e += STATE_THREADS) {
      const float f = dec[e >> 2];
      const int at = slot_of(e >> 2) * VS + 4 * (e & 3);
      float4 s = ld4(S + 4 * e), x = ld4(part + at);
#pragma unroll
      for (int p = 1; p < KG; ++p) {
        const float4 y = ld4(part + p * DK * VS + at);
        x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
      }
      s.x = fmaf(f, s.x, x.x); s.y = fmaf(f, s.y, x.y); s.z = fmaf(f, s.z, x.z); s.w = fmaf(f, s.w, x.w);
      st4(S + 4 * e, s);
    }
    __syncthreads();
  }
  for (int e = tid; e < DK * VS; e += STATE_THREADS) {
    const int d = e / VS, c = c0 + e % VS;
    if (d < dk && c < dv) state[(size_t)d * dv + c] = S[e];
  }
}

// ---------------------------------------------------------------------------------
// The outputs of a chunk of a head.  grid (chunks, heads), 8 x TC outputs per thread; both operands come in slices of 32 rows,
// two deep.  The finished rows lie where the slices lay when a head is one tile of columns: four CTAs per SM then, which is
// what hides the latency of the loads from shared memory (two CTAs of 128 threads with 8 x 8: 135 us where this takes 57 us).
// ---------------------------------------------------------------------------------
template <int TC>
size_t out_smem(int dvp) {
  const size_t stages = 2 * 32 * (CH + 32 * TC), rows = (size_t)CH * (dvp + 4);
  return sizeof(float) * (dvp <= 32 * TC ? (stages > rows ? stages : rows) : stages + rows);
}

template <int DK, int TC>
__global__ void __launch_bounds__(THREADS) delta_out_kernel(DeltaIn P, HeadOut E, int B, int base, float* __restrict__ scratch, int dvp) {
  constexpr int W = 32 * TC, SL = 32, STAGE = SL * (CH + W), SLICES = (DK + CH) / SL;
  extern __shared__ __align__(16) float sm[];
  float* os = dvp <= W ? sm : sm + 2 * STAGE;   // [64][dvp + 4]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  co_pdl_wait();
  const int h = blockIdx.y;
  Run R;
  if (!find_run(P.cu_q, B, base + blockIdx.x, false, R)) return;
  const int row0 = R.start + R.chunk * CH, nt = min(CH, R.len - R.chunk * CH);
  const Piece<DK> in(scratch, (size_t)blockIdx.x * P.heads + h, dvp);
  const int la = lane >> 2, col = warp * 4 * TC + (lane & 3) * TC;
  for (int c0 = 0; c0 < dvp; c0 += W) {
    auto stage = [&](int i) {
      float* to = sm + (i & 1) * STAGE;
#pragma unroll
      for (int e = tid; e < SL * CH / 4; e += THREADS) cp16(to + 4 * e, in.qb + i * SL * CH + 4 * e);
      const float* rows = i * SL < DK ? in.s + (size_t)i * SL * dvp : in.u + (size_t)(i * SL - DK) * dvp;
#pragma unroll
      for (int e = tid; e < SL * W / 4; e += THREADS) {
        const int k = e / (W / 4), c = 4 * (e % (W / 4));
        if (c0 + c < dvp) cp16(to + SL * CH + k * W + c, rows + (size_t)k * dvp + c0 + c);
      }
      cp_commit();
    };
    float acc[8][TC];
    zero(acc);
    if (c0) __syncthreads();
    stage(0);
    for (int i = 0; i < SLICES; ++i) {
      if (i + 1 < SLICES) { stage(i + 1); cp_wait<1>(); }
      else cp_wait<0>();
      __syncthreads();
      const float* left = sm + (i & 1) * STAGE + 4 * la;
      const float* right = sm + (i & 1) * STAGE + SL * CH + col;
      const bool low = i * SL < DK + 32;        // tokens 32.. of U do not reach the first half of the rows
#pragma unroll 8
      for (int k = 0; k < SL; ++k) mac<TC>(acc, left + k * CH, right + k * W, low);
      __syncthreads();
    }
    if (c0 + col < dvp) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float* o = os + row_of(i, la) * (dvp + 4) + c0 + col;
#pragma unroll
        for (int c = 0; c < TC; c += 2) *reinterpret_cast<float2*>(o + c) = make_float2(acc[i][c], acc[i][c + 1]);
      }
    }
  }
  __syncthreads();
  head_out_chunk(E, os, dvp + 4, P.dv, nt, row0, h);
}

int padded(int dv) { return (dv + VS - 1) / VS * VS; }

template <int DK>
int launch(const DeltaIn& P, const HeadOut& E, int B, int chunks, int runs, float* scratch, cudaStream_t stream) {
  const int dvp = padded(P.dv), at_once = chunks_at_once(P.heads * Piece<DK>::floats(dvp));
  auto out = dvp <= 64 ? delta_out_kernel<DK, 2> : delta_out_kernel<DK, 4>;
  const size_t smem = dvp <= 64 ? out_smem<2>(dvp) : out_smem<4>(dvp);
  cudaFuncSetAttribute(delta_chunk_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CHUNK_SMEM);
  cudaFuncSetAttribute(delta_solve_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve_smem<DK>());
  cudaFuncSetAttribute(delta_state_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)state_smem<DK>());
  cudaFuncSetAttribute(out, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  for (int base = 0; base < chunks; base += at_once) {
    const int count = chunks - base < at_once ? chunks - base : at_once;
    co_launch(delta_chunk_kernel<DK>, dim3(count, P.heads), dim3(THREADS), CHUNK_SMEM, stream, P, B, base, scratch, dvp);
    CO_CHECK_LAUNCH("delta_chunk");
    co_launch(delta_solve_kernel<DK>, dim3(count, P.heads), dim3(THREADS), solve_smem<DK>(), stream, P, B, base, scratch, dvp);
    CO_CHECK_LAUNCH("delta_solve");
    co_launch(delta_state_kernel<DK>, dim3(dvp / VS, P.heads, runs), dim3(STATE_THREADS), state_smem<DK>(), stream, P, B, base, count, scratch, dvp);
    CO_CHECK_LAUNCH("delta_state");
    co_launch(out, dim3(count, P.heads), dim3(THREADS), smem, stream, P, E, B, base, scratch, dvp);
    CO_CHECK_LAUNCH("delta_out");
  }
  return 0;
}

}  // namespace

// Up to 128 key channels the state kernel's stages fit an SM; beyond that the scan stays.
bool co_delta_chunks_take(int dk, int dv) { return dk >= 1 && dk <= 128 && dv >= 1 && dv <= 256; }

long co_delta_chunk_floats(int chunks, int heads, int dk, int dv) {
  const size_t each = heads * (dk <= 64 ? Piece<64>::floats(padded(dv)) : Piece<128>::floats(padded(dv)));
  const int at_once = chunks_at_once(each);
  return (long)((size_t)(chunks < at_once ? chunks : at_once) * each);
}

int co_delta_chunks(const DeltaIn& P, const HeadOut& E, int B, int chunks, int runs, float* scratch, cudaStream_t stream) {
  return P.dk <= 64 ? launch<64>(P, E, B, chunks, runs, scratch, stream) : launch<128>(P, E, B, chunks, runs, scratch, stream);
}
