// The gated delta rule (see recurrent.cu) for portions of many tokens, 64 tokens at a time.  Inside a chunk, with L_t the
// running sum of log decays, k and q scaled to unit length and S the state before the chunk:
//     u_t = beta_t (v_t - e^(L_t) S^T k_t - sum_{i<t} e^(L_t - L_i) (k_t . k_i) u_i)        a triangular system
//     o_t = e^(L_t) S^T q_t + sum_{i<=t} e^(L_t - L_i) (q_t . k_i) u_i
//     S  <- e^(L_end) S + sum_i e^(L_end - L_i) k_i u_i^T
// Everything that does not know S is worked out for all chunks side by side (delta_chunk_prepare: the system solved for its
// two right sides, U = WV - WK S, and the factors of the other two lines); what is left of the serial walk is U and the state's own line, two
// small products a chunk (delta_chunk_walk, which leaves every chunk's U and first state behind); the outputs are again worked out for
// all chunks side by side (delta_chunk_outputs).  All of it float32 multiply-adds; the running sums are kept in 64 bits, because a
// difference of two of them is the exponent of a decay.  A portion with an input that is no finite number (or whose length
// squared is none) is walked token by token instead: in the products it would reach its chunk's earlier tokens, as 0 times it.
//
// The token-by-token walk is bound by the latency of its chain, 0.36 us a token at heads of 128 x 128: 738 us for
// 2,048 tokens, whatever the number of SMs.  Here 8 heads of that size take 40 us (prepare: the chains of the 64 x 64 systems,
// two blocks an SM), 61 us (walk: 32 dependent chunks, 128 blocks, one an SM) and 27 us (outputs); with the outputs in the walk and copies of 16
// bytes that took 124 us.  The error against 64 bits is the walk's or less.
#include "long_portions.cuh"
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

namespace ptl {

constexpr int kDcTokens = 64, kDcThreads = 256, kDcCols = 8;
constexpr int kDcSysLd = kDcTokens + 4;

__device__ __forceinline__ float dc_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// A (chunk, head) in the workspace: WK [64][D + 4] and the decayed keys [D][68] (rows as the walk wants them in shared memory, so that a
// chunk is one run of bytes), the decayed queries and the read-out's weights side by side [64][D + 64], WV [64][dv], the chunk's decay, 1 where an
// input is not finite, 1 where the portion was walked token by token (padded to 16 bytes), and by columns what the outputs are made
// of, the state before the chunk and U: [dv][D + 64].
__host__ __device__ constexpr size_t dc_keys_at(int D) { return (size_t)kDcTokens * (D + 4); }
__host__ __device__ constexpr size_t dc_walk_floats(int D) { return dc_keys_at(D) + (size_t)D * kDcSysLd; }
__host__ __device__ constexpr size_t dc_values_at(int D) { return dc_walk_floats(D) + (size_t)kDcTokens * (D + kDcTokens); }
__host__ __device__ constexpr size_t dc_flags_at(int D, int dv) { return dc_values_at(D) + (size_t)kDcTokens * dv; }
__host__ __device__ constexpr size_t dc_columns_at(int D, int dv) { return dc_flags_at(D, dv) + 4; }
__host__ __device__ constexpr size_t dc_floats(int D, int dv) { return dc_columns_at(D, dv) + (size_t)(D + kDcTokens) * dv; }
constexpr size_t dc_prepare_smem(int D) { return sizeof(float) * (2 * kDcTokens * (D + 4) + kDcTokens * kDcSysLd); }
constexpr size_t dc_walk_smem(int D) {
  return sizeof(float) * (2 * dc_walk_floats(D) + kDcCols * (D + 4) + kDcCols * kDcSysLd) + 32;
}
constexpr int kDcOutCols = 64;                     // columns of a block of the outputs
constexpr size_t dc_outputs_smem(int D) { return sizeof(float) * (kDcTokens + kDcOutCols) * (D + kDcTokens + 4) + 16; }

// Bound by its multiply-adds (2.1 M a chunk and head of 128 x 128) and the 64 steps of the substitution, a column per thread
// held in registers, which update all later rows at once.
template <typename T, int D>
__global__ void __launch_bounds__(kDcThreads, 2)
delta_chunk_prepare_kernel(float* __restrict__ work, const T* __restrict__ qkv, const float* __restrict__ ba, const float* __restrict__ rate,
                           const float* __restrict__ dt_bias, const int* __restrict__ q_start, const int* __restrict__ state_slot,
                           int requests, int heads, int kv_heads, int dv, float unit_eps, float q_scale, int walk_max) {
  constexpr int LD = D + 4;
  extern __shared__ __align__(16) float dp_smem[];
  float* s_k = dp_smem;                            // [64][LD], as projected: the lengths are applied to what is made of them,
  float* s_q = s_k + kDcTokens * LD;               // [64][LD]  which is then rounded once
  float* s_sys = s_q + kDcTokens * LD;             // [i][t]: what u_i takes off row t > i
  __shared__ double s_log[kDcTokens];
  __shared__ float s_beta[kDcTokens], s_decay[kDcTokens], s_kn[kDcTokens], s_qn[kDcTokens];
  __shared__ int s_at[2];
  pdl_wait();
  pdl_launch_dependents();
  const LongPortion at = locate_portion<false, kDcTokens>(q_start, requests, walk_max, blockIdx.x);
  if (at.r < 0 || state_slot[at.r] < 0) return;
  const int first = ((int)blockIdx.x - at.piece0) * kDcTokens, row0 = at.lo + first;
  const int h = blockIdx.y, c = h / (heads / kv_heads), n = min(kDcTokens, at.n - first);
  if (threadIdx.x == 0) { s_at[0] = row0; s_at[1] = n; }       // (for the values' turn, which has no register to spare)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ld = 2 * kv_heads * D + heads * dv;
  const T* rows = qkv + (size_t)row0 * ld;
  float* wk = work + ((size_t)blockIdx.x * heads + h) * dc_floats(D, dv);
  float* kdt = wk + dc_keys_at(D);
  float* qg = wk + dc_walk_floats(D);
  constexpr int LQ = D + kDcTokens;
  float* mix = qg + D;
  float* wv = wk + dc_values_at(D);
  // q and k of a token per warp and turn; rows past the portion are zero throughout
  for (int t = warp; t < kDcTokens; t += kDcThreads / 32) {
    float q[D / 32], k[D / 32], qq = 0.f, kk = 0.f;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) {
      q[i] = t < n ? to_f32(rows[(size_t)t * ld + c * D + lane + 32 * i]) : 0.f;
      k[i] = t < n ? to_f32(rows[(size_t)t * ld + (kv_heads + c) * D + lane + 32 * i]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < D / 32; ++i) { qq = fmaf(q[i], q[i], qq); kk = fmaf(k[i], k[i], kk); }
    qq = warp_sum(qq);
    kk = warp_sum(kk);
    if (lane == 0) {
      s_qn[t] = t < n ? q_scale / sqrtf(qq + unit_eps) : 0.f;
      s_kn[t] = t < n ? 1.0f / sqrtf(kk + unit_eps) : 0.f;
      if (!isfinite(qq + kk)) s_kn[t] = NAN;       // (a length of infinity would pass as a factor of zero)
    }
#pragma unroll
    for (int i = 0; i < D / 32; ++i) {
      s_q[t * LD + lane + 32 * i] = q[i];
      s_k[t * LD + lane + 32 * i] = k[i];
    }
  }
  if (warp == 0) {
    double run = 0.0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int t = lane + 32 * half;
      double x = 0.0;
      float beta = 0.f;
      if (t < n) {
        const float* g = ba + (size_t)(row0 + t) * 2 * heads;
        beta = 1.0f / (1.0f + expf(-g[h]));
        x = (double)(-rate[h] * dc_softplus(g[heads + h] + dt_bias[h]));
        if (x < -1e4) x = -1e4;                    // a decay of zero either way; differences of the sums stay numbers
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double before = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += before;
      }
      x += run;
      run = __shfl_sync(0xffffffffu, x, 31);
      s_log[t] = x;
      s_beta[t] = beta;
      s_decay[t] = expf((float)x);
    }
  }
  __syncthreads();
  {
    // k_t . k_i and q_t . k_i, four by four per thread
    const int tx = tid & 15, ty = tid >> 4;
    float kk[4][4], qk[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) { kk[a][b] = 0.f; qk[a][b] = 0.f; }
#pragma unroll 1
    for (int e0 = 0; e0 < D; e0 += 16) {       // sixteen products a chain, the chains' sums added up: shorter chains round less
      float k16[4][4], q16[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) { k16[a][b] = 0.f; q16[a][b] = 0.f; }
#pragma unroll 2
      for (int e = e0; e < e0 + 16; e += 4) {
        float4 col[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) col[b] = *reinterpret_cast<const float4*>(s_k + (tx + 16 * b) * LD + e);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float4 kt = *reinterpret_cast<const float4*>(s_k + (ty + 16 * a) * LD + e);
          const float4 qt = *reinterpret_cast<const float4*>(s_q + (ty + 16 * a) * LD + e);
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            k16[a][b] = fmaf(kt.x, col[b].x, fmaf(kt.y, col[b].y, fmaf(kt.z, col[b].z, fmaf(kt.w, col[b].w, k16[a][b]))));
            q16[a][b] = fmaf(qt.x, col[b].x, fmaf(qt.y, col[b].y, fmaf(qt.z, col[b].z, fmaf(qt.w, col[b].w, q16[a][b]))));
          }
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) { kk[a][b] += k16[a][b]; qk[a][b] += q16[a][b]; }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int t = ty + 16 * a, i = tx + 16 * b;
        const float decay = i <= t ? expf((float)(s_log[t] - s_log[i])) : 0.f;
        s_sys[i * kDcSysLd + t] = i < t ? s_beta[t] * decay * (s_kn[t] * s_kn[i]) * kk[a][b] : 0.f;
        mix[t * LQ + i] = i <= t ? decay * (s_qn[t] * s_kn[i]) * qk[a][b] : 0.f;
      }
  }
  const double end = s_log[kDcTokens - 1];
  for (int i = tid; i < kDcTokens * D; i += kDcThreads) {
    const int t = i / D, e = i % D;
    qg[t * LQ + e] = s_decay[t] * s_qn[t] * s_q[t * LD + e];
    const int t2 = i % kDcTokens, e2 = i / kDcTokens;
    kdt[e2 * kDcSysLd + t2] = expf((float)(end - s_log[t2])) * s_kn[t2] * s_k[t2 * LD + e2];
  }
  __syncthreads();
  bool finite = tid >= kDcTokens || (isfinite(s_kn[tid] + s_qn[tid] + s_beta[tid]) && !isnan(s_log[tid]));
  for (int col = tid; col < D + dv; col += kDcThreads) {
    float u[kDcTokens];
    if (col < D) {
#pragma unroll
      for (int t = 0; t < kDcTokens; ++t) u[t] = s_beta[t] * s_decay[t] * s_kn[t] * s_k[t * LD + col];
    } else {
      const T* v = qkv + (size_t)s_at[0] * ld + 2 * kv_heads * D + (size_t)h * dv + (col - D);
      const int tokens = s_at[1];
#pragma unroll
      for (int t = 0; t < kDcTokens; ++t) {
        const float x = t < tokens ? to_f32(v[(size_t)t * ld]) : 0.f;
        finite = finite && isfinite(x);
        u[t] = s_beta[t] * x;
      }
    }
#pragma unroll
    for (int i = 0; i < kDcTokens - 1; ++i) {
      asm volatile("" ::: "memory");               // (a row's loads are not all moved ahead: two blocks per SM need the registers)
#pragma unroll
      for (int t4 = (i + 1) & ~3; t4 < kDcTokens; t4 += 4) {      // (rows up to i have a zero there)
        const float4 a = *reinterpret_cast<const float4*>(s_sys + i * kDcSysLd + t4);
        u[t4] = t4 > i ? fmaf(-a.x, u[i], u[t4]) : u[t4];
        u[t4 + 1] = t4 + 1 > i ? fmaf(-a.y, u[i], u[t4 + 1]) : u[t4 + 1];
        u[t4 + 2] = t4 + 2 > i ? fmaf(-a.z, u[i], u[t4 + 2]) : u[t4 + 2];
        u[t4 + 3] = fmaf(-a.w, u[i], u[t4 + 3]);
      }
    }
    float* dst = col < D ? wk + col : wv + (col - D);
    const int step = col < D ? LD : dv;
#pragma unroll
    for (int t = 0; t < kDcTokens; ++t) dst[(size_t)t * step] = u[t];
  }
  const int bad = __syncthreads_or(!finite);
  if (tid == 0) {
    wk[dc_flags_at(D, dv)] = s_decay[kDcTokens - 1];
    wk[dc_flags_at(D, dv) + 1] = bad ? 1.f : 0.f;
  }
}

// Eight columns of one head's state per block.  Eight lanes share a row of a product: lane s takes the entries 4 s .. 4 s + 3 of
// every 32 (a quarter warp reads 128 bytes of one row, the state's column packets are the same for the whole warp) against
// all eight columns, and the lanes' sums meet by halves, so that lane s ends up with column s.  The next chunk's WK and decayed keys
// are on their way while a chunk is worked.  Bound by the chain of the two products and by L2: 64 KB a chunk and block.
template <int ROWS>
__device__ __forceinline__ void dc_meet(float (&acc)[ROWS][kDcCols], int s, float (&sum)[ROWS]) {
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    float h4[4], h2[2];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float mine = s & 4 ? acc[j][c + 4] : acc[j][c], theirs = s & 4 ? acc[j][c] : acc[j][c + 4];
      h4[c] = mine + __shfl_xor_sync(0xffffffffu, theirs, 4);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float mine = s & 2 ? h4[c + 2] : h4[c], theirs = s & 2 ? h4[c] : h4[c + 2];
      h2[c] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2);
    }
    const float mine = s & 1 ? h2[1] : h2[0], theirs = s & 1 ? h2[0] : h2[1];
    sum[j] = mine + __shfl_xor_sync(0xffffffffu, theirs, 1);
  }
}

template <int ROWS, int K, int LDA, int LDB>
__device__ __forceinline__ void dc_product(const float* __restrict__ a, const float* __restrict__ b, int s, float (&sum)[ROWS]) {
  float2 acc[ROWS][kDcCols];                        // sums of even and of odd entries
#pragma unroll
  for (int j = 0; j < ROWS; ++j)
#pragma unroll
    for (int c = 0; c < kDcCols; ++c) acc[j][c] = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < K; k += 32) {
    float4 x[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) x[j] = *reinterpret_cast<const float4*>(a + 32 * j * LDA + k + 4 * s);
#pragma unroll
    for (int c = 0; c < kDcCols; ++c) {
      const float4 y = *reinterpret_cast<const float4*>(b + c * LDB + k + 4 * s);
#pragma unroll
      for (int j = 0; j < ROWS; ++j) {
        acc[j][c] = fma2(make_float2(x[j].x, x[j].y), make_float2(y.x, y.y), acc[j][c]);
        acc[j][c] = fma2(make_float2(x[j].z, x[j].w), make_float2(y.z, y.w), acc[j][c]);
      }
    }
  }
  float both[ROWS][kDcCols];
#pragma unroll
  for (int j = 0; j < ROWS; ++j)
#pragma unroll
    for (int c = 0; c < kDcCols; ++c) both[j][c] = acc[j][c].x + acc[j][c].y;
  dc_meet<ROWS>(both, s, sum);
}

// The tokens of a portion one by one, for the eight columns of the state in shared memory (`scratch`: 2 D + 128 floats): the
// walk's own steps (recurrent.cu).  Rare, so that its speed does not matter.
template <typename T, int D>
__device__ __noinline__ void dc_walk_tokens(float* __restrict__ out, const T* __restrict__ rows, const float* __restrict__ ba, int tokens,
                                            float rate, float dt_bias, int heads, int kv_heads, int dv, int h, int j0, float unit_eps,
                                            float q_scale, float* s_s, float* scratch) {
  constexpr int LD = D + 4;
  float *s_q = scratch, *s_k = scratch + D, *s_part = scratch + 2 * D;      // [2][8 warps][8 columns]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = tid & 7, e0 = tid >> 3;       // column, first entry of every 32nd
  const int ld = 2 * kv_heads * D + heads * dv, head = h / (heads / kv_heads);
  for (int t = 0; t < tokens; ++t) {
    const T* row = rows + (size_t)t * ld;
    __syncthreads();
    for (int e = tid; e < 2 * D; e += kDcThreads) scratch[e] = to_f32(e < D ? row[head * D + e] : row[(kv_heads + head) * D + e - D]);
    __syncthreads();
    float qq = 0.f, kk = 0.f;
    for (int e = lane; e < D; e += 32) { qq = fmaf(s_q[e], s_q[e], qq); kk = fmaf(s_k[e], s_k[e], kk); }
    const float qn = q_scale / sqrtf(warp_sum(qq) + unit_eps), kn = 1.0f / sqrtf(warp_sum(kk) + unit_eps);
    const float* gates = ba + (size_t)t * 2 * heads;
    const float beta = 1.0f / (1.0f + expf(-gates[h])), g = expf(-rate * dc_softplus(gates[heads + h] + dt_bias));
    auto over_entries = [&](float v, int which) {                 // a column's sum over the block
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (lane < 8) s_part[which * 64 + warp * 8 + c] = v;
      __syncthreads();
      float sum = 0.f;
      for (int w = 0; w < 8; ++w) sum += s_part[which * 64 + w * 8 + c];
      return sum;
    };
    float part = 0.f;
    for (int e = e0; e < D; e += 32) {
      s_s[c * LD + e] *= g;
      part = fmaf(s_s[c * LD + e], s_k[e], part);
    }
    const float u = beta * (to_f32(row[2 * kv_heads * D + h * dv + j0 + c]) - kn * over_entries(part, 0)) * kn;
    part = 0.f;
    for (int e = e0; e < D; e += 32) {
      s_s[c * LD + e] = fmaf(s_k[e], u, s_s[c * LD + e]);
      part = fmaf(s_s[c * LD + e], s_q[e], part);
    }
    const float o = over_entries(part, 1) * qn;
    if (tid < 8) out[((size_t)t * heads + h) * dv + j0 + c] = o;
  }
}

template <typename T, int D>
__global__ void __launch_bounds__(kDcThreads, 1)
delta_chunk_walk_kernel(float* __restrict__ out, float* __restrict__ state, float* work, const T* __restrict__ qkv,
                        const float* __restrict__ ba, const float* __restrict__ rate, const float* __restrict__ dt_bias, int kv_heads,
                        float unit_eps, float q_scale, const int* __restrict__ q_start, const int* __restrict__ positions,
                        const int* __restrict__ state_slot, int requests, int heads, int dv, int walk_max, int* status, CopyWaits waits) {
  constexpr int LD = D + 4, RB = D / 32;
  extern __shared__ __align__(16) float dw_smem[];
  constexpr int kChunk = (int)dc_walk_floats(D);
  float* s_c = dw_smem;                                  // [2][WK 64 rows of LD | keys D rows of 68]
  float* s_s = s_c + 2 * kChunk;                         // [8][LD]: the state's columns
  float* s_u = s_s + kDcCols * LD;                       // [8][68]
  // before the wait only the step's own integers, which the kernel before this one reads too; no block leaves before it
  const LongPortion at = locate_portion<true, kDcTokens>(q_start, requests, walk_max, blockIdx.z);
  const int slot = at.r < 0 ? -1 : state_slot[at.r];
  const int lo = at.lo, n = at.n, chunk0 = at.piece0, h = blockIdx.y, j0 = blockIdx.x * kDcCols;
  const int chunks = (n + kDcTokens - 1) / kDcTokens;
  const int tid = threadIdx.x, lane = tid & 31, s = lane & 7, rg = (tid >> 5) * 4 + (lane >> 3);
  const size_t stride = (size_t)heads * dc_floats(D, dv);
  float* base = work + ((size_t)chunk0 * heads + h) * dc_floats(D, dv);
  float* st = state + (((size_t)slot * heads + h) * D) * dv + j0;
  const bool from_zero = slot >= 0 && positions[lo] == 0;
  // one bulk copy a chunk (as copies of 16 bytes, 17 a thread, issuing them took 1,140 of a chunk's 4,400 cycles)
  const uint32_t full = smem_u32(s_u + kDcCols * kDcSysLd);
  volatile int* const abort_flag = reinterpret_cast<volatile int*>(s_u + kDcCols * kDcSysLd + 4);
  if (tid == 0) {
    mbar_init(full, 1);
    mbar_init(full + 8, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();
  pdl_launch_dependents();
  if (slot < 0) return;
  auto fetch = [&](int chunk) {
    if (tid != 0 || chunk == waits.withheld) return;
    const uint32_t bar = full + 8 * (chunk & 1);
    mbar_expect_tx(bar, kChunk * 4);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(s_c + (chunk & 1) * kChunk)), "l"(base + chunk * stride), "r"(kChunk * 4), "r"(bar) : "memory");
  };
  // Waits for a chunk, the whole block.  One that does not come ends the walk with the status set: nothing else is in flight then, and the
  // state in memory stays what it was.
  auto here = [&](int chunk) {
    const uint32_t bar = full + 8 * (chunk & 1), parity = chunk >> 1 & 1;
    const bool came = mbar_wait(bar, parity, abort_flag, status, 31, waits.polls);
    const bool lost = __syncthreads_or(!came);
    if (lost && tid == 0) mbar_drain(bar, parity);
    return !lost;
  };
  fetch(0);
  for (int i = tid; i < D * kDcCols; i += kDcThreads) {
    const int e = i / kDcCols, c = i % kDcCols;
    s_s[c * LD + e] = from_zero ? 0.f : st[(size_t)e * dv + c];
  }
  bool bad = false;
  for (int i = tid; i < chunks; i += kDcThreads) bad = bad || base[i * stride + dc_flags_at(D, dv) + 1] != 0.f;
  const bool walk = __syncthreads_or(bad);
  if (blockIdx.x == 0)
    for (int i = tid; i < chunks; i += kDcThreads) base[i * stride + dc_flags_at(D, dv) + 2] = walk ? 1.f : 0.f;
  if (walk) {
    if (!here(0)) return;                  // (the tokens' walk takes the chunk's place)
    dc_walk_tokens<T, D>(out + (size_t)lo * heads * dv, qkv + (size_t)lo * (2 * kv_heads * D + heads * dv), ba + (size_t)lo * 2 * heads, n,
                         rate[h], dt_bias[h], heads, kv_heads, dv, h, j0, unit_eps, q_scale, s_s, s_c);
  }
  for (int chunk = walk ? chunks : 0; chunk < chunks; ++chunk) {
    const float* wv = base + chunk * stride + dc_values_at(D);
    float* columns = base + chunk * stride + dc_columns_at(D, dv) + (size_t)j0 * (D + kDcTokens);
    const float v0 = wv[(size_t)rg * dv + j0 + s], v1 = wv[(size_t)(rg + 32) * dv + j0 + s], decay = wv[(size_t)kDcTokens * dv];
    if (!here(chunk)) return;              // this chunk is here; the chunk before has been read and its state written
    if (chunk + 1 < chunks) fetch(chunk + 1);
    float first[2];
    dc_product<2, D, LD, LD>(s_c + (chunk & 1) * kChunk + rg * LD, s_s, s, first);
    s_u[s * kDcSysLd + rg] = v0 - first[0];
    s_u[s * kDcSysLd + rg + 32] = v1 - first[1];
    if (tid < D * kDcCols / 4) {           // the state before the chunk, for the outputs
      const int c = tid / (D / 4), e = tid % (D / 4) * 4;
      *reinterpret_cast<float4*>(columns + (size_t)c * (D + kDcTokens) + e) = *reinterpret_cast<const float4*>(s_s + c * LD + e);
    }
    __syncthreads();                       // U is whole, and everyone has read the state
    float second[RB];
    dc_product<RB, kDcTokens, kDcSysLd, kDcSysLd>(s_c + (chunk & 1) * kChunk + dc_keys_at(D) + rg * kDcSysLd, s_u, s, second);
    if (tid < kDcTokens * kDcCols / 4) {
      const int c = tid / (kDcTokens / 4), e = tid % (kDcTokens / 4) * 4;
      *reinterpret_cast<float4*>(columns + (size_t)c * (D + kDcTokens) + D + e) = *reinterpret_cast<const float4*>(s_u + c * kDcSysLd + e);
    }
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      float* e = s_s + s * LD + rg + 32 * j;
      *e = fmaf(decay, *e, second[j]);
    }
  }
  __syncthreads();
  for (int i = tid; i < D * kDcCols; i += kDcThreads) {
    const int e = i / kDcCols, c = i % kDcCols;
    st[(size_t)e * dv + c] = s_s[c * LD + e];
  }
}

// A chunk's outputs, 64 columns a block: [queries | read-out weights] times [the state before the chunk; U], four rows by four columns a
// thread, sums of 32 terms added up (shorter chains round less).  Bound by the multiply-adds.
template <int D>
__global__ void __launch_bounds__(kDcThreads, 2)
delta_chunk_outputs_kernel(float* __restrict__ out, const float* __restrict__ work, const int* __restrict__ q_start, const int* __restrict__ state_slot,
                           int requests, int heads, int dv, int walk_max, int* status, CopyWaits waits) {
  constexpr int K = D + kDcTokens, LA = K + 4;
  extern __shared__ __align__(16) float do_smem[];
  float* s_a = do_smem;                                  // [64 tokens][queries D | weights 64]
  float* s_b = s_a + kDcTokens * LA;                     // [64 columns][state D | U 64]
  // (before the wait as in the walk)
  const LongPortion at = locate_portion<false, kDcTokens>(q_start, requests, walk_max, blockIdx.x);
  const bool there = at.r >= 0 && state_slot[at.r] >= 0;
  const int first = ((int)blockIdx.x - at.piece0) * kDcTokens, h = blockIdx.y, n = min(kDcTokens, at.n - first), j0 = blockIdx.z * kDcOutCols;
  const int cols = min(kDcOutCols, dv - j0), tid = threadIdx.x;
  // (a warp is four rows by eight columns: a packet of either operand takes two turns of the shared memory, of sixteen columns four)
  const int tx = (tid >> 7) * 8 + (tid & 7), ty = (tid >> 5 & 3) * 4 + (tid >> 3 & 3);
  const float* base = work + ((size_t)blockIdx.x * heads + h) * dc_floats(D, dv);
  const float *queries = base + dc_walk_floats(D), *columns = base + dc_columns_at(D, dv) + (size_t)j0 * K;
  // a bulk copy per row, all of them counted on one barrier
  const uint32_t full = smem_u32(s_b + kDcOutCols * LA);
  volatile int* const abort_flag = reinterpret_cast<volatile int*>(s_b + kDcOutCols * LA + 2);
  if (tid == 0) {
    mbar_init(full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(full, (kDcTokens + cols) * K * 4);
  }
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();
  if (!there) return;
  const float walked = base[dc_flags_at(D, dv) + 2];     // (on its way while the copies are)
  if (tid < kDcTokens + cols && tid != waits.withheld) {
    const bool is_a = tid < kDcTokens;
    const int r = is_a ? tid : tid - kDcTokens;
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32((is_a ? s_a : s_b) + r * LA)), "l"((is_a ? queries : columns) + (size_t)r * K), "r"(K * 4), "r"(full) : "memory");
  }
  if (tid >= kDcTokens + cols && tid < kDcTokens + kDcOutCols)          // columns that there are not
    for (int k = 0; k < K; ++k) s_b[(tid - kDcTokens) * LA + k] = 0.f;
  const bool came = mbar_wait(full, 0, abort_flag, status, 32, waits.polls);
  if (__syncthreads_or(!came)) {                         // (nothing is written; the status says so)
    if (tid == 0) mbar_drain(full, 0);
    return;
  }
  if (walked != 0.f) return;                             // token by token, the outputs with it
  float sum[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) sum[a][c] = 0.f;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 32) {
    float2 acc[4][4];                                    // of even and of odd terms
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int k = k0; k < k0 + 32; k += 4) {
      float4 x[4], y[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) x[a] = *reinterpret_cast<const float4*>(s_a + (ty + 16 * a) * LA + k);
#pragma unroll
      for (int c = 0; c < 4; ++c) y[c] = *reinterpret_cast<const float4*>(s_b + (tx + 16 * c) * LA + k);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][c] = fma2(make_float2(x[a].x, x[a].y), make_float2(y[c].x, y[c].y), acc[a][c]);
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[a][c] = fma2(make_float2(x[a].z, x[a].w), make_float2(y[c].z, y[c].w), acc[a][c]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[a][c] += acc[a][c].x + acc[a][c].y;
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (ty + 16 * a < n && tx + 16 * c < cols) out[((size_t)(at.lo + first + ty + 16 * a) * heads + h) * dv + j0 + tx + 16 * c] = sum[a][c];
}

template <typename T, int D>
int delta_chunks(float* out, float* work, int chunks, int portions, const void* qkv, const float* ba, const float* rate, const float* dt_bias, float* state,
                 const int* q_start, const int* positions, const int* state_slot, int requests, int heads, int kv_heads, int dv,
                 float unit_eps, float q_scale, int walk_max, int* status, void* stream, CopyWaits walk_waits, CopyWaits output_waits) {
  static SmemRaised raised_p, raised_w, raised_o;
  if (int rc = raise_shared_memory("delta_chunk_prepare", delta_chunk_prepare_kernel<T, D>, (int)dc_prepare_smem(D), raised_p)) return rc;
  if (int rc = raise_shared_memory("delta_chunk_walk", delta_chunk_walk_kernel<T, D>, (int)dc_walk_smem(D), raised_w)) return rc;
  if (int rc = launch_kernel("delta_chunk_prepare", delta_chunk_prepare_kernel<T, D>, dim3(chunks, heads), dim3(kDcThreads), dc_prepare_smem(D),
                             as_stream(stream), work, (const T*)qkv, ba, rate, dt_bias, q_start, state_slot, requests, heads, kv_heads, dv,
                             unit_eps, q_scale, walk_max))
    return rc;
  if (int rc = raise_shared_memory("delta_chunk_outputs", delta_chunk_outputs_kernel<D>, (int)dc_outputs_smem(D), raised_o)) return rc;
  if (int rc = launch_kernel("delta_chunk_walk", delta_chunk_walk_kernel<T, D>, dim3(dv / kDcCols, heads, portions), dim3(kDcThreads), dc_walk_smem(D),
                             as_stream(stream), out, state, work, (const T*)qkv, ba, rate, dt_bias, kv_heads, unit_eps, q_scale, q_start,
                             positions, state_slot, requests, heads, dv, walk_max, status, walk_waits))
    return rc;
  return launch_kernel("delta_chunk_outputs", delta_chunk_outputs_kernel<D>, dim3(chunks, heads, (dv + kDcOutCols - 1) / kDcOutCols),
                       dim3(kDcThreads), dc_outputs_smem(D), as_stream(stream), out, (const float*)work, q_start, state_slot, requests, heads, dv,
                       walk_max, status, output_waits);
}

template <typename T>
int delta_chunks_any(float* out, float* work, int chunks, int portions, const void* qkv, const float* ba, const float* rate, const float* dt_bias,
                     float* state, const int* q_start, const int* positions, const int* state_slot, int requests, int heads, int kv_heads,
                     int d, int dv, float unit_eps, float q_scale, int walk_max, int* status, void* stream, CopyWaits walk_waits = {},
                     CopyWaits output_waits = {}) {
  PTL_REQUIRE(requests >= 0 && requests <= 65535 && portions >= 0 && portions <= requests && heads > 0 && heads <= 65535 && kv_heads > 0 && heads % kv_heads == 0 && chunks >= 0 && walk_max >= 0 &&
                  (d == 64 || d == 128) && dv > 0 && dv % kDcCols == 0 && aligned16(work),
              "gated_delta_rule in chunks: bad sizes heads=%d kv_heads=%d d=%d (64 or 128) dv=%d", heads, kv_heads, d, dv);
  if (requests == 0 || chunks == 0 || portions == 0) return 0;
  const auto fn = d == 64 ? delta_chunks<T, 64> : delta_chunks<T, 128>;
  return fn(out, work, chunks, portions, qkv, ba, rate, dt_bias, state, q_start, positions, state_slot, requests, heads, kv_heads, dv, unit_eps,
            q_scale, walk_max, status, stream, walk_waits, output_waits);
}

}  // namespace ptl

PTL_EXPORT long long ptl_delta_chunk_floats(int d, int dv) { return (long long)ptl::dc_floats(d, dv); }

#define PTL_DELTA_CHUNKS(SUFFIX, TYPE)                                                                                                \
  PTL_EXPORT int ptl_gated_delta_chunks##SUFFIX(float* out, float* work, int chunks, int portions, const void* qkv, const float* ba, const float* rate, \
                                                const float* dt_bias, float* state, const int* q_start, const int* positions,         \
                                                const int* state_slot, int requests, int heads, int kv_heads, int d, int dv,          \
                                                float unit_eps, float q_scale, int walk_max, void* status, void* stream) {            \
    return ptl::delta_chunks_any<TYPE>(out, work, chunks, portions, qkv, ba, rate, dt_bias, state, q_start, positions, state_slot, requests,    \
                                       heads, kv_heads, d, dv, unit_eps, q_scale, walk_max, (int*)status, stream);                    \
  }
PTL_DELTA_CHUNKS(_f32, float)
PTL_DELTA_CHUNKS(_bf16, __nv_bfloat16)

// Self-test of the bounded waits: the float32 form whose waits give up after `polls` polls and in which every walk leaves out the copy of
// chunk `no_chunk`, or every block of the outputs that of row `no_row` (-1: none).  The kernel must then write *status (31: the walk, 32: the
// outputs) and return; a walk that gives up leaves the state as it was, and `out` holds nothing of value.
PTL_EXPORT int ptl_gated_delta_chunks_wait_selftest(float* out, float* work, int chunks, int portions, const void* qkv, const float* ba,
                                                    const float* rate, const float* dt_bias, float* state, const int* q_start,
                                                    const int* positions, const int* state_slot, int requests, int heads, int kv_heads, int d,
                                                    int dv, float unit_eps, float q_scale, int walk_max, void* status, void* stream,
                                                    unsigned polls, int no_chunk, int no_row) {
  PTL_REQUIRE(status && polls >= 1 && polls <= (1u << 16), "gated_delta_chunks_wait_selftest: a status word, and between 1 and 65536 polls");
  return ptl::delta_chunks_any<float>(out, work, chunks, portions, qkv, ba, rate, dt_bias, state, q_start, positions, state_slot, requests, heads,
                                      kv_heads, d, dv, unit_eps, q_scale, walk_max, (int*)status, stream, {polls, no_chunk}, {polls, no_row});
}
