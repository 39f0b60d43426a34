// Generalized delta rule: per head a float32 state S [d, d] (rows: key channels, columns: value channels),
//   S <- diag(w_t) S - (a_t * u_t) (u_t^T S) + k_t v_t^T,   o_t = S^T r_t,   u_t = k_t / sqrt(|k_t|^2 + unit_eps),
// both products on the right reading the old S, with per key channel
//   w_t = exp(-decay_limit * sigmoid(z_t + w_bias)),   a_t = sigmoid(a_pre_t + a_bias).
//
// proj is the projection's output [T, r | k | v | ...] (H heads of d each), a_pre the first H*d columns of a float32
// array with rows of a_ld floats, z float32 [T, H*d] (the decay's argument before its bias, made by
// lowrank_tanh_linear below).  The layout of the walk is that of the gated delta rule (recurrent.cu): eight lanes
// share a column of the state, lane l holding the row pairs (16 m + 2 l, 16 m + 2 l + 1) as float2; a block of 128
// threads walks 16 columns of one head of one request through its tokens in order.  Tokens come in batches of
// kGdBatch: all threads bring a batch's r and k of the head, its decays, removal rates and 16 values into shared
// memory (sigmoids and exponentials worked out while staging; the next batch's inputs are held in registers while
// this one is walked).  With c = -(u^T S) / sqrt(|k|^2 + unit_eps) per column, a row's update is
//   S <- w S + (a k) c + k v,
// three two-wide fused multiply-adds per row pair.  Everything after the loads is float32; a token's result does
// not depend on how the request was cut into steps or on what else the step holds.  The state of a request is read
// from its slot unless the portion starts at position 0, and written back at the end.
#include "common.cuh"

namespace ptl {

constexpr int kGdBatch = 16;

__device__ __forceinline__ float sigmoid_f32(float x) { return 1.0f / (1.0f + expf(-x)); }

template <typename T, int RPL>
__global__ void __launch_bounds__(128)
general_delta_kernel(float* __restrict__ out, const T* __restrict__ proj, int ld, const float* __restrict__ a_pre, int a_ld,
                     const float* __restrict__ a_bias, const float* __restrict__ z, const float* __restrict__ w_bias,
                     float decay_limit, float* __restrict__ state, const int* __restrict__ q_start,
                     const int* __restrict__ positions, const int* __restrict__ state_slot, int heads, int d, float unit_eps) {
  static_assert(RPL % 2 == 0, "a lane holds pairs of rows");
  constexpr int DS = 8 * RPL;                       // floats between tokens' rows in shared memory
  constexpr int HP = RPL / 2;                       // row pairs of a lane
  extern __shared__ __align__(16) float gd_smem[];
  float* s_r = gd_smem;                            // [batch][DS]
  float* s_k = s_r + kGdBatch * DS;
  float* s_w = s_k + kGdBatch * DS;                // decay per row
  float* s_ak = s_w + kGdBatch * DS;               // removal rate times key per row
  float* s_v = s_ak + kGdBatch * DS;               // [batch][16]
  float* s_kn = s_v + kGdBatch * 16;               // 1 / (|k|^2 + unit_eps) per token
  pdl_wait();
  pdl_launch_dependents();
  const int r = blockIdx.z, h = blockIdx.y;
  const int lo = q_start[r], hi = q_start[r + 1];
  if (hi <= lo || state_slot[r] < 0) return;
  const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j0 = blockIdx.x * 16;
  const bool live = j0 + grp < d;
  const int j = live ? j0 + grp : d - 1;
  const int n = heads * d;
  float* st = state + (((size_t)state_slot[r] * heads + h) * d) * d + j;
  const bool from_zero = positions[lo] == 0;
  float2 S[HP];
#pragma unroll
  for (int m = 0; m < HP; ++m) {
    const int row = 16 * m + 2 * sub;
    S[m].x = (row < d && !from_zero) ? st[(size_t)row * d] : 0.f;
    S[m].y = (row + 1 < d && !from_zero) ? st[(size_t)(row + 1) * d] : 0.f;
  }
  for (int i = threadIdx.x; i < 4 * kGdBatch * DS; i += blockDim.x) s_r[i] = 0.f;   // (s_k, s_w, s_ak follow s_r) zero beyond d for good
  // Element i of a thread's share of a batch: flat index threadIdx.x + 128 * i over [batch][d]; RPL of them cover
  // kGdBatch * d = 16 d <= 128 * RPL (d <= 8 * RPL).  They are kept as fetched and converted when they go to shared
  // memory, after the walk over the batch before: the loads are in flight during that walk.
  T pr[RPL], pk[RPL], pv[2];
  float pz[RPL], pa[RPL];
  const int tok_first = threadIdx.x / d, e_first = threadIdx.x % d, tok_step = 128 / d, e_step = 128 % d;
  auto fetch = [&](int t0) {
    const int nb = min(kGdBatch, hi - t0);
    int tok = tok_first, e = e_first;
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      if (tok < nb) {
        const size_t t = (size_t)(t0 + tok);
        pr[i] = proj[t * ld + h * d + e];
        pk[i] = proj[t * ld + n + h * d + e];
        pz[i] = z[t * n + h * d + e];
        pa[i] = a_pre[t * a_ld + h * d + e];
      }
      tok += tok_step;
      e += e_step;
      if (e >= d) { e -= d; ++tok; }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int idx = threadIdx.x + 128 * i;
      if ((idx >> 4) < nb) pv[i] = proj[(size_t)(t0 + (idx >> 4)) * ld + 2 * n + h * d + min(j0 + (idx & 15), d - 1)];
    }
  };
  fetch(lo);
  for (int t0 = lo; t0 < hi; t0 += kGdBatch) {
    const int nb = min(kGdBatch, hi - t0);
    __syncthreads();                                  // the batch before has been walked (and the rows are zeroed)
    {
      int tok = tok_first, e = e_first;
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        if (tok < nb) {
          const float kf = to_f32(pk[i]);
          s_r[tok * DS + e] = to_f32(pr[i]);
          s_k[tok * DS + e] = kf;
          s_w[tok * DS + e] = expf(-decay_limit * sigmoid_f32(pz[i] + w_bias[h * d + e]));
          s_ak[tok * DS + e] = sigmoid_f32(pa[i] + a_bias[h * d + e]) * kf;
        }
        tok += tok_step;
        e += e_step;
        if (e >= d) { e -= d; ++tok; }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int idx = threadIdx.x + 128 * i;
      if ((idx >> 4) < nb) s_v[idx] = to_f32(pv[i]);
    }
    __syncthreads();
    if (t0 + kGdBatch < hi) fetch(t0 + kGdBatch);     // in flight while this batch is walked
    {
      // the squared lengths of the keys: warp w takes tokens w, w + 4, w + 8, w + 12
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int tok = warp + 4 * m;
        if (tok < nb) {
          float kk = 0.f;
          for (int e = lane; e < d; e += 32) kk = fmaf(s_k[tok * DS + e], s_k[tok * DS + e], kk);
          kk = warp_sum(kk);
          if (lane == 0) s_kn[tok] = 1.0f / (kk + unit_eps);
        }
      }
    }
    __syncthreads();
#pragma unroll (RPL <= 16 ? 2 : 1)
    for (int tok = 0; tok < nb; ++tok) {
      const float2* kp = reinterpret_cast<const float2*>(s_k + tok * DS) + sub;     // pair m of this lane: kp[8 * m]
      const float2* rp = reinterpret_cast<const float2*>(s_r + tok * DS) + sub;
      const float2* wp = reinterpret_cast<const float2*>(s_w + tok * DS) + sub;
      const float2* ap = reinterpret_cast<const float2*>(s_ak + tok * DS) + sub;
      float2 k[HP];
      float2 dot0 = make_float2(0.f, 0.f), dot1 = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < HP; ++m) {
        k[m] = kp[8 * m];
        if (m & 1) dot1 = __ffma2_rn(S[m], k[m], dot1); else dot0 = __ffma2_rn(S[m], k[m], dot0);
      }
      float dot = (dot0.x + dot0.y) + (dot1.x + dot1.y);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      const float c = -dot * s_kn[tok];
      const float v = s_v[tok * 16 + grp];
      const float2 c2 = make_float2(c, c), v2 = make_float2(v, v);
      float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
      for (int m = 0; m < HP; ++m) {
        S[m] = __ffma2_rn(wp[8 * m], S[m], __ffma2_rn(ap[8 * m], c2, __fmul2_rn(k[m], v2)));
        const float2 rv = rp[8 * m];
        if (m & 1) acc1 = __ffma2_rn(S[m], rv, acc1); else acc0 = __ffma2_rn(S[m], rv, acc0);
      }
      float acc = (acc0.x + acc0.y) + (acc1.x + acc1.y);
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (sub == 0 && live) out[(size_t)(t0 + tok) * n + h * d + j] = acc;
    }
  }
  if (live) {
#pragma unroll
    for (int m = 0; m < HP; ++m) {
      const int row = 16 * m + 2 * sub;
      if (row < d) st[(size_t)row * d] = S[m].x;
      if (row + 1 < d) st[(size_t)(row + 1) * d] = S[m].y;
    }
  }
}

// The same for heads of 17 to 64 channels, with two columns per group of lanes and the staging by warps of its own: warps 0 to 3
// walk batch i while warps 4 to 7 put batch i + 1 into the other half of shared memory and fetch batch i + 2.  The walk is
// bound by the latency of its chain (two sums over eight lanes a token); in the kernel above every warp also works
// exponentials and quotients out between two batches and meets the others three times a batch, and the four blocks of a
// head do so four times.  A column's sums are the same, in the same order.
// Eight prompts of 65 to 440 tokens, 16 heads of 64: 154 us, the kernel above 235 (with two columns a group alone 219, four 240);
// eight single tokens 6.0 us and 9.8.
template <typename T, int RPL>
__global__ void __launch_bounds__(256, 2)
general_delta_pairs_kernel(float* __restrict__ out, const T* __restrict__ proj, int ld, const float* __restrict__ a_pre, int a_ld,
                           const float* __restrict__ a_bias, const float* __restrict__ z, const float* __restrict__ w_bias,
                           float decay_limit, float* __restrict__ state, const int* __restrict__ q_start,
                           const int* __restrict__ positions, const int* __restrict__ state_slot, int heads, int d, float unit_eps) {
  constexpr int DS = 8 * RPL, HP = RPL / 2, COLS = 32;
  constexpr int kBatchFloats = kGdBatch * (4 * DS + COLS + 1);
  __shared__ __align__(16) float smem[2 * kBatchFloats];
  // floats of a batch: r, k, decay, rate times key [batch][DS]; values [batch][COLS]; 1 / (|k|^2 + unit_eps) [batch]
  constexpr int kKey = kGdBatch * DS, kDecay = 2 * kKey, kRate = 3 * kKey, kValue = 4 * kKey, kNorm = kValue + kGdBatch * COLS;
  pdl_wait();
  pdl_launch_dependents();
  const int r = blockIdx.z, h = blockIdx.y;
  const int lo = q_start[r], hi = q_start[r + 1];
  if (hi <= lo || state_slot[r] < 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j0 = blockIdx.x * COLS;
  const int n = heads * d;
  const int batches = (hi - lo + kGdBatch - 1) / kGdBatch;
  for (int i = threadIdx.x; i < 2 * kBatchFloats; i += 256) smem[i] = 0.f;       // zero beyond d for good
  __syncthreads();
  if (warp >= 4) {
    // element i of a thread's share of a batch: flat index tid + 128 i over [batch][d]
    const int tid = threadIdx.x - 128;
    T pr[RPL], pk[RPL], pv[4];
    float pz[RPL], pa[RPL];
    const int tok_first = tid / d, e_first = tid % d, tok_step = 128 / d, e_step = 128 % d;
    auto fetch = [&](int t0) {
      const int nb = min(kGdBatch, hi - t0);
      int tok = tok_first, e = e_first;
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        if (tok < nb) {
          const size_t t = (size_t)(t0 + tok);
          pr[i] = proj[t * ld + h * d + e];
          pk[i] = proj[t * ld + n + h * d + e];
          pz[i] = z[t * n + h * d + e];
          pa[i] = a_pre[t * a_ld + h * d + e];
        }
        tok += tok_step;
        e += e_step;
        if (e >= d) { e -= d; ++tok; }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = tid + 128 * i;
        if (idx / COLS < nb) pv[i] = proj[(size_t)(t0 + idx / COLS) * ld + 2 * n + h * d + min(j0 + idx % COLS, d - 1)];
      }
    };
    auto stage = [&](int t0, float* dst) {
      const int nb = min(kGdBatch, hi - t0);
      int tok = tok_first, e = e_first;
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        if (tok < nb) {
          const float kf = to_f32(pk[i]);
          dst[tok * DS + e] = to_f32(pr[i]);
          dst[kKey + tok * DS + e] = kf;
          dst[kDecay + tok * DS + e] = expf(-decay_limit * sigmoid_f32(pz[i] + w_bias[h * d + e]));
          dst[kRate + tok * DS + e] = sigmoid_f32(pa[i] + a_bias[h * d + e]) * kf;
        }
        tok += tok_step;
        e += e_step;
        if (e >= d) { e -= d; ++tok; }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = tid + 128 * i;
        if (idx / COLS < nb) dst[kValue + idx] = to_f32(pv[i]);
      }
      if (t0 + kGdBatch < hi) fetch(t0 + kGdBatch);
      asm volatile("bar.sync 1, 128;" ::: "memory");           // the staging warps: the keys are in place
#pragma unroll
      for (int m = 0; m < 4; ++m) {                             // warp w takes tokens w, w + 4, w + 8, w + 12
        const int tk = warp - 4 + 4 * m;
        if (tk < nb) {
          float kk = 0.f;
          for (int e2 = lane; e2 < d; e2 += 32) kk = fmaf(dst[kKey + tk * DS + e2], dst[kKey + tk * DS + e2], kk);
          kk = warp_sum(kk);
          if (lane == 0) dst[kNorm + tk] = 1.0f / (kk + unit_eps);
        }
      }
    };
    fetch(lo);
    stage(lo, smem);
    __syncthreads();
    for (int b = 0; b < batches; ++b) {
      if (b + 1 < batches) stage(lo + (b + 1) * kGdBatch, smem + ((b + 1) & 1) * kBatchFloats);
      __syncthreads();
    }
    return;
  }
  const int sub = threadIdx.x & 7, grp = threadIdx.x >> 3;     // columns j0 + grp and j0 + grp + 16
  float* st = state + (((size_t)state_slot[r] * heads + h) * d) * d + j0 + grp;
  const bool from_zero = positions[lo] == 0;
  float2 S[2][HP];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int m = 0; m < HP; ++m) {
      const int row = 16 * m + 2 * sub;
      const bool live = !from_zero && j0 + grp + 16 * c < d;
      S[c][m].x = row < d && live ? st[(size_t)row * d + 16 * c] : 0.f;
      S[c][m].y = row + 1 < d && live ? st[(size_t)(row + 1) * d + 16 * c] : 0.f;
    }
  __syncthreads();
  for (int b = 0; b < batches; ++b) {
    const int t0 = lo + b * kGdBatch, nb = min(kGdBatch, hi - t0);
    const float* src = smem + (b & 1) * kBatchFloats;
#pragma unroll 2
    for (int tok = 0; tok < nb; ++tok) {
      const float2* rp = reinterpret_cast<const float2*>(src + tok * DS) + sub;                // pair m of this lane: rp[8 * m]
      float2 k[HP], w[HP], ak[HP], rv[HP];
#pragma unroll
      for (int m = 0; m < HP; ++m) {
        k[m] = rp[kKey / 2 + 8 * m];
        w[m] = rp[kDecay / 2 + 8 * m];
        ak[m] = rp[kRate / 2 + 8 * m];
        rv[m] = rp[8 * m];
      }
      float dot[2], acc[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float2 dot0 = make_float2(0.f, 0.f), dot1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int m = 0; m < HP; ++m) {
          if (m & 1) dot1 = __ffma2_rn(S[c][m], k[m], dot1); else dot0 = __ffma2_rn(S[c][m], k[m], dot0);
        }
        dot[c] = (dot0.x + dot0.y) + (dot1.x + dot1.y);
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], o);
        dot[1] += __shfl_xor_sync(0xffffffffu, dot[1], o);
      }
      const float kn = src[kNorm + tok];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float cc = -dot[c] * kn, v = src[kValue + tok * COLS + grp + 16 * c];
        const float2 c2 = make_float2(cc, cc), v2 = make_float2(v, v);
        float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int m = 0; m < HP; ++m) {
          S[c][m] = __ffma2_rn(w[m], S[c][m], __ffma2_rn(ak[m], c2, __fmul2_rn(k[m], v2)));
          if (m & 1) acc1 = __ffma2_rn(S[c][m], rv[m], acc1); else acc0 = __ffma2_rn(S[c][m], rv[m], acc0);
        }
        acc[c] = (acc0.x + acc0.y) + (acc1.x + acc1.y);
      }
      // both sums at once: even lanes of a group end with column 0's, odd lanes with column 1's
      const bool odd = sub & 1;
      float sum = (odd ? acc[1] : acc[0]) + __shfl_xor_sync(0xffffffffu, odd ? acc[0] : acc[1], 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      sum += __shfl_xor_sync(0xffffffffu, sum, 4);
      if (sub < 2 && j0 + grp + 16 * sub < d) out[(size_t)(t0 + tok) * n + h * d + j0 + grp + 16 * sub] = sum;
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
    if (j0 + grp + 16 * c < d) {
#pragma unroll
      for (int m = 0; m < HP; ++m) {
        const int row = 16 * m + 2 * sub;
        if (row < d) st[(size_t)row * d + 16 * c] = S[c][m].x;
        if (row + 1 < d) st[(size_t)(row + 1) * d + 16 * c] = S[c][m].y;
      }
    }
}

template <typename T>
int general_delta_scan(float* out, const void* proj, int ld, const float* a_pre, int a_ld, const float* a_bias, const float* z,
                       const float* w_bias, float decay_limit, float* state, const int* q_start, const int* positions,
                       const int* state_slot, int requests, int heads, int d, float unit_eps, void* stream) {
  PTL_REQUIRE(requests >= 0 && heads > 0 && d > 0 && d <= 256, "general_delta_scan: bad sizes heads=%d d=%d (at most 256)", heads, d);
  PTL_REQUIRE(ld >= 3 * heads * d && a_ld >= heads * d, "general_delta_scan: rows are too short");
  PTL_REQUIRE(requests <= 65535 && heads <= 65535, "general_delta_scan: at most 65535 requests and heads");
  if (requests == 0) return 0;
  const dim3 grid((d + 15) / 16, heads, requests), block(128);
  if (d > 16 && d <= 64)
    return launch_kernel("general_delta_scan", d <= 32 ? general_delta_pairs_kernel<T, 4> : general_delta_pairs_kernel<T, 8>,
                         dim3((d + 31) / 32, heads, requests), dim3(256), 0, as_stream(stream), out, (const T*)proj, ld, a_pre, a_ld, a_bias,
                         z, w_bias, decay_limit, state, q_start, positions, state_slot, heads, d, unit_eps);
  static SmemRaised raised[4];
#define PTL_GD(RPL, SLOT)                                                                                                      \
  {                                                                                                                            \
    const size_t smem = (size_t)kGdBatch * (4 * 8 * RPL + 16 + 1) * sizeof(float);                                             \
    if (smem > 48 * 1024)                                                                                                      \
      if (int rc = raise_shared_memory("general_delta_scan", general_delta_kernel<T, RPL>, (int)smem, raised[SLOT])) return rc; \
    return launch_kernel("general_delta_scan", general_delta_kernel<T, RPL>, grid, block, smem, as_stream(stream), out,        \
                         (const T*)proj, ld, a_pre, a_ld, a_bias, z, w_bias, decay_limit, state, q_start, positions,           \
                         state_slot, heads, d, unit_eps);                                                                      \
  }
  const int per_lane = (d + 7) / 8;
  if (per_lane <= 2) PTL_GD(2, 0)
  if (per_lane <= 12) PTL_GD(12, 1)
  if (per_lane <= 16) PTL_GD(16, 2)
  PTL_GD(32, 3)
#undef PTL_GD
}

// z[t, c] = sum_j w2[c, j] * tanh(x[t, column + j]), float32 throughout; with `decay_bias` the result is the decay
// exp(-exp(z + decay_bias[c])) instead.  Every result is one chain of fused
// multiply-adds, j ascending, whatever the tile it falls into, so a token's row has the same bits in a prompt
// portion and alone.  A block of 128 threads takes kLtTokens tokens and COLS columns: the inner inputs' tanh and a slab of w2
// (RANK values of j at a time, transposed so that neighbouring threads read neighbouring words) go through shared
// memory; a thread holds one column's sums for COLS / 8 of the block's tokens.  The first slab of w2 is fetched before the wait on the
// predecessor.  Narrow blocks where wide ones leave SMs idle: 8 tokens,
// 1,024 columns, rank 64: 15 us in 8 wide blocks, 4.8 in 32 narrow ones; 2,020 tokens 22 us in wide ones.
constexpr int kLtTokens = 16, kLtThreads = 128;

template <int COLS, int RANK>
__global__ void __launch_bounds__(kLtThreads)
lowrank_tanh_linear_kernel(float* __restrict__ z, const float* __restrict__ x, int tokens, int x_ld, int column, int rank,
                           const float* __restrict__ w2, int n, const float* __restrict__ decay_bias) {
  constexpr int TPT = COLS / 8;                                    // tokens of a thread: 128 / COLS groups share the block's sixteen
  __shared__ __align__(16) float s_hid[RANK][kLtTokens];           // tanh of the inner inputs, tokens side by side
  __shared__ float s_w[RANK][COLS + 1];
  const int t0 = blockIdx.y * kLtTokens, c0 = blockIdx.x * COLS;
  const int col = threadIdx.x % COLS, first = threadIdx.x / COLS * TPT;
  const int c = c0 + col;
  auto fetch_weights = [&](int j0) {
#pragma unroll 8
    for (int e = threadIdx.x; e < COLS * RANK; e += kLtThreads) {
      const int cc = e / RANK, jj = e % RANK;
      s_w[jj][cc] = (c0 + cc < n && j0 + jj < rank) ? w2[(size_t)(c0 + cc) * rank + j0 + jj] : 0.f;
    }
  };
  fetch_weights(0);
  pdl_wait();
  pdl_launch_dependents();
  float acc[TPT];
#pragma unroll
  for (int t = 0; t < TPT; ++t) acc[t] = 0.f;
  for (int j0 = 0; j0 < rank; j0 += RANK) {
    const int nj = min(RANK, rank - j0);
    if (j0) {
      __syncthreads();                                             // the slab before has been used
      fetch_weights(j0);
    }
#pragma unroll
    for (int e = threadIdx.x; e < kLtTokens * RANK; e += kLtThreads) {
      const int t = e / RANK, jj = e % RANK;
      s_hid[jj][t] = (t0 + t < tokens && jj < nj) ? tanhf(x[(size_t)(t0 + t) * x_ld + column + j0 + jj]) : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int jj = 0; jj < nj; ++jj) {
      const float w = s_w[jj][col];
      const float4* hp = reinterpret_cast<const float4*>(s_hid[jj] + first);
#pragma unroll
      for (int q = 0; q < TPT / 4; ++q) {
        const float4 hv = hp[q];
        acc[4 * q + 0] = fmaf(w, hv.x, acc[4 * q + 0]);
        acc[4 * q + 1] = fmaf(w, hv.y, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(w, hv.z, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(w, hv.w, acc[4 * q + 3]);
      }
    }
  }
  if (c < n) {
    const float bias = decay_bias ? decay_bias[c] : 0.f;
#pragma unroll
    for (int t = 0; t < TPT; ++t)
      if (t0 + first + t < tokens)
        z[(size_t)(t0 + first + t) * n + c] = decay_bias ? decay_exp(-expf(acc[t] + bias)) : acc[t];
  }
}

}  // namespace ptl

PTL_EXPORT int ptl_lowrank_tanh_linear(float* z, const float* x, int tokens, int x_ld, int column, int rank, const float* w2, int n,
                                       const float* decay_bias, void* stream) {
  PTL_REQUIRE(tokens >= 0 && rank > 0 && n > 0 && column >= 0 && column + rank <= x_ld,
              "lowrank_tanh_linear: bad sizes rank=%d n=%d column=%d ld=%d", rank, n, column, x_ld);
  if (tokens == 0) return 0;
  const int rows = (tokens + ptl::kLtTokens - 1) / ptl::kLtTokens;
  PTL_REQUIRE(rows <= 65535, "lowrank_tanh_linear: %d tokens in one call", tokens);
  const bool narrow = (long long)rows * ((n + 127) / 128) < 148;
  return ptl::launch_kernel("lowrank_tanh_linear", narrow ? ptl::lowrank_tanh_linear_kernel<32, 64> : ptl::lowrank_tanh_linear_kernel<128, 32>,
                            narrow ? dim3((n + 31) / 32, rows) : dim3((n + 127) / 128, rows), dim3(ptl::kLtThreads), 0,
                            ptl::as_stream(stream), z, x, tokens, x_ld, column, rank, w2, n, decay_bias);
}

#define PTL_GENERAL_DELTA(SUFFIX, TYPE)                                                                                          \
  PTL_EXPORT int ptl_general_delta_scan##SUFFIX(float* out, const void* proj, int ld, const float* a_pre, int a_ld,               \
                                                const float* a_bias, const float* z, const float* w_bias, float decay_limit,     \
                                                float* state, const int* q_start, const int* positions, const int* state_slot,   \
                                                int requests, int heads, int d, float unit_eps, void* stream) {                  \
    return ptl::general_delta_scan<TYPE>(out, proj, ld, a_pre, a_ld, a_bias, z, w_bias, decay_limit, state, q_start, positions,   \
                                         state_slot, requests, heads, d, unit_eps, stream);                                      \
  }
PTL_GENERAL_DELTA(_f32, float)
PTL_GENERAL_DELTA(_bf16, __nv_bfloat16)
