// The token-indexed side term of a layer (see token_side_kernel in stream_ops.cu) for 16-bit weights, sixteen tokens per cluster of eight
// blocks: s = residual + x + bias;  z = W_gate s;  g = gelu_tanh(z) * table[token, column + j];  y = W_proj g;
// residual = s + y * rsqrt(mean(y^2) + eps) * norm.
// Block b owns an eighth of the width: its columns of s and of W_gate give partial sums of all z, block b adds up and
// activates its eighth of the dims, and its rows of W_proj give its columns of y.  Partial sums, g and the sums of squares cross
// the cluster through distributed shared memory.  Both products run on the tensor cores; s and g are float32 and go there as three
// bfloat16 terms each (24 bits).  The weights' parts (32 KB a block at 1,024 x 64) are fetched before the wait on the
// predecessor.  Bound by the latency of three cluster barriers at a few tokens.  2,048 tokens of width 1,024: 91 us
// as one block per token, 32 here; 8 tokens: 22.4 and 7.7.
#include "mma_utils.cuh"

namespace ptl {

constexpr int kTsBlocks = 8, kTsTokens = 16, kTsThreads = 256, kTsMaxDim = 128;

__device__ __forceinline__ float ts_gelu_tanh(float z) {
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ void ts_split(float x, __nv_bfloat16* at, int stride) {      // three terms, `stride` elements apart
#pragma unroll
  for (int w = 0; w < 3; ++w) {
    const __nv_bfloat16 t = __float2bfloat16_rn(x);
    at[w * stride] = t;
    x -= __bfloat162float(t);
  }
}
// bytes: s float32, s in three terms, W_gate part, W_proj part, partial sums, g float32, g in three terms
__host__ __device__ constexpr size_t ts_smem(int sl, int dim) {
  return (size_t)4 * kTsTokens * (sl + 4) + 6 * kTsTokens * (sl + 8) + 2 * dim * (sl + 8) + 2 * sl * (dim + 8) + 4 * kTsTokens * dim +
         4 * kTsTokens * dim + 6 * kTsTokens * (dim + 8);
}

template <int SL>
__global__ void __launch_bounds__(kTsThreads)
token_side_cluster_kernel(float* __restrict__ residual, const __nv_bfloat16* __restrict__ x, const float* __restrict__ bias,
                          const int* __restrict__ tokens, const __nv_bfloat16* __restrict__ table, int table_ld, int column, int dim,
                          int vocab, const __nv_bfloat16* __restrict__ w_gate, const __nv_bfloat16* __restrict__ w_proj,
                          const float* __restrict__ norm_w, float eps, int n_tokens) {
  constexpr int width = SL * kTsBlocks, LS = SL + 4, LB = SL + 8;
  extern __shared__ __align__(16) unsigned char ts_raw[];
  float* s32 = reinterpret_cast<float*>(ts_raw);                                     // [16][LS]
  __nv_bfloat16* s16 = reinterpret_cast<__nv_bfloat16*>(s32 + kTsTokens * LS);       // [3][16][LB]
  __nv_bfloat16* wg = s16 + 3 * kTsTokens * LB;                                      // [dim][LB]
  __nv_bfloat16* wp = wg + dim * LB;                                                 // [SL][dim + 8]
  const int LD = dim + 8, per = dim / kTsBlocks;
  float* zrecv = reinterpret_cast<float*>(wp + SL * LD);                             // [8 sources][16][per]
  float* g32 = zrecv + kTsTokens * dim;                                              // [16][dim]
  __nv_bfloat16* g16 = reinterpret_cast<__nv_bfloat16*>(g32 + kTsTokens * dim);      // [3][16][LD]
  __shared__ float s_ss[kTsThreads / 32][kTsTokens];
  __shared__ float s_recv[kTsBlocks][kTsTokens];
  cluster_arrive();                                     // every block runs before a peer writes into it
  const int rank = blockIdx.x % kTsBlocks, t0 = blockIdx.x / kTsBlocks * kTsTokens, c0 = rank * SL;
  const int nt = min(kTsTokens, n_tokens - t0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  // the weights: written by no kernel of the step
  for (int i = tid; i < dim * (SL / 8); i += kTsThreads)
    cp_async_16(smem_u32(wg + (i / (SL / 8)) * LB + i % (SL / 8) * 8), w_gate + (size_t)(i / (SL / 8)) * width + c0 + i % (SL / 8) * 8, true);
  for (int i = tid; i < SL * (dim / 8); i += kTsThreads)
    cp_async_16(smem_u32(wp + (i / (dim / 8)) * LD + i % (dim / 8) * 8), w_proj + (size_t)(c0 + i / (dim / 8)) * dim + i % (dim / 8) * 8, true);
  cp_async_commit();
  const bool own = tid < kTsTokens * per;
  pdl_wait();
  pdl_launch_dependents();
  // this thread's table entry: a kernel of the step may have written the token; nothing needs the entry before the second barrier
  const bool live = own && tid / per < nt;
  int tok = live ? tokens[t0 + tid / per] : 0;
  for (int i = tid; i < kTsTokens * (SL / 4); i += kTsThreads) {
    const int r = i / (SL / 4), c = i % (SL / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nt) {
      v = *reinterpret_cast<const float4*>(residual + (size_t)(t0 + r) * width + c0 + c);
      if (x) {
        const uint2 raw = *reinterpret_cast<const uint2*>(x + (size_t)(t0 + r) * width + c0 + c);
        const float2 lo = unpack_bf16(raw.x), hi = unpack_bf16(raw.y);
        v.x += lo.x; v.y += lo.y; v.z += hi.x; v.w += hi.y;
      }
      if (bias) {
        const float4 b = *reinterpret_cast<const float4*>(bias + c0 + c);
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
      }
    }
    *reinterpret_cast<float4*>(s32 + r * LS + c) = v;
#pragma unroll
    for (int e = 0; e < 4; ++e) ts_split((&v.x)[e], s16 + r * LB + c + e, kTsTokens * LB);
  }
  if (tok < 0 || tok >= vocab) tok = 0;
  const __nv_bfloat16 entry = live ? table[(size_t)tok * table_ld + column + rank * per + tid % per] : __float2bfloat16_rn(0.f);
  cp_async_wait<0>();
  __syncthreads();
  const int lm_row = lane & 15, lm_half = lane >> 4;
  // partial z: a warp per eight dims
  cluster_wait();
  for (int n = warp; n < dim / 8; n += kTsThreads / 32) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < SL / 16; k += 2) {
      uint32_t b[4];
      ldmatrix_x4(b, smem_u32(wg + (8 * n + (lane & 7)) * LB + 16 * k + 8 * (lane >> 3)));
#pragma unroll
      for (int w = 2; w >= 0; --w) {
        uint32_t a[4];
        ldmatrix_x4(a, smem_u32(s16 + (w * kTsTokens + lm_row) * LB + 16 * k + 8 * lm_half));
        mma_bf16_16816(acc, a, b[0], b[1]);
        ldmatrix_x4(a, smem_u32(s16 + (w * kTsTokens + lm_row) * LB + 16 * k + 16 + 8 * lm_half));
        mma_bf16_16816(acc, a, b[2], b[3]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * n + c2 + (e & 1), row = g + 8 * (e >> 1);
      st_peer_f32(map_to_peer(smem_u32(zrecv + (rank * kTsTokens + row) * per + d % per), d / per), acc[e]);
    }
  }
  cluster_arrive();
  cluster_wait();
  if (own) {
    const int row = tid / per, d = tid % per;
    float z = 0.f;
#pragma unroll
    for (int b = 0; b < kTsBlocks; ++b) z += zrecv[(b * kTsTokens + row) * per + d];
    const float v = ts_gelu_tanh(z) * __bfloat162float(entry);
#pragma unroll
    for (int b = 0; b < kTsBlocks; ++b) st_peer_f32(map_to_peer(smem_u32(g32 + row * dim + rank * per + d), b), v);
  }
  cluster_arrive();
  cluster_wait();
  for (int i = tid; i < kTsTokens * dim; i += kTsThreads) ts_split(g32[i], g16 + i / dim * LD + i % dim, kTsTokens * LD);
  __syncthreads();
  constexpr int NT = SL / 64;                           // blocks of eight columns per warp
  float y[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) y[j][e] = 0.f;
  for (int k = 0; k < dim / 16; ++k) {
    uint32_t a[3][4];
#pragma unroll
    for (int w = 0; w < 3; ++w) ldmatrix_x4(a[w], smem_u32(g16 + (w * kTsTokens + lm_row) * LD + 16 * k + 8 * lm_half));
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      uint32_t b[4];                                    // (the upper half of the lanes names the same rows again)
      ldmatrix_x4(b, smem_u32(wp + (8 * (warp * NT + j) + (lane & 7)) * LD + 16 * k + 8 * ((lane >> 3) & 1)));
#pragma unroll
      for (int w = 2; w >= 0; --w) mma_bf16_16816(y[j], a[w], b[0], b[1]);
    }
  }
  float ss[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) ss[e >> 1] = fmaf(y[j][e], y[j][e], ss[e >> 1]);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 1);
    ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 2);
    if ((lane & 3) == 0) s_ss[warp][g + 8 * i] = ss[i];
  }
  __syncthreads();
  if (tid < kTsTokens * kTsBlocks) {
    const int row = tid % kTsTokens, peer = tid / kTsTokens;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kTsThreads / 32; ++w) v += s_ss[w][row];
    st_peer_f32(map_to_peer(smem_u32(&s_recv[rank][row]), peer), v);
  }
  cluster_arrive();
  cluster_wait();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = g + 8 * i;
    if (row >= nt) continue;
    float total = 0.f;
#pragma unroll
    for (int b = 0; b < kTsBlocks; ++b) total += s_recv[b][row];
    const float rrms = 1.0f / sqrtf(total / (float)width + eps);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int c = 8 * (warp * NT + j) + c2;
      const float2 w = *reinterpret_cast<const float2*>(norm_w + c0 + c);
      *reinterpret_cast<float2*>(residual + (size_t)(t0 + row) * width + c0 + c) =
          make_float2(s32[row * LS + c] + y[j][2 * i] * rrms * w.x, s32[row * LS + c + 1] + y[j][2 * i + 1] * rrms * w.y);
    }
  }
}

template <int SL>
int token_side_cluster(float* residual, const void* x, const float* bias, const int* tokens, const void* table, int table_ld, int column,
                       int dim, int vocab, const void* w_gate, const void* w_proj, const float* norm_w, int n_tokens, float eps,
                       void* stream) {
  static SmemRaised raised;
  if (int rc = raise_shared_memory("token_side", token_side_cluster_kernel<SL>, (int)ts_smem(SL, kTsMaxDim), raised)) return rc;
  return launch_kernel_cluster("token_side", token_side_cluster_kernel<SL>, dim3((n_tokens + kTsTokens - 1) / kTsTokens * kTsBlocks),
                               dim3(kTsThreads), ts_smem(SL, dim), as_stream(stream), kTsBlocks, residual, (const __nv_bfloat16*)x, bias,
                               tokens, (const __nv_bfloat16*)table, table_ld, column, dim, vocab, (const __nv_bfloat16*)w_gate,
                               (const __nv_bfloat16*)w_proj, norm_w, eps, n_tokens);
}

// Many tokens: a block owns sixteen whole rows, and nothing crosses blocks.  Its sixteen warps take, for z, an eighth of the width and half of
// the dims each, then a sixteenth of W_proj's rows; a lane reads the weights in packets of eight values straight from L2 (those of W_gate
// before the wait on the predecessor), and the four lanes of a row trade words until each holds its own of the MMAs' operands.  All
// sums in the cluster form's order (a rank's eighth of z in one chain, the ranks in order; the squares by the cluster's warps), so that a
// token has the same bits in either.  What bounds it: 256 KB of weights a block out of L2, and the reads of the rows before anything can begin.
constexpr int kTrThreads = 512, kTrWarps = kTrThreads / 32;
__host__ __device__ constexpr int tr_ld(int n) { return n + 8; }        // rows of 16-bit terms: eight rows' packets in different banks
__host__ __device__ constexpr size_t tr_smem(int width, int dim) {
  const size_t terms = (size_t)6 * kTsTokens * tr_ld(width), sums = (size_t)4 * kTsBlocks * kTsTokens * dim;
  return (size_t)4 * kTsTokens * (width + 4) + (terms > sums ? terms : sums) + (size_t)6 * kTsTokens * tr_ld(dim);
}
// Words 4 q .. 4 q + 3 of a row's sixteen in lane q of four -> words q, q + 4, q + 8, q + 12.
__device__ __forceinline__ void tr_trade(uint4& v) {
  const bool odd = threadIdx.x & 1, high = threadIdx.x & 2;
  const uint32_t a = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1), b = __shfl_xor_sync(0xffffffffu, odd ? v.z : v.w, 1);
  (odd ? v.x : v.y) = a;
  (odd ? v.z : v.w) = b;
  const uint32_t c = __shfl_xor_sync(0xffffffffu, high ? v.x : v.z, 2), d = __shfl_xor_sync(0xffffffffu, high ? v.y : v.w, 2);
  (high ? v.x : v.z) = c;
  (high ? v.y : v.w) = d;
}

template <int WIDTH, int DIM>
__global__ void __launch_bounds__(kTrThreads, 1)
token_side_rows_kernel(float* __restrict__ residual, const __nv_bfloat16* __restrict__ x, const float* __restrict__ bias,
                       const int* __restrict__ tokens, const __nv_bfloat16* __restrict__ table, int table_ld, int column,
                       int vocab, const __nv_bfloat16* __restrict__ w_gate, const __nv_bfloat16* __restrict__ w_proj,
                       const float* __restrict__ norm_w, float eps, int n_tokens) {
  constexpr int LS = WIDTH + 4, LT = tr_ld(WIDTH), LG = tr_ld(DIM), SL = WIDTH / kTsBlocks, SLICE = WIDTH / kTrWarps, KB = SL / 32, NZ = DIM / 16, NY = SLICE / 8;
  constexpr int NT = SL / 64, CW = kTsBlocks * (kTsThreads / 32);       // of the cluster form: blocks of eight columns per warp, warps
  extern __shared__ __align__(16) unsigned char tr_raw[];
  float* s32 = reinterpret_cast<float*>(tr_raw);                                     // [16][LS]
  __nv_bfloat16* s16 = reinterpret_cast<__nv_bfloat16*>(s32 + kTsTokens * LS);       // [3][16][LT]; then the ranks' sums of z [8][16][DIM]
  float* zpart = reinterpret_cast<float*>(s16);
  constexpr size_t terms = (size_t)3 * kTsTokens * LT, sums = (size_t)2 * kTsBlocks * kTsTokens * DIM;
  __nv_bfloat16* g16 = s16 + (terms > sums ? terms : sums);                          // [3][16][LG]
  __shared__ float s_ss[CW][kTsTokens];
  __shared__ float s_rank[kTsBlocks][kTsTokens];
  const int t0 = blockIdx.x * kTsTokens, nt = min(kTsTokens, n_tokens - t0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q8 = (lane & 3) * 8, c2 = (lane & 3) * 2;
  const int rank = warp >> 1, half = warp & 1, lm_row = lane & 15, lm_half = lane >> 4;
  uint4 wg[KB][NZ];                                     // (written by no kernel of the step)
#pragma unroll
  for (int k = 0; k < KB; ++k)
#pragma unroll
    for (int n = 0; n < NZ; ++n) wg[k][n] = __ldg(reinterpret_cast<const uint4*>(w_gate + (size_t)(8 * (half * NZ + n) + g) * WIDTH + rank * SL + 32 * k + q8));
  pdl_wait();
  pdl_launch_dependents();
  constexpr int PER = DIM * kTsTokens / kTrThreads;     // elements of z that a thread finishes
  int tok[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int row = (tid + i * kTrThreads) / DIM;
    tok[i] = row < nt ? tokens[t0 + row] : 0;
    if (tok[i] < 0 || tok[i] >= vocab) tok[i] = 0;
  }
#pragma unroll 4
  for (int i = tid; i < kTsTokens * (WIDTH / 4); i += kTrThreads) {
    const int r = i / (WIDTH / 4), c = i % (WIDTH / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < nt) {
      v = *reinterpret_cast<const float4*>(residual + (size_t)(t0 + r) * WIDTH + c);
      if (x) {
        const uint2 raw = *reinterpret_cast<const uint2*>(x + (size_t)(t0 + r) * WIDTH + c);
        const float2 lo = unpack_bf16(raw.x), hi = unpack_bf16(raw.y);
        v.x += lo.x; v.y += lo.y; v.z += hi.x; v.w += hi.y;
      }
      if (bias) {
        const float4 b = *reinterpret_cast<const float4*>(bias + c);
        v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
      }
    }
    *reinterpret_cast<float4*>(s32 + r * LS + c) = v;
#pragma unroll
    for (int w = 0; w < 3; ++w) {                       // (the terms of ts_split)
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
      *reinterpret_cast<uint2*>(s16 + (w * kTsTokens + r) * LT + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
      v.x -= a.x; v.y -= a.y; v.z -= b.x; v.w -= b.y;
    }
  }
  __nv_bfloat16 entry[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) entry[i] = table[(size_t)tok[i] * table_ld + column + (tid + i * kTrThreads) % DIM];
  __syncthreads();
  // this warp's share of z
  float acc[NZ][4];
#pragma unroll
  for (int n = 0; n < NZ; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
#pragma unroll
  for (int k = 0; k < KB; ++k) {
#pragma unroll
    for (int n = 0; n < NZ; ++n) tr_trade(wg[k][n]);
#pragma unroll
    for (int w = 2; w >= 0; --w) {
      uint32_t a0[4], a1[4];
      const uint32_t at = smem_u32(s16 + (w * kTsTokens + lm_row) * LT + rank * SL + 32 * k + 8 * lm_half);
      ldmatrix_x4(a0, at);
      ldmatrix_x4(a1, at + 32);
#pragma unroll
      for (int n = 0; n < NZ; ++n) {
        mma_bf16_16816(acc[n], a0, wg[k][n].x, wg[k][n].y);
        mma_bf16_16816(acc[n], a1, wg[k][n].z, wg[k][n].w);
      }
    }
  }
  // this warp's rows of W_proj, while the shares are added up
  uint4 wp[NY][DIM / 32];
#pragma unroll
  for (int j = 0; j < NY; ++j)
#pragma unroll
    for (int k = 0; k < DIM / 32; ++k) wp[j][k] = __ldg(reinterpret_cast<const uint4*>(w_proj + (size_t)(warp * SLICE + 8 * j + g) * DIM + 32 * k + q8));
  __syncthreads();                                      // the terms have been read
#pragma unroll
  for (int n = 0; n < NZ; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      *reinterpret_cast<float2*>(zpart + (rank * kTsTokens + g + 8 * i) * DIM + 8 * (half * NZ + n) + c2) = make_float2(acc[n][2 * i], acc[n][2 * i + 1]);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int at = tid + i * kTrThreads;
    float z = 0.f;
#pragma unroll
    for (int b = 0; b < kTsBlocks; ++b) z += zpart[b * kTsTokens * DIM + at];
    const float v = at / DIM < nt ? ts_gelu_tanh(z) * __bfloat162float(entry[i]) : 0.f;
    ts_split(v, g16 + at / DIM * LG + at % DIM, kTsTokens * LG);
  }
  __syncthreads();
  float y[NY][4];
#pragma unroll
  for (int j = 0; j < NY; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) y[j][e] = 0.f;
#pragma unroll
  for (int k = 0; k < DIM / 32; ++k) {
#pragma unroll
    for (int j = 0; j < NY; ++j) tr_trade(wp[j][k]);
#pragma unroll
    for (int step = 0; step < 2; ++step)
#pragma unroll
      for (int w = 2; w >= 0; --w) {
        uint32_t a[4];
        ldmatrix_x4(a, smem_u32(g16 + (w * kTsTokens + lm_row) * LG + 32 * k + 16 * step + 8 * lm_half));
#pragma unroll
        for (int j = 0; j < NY; ++j) mma_bf16_16816(y[j], a, step ? wp[j][k].z : wp[j][k].x, step ? wp[j][k].w : wp[j][k].y);
      }
  }
#pragma unroll
  for (int j0 = 0; j0 < NY; j0 += NT) {
    float ss[2] = {0.f, 0.f};
#pragma unroll
    for (int j = j0; j < j0 + NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) ss[e >> 1] = fmaf(y[j][e], y[j][e], ss[e >> 1]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 1);
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 2);
      if ((lane & 3) == 0) s_ss[(warp * NY + j0) / NT][g + 8 * i] = ss[i];
    }
  }
  __syncthreads();
  if (tid < kTsTokens * kTsBlocks) {
    const int row = tid % kTsTokens, peer = tid / kTsTokens;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kTsThreads / 32; ++w) v += s_ss[peer * (kTsThreads / 32) + w][row];
    s_rank[peer][row] = v;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = g + 8 * i;
    if (row >= nt) continue;
    float total = 0.f;
#pragma unroll
    for (int b = 0; b < kTsBlocks; ++b) total += s_rank[b][row];
    const float rrms = 1.0f / sqrtf(total / (float)WIDTH + eps);
#pragma unroll
    for (int j = 0; j < NY; ++j) {
      const int c = warp * SLICE + 8 * j + c2;
      const float2 w = *reinterpret_cast<const float2*>(norm_w + c), s = *reinterpret_cast<const float2*>(s32 + row * LS + c);
      *reinterpret_cast<float2*>(residual + (size_t)(t0 + row) * WIDTH + c) = make_float2(s.x + y[j][2 * i] * rrms * w.x, s.y + y[j][2 * i + 1] * rrms * w.y);
    }
  }
}

template <int WIDTH, int DIM>
int token_side_rows(float* residual, const void* x, const float* bias, const int* tokens, const void* table, int table_ld, int column, int vocab,
                    const void* w_gate, const void* w_proj, const float* norm_w, int n_tokens, float eps, void* stream) {
  static SmemRaised raised;
  auto kernel = token_side_rows_kernel<WIDTH, DIM>;
  if (int rc = raise_shared_memory("token_side", kernel, (int)tr_smem(WIDTH, DIM), raised)) return rc;
  return launch_kernel("token_side", kernel, dim3((n_tokens + kTsTokens - 1) / kTsTokens), dim3(kTrThreads), tr_smem(WIDTH, DIM),
                       as_stream(stream), residual, (const __nv_bfloat16*)x, bias, tokens, (const __nv_bfloat16*)table, table_ld, column, vocab,
                       (const __nv_bfloat16*)w_gate, (const __nv_bfloat16*)w_proj, norm_w, eps, n_tokens);
}

}  // namespace ptl

// -2: widths other than 512, 1,024 and 2,048, dims that are no whole sixteens up to 128, or rows off their boundaries.
PTL_EXPORT int ptl_token_side_cluster_bf16(float* residual, const void* x, const float* bias, const int* tokens, const void* table,
                                           int table_ld, int column, int dim, int vocab, const void* w_gate, const void* w_proj,
                                           const float* norm_w, int n_tokens, int width, float eps, void* stream) {
  using namespace ptl;
  if ((width != 512 && width != 1024 && width != 2048) || dim < 16 || dim % 16 || dim > kTsMaxDim || !aligned16(residual) ||
      (x && !aligned16(x)) || (bias && !aligned16(bias)) || !aligned16(w_gate) || !aligned16(w_proj) || !aligned16(norm_w))
    return -2;
  PTL_REQUIRE(n_tokens >= 0 && n_tokens <= (1 << 27) && column >= 0 && column + dim <= table_ld && eps > 0.f && vocab > 0,
              "token_side: bad sizes width=%d dim=%d column=%d of %d", width, dim, column, table_ld);
  if (n_tokens == 0) return 0;
  // The rows' form from where the cluster form needs another turn of clusters; its own time is that of one block an SM up to 2,368 tokens.  Width
  // 1,024: 64 dims 11.8 us by clusters and 14.6 by rows at 768 tokens, 15.9 and 14.5 at 784; 32 dims 10.9 and 11.3 at 1,072, 11.8 and 11.2 at
  // 1,088; 2,048 tokens of 64 dims 32.3 and 14.9.  Width 512: 64 dims 9.0 and 9.2 at 560, 10.2 and 9.2 at 576; 32 dims 6.8 both from 560 to 576, 7.0 and 6.8 at 592.
  if (n_tokens > (width == 512 ? 560 : dim == 64 ? 768 : 1072) && width <= 1024 && (dim == 32 || dim == 64)) {
    const auto rows = width == 512 ? dim == 32 ? token_side_rows<512, 32> : token_side_rows<512, 64>
                                   : dim == 32 ? token_side_rows<1024, 32> : token_side_rows<1024, 64>;
    return rows(residual, x, bias, tokens, table, table_ld, column, vocab, w_gate, w_proj, norm_w, n_tokens, eps, stream);
  }
  const auto fn = width == 512 ? token_side_cluster<64> : width == 1024 ? token_side_cluster<128> : token_side_cluster<256>;
  return fn(residual, x, bias, tokens, table, table_ld, column, dim, vocab, w_gate, w_proj, norm_w, n_tokens, eps, stream);
}
