// Attention over the paged cache on the CUDA cores, for any mix of prompt portions and single
// decoded tokens: one or four warps per (token, query head), optional split of the key range
// over blockIdx.z with a merge kernel.  Everything but the stored q/k/v is float32: scores, running
// maximum, sum, accumulator, merge.  It is the float32 path's attention and the reference
// against which faster kernels are checked.
//
// With float32 inputs the two sums of attention are compensated, still in 32-bit arithmetic: the
// score q.k keeps the rounding error of every product and partial sum in a second float (a dot
// product as if summed in twice the precision), and the accumulator of P.V and the softmax sum are
// (high, low) pairs of floats.  Scores of size 10 make softmax weights as wrong (relatively) as the
// score is (absolutely), and a plain 64-term sum is wrong by a few 1e-7 there: over 16 layers of a
// 2,048-wide model these sums, not the matrix products, were what kept logits 8e-5 from a float64
// computation.  bfloat16 inputs (this kernel as the fallback for head sizes the tensor-core
// kernels leave) take plain sums: their inputs are a thousand times coarser than that.
//
// Token t (request r = tok_req[t], position p = positions[t]) sees keys lo..p of its request,
// lo = max(0, p - window + 1) when window > 0, else 0.  Key n lives in page
// block_table[r][n / page_size] at offset n % page_size of the layer's cache
// [pages][2 (k,v)][nkv][page_size][d].  Query head h reads kv head h / (nq / nkv).
#include "common.cuh"

namespace ptl {

constexpr int kMaxDimPerLane = 8;   // head sizes up to 256

// (hi, lo) += a * b without losing the rounding error of the product or of the sum
__device__ __forceinline__ void two_fma(float& hi, float& lo, float a, float b) {
  const float h = __fmul_rn(a, b);
  const float r = fmaf(a, b, -h);                             // the product's rounding error, exactly
  const float t = __fadd_rn(hi, h);
  const float z = __fsub_rn(t, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, z)), __fsub_rn(h, z));   // the sum's rounding error, exactly
  hi = t;
  lo = __fadd_rn(lo, __fadd_rn(e, r));
}
// (hi, lo) *= c
__device__ __forceinline__ void two_scale(float& hi, float& lo, float c) {
  const float h = __fmul_rn(hi, c);
  lo = fmaf(lo, c, fmaf(hi, c, -h));
  hi = h;
}

// (hi, lo) += (h, l)
__device__ __forceinline__ void two_add(float& hi, float& lo, float h, float l) {
  const float t = __fadd_rn(hi, h);
  const float z = __fsub_rn(t, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, z)), __fsub_rn(h, z));
  hi = t;
  lo = __fadd_rn(lo, __fadd_rn(l, e));
}

// The same on two sums at once, by the packed float32 instructions (half the issue slots, the same roundings); `minus_a` is -a.
__device__ __forceinline__ void two_fma_pair(float2& hi, float2& lo, float2 a, float2 minus_a, float2 b) {
  const float2 h = mul2(a, b);
  const float2 r = fma2(minus_a, b, h);                       // minus the products' rounding errors, exactly
  const float2 t = add2(hi, h);
  const float2 z = sub2(t, hi);
  const float2 e = add2(sub2(hi, sub2(t, z)), sub2(h, z));
  hi = t;
  lo = add2(lo, sub2(e, r));
}

// A head's keys in groups of 32, one after the other: the group's scores, a lane a key; the running maximum, to which what was summed
// so far shrinks; then the keys' weights times their values, an entry a lane.  Two kernels with the same sums in the same order, so that
// a token's bits are the same whatever else the step holds.
constexpr int kPacketsAhead = 16;     // packets of a key per lane: the whole key up to 64 floats
__host__ __device__ constexpr int values_ahead(int dpl) { return dpl <= 2 ? 16 : dpl <= 4 ? 8 : 4; }

// The score of a key row with the query in shared memory (16-bit inputs: scaled already).  float32: the even and the odd entries'
// compensated sums side by side, two entries an instruction.
template <typename T>
__device__ __forceinline__ float simt_score(const T* __restrict__ kp, const float* qs, int d, float scale) {
  constexpr int VN = Vec16<T>::N;
  constexpr bool kCompensated = sizeof(T) == 4;
  float dot = 0.f;
  float2 dot2 = make_float2(0.f, 0.f), low2 = dot2;
  for (int i0 = 0; i0 < d; i0 += kPacketsAhead * VN) {
    Vec16<T> kv[kPacketsAhead];
#pragma unroll
    for (int j = 0; j < kPacketsAhead; ++j) kv[j] = load16(kp + min(i0 + j * VN, d - VN));
#pragma unroll
    for (int j = 0; j < kPacketsAhead; ++j) {
      const int i = i0 + j * VN;
      if (i >= d) break;
      if constexpr (kCompensated) {
        const float4 a = *reinterpret_cast<const float4*>(qs + i);
        two_fma_pair(dot2, low2, make_float2(a.x, a.y), make_float2(-a.x, -a.y), make_float2(kv[j].get(0), kv[j].get(1)));
        two_fma_pair(dot2, low2, make_float2(a.z, a.w), make_float2(-a.z, -a.w), make_float2(kv[j].get(2), kv[j].get(3)));
      } else {
#pragma unroll
        for (int e = 0; e < VN; ++e) dot = fmaf(qs[i + e], kv[j].get(e), dot);
      }
    }
  }
  if constexpr (!kCompensated) return dot;
  two_add(dot2.x, low2.x, dot2.y, low2.y);
  return __fmul_rn(__fadd_rn(dot2.x, low2.x), scale);      // (rounded here in both kernels, not folded into what follows)
}
// What was summed so far to a new maximum.
template <bool COMPENSATED>
__device__ __forceinline__ void simt_shrink(float& hi, float& lo, float alpha) {
  if constexpr (COMPENSATED) two_scale(hi, lo, alpha);
  else hi *= alpha;
}
__device__ __forceinline__ float simt_alpha(float m, float m_new) {
  return m_new == -INFINITY ? 1.f : expf(m - m_new);       // m = -inf on the first group gives 0; no score yet: nothing to shrink
}

struct SimtKeys { int r, k_begin, k_end; };                // r < 0: a padding row of a fixed-size batch; it sees no key and yields zeros
__device__ __forceinline__ SimtKeys simt_keys(const int* tok_req, const int* positions, int t, int window, int splits, int split) {
  const int r = tok_req[t], p = positions[t];
  const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
  const int nkeys = r < 0 ? 0 : p - lo + 1;
  const int chunk = ((nkeys + splits - 1) / splits + 31) & ~31;
  const int k_begin = lo + split * chunk;
  return {r, k_begin, r < 0 ? k_begin : min(lo + (split + 1) * chunk, p + 1)};
}

// A warp per head, everything in registers.  Bound by a group's chain: a key's products with their errors, then 32 keys' values, some
// 1,500 instructions and two trips to memory, and for heads that share no keys by the bytes: 600 tokens of 32 heads of 64 620 us (690 with scalar sums), 64 tokens
// of 8 heads of 128 at contexts of 4,000 497 (2.1 GB of keys and values).  It needs L1, since a lane reads its key 16 bytes at a time: with the
// scores and sums of 512 keys in shared memory instead (8.8 KB a head of 128) those took 925 us.
constexpr int kWarpsPerBlock = 4;
template <typename T, int DPL>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
paged_attention_simt_kernel(T* __restrict__ out, float* __restrict__ part_acc, float* __restrict__ part_ml,
                            const T* __restrict__ q, const T* __restrict__ cache,
                            const int* __restrict__ block_table, const int* __restrict__ tok_req,
                            const int* __restrict__ positions, int q_stride, int out_stride,
                            int bt_stride, int nq, int nkv, int d, int page_size, float scale,
                            int window, int splits, int num_pages) {
  extern __shared__ __align__(16) float qs_all[];  // [warps][d] scaled query
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x;
  const int h = blockIdx.y * kWarpsPerBlock + warp;
  if (h >= nq) return;
  const int split = blockIdx.z;
  float* qs = qs_all + warp * d;
  const T* qrow = q + (size_t)t * q_stride + (size_t)h * d;
  constexpr bool kCompensated = sizeof(T) == 4;
  for (int i = lane; i < d; i += 32) qs[i] = kCompensated ? to_f32(qrow[i]) : to_f32(qrow[i]) * scale;
  __syncwarp();

  const SimtKeys keys = simt_keys(tok_req, positions, t, window, splits, split);
  const int kvh = h / (nq / nkv);
  const size_t plane = (size_t)nkv * page_size * d;
  const int* bt = block_table + (size_t)max(keys.r, 0) * bt_stride;

  constexpr int PAIRS = DPL / 2;
  float m = -INFINITY, l = 0.f, l_lo = 0.f;
  float2 acc[PAIRS], low[PAIRS];     // entries lane, lane + 32 of the value; lane + 64, ...
#pragma unroll
  for (int i = 0; i < PAIRS; ++i) acc[i] = low[i] = make_float2(0.f, 0.f);

  for (int k0 = keys.k_begin; k0 < keys.k_end; k0 += 32) {
    const int key = k0 + lane;
    bool valid = key < keys.k_end;
    size_t base = 0;  // element offset of this lane's key row (k plane)
    float s = -INFINITY;
    const int page = valid ? bt[key / page_size] : 0;
    if (page < 0 || page >= num_pages) valid = false;  // never follow a table entry outside the pool
    if (valid) {
      base = ((size_t)page * 2) * plane + ((size_t)kvh * page_size + key % page_size) * d;
      s = simt_score(cache + base, qs, d, scale);
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float pr = valid ? expf(s - m_new) : 0.f;
    const float alpha = simt_alpha(m, m_new);
    const float sum = warp_sum(pr);
    if constexpr (!kCompensated) l = fmaf(l, alpha, sum);
    else if (alpha != 1.f) two_scale(l, l_lo, alpha);
    if constexpr (kCompensated) two_fma(l, l_lo, sum, 1.f);
    if (!kCompensated || alpha != 1.f) {                // (uniform over the warp)
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) {
        simt_shrink<kCompensated>(acc[i].x, low[i].x, alpha);
        simt_shrink<kCompensated>(acc[i].y, low[i].y, alpha);
      }
    }
    m = m_new;
    const int nvalid = min(32, keys.k_end - k0);
    constexpr int kValuesAhead = values_ahead(DPL);
    for (int j0 = 0; j0 < nvalid; j0 += kValuesAhead) {
      float pj[kValuesAhead];
      T v[kValuesAhead][DPL];
#pragma unroll
      for (int u = 0; u < kValuesAhead; ++u) {
        pj[u] = __shfl_sync(0xffffffffu, pr, j0 + u);         // 0 behind the last key, and for a key without a page
        const unsigned long long bj = __shfl_sync(0xffffffffu, (unsigned long long)base, j0 + u);
        const T* vp = cache + (size_t)bj + plane;
#pragma unroll
        for (int i = 0; i < DPL; ++i)
          if (pj[u] != 0.f && lane + 32 * i < d) v[u][i] = vp[lane + 32 * i];
      }
#pragma unroll
      for (int u = 0; u < kValuesAhead; ++u) {
        if (pj[u] == 0.f) continue;                           // (uniform over the warp)
#pragma unroll
        for (int i = 0; i < PAIRS; ++i) {
          if constexpr (kCompensated) {                       // (an entry past the head's last is not stored)
            two_fma_pair(acc[i], low[i], make_float2(pj[u], pj[u]), make_float2(-pj[u], -pj[u]), make_float2(to_f32(v[u][2 * i]), to_f32(v[u][2 * i + 1])));
          } else {
            if (lane + 64 * i < d) acc[i].x = fmaf(pj[u], to_f32(v[u][2 * i]), acc[i].x);
            if (lane + 64 * i + 32 < d) acc[i].y = fmaf(pj[u], to_f32(v[u][2 * i + 1]), acc[i].y);
          }
        }
      }
    }
  }
  if constexpr (kCompensated) {
    l = __fadd_rn(l, l_lo);
#pragma unroll
    for (int i = 0; i < PAIRS; ++i) { acc[i].x = __fadd_rn(acc[i].x, low[i].x); acc[i].y = __fadd_rn(acc[i].y, low[i].y); }
  }

  if (splits == 1) {
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    T* o = out + (size_t)t * out_stride + (size_t)h * d;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int dd = lane + 32 * i;
      if (dd < d) o[dd] = from_f32<T>((i & 1 ? acc[i / 2].y : acc[i / 2].x) * inv);
    }
  } else {
    const size_t idx = ((size_t)t * nq + h) * splits + split;
    float* pa = part_acc + idx * d;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int dd = lane + 32 * i;
      if (dd < d) pa[dd] = i & 1 ? acc[i / 2].y : acc[i / 2].x;
    }
    if (lane == 0) { part_ml[idx * 2] = m; part_ml[idx * 2 + 1] = l; }
  }
}

// Four warps per head, for steps of few heads, which leave the SMs' schedulers a warp each at best: the warps score the groups of up to 512
// keys in turn and turn them into weights, each group to the running maximum that it would meet in the walk above; then a thread an entry (or
// two) adds the values up, key after key.  Bound by the same chains, side by side: four tokens of 32 heads of 64 at contexts of 134 14.4 us,
// one warp a head 30.
constexpr int kWideTurns = 4, kWideGroups = kWarpsPerBlock * kWideTurns;
template <typename T, int EPT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
paged_attention_simt_wide_kernel(T* __restrict__ out, float* __restrict__ part_acc, float* __restrict__ part_ml,
                                 const T* __restrict__ q, const T* __restrict__ cache,
                                 const int* __restrict__ block_table, const int* __restrict__ tok_req,
                                 const int* __restrict__ positions, int q_stride, int out_stride,
                                 int bt_stride, int nq, int nkv, int d, int page_size, float scale,
                                 int window, int splits, int num_pages) {
  extern __shared__ __align__(16) float qs[];                 // [d] scaled query
  __shared__ float s_p[kWideGroups * 32];                     // scores, then weights
  __shared__ long long s_at[kWideGroups * 32];                // element offset of the keys' rows; -1: no page
  __shared__ float s_max[kWideGroups], s_sum[kWideGroups], s_alpha[kWideGroups];
  pdl_wait();
  pdl_launch_dependents();
  constexpr int THREADS = kWarpsPerBlock * 32, AHEAD = 32 / EPT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t = blockIdx.x, h = blockIdx.y, split = blockIdx.z;
  const T* qrow = q + (size_t)t * q_stride + (size_t)h * d;
  constexpr bool kCompensated = sizeof(T) == 4;
  for (int i = tid; i < d; i += THREADS) qs[i] = kCompensated ? to_f32(qrow[i]) : to_f32(qrow[i]) * scale;
  const SimtKeys keys = simt_keys(tok_req, positions, t, window, splits, split);
  const int kvh = h / (nq / nkv);
  const size_t plane = (size_t)nkv * page_size * d;
  const int* bt = block_table + (size_t)max(keys.r, 0) * bt_stride;
  float m = -INFINITY, l = 0.f, l_lo = 0.f, acc[EPT], low[EPT];
#pragma unroll
  for (int i = 0; i < EPT; ++i) acc[i] = low[i] = 0.f;
  __syncthreads();

  for (int c0 = keys.k_begin; c0 < keys.k_end; c0 += kWideGroups * 32) {
    const int groups = min(kWideGroups, (keys.k_end - c0 + 31) / 32);
#pragma unroll 1
    for (int gr = warp; gr < groups; gr += kWarpsPerBlock) {
      const int key = c0 + gr * 32 + lane;
      const int page = key < keys.k_end ? bt[key / page_size] : -1;
      long long at = -1;
      float s = -INFINITY;
      if (page >= 0 && page < num_pages) {                    // never follow a table entry outside the pool
        at = (long long)((size_t)page * 2 * plane + ((size_t)kvh * page_size + key % page_size) * d);
        for (int i = 0; i < d; i += 128 / (int)sizeof(T))     // the key's value, wanted when all weights are known
          asm volatile("prefetch.global.L2 [%0];" ::"l"(cache + at + plane + i));
        s = simt_score(cache + at, qs, d, scale);
      }
      s_p[gr * 32 + lane] = s;
      s_at[gr * 32 + lane] = at;
      const float top = warp_max(s);
      if (lane == 0) s_max[gr] = top;
    }
    __syncthreads();
    // values on their way while those before them are added up: a group's, or half a group's where a thread has two entries
    T v[AHEAD][EPT], next[AHEAD][EPT];
    const auto ask = [&](int key, T (&to)[AHEAD][EPT]) {
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const long long at = s_at[key + u];
#pragma unroll
        for (int i = 0; i < EPT; ++i)
          if (at >= 0 && tid + THREADS * i < d) to[u][i] = cache[(size_t)at + plane + tid + THREADS * i];
      }
    };
    ask(0, v);
#pragma unroll 1
    for (int gr = warp; gr < groups; gr += kWarpsPerBlock) {
      float before = m;
      for (int i = 0; i < gr; ++i) before = fmaxf(before, s_max[i]);
      const float m_new = fmaxf(before, s_max[gr]);
      const float pr = s_at[gr * 32 + lane] >= 0 ? expf(s_p[gr * 32 + lane] - m_new) : 0.f;
      s_p[gr * 32 + lane] = pr;                               // (0 behind the last key, and for a key without a page)
      const float sum = warp_sum(pr);
      if (lane == 0) { s_sum[gr] = sum; s_alpha[gr] = simt_alpha(before, m_new); }
    }
    __syncthreads();
#pragma unroll 1
    for (int key = 0; key < groups * 32; key += AHEAD) {
      if (key + AHEAD < groups * 32) ask(key + AHEAD, next);
      if (AHEAD == 32 || key % 32 == 0) {
        const int gr = key / 32;
        const float alpha = s_alpha[gr];
        m = fmaxf(m, s_max[gr]);
        if constexpr (!kCompensated) l = fmaf(l, alpha, s_sum[gr]);
        else if (alpha != 1.f) two_scale(l, l_lo, alpha);
        if constexpr (kCompensated) two_fma(l, l_lo, s_sum[gr], 1.f);
        if (!kCompensated || alpha != 1.f) {
#pragma unroll
          for (int i = 0; i < EPT; ++i) simt_shrink<kCompensated>(acc[i], low[i], alpha);
        }
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const float pj = s_p[key + u];
        if (pj == 0.f) continue;                              // (uniform over the block)
#pragma unroll
        for (int i = 0; i < EPT; ++i) {                       // (an entry past the head's last is not stored)
          if constexpr (kCompensated) two_fma(acc[i], low[i], pj, to_f32(v[u][i]));
          else acc[i] = fmaf(pj, to_f32(v[u][i]), acc[i]);
        }
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
#pragma unroll
        for (int i = 0; i < EPT; ++i) v[u][i] = next[u][i];
    }
    __syncthreads();                                          // (the next keys' scores and maxima take these places)
  }
  if constexpr (kCompensated) {
    l = __fadd_rn(l, l_lo);
#pragma unroll
    for (int i = 0; i < EPT; ++i) acc[i] = __fadd_rn(acc[i], low[i]);
  }
  const size_t idx = ((size_t)t * nq + h) * splits + split;
  const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int dd = tid + THREADS * i;
    if (dd >= d) continue;
    if (splits == 1) out[(size_t)t * out_stride + (size_t)h * d + dd] = from_f32<T>(acc[i] * inv);
    else part_acc[idx * d + dd] = acc[i];
  }
  if (splits > 1 && tid == 0) { part_ml[idx * 2] = m; part_ml[idx * 2 + 1] = l; }
}

// Merge of the per-split partial results: out = sum_z e^{m_z - M} acc_z / sum_z e^{m_z - M} l_z.
// One warp per (token, head); the lanes share the weights of the splits and split the head's
// dimensions among them.
constexpr int kMergeWarps = 4;
template <typename T>
__global__ void __launch_bounds__(kMergeWarps * 32)
attention_merge_kernel(T* __restrict__ out, const float* __restrict__ part_acc,
                       const float* __restrict__ part_ml, int out_stride, int nq, int d,
                       int splits, const int* __restrict__ items, int n_rows) {
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = blockIdx.x * kMergeWarps + warp;       // (row, head) pair
  if (pair >= n_rows * nq) return;
  const int ti = pair / nq, h = pair % nq;
  const int t = items ? items[ti] : ti;
  const size_t idx0 = ((size_t)t * nq + h) * splits;
  // lane z holds the (max, sum) pair of split z, 32 splits at a time; the weights are then handed
  // round by shuffles, so the loads of the partial accumulators below do not wait on one another
  float M = -INFINITY;
  for (int z = lane; z < splits; z += 32) M = fmaxf(M, part_ml[(idx0 + z) * 2]);
  M = warp_max(M);
  float L = 0.f;
  float acc[kMaxDimPerLane];
#pragma unroll
  for (int i = 0; i < kMaxDimPerLane; ++i) acc[i] = 0.f;
  for (int z0 = 0; z0 < splits; z0 += 32) {
    const int z = z0 + lane;
    float wz = 0.f;
    if (z < splits) {
      const float mz = part_ml[(idx0 + z) * 2];
      if (mz > -INFINITY) {
        wz = expf(mz - M);
        L += wz * part_ml[(idx0 + z) * 2 + 1];
      }
    }
    const int n = min(32, splits - z0);
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
      const float wj = __shfl_sync(0xffffffffu, wz, j);
      const float* pa = part_acc + (idx0 + z0 + j) * d;      // an empty split wrote zeros here
#pragma unroll
      for (int i = 0; i < kMaxDimPerLane; ++i) {
        const int dd = lane + 32 * i;
        if (dd < d) acc[i] = fmaf(wj, pa[dd], acc[i]);
      }
    }
  }
  L = warp_sum(L);
  const float inv = L > 0.f ? 1.0f / L : 0.f;
  T* o = out + (size_t)t * out_stride + (size_t)h * d;
#pragma unroll
  for (int i = 0; i < kMaxDimPerLane; ++i) {
    const int dd = lane + 32 * i;
    if (dd < d) o[dd] = from_f32<T>(acc[i] * inv);
  }
}

template <typename T>
int paged_attention_simt(void* out, const void* q, const void* cache, const int* block_table,
                         const int* tok_req, const int* positions, float* part_acc, float* part_ml,
                         int tokens, int q_stride, int out_stride, int bt_stride, int nq, int nkv, int d,
                         int page_size, float scale, int window, int splits, int num_pages, void* stream) {
  PTL_REQUIRE(tokens >= 0 && nq > 0 && nkv > 0 && page_size > 0, "paged_attention: bad sizes");
  PTL_REQUIRE(nq % nkv == 0, "paged_attention: %d query heads are no multiple of %d kv heads", nq, nkv);
  PTL_REQUIRE(d % 16 == 0 && d >= 16 && d <= 32 * kMaxDimPerLane, "paged_attention: head size %d must be a multiple of 16 in [16, %d]", d, 32 * kMaxDimPerLane);
  PTL_REQUIRE(splits >= 1 && splits <= 65535, "paged_attention: splits=%d", splits);
  PTL_REQUIRE(splits == 1 || (part_acc && part_ml), "paged_attention: splits > 1 need scratch buffers");
  PTL_REQUIRE(window >= 0 && num_pages > 0, "paged_attention: window must be >= 0 and the pool non-empty");
  PTL_REQUIRE(aligned16(q) && aligned16(cache) && (q_stride * sizeof(T)) % 16 == 0, "paged_attention: q and cache must be 16-byte aligned");
  if (tokens == 0) return 0;
  const auto launch = [&](auto kernel, int heads) {
    return launch_kernel("paged_attention", kernel, dim3(tokens, (nq + heads - 1) / heads, splits), dim3(kWarpsPerBlock * 32), (size_t)heads * d * sizeof(float),
                         as_stream(stream), (T*)out, part_acc, part_ml, (const T*)q, (const T*)cache, block_table, tok_req, positions, q_stride, out_stride,
                         bt_stride, nq, nkv, d, page_size, scale, window, splits, num_pages);
  };
  // A warp per head from three heads an SM on (neighbouring heads of a block read the same keys, out of L1), from six or eight where a
  // value's entries keep the four warps' threads busy.  One warp and four, us, 32 heads over 8 kv heads,
  // 24 tokens at contexts of 300 (5.2 heads an SM): heads of 64 51 and 58, of 128 87 and 80, of 256 264 and 153; 32 tokens (6.9): of 128 102
  // and 117, of 256 261 and 216.  16 tokens at 500 (3.5): of 32 56 and 62, of 64 77 and 75; bfloat16, of 48 44 and 63, of 80 64 and 70, of 256 162 and 77.
  const int wide_heads = d > 128 ? 8 : d > 64 && sizeof(T) == 4 ? 6 : 3;
  int rc;
  if ((long long)tokens * nq * splits < (long long)wide_heads * sm_count_of_device())
    rc = launch(d <= kWarpsPerBlock * 32 ? paged_attention_simt_wide_kernel<T, 1> : paged_attention_simt_wide_kernel<T, 2>, 1);
  else
    rc = launch(d <= 64 ? paged_attention_simt_kernel<T, 2> : d <= 128 ? paged_attention_simt_kernel<T, 4> : paged_attention_simt_kernel<T, kMaxDimPerLane>,
                kWarpsPerBlock);
  if (rc) return rc;
  if (splits > 1) {
    const long long pairs = (long long)tokens * nq;
    rc = launch_kernel("attention_merge", attention_merge_kernel<T>, dim3((unsigned)((pairs + kMergeWarps - 1) / kMergeWarps)),
                       dim3(kMergeWarps * 32), 0, as_stream(stream), (T*)out, (const float*)part_acc, (const float*)part_ml,
                       out_stride, nq, d, splits, (const int*)nullptr, tokens);
  }
  return rc;
}

// Merge for the tensor-core decode kernel: `items` (or 0..tokens-1) names the token rows.
int attention_merge_bf16(void* out, const float* part_acc, const float* part_ml, int tokens, int out_stride,
                         int nq, int d, int splits, const int* items, void* stream) {
  const long long pairs = (long long)tokens * nq;
  return launch_kernel("attention_merge", attention_merge_kernel<__nv_bfloat16>,
                       dim3((unsigned)((pairs + kMergeWarps - 1) / kMergeWarps)), dim3(kMergeWarps * 32), 0, as_stream(stream),
                       (__nv_bfloat16*)out, part_acc, part_ml, out_stride, nq, d, splits, items, tokens);
}

}  // namespace ptl

PTL_EXPORT int ptl_paged_attention_simt_f32(void* out, const void* q, const void* cache, const int* block_table, const int* tok_req, const int* positions, float* part_acc, float* part_ml, int tokens, int q_stride, int out_stride, int bt_stride, int nq, int nkv, int d, int page_size, float scale, int window, int splits, int num_pages, void* stream) {
  return ptl::paged_attention_simt<float>(out, q, cache, block_table, tok_req, positions, part_acc, part_ml, tokens, q_stride, out_stride, bt_stride, nq, nkv, d, page_size, scale, window, splits, num_pages, stream);
}
PTL_EXPORT int ptl_paged_attention_simt_bf16(void* out, const void* q, const void* cache, const int* block_table, const int* tok_req, const int* positions, float* part_acc, float* part_ml, int tokens, int q_stride, int out_stride, int bt_stride, int nq, int nkv, int d, int page_size, float scale, int window, int splits, int num_pages, void* stream) {
  return ptl::paged_attention_simt<__nv_bfloat16>(out, q, cache, block_table, tok_req, positions, part_acc, part_ml, tokens, q_stride, out_stride, bt_stride, nq, nkv, d, page_size, scale, window, splits, num_pages, stream);
}
