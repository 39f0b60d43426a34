// Attention over the paged cache on the CUDA cores, for any mix of prompt portions and single
// decoded tokens: four warps per (token, query head) that take groups of 32 keys in turns, optional split of the key range
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

// A head's keys in groups of 32, the groups dealt to kParts parts in turn; the scores of up to kPartTurns turns (512 keys) are kept in
// shared memory until their common maximum is known, so no weight of theirs is rescaled.  The parts' sums meet, as pairs of floats,
// in their order.  Which part a group goes to depends on its place in the context alone, so a token's bits are the same
// whatever else the step holds, and whether its parts are worked side by side (WARPS = 4) or one after the other (WARPS = 1).
//
// Bound by a group's chain: a key's 64 products with their errors, then 32 keys' values, some 1,500 instructions and two trips to L2.  A few
// tokens leave the SMs' schedulers a warp each at best, so there a head's parts go to four warps, a head to a block: four tokens of 32 heads at contexts
// of 40 to 134, one warp walking a head's groups one after the other took 30 us, 15 so.  With enough blocks (a prompt) a warp takes
// a whole head and no warp waits for another: prompts of 33 to 127 tokens 82 us before, 75 now (89 where the values are asked for early
// there too).
constexpr int kPacketsAhead = 16;     // packets of a key per lane: the whole key up to 64 floats
constexpr int kParts = 4, kPartTurns = 4;
__host__ __device__ constexpr int values_ahead(int dpl) { return dpl <= 2 ? 16 : dpl <= 4 ? 8 : 4; }
// floats of a part: its sums (hi, lo) of values and of weights, its maximum, its keys' scores and pages.  Of a head: the scaled query and its parts
__host__ __device__ constexpr int simt_part_floats(int d) { return 2 * d + 4 + 2 * kPartTurns * 32; }
__host__ __device__ constexpr int simt_head_floats(int d) { return d + kParts * simt_part_floats(d); }

template <typename T, int DPL, int HEADS, int WARPS>
__global__ void __launch_bounds__(HEADS * WARPS * 32)
paged_attention_simt_kernel(T* __restrict__ out, float* __restrict__ part_acc, float* __restrict__ part_ml,
                            const T* __restrict__ q, const T* __restrict__ cache,
                            const int* __restrict__ block_table, const int* __restrict__ tok_req,
                            const int* __restrict__ positions, int q_stride, int out_stride,
                            int bt_stride, int nq, int nkv, int d, int page_size, float scale,
                            int window, int splits, int num_pages) {
  static_assert(WARPS == 1 || (WARPS == kParts && HEADS == 1), "a head's warps meet at the block's barrier");
  extern __shared__ __align__(16) float simt_smem[];
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = WARPS == 1 ? 0 : threadIdx.x >> 5, slot = WARPS == 1 ? threadIdx.x >> 5 : 0;
  const int t = blockIdx.x;
  const int h = blockIdx.y * HEADS + slot;
  if (h >= nq) return;                 // (a whole head's warps: those that stay do not wait for it)
  const int split = blockIdx.z;
  const auto meet = [] {
    if constexpr (WARPS == 1) __syncwarp();
    else __syncthreads();
  };
  float* qs = simt_smem + slot * simt_head_floats(d);        // [d], then the parts' [hi d | lo d | weights hi, lo, maximum | scores | pages]
  const auto part_of = [&](int part) { return qs + d + part * simt_part_floats(d); };
  const T* qrow = q + (size_t)t * q_stride + (size_t)h * d;
  constexpr bool kCompensated = sizeof(T) == 4;
  for (int i = warp * 32 + lane; i < d; i += WARPS * 32) qs[i] = kCompensated ? to_f32(qrow[i]) : to_f32(qrow[i]) * scale;

  const int r = tok_req[t];        // r < 0: a padding row of a fixed-size batch; it sees no key and yields zeros
  const int p = positions[t];
  const int lo = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
  const int nkeys = r < 0 ? 0 : p - lo + 1;
  int chunk = (nkeys + splits - 1) / splits;
  chunk = (chunk + 31) & ~31;
  const int k_begin = lo + split * chunk;
  const int k_end = r < 0 ? k_begin : min(lo + (split + 1) * chunk, p + 1);
  const int kvh = h / (nq / nkv);
  const size_t plane = (size_t)nkv * page_size * d;
  const int* bt = block_table + (size_t)(r < 0 ? 0 : r) * bt_stride;
  constexpr int VN = Vec16<T>::N;
  constexpr int PAIRS = (DPL + 1) / 2;
  meet();

  float m = -INFINITY;
  for (int c0 = k_begin; c0 < k_end; c0 += kParts * kPartTurns * 32) {      // (the same for all warps of the head)
    float top = -INFINITY;
#pragma unroll 1
    for (int part = warp; part < kParts; part += WARPS) {
      float* scores = part_of(part) + 2 * d + 4 + lane;                     // [turn][32]
      int* pages = reinterpret_cast<int*>(scores + kPartTurns * 32);
#pragma unroll 1
      for (int turn = 0; turn < kPartTurns; ++turn) {
        const int k0 = c0 + (turn * kParts + part) * 32, key = k0 + lane;
        if (k0 >= k_end) break;
        float score = -INFINITY;
        int page = key < k_end ? bt[key / page_size] : -1;
        if (page >= num_pages) page = -1;                 // never follow a table entry outside the pool
        if (page >= 0) {
          const T* kp = cache + (size_t)page * 2 * plane + ((size_t)kvh * page_size + key % page_size) * d;
          float dot = 0.f;
          float2 dot2 = make_float2(0.f, 0.f), low2 = dot2;                 // sums of the even and the odd entries
          for (int i0 = 0; i0 < d; i0 += kPacketsAhead * VN) {
            Vec16<T> kv[kPacketsAhead];
#pragma unroll
            for (int j = 0; j < kPacketsAhead; ++j) kv[j] = load16(kp + min(i0 + j * VN, d - VN));
            if (WARPS > 1 && i0 == 0)                                        // the key's value, wanted when all scores are known
              for (int i = 0; i < d; i += 128 / (int)sizeof(T)) asm volatile("prefetch.global.L2 [%0];" ::"l"(kp + plane + i));
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
          if constexpr (kCompensated) {
            two_add(dot2.x, low2.x, dot2.y, low2.y);
            score = __fadd_rn(dot2.x, low2.x) * scale;
          } else {
            score = dot;
          }
        }
        scores[turn * 32] = score;
        pages[turn * 32] = page;
        top = fmaxf(top, score);
      }
    }
    // the maximum over the head's parts
    top = warp_max(top);
    float m_new = fmaxf(m, top);
    if constexpr (WARPS > 1) {
      if (lane == 0) part_of(warp)[2 * d + 2] = top;
      meet();
#pragma unroll
      for (int w = 0; w < kParts; ++w) m_new = fmaxf(m_new, part_of(w)[2 * d + 2]);
      meet();                            // (the maxima are written again by the next 512 keys)
    }
    const float alpha = m_new == -INFINITY ? 1.f : expf(m - m_new);  // m = -inf at first gives 0; no score above it yet: nothing to shrink
    m = m_new;
    const bool begin = c0 == k_begin;
#pragma unroll 1
    for (int part = warp; part < kParts; part += WARPS) {
      float* own = part_of(part);
      float2 acc[PAIRS], low[PAIRS];     // entries lane, lane + 32 of the value; lane + 64, ...
      float l = begin ? 0.f : own[2 * d], l_lo = begin ? 0.f : own[2 * d + 1];
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) {
        acc[i] = low[i] = make_float2(0.f, 0.f);
        if (!begin) {
          if (lane + 64 * i < d) { acc[i].x = own[lane + 64 * i]; low[i].x = own[d + lane + 64 * i]; }
          if (lane + 64 * i + 32 < d) { acc[i].y = own[lane + 64 * i + 32]; low[i].y = own[d + lane + 64 * i + 32]; }
        }
      }
      if (!begin && alpha != 1.f) {      // the maximum grew: everything so far shrinks
        if constexpr (kCompensated) {
          two_scale(l, l_lo, alpha);
#pragma unroll
          for (int i = 0; i < PAIRS; ++i) { two_scale(acc[i].x, low[i].x, alpha); two_scale(acc[i].y, low[i].y, alpha); }
        } else {
          l *= alpha;
#pragma unroll
          for (int i = 0; i < PAIRS; ++i) { acc[i].x *= alpha; acc[i].y *= alpha; }
        }
      }
      const float* scores = own + 2 * d + 4 + lane;
      const int* pages = reinterpret_cast<const int*>(scores + kPartTurns * 32);
#pragma unroll 1
      for (int turn = 0; turn < kPartTurns; ++turn) {
        const int k0 = c0 + (turn * kParts + part) * 32;
        if (k0 >= k_end) break;
        const int page = pages[turn * 32];
        const long long base = (long long)((size_t)max(page, 0) * 2 * plane + ((size_t)kvh * page_size + (k0 + lane) % page_size) * d + plane);
        const float pr = page >= 0 ? expf(scores[turn * 32] - m) : 0.f;
        if constexpr (kCompensated) two_fma(l, l_lo, warp_sum(pr), 1.f);
        else l += warp_sum(pr);
        const int nvalid = min(32, k_end - k0);
        constexpr int kValuesAhead = values_ahead(DPL);
        for (int j0 = 0; j0 < nvalid; j0 += kValuesAhead) {
          float pj[kValuesAhead];
          T v[kValuesAhead][2 * PAIRS];
#pragma unroll
          for (int u = 0; u < kValuesAhead; ++u) {
            pj[u] = __shfl_sync(0xffffffffu, pr, j0 + u);         // 0 behind the last key, and for a key without a page
            const T* vp = cache + __shfl_sync(0xffffffffu, base, j0 + u);
#pragma unroll
            for (int i = 0; i < 2 * PAIRS; ++i) {
              v[u][i] = from_f32<T>(0.f);
              if (pj[u] != 0.f && lane + 32 * i < d) v[u][i] = vp[lane + 32 * i];
            }
          }
#pragma unroll
          for (int u = 0; u < kValuesAhead; ++u) {
            if (pj[u] == 0.f) continue;                           // (uniform over the warp)
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
              const float2 b = make_float2(to_f32(v[u][2 * i]), to_f32(v[u][2 * i + 1]));
              if constexpr (kCompensated) two_fma_pair(acc[i], low[i], make_float2(pj[u], pj[u]), make_float2(-pj[u], -pj[u]), b);
              else acc[i] = fma2(make_float2(pj[u], pj[u]), b, acc[i]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) {
        if (lane + 64 * i < d) { own[lane + 64 * i] = acc[i].x; own[d + lane + 64 * i] = low[i].x; }
        if (lane + 64 * i + 32 < d) { own[lane + 64 * i + 32] = acc[i].y; own[d + lane + 64 * i + 32] = low[i].y; }
      }
      __syncwarp();                      // (every lane has read the sums of weights)
      if (lane == 0) { own[2 * d] = l; own[2 * d + 1] = l_lo; }
    }
  }
  // the parts' sums, all to the same maximum, in their order
  meet();
  if (warp) return;
  float l = 0.f, l_lo = 0.f, acc[DPL], acc_lo[DPL];
#pragma unroll
  for (int i = 0; i < DPL; ++i) { acc[i] = 0.f; acc_lo[i] = 0.f; }
  if (k_begin < k_end) {
#pragma unroll
    for (int part = 0; part < kParts; ++part) {
      const float* from = part_of(part);
      two_add(l, l_lo, from[2 * d], from[2 * d + 1]);
#pragma unroll
      for (int i = 0; i < DPL; ++i)
        if (lane + 32 * i < d) two_add(acc[i], acc_lo[i], from[lane + 32 * i], from[d + lane + 32 * i]);
    }
  }
  l = __fadd_rn(l, l_lo);
#pragma unroll
  for (int i = 0; i < DPL; ++i) acc[i] = __fadd_rn(acc[i], acc_lo[i]);

  if (splits == 1) {
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    T* o = out + (size_t)t * out_stride + (size_t)h * d;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int dd = lane + 32 * i;
      if (dd < d) o[dd] = from_f32<T>(acc[i] * inv);
    }
  } else {
    const size_t idx = ((size_t)t * nq + h) * splits + split;
    float* pa = part_acc + idx * d;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int dd = lane + 32 * i;
      if (dd < d) pa[dd] = acc[i];
    }
    if (lane == 0) { part_ml[idx * 2] = m; part_ml[idx * 2 + 1] = l; }
  }
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
  const auto launch = [&](auto kernel, int heads, int warps) {
    return launch_kernel("paged_attention", kernel, dim3(tokens, (nq + heads - 1) / heads, splits), dim3(heads * warps * 32),
                         (size_t)heads * simt_head_floats(d) * sizeof(float), as_stream(stream), (T*)out, part_acc, part_ml, (const T*)q,
                         (const T*)cache, block_table, tok_req, positions, q_stride, out_stride, bt_stride, nq, nkv, d, page_size, scale, window,
                         splits, num_pages);
  };
  // a warp per head from eight heads an SM on (neighbouring heads of a block read the same keys, out of L1)
  const bool many = (long long)tokens * nq * splits >= 8LL * sm_count_of_device();
  int rc = d <= 64    ? many ? launch(paged_attention_simt_kernel<T, 2, 4, 1>, 4, 1) : launch(paged_attention_simt_kernel<T, 2, 1, kParts>, 1, kParts)
           : d <= 128 ? many ? launch(paged_attention_simt_kernel<T, 4, 2, 1>, 2, 1) : launch(paged_attention_simt_kernel<T, 4, 1, kParts>, 1, kParts)
           : many     ? launch(paged_attention_simt_kernel<T, kMaxDimPerLane, 2, 1>, 2, 1)
                      : launch(paged_attention_simt_kernel<T, kMaxDimPerLane, 1, kParts>, 1, kParts);
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
