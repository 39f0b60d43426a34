// Attention inside blocks of positions over the paged cache, with a distance bias on the scores, weights
// mixed between heads after the softmax, and values that are normed before they are stored.
//
// A page of the cache holds its keys, then its values: element (g, offset, e) of the keys lies at
// page * page_stride + (g * page_size + offset) * d + e, of the values at
// page * page_stride + G * page_size * d + (g * page_size + offset) * dv + e, page_stride = G * page_size * (d + dv).
// Scores, weights and all sums are float32; T is the element type of q, of the cache and of the result.
#include "mma_utils.cuh"

namespace ptl {

// k (+ bias) and v (+ bias, then divided by its root mean square per head when eps > 0) of every token go to
// the token's slot (page * page_size + offset; -1: not stored).  qkv rows: [q: H * d | k: G * d | v: G * dv].
template <typename T>
__global__ void __launch_bounds__(128)
kv_write_normed_kernel(T* __restrict__ cache, const T* __restrict__ qkv, const float* __restrict__ bias,
                       const int* __restrict__ slots, int H, int G, int d, int dv, int page_size, long long num_slots, float eps) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const long long slot = slots[t];
  if (slot < 0 || slot >= num_slots) return;
  const size_t page = (size_t)(slot / page_size), off = (size_t)(slot % page_size);
  const int ld = H * d + G * (d + dv);
  const T* row = qkv + (size_t)t * ld;
  T* kp = cache + page * (size_t)G * page_size * (d + dv);
  T* vp = kp + (size_t)G * page_size * d;
#pragma unroll 4
  for (int i = threadIdx.x; i < G * d; i += blockDim.x) {
    const int g = i / d, e = i % d;
    const float v = to_f32(row[H * d + i]) + (bias ? bias[H * d + i] : 0.f);
    kp[((size_t)g * page_size + off) * d + e] = from_f32<T>(v);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int g = warp; g < G; g += nwarps) {
    const int base = (H + G) * d + g * dv;
    float ss = 0.f;
#pragma unroll 4
    for (int e = lane; e < dv; e += 32) {
      const float v = to_f32(row[base + e]) + (bias ? bias[base + e] : 0.f);
      ss = fmaf(v, v, ss);
    }
    ss = warp_sum(ss);
    const float f = eps > 0.f ? 1.0f / sqrtf(ss / (float)dv + eps) : 1.0f;
#pragma unroll 4
    for (int e = lane; e < dv; e += 32) {
      const float v = to_f32(row[base + e]) + (bias ? bias[base + e] : 0.f);
      vp[((size_t)g * page_size + off) * dv + e] = from_f32<T>(v * f);
    }
  }
}

constexpr int kMaxMixedHeads = 128;     // heads whose weights can be mixed (a thread holds one key's column of them)

// One block per query token (`items`: the token rows, else rows 0 .. tokens - 1).  Keys j = lo .. p of the token's request, lo = p - p % chunk (0 without chunks):
//   score_h(j) = (q_h + bias) . k_j * scale - r1[h] * log1p(r2[h] * (p - j));   w_h = softmax_j;
//   w'_h = sum_g talk[h, g] w_g;   out_h = out_scale * sum_j w'_h(j) v_j.
// Shared memory: max_keys page addresses, the query (H * d floats), H * max_keys weights.
template <typename T>
__global__ void __launch_bounds__(256)
chunk_attention_kernel(T* __restrict__ out, int out_ld, int column, const T* __restrict__ qkv, int q_ld,
                       const float* __restrict__ q_bias, const T* __restrict__ cache, const int* __restrict__ block_table,
                       int table_width, const int* __restrict__ tok_req, const int* __restrict__ positions, int H, int G, int d,
                       int dv, int page_size, float scale, int chunk, const float* __restrict__ r1, const float* __restrict__ r2,
                       const float* __restrict__ talk, int max_keys, int num_pages, float out_scale, int vec_ok,
                       const int* __restrict__ items) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  long long* page_at = reinterpret_cast<long long*>(smem_raw);       // first element of the page that holds key j, -1: none
  float* q = reinterpret_cast<float*>(page_at + max_keys);
  float* w = q + H * d;
  pdl_wait();
  pdl_launch_dependents();
  const int t = items ? items[blockIdx.x] : blockIdx.x;
  const int r = tok_req[t];
  if (r < 0) return;
  const int p = positions[t];
  const int lo = chunk > 0 ? p - p % chunk : 0;
  const int n = min(p - lo + 1, max_keys);
  const int group = H / G;
  const size_t page_stride = (size_t)G * page_size * (d + dv);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll 4
  for (int i = threadIdx.x; i < H * d; i += blockDim.x)      // (four turns' loads are issued together)
    q[i] = to_f32(qkv[(size_t)t * q_ld + i]) + (q_bias ? q_bias[i] : 0.f);
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const int pos = lo + j;
    const int page = block_table[(size_t)r * table_width + pos / page_size];
    page_at[j] = (page >= 0 && page < num_pages) ? (long long)((size_t)page * page_stride) : -1;
  }
  __syncthreads();
  // scores: one (kv head, key) pair per thread and turn, for up to four of the kv head's query heads at a time, so that
  // a key row is fetched once for them; consecutive threads take consecutive keys
  for (int i = threadIdx.x; i < G * n; i += blockDim.x) {
    const int c = i / n, j = i % n;
    const bool there = page_at[j] >= 0;
    const T* kr = cache + (there ? page_at[j] : 0) + ((size_t)c * page_size + (lo + j) % page_size) * d;
    for (int h0 = c * group; h0 < (c + 1) * group; h0 += 4) {
      const int nh = min(4, (c + 1) * group - h0);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      if (there && vec_ok) {                            // 16-byte packets of the key row and of the queries
        constexpr int VN = Vec16<T>::N;
#pragma unroll 8
        for (int e = 0; e < d; e += VN) {
          const Vec16<T> kv = load16(kr + e);
#pragma unroll
          for (int a4 = 0; a4 < 4; ++a4) {
            if (a4 < nh) {
#pragma unroll
              for (int u = 0; u < VN; u += 4) {
                const float4 qv = *reinterpret_cast<const float4*>(q + (h0 + a4) * d + e + u);
                acc[a4] = fmaf(qv.x, kv.get(u), acc[a4]);
                acc[a4] = fmaf(qv.y, kv.get(u + 1), acc[a4]);
                acc[a4] = fmaf(qv.z, kv.get(u + 2), acc[a4]);
                acc[a4] = fmaf(qv.w, kv.get(u + 3), acc[a4]);
              }
            }
          }
        }
      } else if (there) {
        for (int e = 0; e < d; ++e) {
          const float kv = to_f32(kr[e]);
#pragma unroll
          for (int a4 = 0; a4 < 4; ++a4)
            if (a4 < nh) acc[a4] = fmaf(q[(h0 + a4) * d + e], kv, acc[a4]);
        }
      }
#pragma unroll
      for (int a4 = 0; a4 < 4; ++a4) {
        if (a4 >= nh) continue;
        const int h = h0 + a4;
        float sc = -INFINITY;
        if (there) {
          sc = acc[a4] * scale;
          if (r1) sc -= r1[h] * log1pf(r2[h] * (float)(p - lo - j));
        }
        w[(size_t)h * max_keys + j] = sc;
      }
    }
  }
  __syncthreads();
  for (int h = warp; h < H; h += nwarps) {
    float* wh = w + (size_t)h * max_keys;
    float m = -INFINITY;
    for (int j = lane; j < n; j += 32) m = fmaxf(m, wh[j]);
    m = warp_max(m);
    float sum = 0.f;
    for (int j = lane; j < n; j += 32) {
      const float e = wh[j] == -INFINITY ? 0.f : expf(wh[j] - m);
      wh[j] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    const float inv = sum > 0.f ? 1.0f / sum : 0.f;
    for (int j = lane; j < n; j += 32) wh[j] *= inv;
  }
  __syncthreads();
  if (talk) {
    // in place, a key's column of weights at a time: the thread that owns the key reads all heads' weights, then writes the mixed ones
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      float col[kMaxMixedHeads];
      for (int g = 0; g < H; ++g) col[g] = w[(size_t)g * max_keys + j];
      for (int h = 0; h < H; ++h) {
        float acc = 0.f;
        for (int g = 0; g < H; ++g) acc = fmaf(talk[h * H + g], col[g], acc);
        w[(size_t)h * max_keys + j] = acc;
      }
    }
    __syncthreads();
  }
  const float* use = w;
  // outputs: one (kv head, value element) pair per thread and turn, for up to four of the kv head's query heads at a
  // time, so that a value is fetched once for them; consecutive threads take consecutive elements
  for (int i = threadIdx.x; i < G * dv; i += blockDim.x) {
    const int c = i / dv, e = i % dv;
    const size_t head_off = (size_t)G * page_size * d + (size_t)c * page_size * dv + e;
    for (int h0 = c * group; h0 < (c + 1) * group; h0 += 4) {
      const int nh = min(4, (c + 1) * group - h0);
      const float* w0 = use + (size_t)h0 * max_keys;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
      for (int j = 0; j < n; ++j) {                   // (eight keys per turn: their values are fetched side by side)
        // no branch in here: a key without a page (its weight is zero already) reads the first page's value
        const long long pg = page_at[j];
        const T raw = cache[(size_t)(pg < 0 ? 0 : pg) + head_off + (size_t)((lo + j) % page_size) * dv];
        const float v = pg < 0 ? 0.f : to_f32(raw);
#pragma unroll
        for (int a4 = 0; a4 < 4; ++a4)
          if (a4 < nh) acc[a4] = fmaf(w0[(size_t)a4 * max_keys + j], v, acc[a4]);
      }
#pragma unroll
      for (int a4 = 0; a4 < 4; ++a4)
        if (a4 < nh) out[(size_t)t * out_ld + column + (h0 + a4) * dv + e] = from_f32<T>(acc[a4] * out_scale);
    }
  }
}

// Single tokens of a bfloat16 cache with up to eight query heads over up to two kv heads of 64 or 128 entries, blocks of up to 256
// positions: the same sums, a block per token whose sixteen warps share the keys.  A lane owns four (heads of 64: two) neighbouring entries of
// every head: four keys' products with eight heads meet in one butterfly that leaves a (key, head) in every lane, and for the
// values the warps' sums meet in shared memory.  What bounds it: the trips to memory of its five steps, one after the other, and from some
// hundred keys on their 512 bytes each through one SM.  Eight tokens of 8 heads of 128 at the end of 256 positions: 15.8 us, the kernel above
// (a thread per key) 43.8; at the 17th 6.3 and 14.6.
constexpr int kCsThreads = 512, kCsWarps = kCsThreads / 32, kCsHeads = 8, kCsMaxBlock = 256;

template <int D, int G>
__global__ void __launch_bounds__(kCsThreads)
chunk_attention_single_kernel(__nv_bfloat16* __restrict__ out, int out_ld, int column, const __nv_bfloat16* __restrict__ qkv, int q_ld,
                              const float* __restrict__ q_bias, const __nv_bfloat16* __restrict__ cache, const int* __restrict__ block_table,
                              int table_width, const int* __restrict__ tok_req, const int* __restrict__ positions, int H, int page_size,
                              float scale, int chunk, const float* __restrict__ r1, const float* __restrict__ r2, const float* __restrict__ talk,
                              int num_pages, float out_scale, const int* __restrict__ items) {
  constexpr int HG = kCsHeads / G, E = D / 32;                // places for a kv head's query heads, entries of a lane
  extern __shared__ __align__(16) float cs_smem[];
  float* s_w = cs_smem;                                       // [256 keys][8 heads]: scores, weights, mixed weights
  float* s_sum = s_w + kCsMaxBlock * kCsHeads;                // [16 warps][8 heads][D]
  __shared__ long long s_at[kCsMaxBlock];
  __shared__ float s_talk[kCsHeads * kCsHeads];
  pdl_wait();
  pdl_launch_dependents();
  const int t = items ? items[blockIdx.x] : blockIdx.x;
  const int r = tok_req[t];
  if (r < 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, group = H / G;
  const int p = positions[t], lo = p - p % chunk, n = min(p - lo + 1, table_width * page_size);      // (no more keys than the table can name)
  const size_t page_stride = (size_t)G * page_size * 2 * D, plane = (size_t)page_size * D;
  // asked for together: the key's page, and the queries (with their bias) of this lane's entries, for the warps that have keys to score; a place
  // without a head holds zeros
  const int pos = lo + tid, page = tid < n ? block_table[(size_t)r * table_width + pos / page_size] : -1;
  uint32_t raw[kCsHeads][E / 2];
  float2 bias[kCsHeads][E / 2];
#pragma unroll
  for (int a = 0; a < kCsHeads; ++a) {
    const bool there = 4 * warp < n && a % HG < group;
    const int at = (a / HG * group + a % HG) * D + lane * E;
#pragma unroll
    for (int e = 0; e < E / 2; ++e) {
      raw[a][e] = 0u;
      bias[a][e] = make_float2(0.f, 0.f);
    }
    if (there) {
      if constexpr (E == 4) *reinterpret_cast<uint2*>(raw[a]) = *reinterpret_cast<const uint2*>(qkv + (size_t)t * q_ld + at);
      else raw[a][0] = *reinterpret_cast<const uint32_t*>(qkv + (size_t)t * q_ld + at);
      if (q_bias) {
#pragma unroll
        for (int e = 0; e < E / 2; ++e) bias[a][e] = *reinterpret_cast<const float2*>(q_bias + at + 2 * e);
      }
    }
  }
  if (tid < n) s_at[tid] = page >= 0 && page < num_pages ? (long long)((size_t)page * page_stride + (size_t)(pos % page_size) * D) : -1;
  float q[kCsHeads][E];
#pragma unroll
  for (int a = 0; a < kCsHeads; ++a)
#pragma unroll
    for (int e = 0; e < E; e += 2) {
      const float2 v = unpack_bf16(raw[a][e / 2]);
      q[a][e] = v.x + bias[a][e / 2].x;
      q[a][e + 1] = v.y + bias[a][e / 2].y;
    }
  if (talk && tid < H * H) s_talk[tid] = talk[tid];
  __syncthreads();
  // a lane's entries of a row of the cache
  const auto entries = [&](long long at, float (&x)[E]) {
    if (at < 0) {
#pragma unroll
      for (int e = 0; e < E; ++e) x[e] = 0.f;
      return;
    }
    const __nv_bfloat162* src = reinterpret_cast<const __nv_bfloat162*>(cache + at + lane * E);
    __nv_bfloat162 raw[E / 2];
    if constexpr (E == 4) *reinterpret_cast<uint2*>(raw) = *reinterpret_cast<const uint2*>(src);
    else raw[0] = *src;
#pragma unroll
    for (int e = 0; e < E / 2; ++e) {
      const float2 v = __bfloat1622float2(raw[e]);
      x[2 * e] = v.x;
      x[2 * e + 1] = v.y;
    }
  };
  // scores, four keys at a time: lane 8 k + a ends up with key k's of head place a
  const int a0 = lane & 7, my_head = a0 / HG * group + a0 % HG;
  const bool my_there = a0 % HG < group;
  const float f1 = r1 && my_there ? r1[my_head] : 0.f, f2 = r1 && my_there ? r2[my_head] : 0.f;
#pragma unroll 2
  for (int j0 = 4 * warp; j0 < n; j0 += 4 * kCsWarps) {
    float x[4][G][E], v[32];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long at = j0 + k < n ? s_at[j0 + k] : -1;
#pragma unroll
      for (int c = 0; c < G; ++c) entries(at < 0 ? -1 : at + (long long)(c * plane), x[k][c]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int a = 0; a < kCsHeads; ++a) {
        float sum = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) sum = fmaf(q[a][e], x[k][a / HG][e], sum);
        v[8 * k + a] = sum;
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const int j = j0 + (lane >> 3);
    if (j < n) {
      float sc = -INFINITY;
      if (my_there && s_at[j] >= 0) {
        sc = v[0] * scale;
        if (r1) sc -= f1 * log1pf(f2 * (float)(p - lo - j));
      }
      s_w[j * kCsHeads + a0] = sc;
    }
  }
  __syncthreads();
  if (warp < kCsHeads) {                                       // softmax, a warp per head place
    float x[kCsMaxBlock / 32], m = -INFINITY, sum = 0.f;
#pragma unroll
    for (int i = 0; i < kCsMaxBlock / 32; ++i) {
      x[i] = lane + 32 * i < n ? s_w[(lane + 32 * i) * kCsHeads + warp] : -INFINITY;
      m = fmaxf(m, x[i]);
    }
    m = warp_max(m);
#pragma unroll
    for (int i = 0; i < kCsMaxBlock / 32; ++i) {
      x[i] = x[i] == -INFINITY ? 0.f : expf(x[i] - m);
      sum += x[i];
    }
    sum = warp_sum(sum);
    const float inv = sum > 0.f ? 1.0f / sum : 0.f;
#pragma unroll
    for (int i = 0; i < kCsMaxBlock / 32; ++i)
      if (lane + 32 * i < n) s_w[(lane + 32 * i) * kCsHeads + warp] = x[i] * inv;
  }
  __syncthreads();
  if (talk) {                                                  // a key's column of weights per thread
    if (tid < n) {
      float x[kCsHeads], y[kCsHeads];
#pragma unroll
      for (int a = 0; a < kCsHeads; ++a) x[a] = s_w[tid * kCsHeads + a];
#pragma unroll
      for (int b = 0; b < kCsHeads; ++b) {
        y[b] = 0.f;
        if (b % HG >= group) continue;
        const float* row = s_talk + (b / HG * group + b % HG) * H;
#pragma unroll
        for (int a = 0; a < kCsHeads; ++a)
          if (a % HG < group) y[b] = fmaf(row[a / HG * group + a % HG], x[a], y[b]);
      }
#pragma unroll
      for (int b = 0; b < kCsHeads; ++b) s_w[tid * kCsHeads + b] = y[b];
    }
    __syncthreads();
  }
  // outputs: a warp's keys, all heads
  float acc[kCsHeads][E];
#pragma unroll
  for (int a = 0; a < kCsHeads; ++a)
#pragma unroll
    for (int e = 0; e < E; ++e) acc[a][e] = 0.f;
#pragma unroll 4
  for (int j = warp; j < n; j += kCsWarps) {
    const long long at = s_at[j];
    float x[G][E];
#pragma unroll
    for (int c = 0; c < G; ++c) entries(at < 0 ? -1 : at + (long long)((G + c) * plane), x[c]);
    const float4 w0 = *reinterpret_cast<const float4*>(s_w + j * kCsHeads), w1 = *reinterpret_cast<const float4*>(s_w + j * kCsHeads + 4);
    const float w[kCsHeads] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int a = 0; a < kCsHeads; ++a)
#pragma unroll
      for (int e = 0; e < E; ++e) acc[a][e] = fmaf(w[a], x[a / HG][e], acc[a][e]);
  }
#pragma unroll
  for (int a = 0; a < kCsHeads; ++a)
#pragma unroll
    for (int e = 0; e < E; e += 2) *reinterpret_cast<float2*>(s_sum + (warp * kCsHeads + a) * D + lane * E + e) = make_float2(acc[a][e], acc[a][e + 1]);
  __syncthreads();
  for (int i = tid; i < kCsHeads * D; i += kCsThreads) {
    const int a = i / D, e = i % D;
    if (a % HG >= group) continue;
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kCsWarps; ++w) sum += s_sum[w * kCsHeads * D + i];
    out[(size_t)t * out_ld + column + (a / HG * group + a % HG) * D + e] = __float2bfloat16_rn(sum * out_scale);
  }
}

template <int D, int G>
int chunk_attention_single(void* out, int out_ld, int column, const void* qkv, int q_ld, const float* q_bias, const void* cache, const int* bt,
                           int table_width, const int* tok_req, const int* positions, int rows, int H, int page_size, float scale, int chunk,
                           const float* r1, const float* r2, const float* talk, int num_pages, float out_scale, const int* items, void* stream) {
  static SmemRaised raised;
  constexpr int smem = (kCsMaxBlock * kCsHeads + kCsWarps * kCsHeads * D) * (int)sizeof(float);
  if (int rc = raise_shared_memory("chunk_attention_single", chunk_attention_single_kernel<D, G>, smem, raised)) return rc;
  return launch_kernel("chunk_attention_single", chunk_attention_single_kernel<D, G>, dim3(rows), dim3(kCsThreads), smem, as_stream(stream),
                       (__nv_bfloat16*)out, out_ld, column, (const __nv_bfloat16*)qkv, q_ld, q_bias, (const __nv_bfloat16*)cache, bt,
                       table_width, tok_req, positions, H, page_size, scale, chunk, r1, r2, talk, num_pages, out_scale, items);
}

template <typename T>
int kv_write_normed(void* cache, const void* qkv, const float* bias, const int* slots, int tokens, int H, int G, int d, int dv,
                    int page_size, long long num_slots, float eps, void* stream) {
  PTL_REQUIRE(tokens >= 0 && H > 0 && G > 0 && d > 0 && dv > 0 && page_size > 0 && eps >= 0.f,
              "kv_write_normed: bad sizes tokens=%d H=%d G=%d d=%d dv=%d page=%d", tokens, H, G, d, dv, page_size);
  if (tokens == 0) return 0;
  return launch_kernel("kv_write_normed", kv_write_normed_kernel<T>, dim3(tokens), dim3(128), 0, as_stream(stream), (T*)cache,
                       (const T*)qkv, bias, slots, H, G, d, dv, page_size, num_slots, eps);
}

template <typename T>
int chunk_attention(void* out, int out_ld, int column, const void* qkv, int q_ld, const float* q_bias, const void* cache,
                    const int* block_table, int table_width, const int* tok_req, const int* positions, int tokens, int H, int G,
                    int d, int dv, int page_size, float scale, int chunk, const float* r1, const float* r2, const float* talk,
                    int max_keys, int num_pages, float out_scale, const int* items, void* stream) {
  PTL_REQUIRE(tokens >= 0 && H > 0 && G > 0 && H % G == 0 && d > 0 && dv > 0 && page_size > 0 && chunk >= 0 && max_keys > 0,
              "chunk_attention: bad sizes tokens=%d H=%d G=%d d=%d dv=%d page=%d chunk=%d keys=%d", tokens, H, G, d, dv, page_size,
              chunk, max_keys);
  PTL_REQUIRE((r1 == nullptr) == (r2 == nullptr), "chunk_attention: the distance bias needs both of its factors");
  PTL_REQUIRE(column >= 0 && column + H * dv <= out_ld && q_ld >= H * d, "chunk_attention: rows too short for the heads");
  if (tokens == 0) return 0;
  max_keys += max_keys & 1;            // the queries behind the page addresses start on a 16-byte boundary
  PTL_REQUIRE(!talk || H <= kMaxMixedHeads, "chunk_attention: weights of at most %d heads can be mixed, got %d", kMaxMixedHeads, H);
  const size_t smem = (size_t)max_keys * sizeof(long long) + ((size_t)H * d + (size_t)H * max_keys) * sizeof(float);
  PTL_REQUIRE(smem <= 200 * 1024, "chunk_attention: %d heads over %d keys do not fit the shared memory of a block (%zu bytes)", H,
              max_keys, smem);
  static SmemRaised raised = {};
  if (smem > 48 * 1024)
    if (int rc = raise_shared_memory("chunk_attention", chunk_attention_kernel<T>, 200 * 1024, raised)) return rc;
  const int vec_ok = d % Vec16<T>::N == 0 && dv % Vec16<T>::N == 0 && d % 4 == 0 && aligned16(cache);   // every key row starts on a 16-byte boundary
  return launch_kernel("chunk_attention", chunk_attention_kernel<T>, dim3(tokens), dim3(256), smem, as_stream(stream), (T*)out,
                       out_ld, column, (const T*)qkv, q_ld, q_bias, (const T*)cache, block_table, table_width, tok_req, positions,
                       H, G, d, dv, page_size, scale, chunk, r1, r2, talk, max_keys, num_pages, out_scale, vec_ok, items);
}

}  // namespace ptl

#define PTL_CHUNK_ATTENTION(SUFFIX, TYPE)                                                                                         \
  PTL_EXPORT int ptl_kv_write_normed##SUFFIX(void* cache, const void* qkv, const float* bias, const int* slots, int tokens, int H, \
                                             int G, int d, int dv, int page_size, long long num_slots, float eps, void* stream) { \
    return ptl::kv_write_normed<TYPE>(cache, qkv, bias, slots, tokens, H, G, d, dv, page_size, num_slots, eps, stream);            \
  }                                                                                                                               \
  PTL_EXPORT int ptl_chunk_attention##SUFFIX(void* out, int out_ld, int column, const void* qkv, int q_ld, const float* q_bias,    \
                                             const void* cache, const int* block_table, int table_width, const int* tok_req,      \
                                             const int* positions, int tokens, int H, int G, int d, int dv, int page_size,        \
                                             float scale, int chunk, const float* r1, const float* r2, const float* talk,         \
                                             int max_keys, int num_pages, float out_scale, const int* items, void* stream) { \
    return ptl::chunk_attention<TYPE>(out, out_ld, column, qkv, q_ld, q_bias, cache, block_table, table_width, tok_req, positions, \
                                      tokens, H, G, d, dv, page_size, scale, chunk, r1, r2, talk, max_keys, num_pages, out_scale, \
                                      items, stream);                                                                                    \
  }
PTL_CHUNK_ATTENTION(_f32, float)
PTL_CHUNK_ATTENTION(_bf16, __nv_bfloat16)

// Single tokens.  -2: sizes or addresses for the kernel above.
PTL_EXPORT int ptl_chunk_attention_single_bf16(void* out, int out_ld, int column, const void* qkv, int q_ld, const float* q_bias, const void* cache,
                                               const int* block_table, int table_width, const int* tok_req, const int* positions, int rows, int H,
                                               int G, int d, int page_size, float scale, int chunk, const float* r1, const float* r2,
                                               const float* talk, int num_pages, float out_scale, const int* items, void* stream) {
  using namespace ptl;
  if ((d != 64 && d != 128) || H < 1 || H > kCsHeads || G < 1 || G > 2 || H % G || H / G > kCsHeads / G || chunk < 1 || chunk > kCsMaxBlock ||
      !aligned16(cache) || !aligned16(qkv) || q_ld % 8 || (reinterpret_cast<uintptr_t>(q_bias) & 7u))
    return -2;
  PTL_REQUIRE((r1 == nullptr) == (r2 == nullptr) && page_size > 0 && num_pages > 0 && rows >= 0 && column >= 0 && column + H * d <= out_ld &&
                  q_ld >= H * d, "chunk_attention_single: bad sizes");
  // A block holds an SM (by its registers), and few heads in short blocks of positions have little for sixteen warps: beyond two turns of SMs
  // they are left to the kernel above.  Positions spread over the blocks, us there and here: 4 heads of 64 in blocks of 64, 296 tokens 14.7 and
  // 11.5, 600 17.9 and 22.4; in blocks of 128 28.2 and 28.9; 8 heads of 128 in blocks of 256, 600 tokens 104 and 56 (all at the 17th position 20 and
  // 26, all at the last 137 and 101).
  if (rows > 2 * sm_count_of_device() && H * chunk < 512) return -2;
  if (rows == 0) return 0;
  const auto fn = d == 64 ? G == 1 ? chunk_attention_single<64, 1> : chunk_attention_single<64, 2>
                          : G == 1 ? chunk_attention_single<128, 1> : chunk_attention_single<128, 2>;
  return fn(out, out_ld, column, qkv, q_ld, q_bias, cache, block_table, table_width, tok_req, positions, rows, H, page_size, scale, chunk, r1, r2,
            talk, num_pages, out_scale, items, stream);
}
