// The attention inside blocks of positions (see chunk_attention.cu) for bfloat16 caches on the tensor cores, up to eight query
// heads over up to two kv heads of 64 or 128 entries, blocks of up to 256 positions: sixteen neighbouring positions of one
// request per block, two warps per query head (of the keys' scores, the rows' softmax and the values' entries each takes half).
//
// Scores: a query is bfloat16 plus a float32 bias; the bfloat16 part goes to the tensor cores, the bias's product with a key is the
// same for all queries and is worked out once per head and key, from three bfloat16 terms of the bias (24 bits).  Keys come in tiles of 64 by cp.async.  A head's scores
// of all its keys stay in shared memory as float32; the softmax runs over whole rows, the mixing between heads takes a key's
// column of weights per thread, and the mixed float32 weights go to the tensor cores as three bfloat16 terms each (24 bits).
// Nothing is rounded to 16 bits but the result.  The products also meet the zero weights of a row's later keys, and 0 times a value
// that is no finite number is none: a head whose sums are not all finite is added up again, key by key and row by row.
// Bound by the warp-level tensor instructions of a block's keys (one block per SM).  Replaces, for the portions of such sizes, a
// block per token on the CUDA cores that reads a block's keys and values from L2 once per query: 2,048 tokens of 8 heads of 128
// in blocks of 256 took 221 us.  One warp per head, a logarithm per score and one row of the softmax after the other: 66 us, bound by the chain of
// a block at the end of 256 positions, one block of eight warps per SM.  Two warps per head, the logarithms (of a distance and a head) out of a
// table, the biases' products on the tensor cores and four rows at a time: 41 us (in a step; 33 a block at the end of 256 positions).
#include "mma_utils.cuh"

namespace ptl {

constexpr int kCtRows = 16, kCtKeys = 64, kCtThreads = 512, kCtHeads = 8, kCtMaxBlock = 256;
constexpr int kCtLd = kCtMaxBlock + 8;               // floats of a row of weights: eight rows' pairs in different banks
__host__ __device__ constexpr int ct_row_bytes(int d) { return 2 * d + 16; }
// (the biases of a kv head's query heads, three terms each: a tile of sixteen rows, two where all eight heads share one kv head)
constexpr int ct_smem(int d, int G) {
  return kCtHeads * kCtRows * kCtLd * 4 + 2 * G * kCtKeys * ct_row_bytes(d) + kCtHeads * kCtMaxBlock * 4 + (G == 1 ? 2 : G) * 16 * ct_row_bytes(d);
}

// x as three bfloat16 terms, two neighbours at a time
__device__ __forceinline__ void ct_split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16(x, y);
  float2 back = unpack_bf16(hi);
  x -= back.x; y -= back.y;
  mid = pack_bf16(x, y);
  back = unpack_bf16(mid);
  lo = pack_bf16(x - back.x, y - back.y);
}

template <int D>
__global__ void __launch_bounds__(kCtThreads, 1)
chunk_attention_tc_kernel(__nv_bfloat16* __restrict__ out, int out_ld, int column, const __nv_bfloat16* __restrict__ qkv, int q_ld,
                          const float* __restrict__ q_bias, const __nv_bfloat16* __restrict__ cache, const int* __restrict__ block_table,
                          int table_width, const int* __restrict__ tiles, int H, int G, int page_size, float scale, int chunk, const float* __restrict__ r1,
                          const float* __restrict__ r2, const float* __restrict__ talk, int num_pages, float out_scale) {
  extern __shared__ __align__(128) unsigned char ct_raw[];
  float* s_w = reinterpret_cast<float*>(ct_raw);                                   // [8 heads][16][kCtLd]
  const uint32_t s_kv = smem_u32(ct_raw) + kCtHeads * kCtRows * kCtLd * 4;         // [2][G][64] rows of a head
  float* s_log = reinterpret_cast<float*>(ct_raw + kCtHeads * kCtRows * kCtLd * 4 + 2 * G * kCtKeys * ct_row_bytes(D));    // [heads][distance]
  unsigned char* s_terms = ct_raw + kCtHeads * kCtRows * kCtLd * 4 + 2 * G * kCtKeys * ct_row_bytes(D) + kCtHeads * kCtMaxBlock * 4;
  __shared__ float s_talk[kCtHeads * kCtHeads];
  __shared__ float s_key[2][16][kCtKeys];                                           // the biases' terms times a tile's keys: [tile of rows][row][key]
  __shared__ long long s_at[kCtMaxBlock];                                           // first element of a key's row of kv head 0, -1: no page
  constexpr int RB = ct_row_bytes(D);
  // the block's sixteen positions first .. first + 15, of which those from pos0 to end - 1 are tokens of its tile (inputs of
  // the step: request row, first token row, tokens, first position)
  const int* tile = tiles + 4 * blockIdx.y;
  const int req = tile[0], token0 = tile[1], pos0 = tile[3], end = pos0 + tile[2];
  const int first = pos0 / kCtRows * kCtRows + (int)blockIdx.x * kCtRows;
  pdl_wait();
  pdl_launch_dependents();
  if (req < 0 || first >= end) return;
  const int lo = first - first % chunk;                           // (a block of positions is a whole number of sixteens)
  const int n = min(first + kCtRows, end) - lo;                   // keys
  const int n_tiles = (n + kCtKeys - 1) / kCtKeys;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  const int h = warp & (kCtHeads - 1), part = warp / kCtHeads, group = H / G;      // part: which half of the head's work
  const size_t page_stride = (size_t)G * page_size * 2 * D;
  const int* bt = block_table + (size_t)req * table_width;
  // everything that is read once is asked for together: the queries, the block table, the tables of the heads
  // (tokens of this thread's rows g and g + 8; a row that is no token of the step reads the nearest one's query)
  int token[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) token[i] = token0 + min(max(first + g + 8 * i, pos0), end - 1) - pos0;
  uint32_t q[D / 16][4];
  if (h < H) {
#pragma unroll
    for (int k = 0; k < D / 16; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        q[k][e] = *reinterpret_cast<const uint32_t*>(qkv + (size_t)token[e & 1] * q_ld + h * D + 16 * k + c2 + 8 * (e >> 1));
  }
  if (tid < n_tiles * kCtKeys) {
    const int pos = lo + tid, page = tid < n ? bt[pos / page_size] : -1;
    s_at[tid] = page >= 0 && page < num_pages ? (long long)((size_t)page * page_stride + (size_t)(pos % page_size) * D) : -1;
  }
  if (talk && tid < H * H) s_talk[tid] = talk[tid];
  const int b_tiles = 3 * group > 16 ? 2 : 1;                      // of sixteen rows of bias terms
  if (q_bias) {
    for (int i = tid; i < (b_tiles == 2 ? 2 : G) * 16 * (D / 2); i += kCtThreads) {      // (rows: head of the group * 3 + term)
      const int e = i % (D / 2) * 2, row = i / (D / 2), c = b_tiles == 2 ? 0 : row / 16, in = b_tiles == 2 ? row : row % 16;
      uint32_t terms[3] = {0u, 0u, 0u};
      if (in / 3 < group) {
        const float* v = q_bias + (c * group + in / 3) * D + e;
        ct_split(v[0], v[1], terms[0], terms[1], terms[2]);
      }
      *reinterpret_cast<uint32_t*>(s_terms + row * RB + 2 * e) = terms[in % 3];
    }
  }
  __syncthreads();
  auto fetch = [&](int tile, int values, int stage) {             // 64 keys (or values) of every kv head
    const uint32_t dst = s_kv + stage * G * kCtKeys * RB;
    const size_t plane = (size_t)page_size * D;
#pragma unroll 4
    for (int i = tid; i < G * kCtKeys * (D / 8); i += kCtThreads) {
      const int p = i % (D / 8), row = i / (D / 8), c = row / kCtKeys;
      const long long at = s_at[tile * kCtKeys + row % kCtKeys];
      cp_async_16(dst + row * RB + 16 * p, cache + (at < 0 ? 0 : (size_t)at + (values * G + c) * plane + 8 * p), at >= 0);
    }
    cp_async_commit();
  };
  fetch(0, 0, 0);
  if (r1)
    for (int i = tid; i < H * kCtMaxBlock; i += kCtThreads)
      if (i % kCtMaxBlock < n) s_log[i] = log1pf(r2[i / kCtMaxBlock] * (float)(i % kCtMaxBlock));
  float* w_h = s_w + h * kCtRows * kCtLd;
  const float f1 = r1 && h < H ? r1[h] : 0.f;
  for (int t = 0; t < n_tiles; ++t) {
    if (t + 1 < n_tiles) fetch(t + 1, 0, (t + 1) & 1);
    else fetch(0, 1, (t + 1) & 1);                                // behind the last keys the first values
    cp_async_wait<1>();
    __syncthreads();
    float s[4][4];
    if (h < H) {
      const uint32_t kt = s_kv + (((t & 1) * G + h / group) * kCtKeys + 32 * part) * RB;      // 32 keys of the tile
      const uint32_t ka = kt + ((lane & 7) + 8 * (lane >> 4)) * RB + 16 * ((lane >> 3) & 1);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          uint32_t b[4];
          ldmatrix_x4(b, ka + 8 * j * RB + 32 * k);
          mma_bf16_16816(s[j], q[k], b[0], b[1]);
          mma_bf16_16816(s[j + 1], q[k], b[2], b[3]);
        }
    }
    if (q_bias) {
      // the biases' terms times the keys: a warp takes sixteen keys of a tile of rows
      if (warp < (b_tiles == 2 ? 2 : G) * 4) {
        const int rt = warp >> 2, c = b_tiles == 2 ? 0 : rt, k0 = (warp & 3) * 16;
        const uint32_t ka = s_kv + (((t & 1) * G + c) * kCtKeys + k0 + (lane & 7) + 8 * (lane >> 4)) * RB + 16 * ((lane >> 3) & 1);
        const uint32_t aa = smem_u32(s_terms) + (rt * 16 + (lane & 15)) * RB + 16 * (lane >> 4);
        float acc[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          uint32_t a[4], b[4];
          ldmatrix_x4(a, aa + 32 * k);
          ldmatrix_x4(b, ka + 32 * k);
          mma_bf16_16816(acc[0], a, b[0], b[1]);
          mma_bf16_16816(acc[1], a, b[2], b[3]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i)
            *reinterpret_cast<float2*>(&s_key[rt][g + 8 * i][k0 + 8 * j + c2]) = make_float2(acc[j][2 * i], acc[j][2 * i + 1]);
      }
      __syncthreads();
    }
    if (h < H) {
      const int r0 = 3 * (h % group), rt = b_tiles == 2 ? 0 : h / group;      // this head's rows of bias terms
      const float* key_row[3];
#pragma unroll
      for (int w = 0; w < 3; ++w) key_row[w] = b_tiles == 2 ? s_key[(r0 + w) / 16][(r0 + w) % 16] : s_key[rt][r0 + w];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float2 v;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int in_tile = 32 * part + 8 * j + c2 + e, key = t * kCtKeys + in_tile;
            const int dist = first + g + 8 * i - lo - key;
            float x = (s[j][2 * i + e] + (q_bias ? key_row[0][in_tile] + (key_row[1][in_tile] + key_row[2][in_tile]) : 0.f)) * scale;
            if (r1) x -= f1 * s_log[h * kCtMaxBlock + min(max(dist, 0), n - 1)];
            (&v.x)[e] = dist >= 0 && s_at[key] >= 0 ? x : -INFINITY;
          }
          *reinterpret_cast<float2*>(w_h + (g + 8 * i) * kCtLd + t * kCtKeys + 32 * part + 8 * j + c2) = v;
        }
    }
    __syncthreads();                                              // the tile's stage is free
  }
  const int width = n_tiles * kCtKeys;
  if (h < H) {
    constexpr int RS = 4;                                         // rows at a time: their reductions overlap
#pragma unroll 1
    for (int r0 = part * (kCtRows / 2); r0 < (part + 1) * (kCtRows / 2); r0 += RS) {
      float x[RS][kCtMaxBlock / 32], m[RS], sum[RS];
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        const float* row = w_h + (r0 + r) * kCtLd;
        m[r] = -INFINITY;
#pragma unroll
        for (int i = 0; i < kCtMaxBlock / 32; ++i) {
          x[r][i] = lane + 32 * i < width ? row[lane + 32 * i] : -INFINITY;
          m[r] = fmaxf(m[r], x[r][i]);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < RS; ++r) m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], o));
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        sum[r] = 0.f;
#pragma unroll
        for (int i = 0; i < kCtMaxBlock / 32; ++i) {
          x[r][i] = x[r][i] == -INFINITY ? 0.f : expf(x[r][i] - m[r]);
          sum[r] += x[r][i];
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < RS; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        float* row = w_h + (r0 + r) * kCtLd;
        const float inv = sum[r] > 0.f ? 1.0f / sum[r] : 0.f;
#pragma unroll
        for (int i = 0; i < kCtMaxBlock / 32; ++i)
          if (lane + 32 * i < width) row[lane + 32 * i] = x[r][i] * inv;
      }
    }
  }
  __syncthreads();
  if (talk) {
    float mixes[kCtHeads][kCtHeads];
#pragma unroll
    for (int b = 0; b < kCtHeads; ++b)
#pragma unroll
      for (int a = 0; a < kCtHeads; ++a) mixes[b][a] = a < H && b < H ? s_talk[b * H + a] : 0.f;
    for (int i = tid; i < kCtRows * width; i += kCtThreads) {
      float* at = s_w + (i / width) * kCtLd + i % width;
      float x[kCtHeads];
#pragma unroll
      for (int a = 0; a < kCtHeads; ++a) x[a] = a < H ? at[a * kCtRows * kCtLd] : 0.f;
#pragma unroll
      for (int b = 0; b < kCtHeads; ++b) {
        if (b >= H) break;
        float y = 0.f;
#pragma unroll
        for (int a = 0; a < kCtHeads; ++a)
          y = fmaf(mixes[b][a], x[a], y);
        at[b * kCtRows * kCtLd] = y;
      }
    }
    __syncthreads();
  }
  constexpr int NJ = D / 16;                                      // blocks of eight entries of this warp's half of the values
  const int col0 = part * (D / 2);
  float o[NJ][4];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  const int turn = n_tiles & 1;                                   // the stage that holds the first values
  for (int t = 0; t < n_tiles; ++t) {
    if (t + 1 < n_tiles) fetch(t + 1, 1, (turn + t + 1) & 1); else cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (h < H) {
      const uint32_t va = s_kv + (((turn + t) & 1) * G + h / group) * kCtKeys * RB + (lane & 15) * RB + 16 * (lane >> 4) + 2 * col0;
#pragma unroll
      for (int k = 0; k < kCtKeys / 16; ++k) {
        uint32_t a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 v = *reinterpret_cast<const float2*>(w_h + (g + 8 * (e & 1)) * kCtLd + t * kCtKeys + 16 * k + c2 + 8 * (e >> 1));
          ct_split(v.x, v.y, a[0][e], a[1][e], a[2][e]);
        }
#pragma unroll
        for (int j = 0; j < NJ; j += 2) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, va + 16 * k * RB + 16 * j);
#pragma unroll
          for (int w = 2; w >= 0; --w) {
            mma_bf16_16816(o[j], a[w], b[0], b[1]);
            mma_bf16_16816(o[j + 1], a[w], b[2], b[3]);
          }
        }
      }
    }
    __syncthreads();
  }
  if (h >= H) return;
  bool finite = true;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) finite = finite && isfinite(o[j][e]);
  if (!__all_sync(0xffffffffu, finite)) {
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    const __nv_bfloat16* values = cache + ((size_t)G + h / group) * page_size * D + col0 + c2;
    for (int key = 0; key < n; ++key) {
      if (s_at[key] < 0) continue;
      const int pos = lo + key;
      const __nv_bfloat16* v = values + (size_t)bt[pos / page_size] * page_stride + (size_t)(pos % page_size) * D;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (pos > first + g + 8 * i) continue;
        const float weight = w_h[(g + 8 * i) * kCtLd + key];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float2 x = unpack_bf16(*reinterpret_cast<const uint32_t*>(v + 8 * j));
          o[j][2 * i] = fmaf(weight, x.x, o[j][2 * i]);
          o[j][2 * i + 1] = fmaf(weight, x.y, o[j][2 * i + 1]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int pos = first + g + 8 * i;
    if (pos < pos0 || pos >= end) continue;
    __nv_bfloat16* dst = out + (size_t)(token0 + pos - pos0) * out_ld + column + h * D + col0 + c2;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
      *reinterpret_cast<uint32_t*>(dst + 8 * j) = pack_bf16(o[j][2 * i] * out_scale, o[j][2 * i + 1] * out_scale);
  }
}

template <int D>
int chunk_attention_tc(void* out, int out_ld, int column, const void* qkv, int q_ld, const float* q_bias, const void* cache,
                       const int* bt, int table_width, const int* tiles, dim3 grid, int H, int G, int page_size, float scale, int chunk, const float* r1, const float* r2, const float* talk,
                       int num_pages, float out_scale, void* stream) {
  static SmemRaised raised;
  if (int rc = raise_shared_memory("chunk_attention_tc", chunk_attention_tc_kernel<D>, ct_smem(D, 2), raised)) return rc;
  return launch_kernel("chunk_attention_tc", chunk_attention_tc_kernel<D>, grid, dim3(kCtThreads), ct_smem(D, G), as_stream(stream),
                       (__nv_bfloat16*)out, out_ld, column, (const __nv_bfloat16*)qkv, q_ld, q_bias, (const __nv_bfloat16*)cache, bt,
                       table_width, tiles, H, G, page_size, scale, chunk, r1, r2, talk, num_pages, out_scale);
}

}  // namespace ptl

// The step's portions: n_tiles tiles of up to tile_tokens tokens.  -2: sizes or addresses for the other kernel.
PTL_EXPORT int ptl_chunk_attention_tc_bf16(void* out, int out_ld, int column, const void* qkv, int q_ld, const float* q_bias,
                                           const void* cache, const int* block_table, int table_width, const int* tiles, int n_tiles,
                                           int tile_tokens, int H, int G, int d, int page_size, float scale, int chunk, const float* r1,
                                           const float* r2, const float* talk, int num_pages, float out_scale, void* stream) {
  if ((d != 64 && d != 128) || H < 1 || H > ptl::kCtHeads || G < 1 || G > 2 || H % G || chunk < ptl::kCtRows || chunk % ptl::kCtRows ||
      chunk > ptl::kCtMaxBlock || n_tiles > 65535 || q_ld % 2 || out_ld % 2 || column % 2 || !ptl::aligned16(cache) ||
      (reinterpret_cast<uintptr_t>(qkv) & 3u) || (reinterpret_cast<uintptr_t>(out) & 3u))
    return -2;
  PTL_REQUIRE((r1 == nullptr) == (r2 == nullptr) && page_size > 0 && num_pages > 0 && n_tiles >= 0 && tile_tokens > 0 &&
                  column >= 0 && column + H * d <= out_ld && q_ld >= H * d, "chunk_attention_tc: bad sizes");
  const dim3 grid((tile_tokens + ptl::kCtRows - 1) / ptl::kCtRows + 1, n_tiles);
  if (n_tiles == 0) return 0;
  const auto fn = d == 64 ? ptl::chunk_attention_tc<64> : ptl::chunk_attention_tc<128>;
  return fn(out, out_ld, column, qkv, q_ld, q_bias, cache, block_table, table_width, tiles, grid, H, G, page_size, scale, chunk, r1, r2, talk,
            num_pages, out_scale, stream);
}
