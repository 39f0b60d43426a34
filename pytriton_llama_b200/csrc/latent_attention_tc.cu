// Attention over kept rows [latent (R) | rotated key part (n)] that all heads share (parts/latent_attention.py), bfloat16 on
// the tensor cores, straight from the paged cache: the latent is the key's first R entries and the value.
//   out[t, h, :] = sum_j softmax_j(scale * q[t, h, :] . row_j) * row_j[:R],   j <= position of t
// q [T, H * (R + n)], out [T, H * R].  Two kernels share the layout: a row of 16-byte packets in shared memory has one packet
// more than an even number, so that the eight rows of an ldmatrix start in different banks.
//
// latent_prefill: portions of prompts.  The rows of q, (token, head) after (token, head), are one matrix: a block takes 64 of
// them from a tile of the step's list (128 tokens of one request) and walks the keys up to its last token's position in
// tiles of 32, a ring of three.  Of the scores each of the eight warps works 32 rows by 16 keys over half of the columns (the halves meet through
// shared memory), of the weighted sums 32 rows by a quarter of the latent's columns; the weights (rounded once to bfloat16, as the
// softmax over stored scores did) pass through shared memory.  The rows of keys and queries come by one bulk copy each, a warp's lanes a
// tile (as copies of 16 bytes they held all warps up for 1,200 of a tile's 5,500 cycles).  Bound by the fragments read for the warp-level tensor
// instructions, 303 KB per 64 x 32 scores (16 rows a warp: 434).  8 heads, R 512, n 64, us against copies of 16 bytes and 16 rows a warp: eight
// prompts of 65 to 440 tokens 60 and 71, one of 2,048 242 and 294, of 33 7.8 and 9.3, 128 tokens after 4,000 339 and 414; 16 heads, R 128: 202 and 207,
// of 33 5.1 and 4.8.
//
// latent_decode: single tokens, all heads of a token (up to 16 per block) against a share of its keys, 64 at a time, two
// tiles in flight; the float32 weights go to the tensor cores as three bfloat16 terms each (24 bits), so that nothing of
// them is lost; shares are merged by latent_merge.  Bound by the latency of a tile at eight requests of 1,000 positions: one
// tile a block, 7.6 us and 4.7 us for the merge.
//
// For R of 128, 256 and 512 both replace what was there: per request a gather, two library products around a softmax kernel
// (260 us of kernels a layer for the eight prompts above, and more launches than the host keeps up with: the whole step of
// four such layers 5.52 -> 2.61 ms), and for decoding the CUDA-core kernel with a warp per token, head and share (48 + 30 us
// a layer with dependent launches; a step of eight 731 -> 536 us).
#include "mma_utils.cuh"
#include "tcgen05_utils.cuh"

namespace ptl {

constexpr int kLpRows = 64, kLpKeys = 32, kLpStages = 3, kLpThreads = 256;
constexpr int kLdKeys = 64, kLdStages = 2, kLdThreads = 256, kLdHeads = 16;

__host__ __device__ constexpr int latent_row_bytes(int d) { return d * 2 + 16; }      // d a multiple of 16
constexpr int kLpWeightBytes = kLpKeys * 2 + 16;

// The packets of `rows` keys from `first` on into shared memory, zeros for keys from `limit` on and for pages not held;
// eight threads per key.
template <int KEYS>
__device__ __forceinline__ void latent_fetch(uint32_t dst, const __nv_bfloat16* __restrict__ cache, const int* __restrict__ bt, int first,
                                             int limit, int d, int page_size, int num_pages) {
  constexpr int PASSES = KEYS / 32;      // 256 threads
  const int sub = threadIdx.x & 7;
#pragma unroll
  for (int i = 0; i < PASSES; ++i) {
    const int row = (threadIdx.x >> 3) + 32 * i, key = first + row;
    const int page = key < limit ? bt[key / page_size] : -1;
    const bool ok = page >= 0 && page < num_pages;
    const __nv_bfloat16* src = ok ? cache + ((size_t)page * page_size + key % page_size) * d : cache;
    const uint32_t to = dst + row * latent_row_bytes(d);
    for (int c = sub; c < d / 8; c += 8) cp_async_16(to + 16 * c, src + (ok ? 8 * c : 0), ok);
  }
}

template <int R>
__global__ void __launch_bounds__(kLpThreads, 1)
latent_prefill_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ cache,
                      const int* __restrict__ block_table, const int* __restrict__ tiles, int bt_stride, int H, int d, int page_size,
                      int num_pages, float scale_log2, int* status, CopyWaits waits) {
  extern __shared__ __align__(128) unsigned char lp_smem[];
  __shared__ uint64_t s_bars[kLpStages + 1];                      // a tile's rows are here; the queries are
  __shared__ int s_abort;
  __shared__ float s_max[2][kLpRows];
  __shared__ float s_sum[2][kLpRows];
  const int* tile = tiles + 4 * blockIdx.y;                       // request row, first token row, tokens, first position (inputs of the step)
  const int req = tile[0], token0 = tile[1], tokens = tile[2], pos0 = tile[3];
  const int row0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * kLpRows;      // the rows that see most keys first
  const int rows = tokens * H;
  pdl_wait();
  pdl_launch_dependents();
  if (req < 0 || row0 >= rows) return;
  const int ld = latent_row_bytes(d);
  const uint32_t sq = smem_u32(lp_smem), sk = sq + kLpRows * ld, sp = sk + kLpStages * kLpKeys * ld, sx = sp + kLpRows * kLpWeightBytes;
  const int* bt = block_table + (size_t)req * bt_stride;
  const int last_row = min(row0 + kLpRows, rows) - 1;
  const int keys = pos0 + last_row / H + 1;                       // keys that the block's last token sees
  const int n_tiles = (keys + kLpKeys - 1) / kLpKeys;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  // scores: 32 rows (wr), 16 keys (wn), half of the dot product (wk), the halves added for 16 of the rows each (wm); weighted sums: 32 rows, a
  // quarter of the columns (wc)
  const int wr = warp & 1, wn = (warp >> 1) & 1, wk = warp >> 2, wm = 2 * wr + wk, wc = warp >> 1;

  const uint32_t bars = smem_u32(s_bars);
  volatile int* const abort_flag = &s_abort;
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i <= kLpStages; ++i) mbar_init(bars + 8 * i, kLpThreads / 32);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Every warp fetches four keys of a tile, a lane each (75 cycles a copy: one warp's 32 would take 2,400); the lane's page is looked up a tile ahead
  constexpr int OWN = kLpKeys / (kLpThreads / 32), OWN_ROWS = kLpRows / (kLpThreads / 32);
  static_assert(OWN <= 32 && OWN_ROWS <= 32, "a lane a row");
  const int own = warp * OWN + lane;
  int key = own, entry = own / page_size, offset = own % page_size, page = -1;
  const int step_entries = kLpKeys / page_size, step_offset = kLpKeys % page_size;
  const auto look_up = [&] {
    page = -1;
    if (lane < OWN && key < keys) asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(page) : "l"(bt + entry));
  };
  look_up();
  __syncthreads();
  const auto copy_row = [&](uint32_t dst, const __nv_bfloat16* src, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(d * 2), "r"(bar) : "memory");
  };
  const auto fetch = [&](int t) {                                 // this warp's keys of tile t; zeros for keys without a page
    if (t == waits.withheld) return;
    const uint32_t stage = sk + (t % kLpStages) * kLpKeys * ld, bar = bars + 8 * (t % kLpStages);
    const bool ok = page >= 0 && page < num_pages;
    const unsigned held = __ballot_sync(0xffffffffu, ok), missing = ((1u << OWN) - 1) & ~held;
    for (unsigned miss = missing; miss; miss &= miss - 1)
      for (int c = lane; c < d / 8; c += 32) st_shared_16(stage + (warp * OWN + __ffs(miss) - 1) * ld + 16 * c, make_uint4(0u, 0u, 0u, 0u));
    if (missing) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // (a later tile's copies come after these)
    __syncwarp();
    if (lane == 0) mbar_expect_tx(bar, __popc(held) * d * 2);
    __syncwarp();
    if (ok) copy_row(stage + own * ld, cache + ((size_t)page * page_size + offset) * d, bar);
    key += kLpKeys;
    entry += step_entries;
    offset += step_offset;
    if (offset >= page_size) { offset -= page_size; ++entry; }
    look_up();
  };
  if (lane == 0) mbar_expect_tx(bars + 8 * kLpStages, OWN_ROWS * d * 2);
  __syncwarp();
  if (lane < OWN_ROWS) {                                          // (rows past the last one hold it again)
    const int r = warp * OWN_ROWS + lane;
    copy_row(sq + r * ld, q + ((size_t)token0 * H + min(row0 + r, rows - 1)) * d, bars + 8 * kLpStages);
  }
  for (int t = 0; t < min(n_tiles, kLpStages - 1); ++t) fetch(t);
  // rows of this thread: wm * 16 + g and + 8; a row past the end sees what the last one sees and is not stored
  int pos[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) pos[i] = pos0 + min(row0 + wm * 16 + g + 8 * i, rows - 1) / H;
  constexpr int NT = R / 32;                                      // 8-column blocks of a warp's quarter of the latent
  float o[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][j][e] = 0.f;
  float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, l[2] = {0.f, 0.f};      // rows wr * 32 + g + 8 i; of the warp's own 16
  const int lm_row = lane & 15, lm_half = lane >> 4;              // rows and packet of an ldmatrix.x4 of 16 x 16

  bool came = mbar_wait(bars + 8 * kLpStages, 0, abort_flag, status, 41, waits.polls);
  for (int t = 0; t < n_tiles; ++t) {
    came = mbar_wait(bars + 8 * (t % kLpStages), (t / kLpStages) & 1, abort_flag, status, 42, waits.polls) && came;
    if (__syncthreads_or(!came)) {                                // (the status says so; nothing is stored)
      if (tid == 0) {
        mbar_drain(bars + 8 * kLpStages, 0);
        for (int i = t; i < min(n_tiles, t + kLpStages - 1); ++i) mbar_drain(bars + 8 * (i % kLpStages), (i / kLpStages) & 1);
      }
      return;
    }
    if (t + kLpStages - 1 < n_tiles) fetch(t + kLpStages - 1);
    const uint32_t kt = sk + (t % kLpStages) * kLpKeys * ld;
    // scores of 32 rows and 16 keys over half of the columns; the other half's come through shared memory
    float part[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[i][j][e] = 0.f;
    const uint32_t qa = sq + (wr * 32 + lm_row) * ld + 16 * lm_half;
    const uint32_t ka = kt + (wn * 16 + (lane & 7) + 8 * lm_half) * ld + 16 * ((lane >> 3) & 1);
    const int k_mid = (d / 16 + 1) / 2, k_end = wk ? d / 16 : k_mid;
#pragma unroll 2
    for (int k = wk ? k_mid : 0; k < k_end; ++k) {
      uint32_t a[2][4], b[4];
      ldmatrix_x4(a[0], qa + 32 * k);
      ldmatrix_x4(a[1], qa + 16 * ld + 32 * k);
      ldmatrix_x4(b, ka + 32 * k);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mma_bf16_16816(part[i][0], a[i], b[0], b[1]);
        mma_bf16_16816(part[i][1], a[i], b[2], b[3]);
      }
    }
    float s[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const float give0 = wk ? part[0][j][e] : part[1][j][e], give1 = wk ? part[0][j][e + 1] : part[1][j][e + 1];
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(sx + (((warp * 4 + 2 * j + e / 2) * 32 + lane) << 3)), "f"(give0), "f"(give1) : "memory");
      }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        float got0, got1;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(got0), "=f"(got1) : "r"(sx + ((((warp ^ 4) * 4 + 2 * j + e / 2) * 32 + lane) << 3)) : "memory");
        s[j][e] = (wk ? part[1][j][e] : part[0][j][e]) + got0;
        s[j][e + 1] = (wk ? part[1][j][e + 1] : part[0][j][e + 1]) + got1;
      }
    // to base 2, the causal bound, the rows' maxima over both halves of the keys
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int key = t * kLpKeys + wn * 16 + j * 8 + c2 + (e & 1);
        s[j][e] = key <= pos[e >> 1] ? s[j][e] * scale_log2 : -INFINITY;
        mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
      }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
      mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
    }
    if ((lane & 3) == 0) {
      s_max[wn][wm * 16 + g] = mx[0];
      s_max[wn][wm * 16 + g + 8] = mx[1];
    }
    __syncthreads();
    float alpha[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = wr * 32 + g + 8 * i;
      const float now = fmaxf(m[i], fmaxf(s_max[0][row], s_max[1][row]));      // (key 0 is in the first tile: finite)
      alpha[i] = exp2f(m[i] - now);
      m[i] = now;
    }
    const float own_m[2] = {wk ? m[2] : m[0], wk ? m[3] : m[1]};
    l[0] *= wk ? alpha[2] : alpha[0];
    l[1] *= wk ? alpha[3] : alpha[1];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float p[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        p[e] = exp2f(s[j][e] - own_m[e >> 1]);
        l[e >> 1] += p[e];
      }
      const uint32_t at = sp + (wm * 16 + g) * kLpWeightBytes + (wn * 16 + j * 8 + c2) * 2;
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(pack_bf16(p[0], p[1])) : "memory");
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + 8 * kLpWeightBytes), "r"(pack_bf16(p[2], p[3])) : "memory");
    }
    if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f || alpha[2] != 1.f || alpha[3] != 1.f)) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          o[i][j][0] *= alpha[2 * i]; o[i][j][1] *= alpha[2 * i];
          o[i][j][2] *= alpha[2 * i + 1]; o[i][j][3] *= alpha[2 * i + 1];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kLpKeys / 16; ++k) {
      uint32_t a[2][4];
      ldmatrix_x4(a[0], sp + (wr * 32 + lm_row) * kLpWeightBytes + 32 * k + 16 * lm_half);
      ldmatrix_x4(a[1], sp + (wr * 32 + 16 + lm_row) * kLpWeightBytes + 32 * k + 16 * lm_half);
      const uint32_t va = kt + (16 * k + lm_row) * ld + wc * (R / 2) + 16 * lm_half;       // (R / 2 bytes: a quarter of the latent's columns)
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, va + 16 * j);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_bf16_16816(o[i][j], a[i], b[0], b[1]);
          mma_bf16_16816(o[i][j + 1], a[i], b[2], b[3]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
  }
  if ((lane & 3) == 0) {
    s_sum[wn][wm * 16 + g] = l[0];
    s_sum[wn][wm * 16 + g + 8] = l[1];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = wr * 32 + g + 8 * i;
    if (row0 + row >= rows) continue;
    const float inv = 1.0f / (s_sum[0][row] + s_sum[1][row]);
    __nv_bfloat16* dst = out + ((size_t)token0 * H + row0 + row) * R + wc * (R / 4) + c2;
#pragma unroll
    for (int j = 0; j < NT; ++j)
      *reinterpret_cast<uint32_t*>(dst + 8 * j) = pack_bf16(o[i >> 1][j][2 * (i & 1)] * inv, o[i >> 1][j][2 * (i & 1) + 1] * inv);
  }
}

// part [items][splits][H][R] float32 (not yet divided), ml [items][splits][H][2] (maximum to base 2, sum); with one share the
// result itself.
template <int R>
__global__ void __launch_bounds__(kLdThreads, 1)
latent_decode_kernel(__nv_bfloat16* __restrict__ out, float* __restrict__ part, float* __restrict__ ml, const __nv_bfloat16* __restrict__ q,
                     const __nv_bfloat16* __restrict__ cache, const int* __restrict__ block_table, const int* __restrict__ tok_req,
                     const int* __restrict__ positions, const int* __restrict__ items, int bt_stride, int H, int d, int page_size,
                     int num_pages, int splits, float scale_log2) {
  extern __shared__ __align__(128) unsigned char ld_smem[];
  __shared__ float s_scores[kLdHeads][kLdKeys + 4];
  __shared__ __align__(16) __nv_bfloat16 s_w[3][kLdHeads][kLdKeys + 8];
  __shared__ float s_alpha[kLdHeads], s_m[kLdHeads], s_l[kLdHeads];
  const int item = blockIdx.y, split = blockIdx.x, h0 = blockIdx.z * kLdHeads;
  const int token = items ? items[item] : item;                   // inputs of the step
  const int req = tok_req[token], keys_all = positions[token] + 1;
  pdl_wait();
  pdl_launch_dependents();
  if (req < 0) return;
  const int heads = min(kLdHeads, H - h0);
  // whole tiles of 64 keys per share; a share without keys leaves a sum of zero
  const int n_all = (keys_all + kLdKeys - 1) / kLdKeys;
  const int each = (n_all + splits - 1) / splits;
  const int tile0 = split * each, n_tiles = max(0, min(each, n_all - tile0));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  const size_t at = ((size_t)item * splits + split) * H + h0;
  if (n_tiles == 0) {
    if (tid < heads) { ml[2 * (at + tid)] = -INFINITY; ml[2 * (at + tid) + 1] = 0.f; }
    return;
  }
  const int ld = latent_row_bytes(d);
  const uint32_t sq = smem_u32(ld_smem), sk = sq + kLdHeads * ld;
  const int* bt = block_table + (size_t)req * bt_stride;
  const __nv_bfloat16* q0 = q + ((size_t)token * H + h0) * d;
  for (int idx = tid; idx < kLdHeads * (d / 8); idx += kLdThreads) {
    const int r = idx / (d / 8), c = idx % (d / 8);
    const bool ok = r < heads;
    cp_async_16(sq + r * ld + 16 * c, q0 + (ok ? (size_t)r * d + 8 * c : 0), ok);
  }
#pragma unroll
  for (int s = 0; s < kLdStages - 1; ++s) {
    if (s < n_tiles) latent_fetch<kLdKeys>(sk + s * kLdKeys * ld, cache, bt, (tile0 + s) * kLdKeys, keys_all, d, page_size, num_pages);
    cp_async_commit();
  }
  if (tid < kLdHeads) { s_m[tid] = -INFINITY; s_l[tid] = 0.f; }
  constexpr int NT = R / 64;                                      // 8-column blocks of a warp's eighth of the latent
  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  const int lm_row = lane & 15, lm_half = lane >> 4;

  for (int t = 0; t < n_tiles; ++t) {
    __syncthreads();                                              // the stage that is filled next has been read
    if (t + kLdStages - 1 < n_tiles)
      latent_fetch<kLdKeys>(sk + ((t + kLdStages - 1) % kLdStages) * kLdKeys * ld, cache, bt, (tile0 + t + kLdStages - 1) * kLdKeys,
                            keys_all, d, page_size, num_pages);
    cp_async_commit();
    cp_async_wait<kLdStages - 1>();
    __syncthreads();
    const uint32_t kt = sk + (t % kLdStages) * kLdKeys * ld;
    // scores of all heads and 8 keys per warp; two products at a time, k ranges side by side in one ldmatrix of the keys
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
    const uint32_t qa = sq + lm_row * ld + 16 * lm_half;
    const uint32_t ka = kt + (warp * 8 + (lane & 7)) * ld + 16 * (lane >> 3);
    int k = 0;
#pragma unroll 4
    for (; k + 1 < d / 16; k += 2) {
      uint32_t a[4], a1[4], b[4];
      ldmatrix_x4(b, ka + 32 * k);
      ldmatrix_x4(a, qa + 32 * k);
      ldmatrix_x4(a1, qa + 32 * k + 32);
      mma_bf16_16816(s0, a, b[0], b[1]);
      mma_bf16_16816(s1, a1, b[2], b[3]);
    }
    if (k < d / 16) {                                             // an odd number of 16s: the last packet pair alone
      uint32_t a[4], b[4];
      ldmatrix_x4(b, kt + (warp * 8 + (lane & 7)) * ld + 32 * k + 16 * ((lane >> 3) & 1));
      ldmatrix_x4(a, qa + 32 * k);
      mma_bf16_16816(s0, a, b[0], b[1]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int col = warp * 8 + c2 + (e & 1);
      const bool seen = (tile0 + t) * kLdKeys + col < keys_all;
      s_scores[g + 8 * (e >> 1)][col] = seen ? (s0[e] + s1[e]) * scale_log2 : -INFINITY;
    }
    __syncthreads();
    // two heads per warp: maximum, weights (three bfloat16 terms each), sum
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int h = warp * 2 + i;
      const float a = s_scores[h][lane], b = s_scores[h][lane + 32];
      const float before = s_m[h];
      const float now = fmaxf(before, warp_max(fmaxf(a, b)));
      const float p[2] = {exp2f(a - now), exp2f(b - now)};
      const float sum = warp_sum(p[0] + p[1]);
      if (lane == 0) {
        const float alpha = exp2f(before - now);
        s_alpha[h] = alpha;
        s_m[h] = now;
        s_l[h] = s_l[h] * alpha + sum;
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float rest = p[e];
#pragma unroll
        for (int w = 0; w < 3; ++w) {
          const __nv_bfloat16 term = __float2bfloat16_rn(rest);
          s_w[w][h][lane + 32 * e] = term;
          rest -= __bfloat162float(term);
        }
      }
    }
    __syncthreads();
    const float al0 = s_alpha[g], al1 = s_alpha[g + 8];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      o[j][0] *= al0; o[j][1] *= al0;
      o[j][2] *= al1; o[j][3] *= al1;
    }
#pragma unroll
    for (int kk = 0; kk < kLdKeys / 16; ++kk) {
      uint32_t a[3][4];
#pragma unroll
      for (int w = 0; w < 3; ++w) ldmatrix_x4(a[w], smem_u32(&s_w[w][lm_row][16 * kk + 8 * lm_half]));
      const uint32_t va = kt + (16 * kk + lm_row) * ld + warp * (R / 8) * 2 + 16 * lm_half;
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, va + 16 * j);
#pragma unroll
        for (int w = 2; w >= 0; --w) {
          mma_bf16_16816(o[j], a[w], b[0], b[1]);
          mma_bf16_16816(o[j + 1], a[w], b[2], b[3]);
        }
      }
    }
  }
  const int col0 = warp * (R / 8) + c2;
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int h = g + 8 * i;
      if (h >= heads) continue;
      const float inv = 1.0f / s_l[h];
      __nv_bfloat16* dst = out + ((size_t)token * H + h0 + h) * R + col0;
#pragma unroll
      for (int j = 0; j < NT; ++j)
        *reinterpret_cast<uint32_t*>(dst + 8 * j) = pack_bf16(o[j][2 * i] * inv, o[j][2 * i + 1] * inv);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int h = g + 8 * i;
    if (h >= heads) continue;
    float* dst = part + (at + h) * R + col0;
#pragma unroll
    for (int j = 0; j < NT; ++j) *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(o[j][2 * i], o[j][2 * i + 1]);
  }
  if (tid < heads) { ml[2 * (at + tid)] = s_m[tid]; ml[2 * (at + tid) + 1] = s_l[tid]; }
}

// One block per (item, head): the shares' sums weighted by 2^(their maximum - the largest), R / 4 threads of four columns.  Bound by
// latency: the maxima and sums come in one round trip and the weights go to shared memory, so that the shares' loads wait for
// nothing and are in flight together (8 requests of 8 heads, 16 shares: 4.7 us; one share after the other 7.9).
constexpr int kLmShares = 256;

__global__ void __launch_bounds__(128)
latent_merge_kernel(__nv_bfloat16* __restrict__ out, const float* __restrict__ part, const float* __restrict__ ml,
                    const int* __restrict__ tok_req, const int* __restrict__ items, int H, int R, int splits) {
  __shared__ float s_m[kLmShares], s_l[kLmShares], s_w[kLmShares];
  const int item = blockIdx.y, h = blockIdx.x;
  const int token = items ? items[item] : item;
  const bool held = tok_req[token] >= 0;
  pdl_wait();
  pdl_launch_dependents();
  if (!held) return;
  const size_t at = (size_t)item * splits * H + h;
  for (int s = threadIdx.x; s < splits; s += blockDim.x) {
    const float2 v = *reinterpret_cast<const float2*>(ml + 2 * (at + (size_t)s * H));
    s_m[s] = v.x;
    s_l[s] = v.y;
  }
  __syncthreads();
  float top = -INFINITY;
  for (int s = 0; s < splits; ++s) top = fmaxf(top, s_m[s]);
  for (int s = threadIdx.x; s < splits; s += blockDim.x) s_w[s] = s_m[s] == -INFINITY ? 0.f : exp2f(s_m[s] - top);
  __syncthreads();
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  float l = 0.f;
  const float* src = part + at * R + 4 * threadIdx.x;
  for (int s0 = 0; s0 < splits; s0 += 8) {
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)                                     // (weight 0: no keys, nothing was written)
      v[i] = s0 + i < splits && s_w[s0 + i] > 0.f ? *reinterpret_cast<const float4*>(src + (size_t)(s0 + i) * H * R)
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (s0 + i >= splits) break;
      const float w = s_w[s0 + i];
      if (w > 0.f) l = fmaf(w, s_l[s0 + i], l);
      sum.x = fmaf(w, v[i].x, sum.x); sum.y = fmaf(w, v[i].y, sum.y);
      sum.z = fmaf(w, v[i].z, sum.z); sum.w = fmaf(w, v[i].w, sum.w);
    }
  }
  const float inv = 1.0f / l;
  uint2 packed = make_uint2(pack_bf16(sum.x * inv, sum.y * inv), pack_bf16(sum.z * inv, sum.w * inv));
  *reinterpret_cast<uint2*>(out + ((size_t)token * H + h) * R + 4 * threadIdx.x) = packed;
}

// What both kernels ask of sizes and addresses (and a grid's 65,535 tiles or single tokens); -2: take another path.
inline bool latent_tc_fits(const void* out, const void* q, const void* cache, int H, int R, int n) {
  return (R == 128 || R == 256 || R == 512) && n >= 0 && n % 16 == 0 && n <= 64 && H > 0 && H <= 512 && aligned16(out) && aligned16(q) &&
         aligned16(cache);
}

template <int R>
int latent_prefill(void* out, const void* q, const void* cache, const int* bt, const int* tiles, int n_tiles, int bt_stride, int H, int d,
                   int page_size, int num_pages, float scale, int tile_tokens, int* status, void* stream, CopyWaits waits) {
  const int smem = (kLpRows + kLpStages * kLpKeys) * latent_row_bytes(d) + kLpRows * kLpWeightBytes + kLpThreads * 32;
  static SmemRaised raised;
  if (int rc = raise_shared_memory("latent_prefill", latent_prefill_kernel<R>, 200 * 1024, raised)) return rc;
  const dim3 grid((tile_tokens * H + kLpRows - 1) / kLpRows, n_tiles);
  return launch_kernel("latent_prefill", latent_prefill_kernel<R>, grid, dim3(kLpThreads), smem, as_stream(stream), (__nv_bfloat16*)out,
                       (const __nv_bfloat16*)q, (const __nv_bfloat16*)cache, bt, tiles, bt_stride, H, d, page_size, num_pages,
                       scale * 1.4426950408889634f, status, waits);
}

template <int R>
int latent_decode(void* out, float* part, float* ml, const void* q, const void* cache, const int* bt, const int* tok_req, const int* positions,
                  const int* items, int n_items, int bt_stride, int H, int d, int page_size, int num_pages, int splits, float scale,
                  void* stream) {
  const int smem = (kLdHeads + kLdStages * kLdKeys) * latent_row_bytes(d);
  static SmemRaised raised;
  if (int rc = raise_shared_memory("latent_decode", latent_decode_kernel<R>, 200 * 1024, raised)) return rc;
  const dim3 grid(splits, n_items, (H + kLdHeads - 1) / kLdHeads);
  if (int rc = launch_kernel("latent_decode", latent_decode_kernel<R>, grid, dim3(kLdThreads), smem, as_stream(stream), (__nv_bfloat16*)out,
                             part, ml, (const __nv_bfloat16*)q, (const __nv_bfloat16*)cache, bt, tok_req, positions, items, bt_stride, H, d,
                             page_size, num_pages, splits, scale * 1.4426950408889634f))
    return rc;
  if (splits == 1) return 0;
  return launch_kernel("latent_merge", latent_merge_kernel, dim3(H, n_items), dim3(R / 4), 0, as_stream(stream), (__nv_bfloat16*)out, part,
                       ml, tok_req, items, H, R, splits);
}

}  // namespace ptl

static int latent_prefill_any(void* out, const void* q, const void* cache, const int* block_table, const int* tiles, int n_tiles, int bt_stride,
                              int H, int R, int n, int page_size, int num_pages, float scale, int tile_tokens, void* status, void* stream,
                              ptl::CopyWaits waits = {}) {
  if (!ptl::latent_tc_fits(out, q, cache, H, R, n) || n_tiles > 65535) return -2;
  PTL_REQUIRE(n_tiles >= 0 && bt_stride > 0 && page_size > 0 && num_pages > 0 && tile_tokens > 0,
              "latent_prefill: bad sizes");
  if (n_tiles == 0) return 0;
  const auto fn = R == 128 ? ptl::latent_prefill<128> : R == 256 ? ptl::latent_prefill<256> : ptl::latent_prefill<512>;
  return fn(out, q, cache, block_table, tiles, n_tiles, bt_stride, H, R + n, page_size, num_pages, scale, tile_tokens, (int*)status, stream, waits);
}
// For callers without a status word: a wait that gives up is not reported.
PTL_EXPORT int ptl_latent_prefill_bf16(void* out, const void* q, const void* cache, const int* block_table, const int* tiles, int n_tiles,
                                       int bt_stride, int H, int R, int n, int page_size, int num_pages, float scale, int tile_tokens,
                                       void* stream) {
  return latent_prefill_any(out, q, cache, block_table, tiles, n_tiles, bt_stride, H, R, n, page_size, num_pages, scale, tile_tokens, nullptr, stream);
}
// `status`: set where a wait inside the kernel gave up.
PTL_EXPORT int ptl_latent_prefill_status_bf16(void* out, const void* q, const void* cache, const int* block_table, const int* tiles, int n_tiles,
                                              int bt_stride, int H, int R, int n, int page_size, int num_pages, float scale, int tile_tokens,
                                              void* status, void* stream) {
  return latent_prefill_any(out, q, cache, block_table, tiles, n_tiles, bt_stride, H, R, n, page_size, num_pages, scale, tile_tokens, status, stream);
}
// Self-test of the bounded waits: they give up after `polls` polls, and no block fetches its tile `no_tile` of keys.  The kernel must then
// write *status (42) and return; `out` holds nothing of value.
PTL_EXPORT int ptl_latent_prefill_wait_selftest(void* out, const void* q, const void* cache, const int* block_table, const int* tiles, int n_tiles,
                                                int bt_stride, int H, int R, int n, int page_size, int num_pages, float scale, int tile_tokens,
                                                void* status, void* stream, unsigned polls, int no_tile) {
  PTL_REQUIRE(status && polls >= 1 && polls <= (1u << 16), "latent_prefill_wait_selftest: a status word, and between 1 and 65536 polls");
  return latent_prefill_any(out, q, cache, block_table, tiles, n_tiles, bt_stride, H, R, n, page_size, num_pages, scale, tile_tokens, status, stream,
                            {polls, no_tile});
}

PTL_EXPORT int ptl_latent_decode_bf16(void* out, float* part, float* ml, const void* q, const void* cache, const int* block_table,
                                      const int* tok_req, const int* positions, const int* items, int n_items, int bt_stride, int H, int R,
                                      int n, int page_size, int num_pages, int splits, float scale, void* stream) {
  if (!ptl::latent_tc_fits(out, q, cache, H, R, n) || n_items > 65535) return -2;
  PTL_REQUIRE(n_items >= 0 && bt_stride > 0 && page_size > 0 && num_pages > 0 && splits >= 1 && splits <= ptl::kLmShares &&
                  (splits == 1 || (part && ml)), "latent_decode: bad sizes");
  if (n_items == 0) return 0;
  const auto fn = R == 128 ? ptl::latent_decode<128> : R == 256 ? ptl::latent_decode<256> : ptl::latent_decode<512>;
  return fn(out, part, ml, q, cache, block_table, tok_req, positions, items, n_items, bt_stride, H, R + n, page_size, num_pages, splits, scale,
            stream);
}
