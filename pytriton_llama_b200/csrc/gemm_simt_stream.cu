// out[M, N] (+)= A[M, K] * W[N, K]^T in float32 for up to 32 rows, K a multiple of 32: the products of a decode step, bound by the
// weights' bytes.  The sums are those of gemm_simt.cu, bit for bit: chunks of 32 k values by two chains of FMAs (even and odd k), chunk sums added in order
// with a compensated addition.
//
// As many blocks as fit at once walk tiles of 8 or 16 weight rows.  A thread of its own asks for turns of 256 k values of a tile's rows by TMA, one tile after the other without a stop, the weights of the first
// ring of turns before the wait on the predecessor (weights that a kernel of the step has written need an ordinary launch); the warps take the
// turns one after the other, and a warp of its own adds the chunk sums of a round of turns while the next is multiplied.  A lane owns
// one chunk for a quarter of the weight rows and all token rows.  A chunk is a 128-byte row of the TMA tile: with the 128-byte swizzle the
// eight chunks of a quarter warp lie in different banks.
// The form by cp.async (gemm_simt_few, which keeps what is no multiple of 32) has a warp copy its own turns, 24 instructions a lane and
// turn, and wait for them with nothing else in flight, us there and here: 4 rows to 16,384 features of 2,048 34 and 24, to 32,000 of 1,024 40 and
// 22, 2,048 features of 8,192 24 and 18; 16 rows to 16,384 features 85 and 48; a row to 16,384 27 and 21.
#include <algorithm>
#include "tcgen05_utils.cuh"

namespace ptl {

constexpr int kStreamTurn = 256;
__host__ __device__ constexpr int stream_sums_ld(int mt, int rows) { return rows * mt + 33; }
__host__ __device__ constexpr int stream_ring_bytes(int mt, int rows, int stages) { return stages * (rows + mt) * 1024; }
constexpr int stream_smem_bytes(int mt, int rows, int warps, int stages) {
  return stream_ring_bytes(mt, rows, stages) + 2 * warps * 8 * stream_sums_ld(mt, rows) * 4 + 16 * stages + 16;
}

__device__ __forceinline__ void stream_kahan(float& sum, float& comp, float chunk) {
  const float y = __fsub_rn(chunk, comp);
  const float t = __fadd_rn(sum, y);
  comp = __fsub_rn(__fsub_rn(t, sum), y);
  sum = t;
}

template <int MT, int ROWS, int WARPS, int STAGES>
__global__ void __launch_bounds__((WARPS + 2) * 32)
gemm_simt_stream_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, float* __restrict__ out,
                        int M, int N, int K, int ldo, int accumulate, int* __restrict__ status, CopyWaits waits) {
  static_assert(STAGES >= WARPS, "a stage's next filling is waited for a round after its last at the earliest");
  constexpr int kStage = (ROWS + MT) * 1024, SUMS_LD = stream_sums_ld(MT, ROWS);
  extern __shared__ __align__(1024) unsigned char stream_smem[];
  float* sums = reinterpret_cast<float*>(stream_smem + STAGES * kStage);      // [2][warp][8 chunks][4 groups][RL rows][MT]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sums + 2 * WARPS * 8 * SUMS_LD);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * STAGES);
  const uint32_t base = smem_addr(stream_smem), bar = smem_addr(bars);
  const auto full = [&](int s) { return bar + 8u * s; };
  const auto empty = [&](int s) { return bar + 8u * (STAGES + s); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int turns = (K + kStreamTurn - 1) / kStreamTurn, tiles = (N + ROWS - 1) / ROWS;
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;      // tiles blockIdx.x, + gridDim.x, ...
  const int all = mine * turns;                                                          // turns of this block, over its tiles
  if (warp == WARPS + 1 && lane == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (base & 1023u) {                                          // never expected (the same in every block)
    pdl_wait();
    if (threadIdx.x == 0 && status) atomicExch(status, 99);
    return;
  }
  if (warp == WARPS + 1) {
    if (lane == 0) {
      const int ahead = min(all, STAGES);
      int turn = 0, n0 = blockIdx.x * ROWS, turn_x = 0;
      const auto weights = [&](int s, int t) {
        if (t != waits.withheld) {
          mbar_expect_tx(full(s), kStage);
          tma_load_3d(base + s * kStage, &w_map, full(s), 0, turn * 8, n0);
        }
        if (++turn == turns) { turn = 0; n0 += gridDim.x * ROWS; }
      };
      const auto tokens = [&](int s, int t) {
        if (t != waits.withheld) tma_load_3d(base + s * kStage + ROWS * 1024, &x_map, full(s), 0, turn_x * 8, 0);
        if (++turn_x == turns) turn_x = 0;
      };
      for (int t = 0; t < ahead; ++t) weights(t, t);
      pdl_wait();
      for (int t = 0; t < ahead; ++t) tokens(t, t);
      int s = 0, round = 0, t = ahead;
      for (; t < all; ++t) {
        if (!mbar_wait(empty(s), round, abort_flag, status, 21, waits.polls)) break;
        weights(s, t);
        tokens(s, t);
        if (++s == STAGES) { s = 0; round ^= 1; }
      }
      // leave no copy in flight behind, also where a warp gives up after the last one was asked for (else they are here by the time the warps are done)
      for (int i = max(0, t - STAGES); i < t; ++i) mbar_drain(full(i % STAGES), (i / STAGES) & 1);
    }
    return;
  }
  pdl_wait();                                                  // (nothing is lost: a turn needs the tokens too)
  pdl_launch_dependents();
  const auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"((WARPS + 1) * 32) : "memory"); };
  const int chunk = lane & 7, group = lane >> 3;
  constexpr int RL = ROWS / 4;                                           // weight rows of a lane
  constexpr int RESULTS = ROWS * MT, PER = (RESULTS + 31) / 32;          // of the last warp's lanes
  float sum[PER], comp[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) { sum[i] = 0.f; comp[i] = 0.f; }
  const bool works = warp < WARPS;
  const int rounds = (turns + WARPS - 1) / WARPS;
  int in_tile = 0, done_round = 0, done_tile = blockIdx.x;      // round of the tile: being multiplied, being added
  int first = 0, buffer = 0;                                                         // this tile's turns before, parity of the rounds
  for (int n = mine * rounds; n >= 0; --n, buffer ^= 1) {
    const int turn = in_tile * WARPS + warp;
    if (works && n > 0 && turn < turns) {
      const int g = first + turn, s = g % STAGES;
      mbar_wait(full(s), (g / STAGES) & 1, abort_flag, status, 22, waits.polls);      // (given up: the flag is set, and the warps go on to their meetings)
      float2 acc[RL][MT];                                               // sums of even and of odd k
#pragma unroll
      for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = make_float2(0.f, 0.f);
      const unsigned char* wp = stream_smem + s * kStage + group * RL * 1024 + chunk * 128;
      const unsigned char* xp = stream_smem + s * kStage + ROWS * 1024 + chunk * 128;
#pragma unroll 2
      for (int k = 0; k < 8; ++k) {
        const int at = (k ^ chunk) << 4;
        float4 w[RL];
#pragma unroll
        for (int r = 0; r < RL; ++r) w[r] = *reinterpret_cast<const float4*>(wp + r * 1024 + at);
        constexpr int MS = MT < 4 ? MT : 4;                              // token rows at a time: their FMAs lie between two of one sum
#pragma unroll
        for (int m0 = 0; m0 < MT; m0 += MS) {
          float4 x[MS];
#pragma unroll
          for (int m = 0; m < MS; ++m) x[m] = *reinterpret_cast<const float4*>(xp + (m0 + m) * 1024 + at);
#pragma unroll
          for (int m = 0; m < MS; ++m)
#pragma unroll
            for (int r = 0; r < RL; ++r) acc[r][m0 + m] = fma2(make_float2(x[m].x, x[m].y), make_float2(w[r].x, w[r].y), acc[r][m0 + m]);
#pragma unroll
          for (int m = 0; m < MS; ++m)
#pragma unroll
            for (int r = 0; r < RL; ++r) acc[r][m0 + m] = fma2(make_float2(x[m].z, x[m].w), make_float2(w[r].z, w[r].w), acc[r][m0 + m]);
        }
      }
      __syncwarp();
      if (lane == 0 && !*abort_flag) mbar_arrive(empty(s));              // (a stage that did not come must not be asked for again)
      float* dst = sums + (size_t)buffer * WARPS * 8 * SUMS_LD + (warp * 8 + chunk) * SUMS_LD + group * (RL * MT + 8);
#pragma unroll
      for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) dst[r * MT + m] = __fadd_rn(acc[r][m].x, acc[r][m].y);
    }
    if (!works && n < mine * rounds) {                                   // the round before, while this one is multiplied
      const float* done = sums + (size_t)(buffer ^ 1) * WARPS * 8 * SUMS_LD;
      const int chunks = min(WARPS * 8, K / 32 - done_round * WARPS * 8);
#pragma unroll 4
      for (int c = 0; c < chunks; ++c)
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int at = min(lane + 32 * i, RESULTS - 1);
          stream_kahan(sum[i], comp[i], done[c * SUMS_LD + at + at / (RL * MT) * 8]);
        }
      if (++done_round == rounds) {
        done_round = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int at = lane + 32 * i, row = done_tile * ROWS + at / MT, m = at % MT;
          if (at < RESULTS && row < N && m < M) {
            float* o = out + (size_t)m * ldo + row;
            *o = accumulate ? sum[i] + *o : sum[i];
          }
          sum[i] = comp[i] = 0.f;
        }
        done_tile += gridDim.x;
      }
    }
    if (++in_tile == rounds) { in_tile = 0; first += turns; }
    meet();
  }
}

// A float32 matrix of rows ld apart as [rows][K / 32][32], fetched in boxes of box_rows x 8 x 32 with the 128-byte swizzle.
struct StreamMapKey {
  const void* base; int rows, chunks, ld, box_rows;
  bool operator==(const StreamMapKey& o) const { return base == o.base && rows == o.rows && chunks == o.chunks && ld == o.ld && box_rows == o.box_rows; }
};
struct StreamMapHash {
  size_t operator()(const StreamMapKey& k) const {
    return reinterpret_cast<size_t>(k.base) ^ ((size_t)k.rows * 0x9E3779B97F4A7C15ull + (size_t)k.chunks * 0xC2B2AE3D27D4EB4Full +
                                               (size_t)k.ld * 0x27D4EB2F165667C5ull + (size_t)k.box_rows * 0x165667B19E3779F9ull);
  }
};
static int stream_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows) {
  static std::unordered_map<StreamMapKey, CUtensorMap, StreamMapHash> cache;
  static std::mutex lock;
  const StreamMapKey key{base, rows, K / 32, ld, box_rows};
  std::lock_guard<std::mutex> guard(lock);
  auto it = cache.find(key);
  if (it != cache.end()) { *map = it->second; return 0; }
  EncodeTiledFn fn = encode_fn();
  PTL_REQUIRE(fn != nullptr, "gemm_simt_stream: the driver has no cuTensorMapEncodeTiled");
  cuuint64_t dims[3] = {32, (cuuint64_t)K / 32, (cuuint64_t)rows}, strides[2] = {128, (cuuint64_t)ld * 4};
  cuuint32_t box[3] = {32, 8, (cuuint32_t)box_rows}, estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  PTL_REQUIRE(r == CUDA_SUCCESS, "gemm_simt_stream: cuTensorMapEncodeTiled failed with %d (rows=%d K=%d ld=%d)", (int)r, rows, K, ld);
  if (cache.size() > 8192) cache.clear();
  cache.emplace(key, *map);
  return 0;
}

template <int MT, int ROWS, int WARPS, int STAGES, int HELD>
static int launch_stream(float* out, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldo, int accumulate, int* status,
                         cudaStream_t stream, CopyWaits waits) {
  static SmemRaised raised;
  auto kernel = gemm_simt_stream_kernel<MT, ROWS, WARPS, STAGES>;
  constexpr int smem = stream_smem_bytes(MT, ROWS, WARPS, STAGES);
  if (int rc = raise_shared_memory("gemm_simt_stream", kernel, smem, raised)) return rc;
  CUtensorMap w_map, x_map;
  int rc = stream_map(&w_map, W, N, K, ldw, ROWS);
  if (!rc) rc = stream_map(&x_map, A, M, K, lda, MT);
  if (rc) return rc;
  return launch_kernel("gemm_simt_stream", kernel, dim3(std::min((N + ROWS - 1) / ROWS, HELD * sm_count_of_device())), dim3((WARPS + 2) * 32), smem, stream, w_map, x_map, out, M, N,
                       K, ldo, accumulate, status, waits);
}

}  // namespace ptl

static int stream_product(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldo, int accumulate, void* status,
                          void* stream, ptl::CopyWaits waits = {}) {
  using namespace ptl;
  const bool narrow = N < 4736;       // fewer than four blocks of eight rows per SM
  if (M < 1 || M > 32 || (M > 16 && !narrow) || N < 1 || K < 32 || K % 32 || lda < K || ldw < K || ldo < N || lda % 4 || ldw % 4 || !aligned16(A) ||
      !aligned16(W))
    return -2;
  // Weights of a few hundred KB are there after one trip, and the kernel that copies them without a ring has less to set up: a row to 8 features
  // of 32 1.5 us there and 1.9 here, to 256 of 1,024 2.0 and 2.3, to 2,048 of 256 2.4 and 2.1, to 512 of 2,048 3.5 both; two rows to 256 of 1,024 2.25 and 2.30.
  if (M <= 2 && N <= (M == 1 ? 1024 : 256) && (long long)N * K <= 1 << 19) return -2;
#define PTL_STREAM(MT, ROWS, WARPS, STAGES, HELD)                                                                               \
  return launch_stream<MT, ROWS, WARPS, STAGES, HELD>((float*)out, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldo, accumulate, \
                                                (int*)status, as_stream(stream), waits)
  if (M <= 1) PTL_STREAM(1, 8, 4, 5, 4);
  if (M <= 2) PTL_STREAM(2, 8, 4, 4, 4);
  if (M <= 4) PTL_STREAM(4, 8, 4, 4, 3);
  if (M <= 8) PTL_STREAM(8, 8, 3, 3, 3);
  if (M <= 16) PTL_STREAM(16, 16, 4, 4, 1);
  PTL_STREAM(32, 8, 2, 3, 1);
#undef PTL_STREAM
}

// -2: sizes that gemm_simt takes.
PTL_EXPORT int ptl_gemm_simt_stream_f32(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldo, int accumulate,
                                        void* status, void* stream) {
  return stream_product(out, A, W, M, N, K, lda, ldw, ldo, accumulate, status, stream);
}
// Self-test of the bounded waits: they give up after `polls` polls, and no block asks for its turn `no_turn` (counted over its tiles).  The
// kernel must then write *status (21 or 22) and return; `out` holds nothing of value.
PTL_EXPORT int ptl_gemm_simt_stream_wait_selftest(void* out, const void* A, const void* W, int M, int N, int K, void* status, void* stream,
                                                  unsigned polls, int no_turn) {
  PTL_REQUIRE(status && polls >= 1 && polls <= (1u << 16), "gemm_simt_stream_wait_selftest: a status word, and between 1 and 65536 polls");
  return stream_product(out, A, W, M, N, K, K, K, N, 0, status, stream, {polls, no_turn});
}
