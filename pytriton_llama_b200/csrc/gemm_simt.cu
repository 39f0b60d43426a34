// out[M, N] (+)= A[M, K] * W[N, K]^T on the CUDA cores in float32: the true 32-bit matrix product
// of the float32 path (no tensor-core mode that drops mantissa bits), and a library-free check for
// the bfloat16 tensor-core kernels.  Any M, N, K; both operands are K-contiguous.
// A launch may hold several products of one shape (blockIdx.z = b): operand and result pointers move on by
// batch_a, batch_w, batch_o elements per b (the heads of an activation [M, heads * x] against weights
// [heads, N, K]); with `gate` the result of row m of product b is multiplied by sigmoid(gate[m * gate_ld + b]).
//
// Summation order, the same for every tile shape, so that a row's result does not depend on how
// many rows the call has (a prompt portion and a single decoded token give the same bits):
// the K range is cut into chunks of 32; inside a chunk the products of even and of odd k are added one by one with
// fused multiply-adds, k ascending, into two fresh accumulators (the two halves of a packed instruction), whose sum is the
// chunk's; the chunk sums are added to the running total with a compensated (Kahan) addition.  A plain running sum over K = 8,192 terms is
// wrong by about K/4 ulp of a term, which over 16 layers of a 2,048-wide model reaches 3e-4 in the
// logits; with chunks the error of a product is that of one chunk, a few ulp.
#include "common.cuh"

namespace ptl {

constexpr int kSimtChunk = 32;       // k values per chunk: the tile depth of every kernel shape

// sum += chunk, with the rounding error of the addition carried in `comp`
__device__ __forceinline__ void kahan_add(float& sum, float& comp, float chunk) {
  const float y = __fsub_rn(chunk, comp);
  const float t = __fadd_rn(sum, y);
  comp = __fsub_rn(__fsub_rn(t, sum), y);
  sum = t;
}
__device__ __forceinline__ void kahan_add_pair(float2& sum, float2& comp, float2 chunk) {
  const float2 y = sub2(chunk, comp);
  const float2 t = add2(sum, y);
  comp = sub2(sub2(t, sum), y);
  sum = t;
}

// What the kernels below cannot read in packets of 16 bytes, and 16-bit operands: any type and alignment.  CHAINS of FMAs a chunk: two
// where another kernel may take other rows of the same product (float32, K a multiple of 4), else one.
template <typename TI, typename TO, int BM, int BN, int TM, int TN, int CHAINS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simt_kernel(TO* __restrict__ out, const TI* __restrict__ A, const TI* __restrict__ W,
                 int M, int N, int K, int lda, int ldw, int ldo, int accumulate,
                 long long batch_a, long long batch_w, long long batch_o, const TI* __restrict__ gate, int gate_ld) {
  constexpr int BK = kSimtChunk;
  constexpr int THREADS = (BM / TM) * (BN / TN);
  static_assert(TM % 4 == 0, "rows per thread, two an instruction");
  pdl_wait();
  pdl_launch_dependents();
  A += (size_t)blockIdx.z * batch_a;
  W += (size_t)blockIdx.z * batch_w;
  out += (size_t)blockIdx.z * batch_o;
  __shared__ __align__(16) float As[BK][BM + 4];
  __shared__ __align__(16) float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN);  // along N
  const int ty = tid / (BN / TN);  // along M
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float2 acc[CHAINS][TM / 2][TN], sum[TM / 2][TN], comp[TM / 2][TN];      // of two rows each
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sum[i][j] = comp[i][j] = make_float2(0.f, 0.f);

  for (int k0 = 0; k0 < K; k0 += BK) {
    // any element type and alignment: consecutive threads walk along K so that global reads coalesce
    for (int e = tid; e < BM * BK; e += THREADS) {
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.f;
    }
    for (int e = tid; e < BN * BK; e += THREADS) {
      const int r = e / BK, c = e % BK;
      const int gn = n0 + r, gk = k0 + c;
      Ws[c][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[0][i][j] = acc[CHAINS - 1][i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float2 a[TM / 2];
      float b[TN];
#pragma unroll
      for (int i = 0; i < TM / 2; ++i) a[i] = *reinterpret_cast<const float2*>(&As[kk][ty * TM + 2 * i]);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[kk % CHAINS][i][j] = fma2(a[i], make_float2(b[j], b[j]), acc[kk % CHAINS][i][j]);
    }
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) kahan_add_pair(sum[i][j], comp[i][j], CHAINS == 2 ? add2(acc[0][i][j], acc[1][i][j]) : acc[0][i][j]);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
    const float row_gate = gate ? 1.0f / (1.0f + expf(-to_f32(gate[(size_t)gm * gate_ld + blockIdx.z]))) : 1.0f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= N) continue;
      TO* o = out + (size_t)gm * ldo + gn;
      float v = (i & 1 ? sum[i / 2][j].y : sum[i / 2][j].x) * row_gate;
      if (accumulate) v += to_f32(*o);
      *o = from_f32<TO>(v);
    }
  }
}

// ---------------------------------------------------------------- float32, rows in packets of 16 bytes
__device__ __forceinline__ void copy16_async(float* dst, const float* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = valid ? 16 : 0;           // 0: the sixteen bytes become zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void store_result(float* __restrict__ out, size_t at, float v, int accumulate) {
  out[at] = accumulate ? v + out[at] : v;
}

// Up to 32 rows (a decode step): bound by the weights' bytes.  A block owns 8 or 16 weight rows; its warps take the K range in
// turns of 256 values (8 chunks).  A lane owns one chunk of 32 values for a quarter of the weight rows and all MT token rows, so
// a chunk's sum is the same chain of FMAs as anywhere else; the chunk sums of a round of turns meet in shared memory, where a
// warp of its own adds them in order while the others are at the next round.  Weights and tokens come by cp.async into rows of 36 floats per chunk (a
// quarter warp reads 8 chunks' packets from 32 different banks); the first turn's weights are asked for before the wait
// on the predecessor (weights that a kernel of the step has written need an ordinary launch), and a warp asks for its next turn as soon as it has multiplied the last.  What a warp cannot do is
// multiply one turn while it waits for the next, so the blocks are small and many warps share an SM: 8 rows and four warps (three blocks an
// SM) against 16 rows and two warps 35 us and 47 (4 rows of 2,048 to 16,384 features), 16 rows and four warps from 9 rows on, where
// the tokens' share of the copies counts (16 rows: 87 us against 101).  The tile kernel with 32 x 16 tiles that stood here
// before read a K range of 32 between two barriers: 4 rows against the 16 layers and the head of the 1B shape 16.2 ms a step, here 1.6.
// From 17 rows on wide weights go to the tiles below (32 rows to 16,384 features: 229 us here, 152 there), narrow ones stay
// (to 2,048 features 49 us here, 62 there).
constexpr int kFewTurn = 8 * kSimtChunk, kFewLd = 8 * 36;
// floats of a chunk's sums: 8 behind every quarter of the rows, 1 behind a chunk, for the banks
__host__ __device__ constexpr int few_sums_ld(int mt, int rows) { return rows * mt + 33; }
constexpr size_t few_smem_bytes(int mt, int rows, int warps) {
  return sizeof(float) * ((size_t)warps * (rows + mt) * kFewLd + (size_t)2 * warps * 8 * few_sums_ld(mt, rows));
}

template <int MT, int ROWS, int WARPS>
__global__ void __launch_bounds__((WARPS + 1) * 32)
gemm_simt_few_kernel(float* __restrict__ out, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K, int lda,
                     int ldw, int ldo, int accumulate, long long batch_a, long long batch_w, long long batch_o,
                     const float* __restrict__ gate, int gate_ld) {
  extern __shared__ __align__(16) float few_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ws = few_smem + (size_t)warp * (ROWS + MT) * kFewLd;       // [ROWS][8 chunks][36]
  float* xs = ws + ROWS * kFewLd;                                    // [MT][8 chunks][36]
  float* sums = few_smem + (size_t)WARPS * (ROWS + MT) * kFewLd;    // [2][warp][8 chunks][4 groups][RL rows][MT]
  A += (size_t)blockIdx.z * batch_a;
  W += (size_t)blockIdx.z * batch_w;
  out += (size_t)blockIdx.z * batch_o;
  const int n0 = blockIdx.x * ROWS;
  const int turns = (K + kFewTurn - 1) / kFewTurn;

  // a row of a turn is 64 packets
  auto copy_rows = [&](float* dst, const float* src, int ld, int rows, int valid_rows, int k0) {
#pragma unroll 4
    for (int e = lane; e < rows * 64; e += 32) {
      const int r = e >> 6, p = e & 63, k = k0 + 4 * p;
      const bool ok = r < valid_rows && k < K;
      copy16_async(dst + r * kFewLd + (p >> 3) * 36 + (p & 7) * 4, ok ? src + (size_t)r * ld + k : src, ok);
    }
  };
  const float* w_rows = W + (size_t)n0 * ldw;
  const int valid_n = min(ROWS, N - n0);
  const bool works = warp < WARPS;                                       // the last warp adds up
  if (works && warp < turns) copy_rows(ws, w_rows, ldw, ROWS, valid_n, warp * kFewTurn);
  pdl_wait();
  pdl_launch_dependents();
  if (works && warp < turns) copy_rows(xs, A, lda, MT, M, warp * kFewTurn);
  copy_commit();

  const int chunk = lane & 7, group = lane >> 3;
  constexpr int RL = ROWS / 4;                                           // weight rows of a lane
  constexpr int SUMS_LD = few_sums_ld(MT, ROWS);
  constexpr int RESULTS = ROWS * MT, PER = (RESULTS + 31) / 32;          // of the last warp's lanes
  float sum[PER], comp[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) { sum[i] = 0.f; comp[i] = 0.f; }

  const int rounds = (turns + WARPS - 1) / WARPS;
  for (int round = 0; round <= rounds; ++round) {
    float* round_sums = sums + (size_t)(round & 1) * WARPS * 8 * SUMS_LD;
    const int turn = round * WARPS + warp;
    if (works && turn < turns) {
      copy_wait<0>();
      __syncwarp();
      float2 acc[RL][MT];
#pragma unroll
      for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[r][m] = make_float2(0.f, 0.f);
      const float* wp = ws + group * RL * kFewLd + chunk * 36;
      const float* xp = xs + chunk * 36;
#pragma unroll 2
      for (int k = 0; k < kSimtChunk; k += 4) {
        float4 w[RL];
#pragma unroll
        for (int r = 0; r < RL; ++r) w[r] = *reinterpret_cast<const float4*>(wp + r * kFewLd + k);
        constexpr int MS = MT < 4 ? MT : 4;                              // token rows at a time: their FMAs lie between two of one sum
#pragma unroll
        for (int m0 = 0; m0 < MT; m0 += MS) {
          float4 x[MS];
#pragma unroll
          for (int m = 0; m < MS; ++m) x[m] = *reinterpret_cast<const float4*>(xp + (m0 + m) * kFewLd + k);
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
      if (turn + WARPS < turns) {
        copy_rows(ws, w_rows, ldw, ROWS, valid_n, (turn + WARPS) * kFewTurn);
        copy_rows(xs, A, lda, MT, M, (turn + WARPS) * kFewTurn);
        copy_commit();
      }
      float* dst = round_sums + (warp * 8 + chunk) * SUMS_LD + group * (RL * MT + 8);
#pragma unroll
      for (int r = 0; r < RL; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) dst[r * MT + m] = __fadd_rn(acc[r][m].x, acc[r][m].y);
    }
    if (!works && round > 0) {                                           // the round before, while this one is multiplied
      const float* done = sums + (size_t)((round - 1) & 1) * WARPS * 8 * SUMS_LD;
      const int chunks = min(WARPS * 8, (K - (round - 1) * WARPS * kFewTurn + kSimtChunk - 1) / kSimtChunk);
#pragma unroll 4
      for (int c = 0; c < chunks; ++c)
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int at = min(lane + 32 * i, RESULTS - 1);
          kahan_add(sum[i], comp[i], done[c * SUMS_LD + at + at / (RL * MT) * 8]);
        }
    }
    __syncthreads();
  }
  if (works) return;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int at = lane + 32 * i;
    const int n = n0 + at / MT, m = at % MT;
    if (at >= RESULTS || n >= N || m >= M) continue;
    const float row_gate = gate ? 1.0f / (1.0f + expf(-gate[(size_t)m * gate_ld + blockIdx.z])) : 1.0f;
    store_result(out, (size_t)m * ldo + n, sum[i] * row_gate, accumulate);
  }
}

// More rows (prompts): bound by the FMAs.  128 threads, TM x TN results each (rows 8 apart, columns 16 apart) with sum, compensation
// and chunk accumulator in registers; a chunk of 32 k values per stage, rows kept along K as they come (cp.async, a ring of
// three stages) with 36 floats a row: a thread reads four k values of a row in one packet, and the eight rows of a quarter
// warp's packets start in different banks.  The products of two neighbouring k values are one packed instruction
// (pairs lie side by side in the packets as they are read), which leaves issue slots for the rest; 8 x 4 results, or fewer for weights
// of few rows, whose tiles leave SMs without work (simt_tile below).  320 rows to 16,384 features of 2,048: 551 us, 39 TFLOP/s, 596
// with scalar FMAs and 8 x 8 results; to 2,048 features 94 and 108.  Packed FMAs with three different operands, and
// nothing else, reach 59 TFLOP/s with 8 x 4 results.  Two halves of a block at neighbouring chunks: 635 us, though 46 in place of 57 where a tile per SM is all there is.
constexpr int kTileLd = kSimtChunk + 4, kTileStages = 3, kTileThreads = 128;

template <int TM, int TN>
__global__ void __launch_bounds__(kTileThreads, TM * TN >= 32 ? 3 : 4)
gemm_simt_tile_kernel(float* __restrict__ out, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K, int lda,
                      int ldw, int ldo, int accumulate, long long batch_a, long long batch_w, long long batch_o,
                      const float* __restrict__ gate, int gate_ld) {
  constexpr int BM = 8 * TM, BN = 16 * TN, ROWS = BM + BN;
  extern __shared__ __align__(16) float tile_smem[];                     // [stage][x BM rows | w BN rows][36]
  A += (size_t)blockIdx.z * batch_a;
  W += (size_t)blockIdx.z * batch_w;
  out += (size_t)blockIdx.z * batch_o;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;                  // the tiles of one set of weight rows run side by side
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int chunks = (K + kSimtChunk - 1) / kSimtChunk;
  pdl_wait();
  pdl_launch_dependents();
  auto fetch = [&](int c) {
    float* stage = tile_smem + (size_t)(c % kTileStages) * ROWS * kTileLd;
    const int p = tid & 7, k = c * kSimtChunk + 4 * p;
#pragma unroll
    for (int i = 0; i < (ROWS + 15) / 16; ++i) {
      const int r = (tid >> 3) + 16 * i;
      if (ROWS % 16 && r >= ROWS) break;
      const bool is_x = r < BM;
      const int row = is_x ? m0 + r : n0 + r - BM;
      const bool ok = k < K && row < (is_x ? M : N);
      const float* src = is_x ? A + (size_t)row * lda + k : W + (size_t)row * ldw + k;
      copy16_async(stage + r * kTileLd + 4 * p, ok ? src : A, ok);
    }
  };
  float2 sum[TM][TN / 2], comp[TM][TN / 2];             // of two columns each
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) sum[i][j] = comp[i][j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int c = 0; c < kTileStages - 1; ++c) {
    if (c < chunks) fetch(c);
    copy_commit();
  }
  for (int c = 0; c < chunks; ++c) {
    copy_wait<kTileStages - 2>();
    __syncthreads();
    if (c + kTileStages - 1 < chunks) fetch(c + kTileStages - 1);
    copy_commit();
    const float* xs = tile_smem + (size_t)(c % kTileStages) * ROWS * kTileLd + ty * kTileLd;
    const float* ws = tile_smem + ((size_t)(c % kTileStages) * ROWS + BM + tx) * kTileLd;
    float2 acc[TM][TN];                                                    // sums of even and of odd k
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll (TM * TN <= 16 ? 4 : 2)
    for (int k = 0; k < kSimtChunk; k += 4) {
      float4 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + 16 * j * kTileLd + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(xs + 8 * i * kTileLd + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma2(make_float2(x.x, x.y), make_float2(w[j].x, w[j].y), acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma2(make_float2(x.z, x.w), make_float2(w[j].z, w[j].w), acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j)
        kahan_add_pair(sum[i][j], comp[i][j],
                       make_float2(__fadd_rn(acc[i][2 * j].x, acc[i][2 * j].y), __fadd_rn(acc[i][2 * j + 1].x, acc[i][2 * j + 1].y)));
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + 8 * i;
    if (m >= M) continue;
    const float row_gate = gate ? 1.0f / (1.0f + expf(-gate[(size_t)m * gate_ld + blockIdx.z])) : 1.0f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n < N) store_result(out, (size_t)m * ldo + n, (j & 1 ? sum[i][j / 2].y : sum[i][j / 2].x) * row_gate, accumulate);
    }
  }
}

// Results per thread (10 TM + TN) of a product: the shape whose blocks the busiest SM is soonest done with, by what 1, 2, ...
// blocks of a shape take side by side on an SM, up to as many as it holds (`us`, for 2,048 k values on a B200; blocks share its
// FMA units, but one alone leaves them idle for its latencies).  Three of 5 x 4 stand for any number above two: the scheduler
// spreads fewer than four per SM unevenly, 416 blocks took 173 us, 444 138.  The times are those of scalar FMAs.  With packed ones even numbers of blocks take 85, 138 and
// 195 us (8 x 4), 60, 94, 133 and 171 (5 x 4), 51, 78, 109 and 141 (4 x 4): the same order but for two of 4 x 4, which a
// single one of 8 x 4 is still preferred to, 8 % slower.  Against the best of the three for 153 sizes of 33 to 2,048 rows, 512 to 16,384
// features and 1,024 to 8,192 k values: 0.9 % slower on average, 8.8 % at most.
inline int simt_tile(int M, int N, int batch) {
  constexpr struct { int tm, tn, held; float us[4]; } shapes[] = {
      {8, 4, 3, {88.f, 193.f, 203.f}}, {5, 4, 4, {64.f, 109.f, 170.f, 181.f}}, {4, 4, 4, {56.f, 98.f, 116.f, 152.f}}};
  const int sms = sm_count_of_device();
  int best = 84;
  float least = 0.f;
  for (const auto& s : shapes) {
    const long long blocks = (long long)batch * ((M + 8 * s.tm - 1) / (8 * s.tm)) * ((N + 16 * s.tn - 1) / (16 * s.tn));
    const long long busiest = (blocks + sms - 1) / sms;
    const float cost = (float)(busiest / s.held) * s.us[s.held - 1] + (busiest % s.held ? s.us[busiest % s.held - 1] : 0.f);
    if (least == 0.f || cost < least) { least = cost; best = 10 * s.tm + s.tn; }
  }
  return best;
}

template <typename TI, typename TO>
int gemm_simt(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldo,
              int accumulate, void* stream, int batch = 1, long long batch_a = 0, long long batch_w = 0, long long batch_o = 0,
              const void* gate_v = nullptr, int gate_ld = 0) {
  PTL_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
  PTL_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm_simt: pitches smaller than rows");
  PTL_REQUIRE(batch >= 1 && batch <= 65535, "gemm_simt: %d products in one launch", batch);
  if (M == 0) return 0;
  const TI* gate = (const TI*)gate_v;
  const int vec_ok = sizeof(TI) == 4 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && aligned16(A) && aligned16(W) &&
                     batch_a % 4 == 0 && batch_w % 4 == 0;
  if constexpr (sizeof(TI) == 4 && sizeof(TO) == 4) {
    if (vec_ok) {
      const auto few = [&](auto kernel, int mt, int rows, int warps, SmemRaised& raised) {
        const size_t smem = few_smem_bytes(mt, rows, warps);
        if (int rc = raise_shared_memory("gemm_simt_few", kernel, (int)smem, raised)) return rc;
        return launch_kernel("gemm_simt_few", kernel, dim3((N + rows - 1) / rows, 1, batch), dim3(warps * 32 + 32), smem,
                             as_stream(stream), (float*)out, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldo, accumulate,
                             batch_a, batch_w, batch_o, (const float*)gate_v, gate_ld);
      };
#define PTL_FEW(MT, ROWS, WARPS)                                                              \
      {                                                                                       \
        static SmemRaised raised;                                                             \
        return few(gemm_simt_few_kernel<MT, ROWS, WARPS>, MT, ROWS, WARPS, raised);           \
      }
      const bool narrow = (long long)N * batch < 4736;       // fewer than four blocks of eight rows per SM
      if (M <= 1) PTL_FEW(1, 8, 4)
      if (M <= 2) PTL_FEW(2, 8, 4)
      if (M <= 4) PTL_FEW(4, 8, 4)
      if (M <= 8 && narrow) PTL_FEW(8, 8, 4)
      if (M <= 8) PTL_FEW(8, 8, 3)
      if (M <= 16) PTL_FEW(16, 16, 4)
      if (M <= 32 && narrow) PTL_FEW(32, 8, 2)
#undef PTL_FEW
      // (weight rows are the grid's second dimension: more of them go to the tiles below, where they are its first)
      const bool tiles = N <= 16 * 4 * 65535;
      const auto tiled = [&](auto kernel, int tm, int tn, SmemRaised& raised) {
        const int smem = kTileStages * (8 * tm + 16 * tn) * kTileLd * (int)sizeof(float);
        if (int rc = raise_shared_memory("gemm_simt_tile", kernel, smem, raised)) return rc;
        const dim3 grid((M + 8 * tm - 1) / (8 * tm), (N + 16 * tn - 1) / (16 * tn), batch);
        return launch_kernel("gemm_simt_tile", kernel, grid, dim3(kTileThreads), smem, as_stream(stream), (float*)out, (const float*)A,
                             (const float*)W, M, N, K, lda, ldw, ldo, accumulate, batch_a, batch_w, batch_o, (const float*)gate_v, gate_ld);
      };
      static SmemRaised r84, r54, r44;
      switch (tiles ? simt_tile(M, N, batch) : 0) {
        case 84: return tiled(gemm_simt_tile_kernel<8, 4>, 8, 4, r84);
        case 54: return tiled(gemm_simt_tile_kernel<5, 4>, 5, 4, r54);
        case 44: return tiled(gemm_simt_tile_kernel<4, 4>, 4, 4, r44);
        default: break;
      }
    }
  }
  // narrow tiles: the rows the kernels above cannot read in packets of 16 bytes, and the library-free check of the
  // bfloat16 products
  const auto narrow_tiles = [&](auto kernel, int bm, int bn, int threads) {
    const dim3 grid((N + bn - 1) / bn, (M + bm - 1) / bm, batch);
    PTL_REQUIRE(grid.y <= 65535, "gemm_simt: M=%d too large", M);
    return launch_kernel("gemm_simt", kernel, grid, dim3(threads), 0, as_stream(stream), (TO*)out, (const TI*)A, (const TI*)W, M, N, K, lda, ldw,
                         ldo, accumulate, batch_a, batch_w, batch_o, gate, gate_ld);
  };
  if (sizeof(TI) == 4 && K % 4 == 0)
    return M > 32 ? narrow_tiles(gemm_simt_kernel<TI, TO, 64, 64, 4, 4, 2>, 64, 64, 256) : narrow_tiles(gemm_simt_kernel<TI, TO, 32, 16, 4, 1, 2>, 32, 16, 128);
  return M > 32 ? narrow_tiles(gemm_simt_kernel<TI, TO, 128, 64, 8, 4, 1>, 128, 64, 256) : narrow_tiles(gemm_simt_kernel<TI, TO, 32, 16, 4, 1, 1>, 32, 16, 128);
}

// The heads' products of a step with few tokens, 16-bit operands: a warp per output feature o of a head reads the weight
// row W[b, o, :] once, in packets of 16 bytes, against up to kHfTok token rows held as float32 in shared memory;
// float32 sums, each (token, feature) by the same chain whatever else the step holds: a lane adds its packets in order,
// the lanes meet in a butterfly.  K a multiple of 8, every row on a 16-byte boundary.
constexpr int kHfTok = 8, kHfWarps = 8;

template <typename T>
__global__ void __launch_bounds__(kHfWarps * 32)
head_linear_few_kernel(T* __restrict__ out, const T* __restrict__ A, const T* __restrict__ W, int M, int N, int K, int lda, int ldo,
                       int batch_a, int batch_o, const T* __restrict__ gate, int gate_ld) {
  extern __shared__ __align__(16) float hf_x[];          // [kHfTok][K]
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.y, m0 = blockIdx.z * kHfTok;
  const int nt = min(kHfTok, M - m0);
  const int packets = K / 8;
  for (int idx = threadIdx.x; idx < kHfTok * packets; idx += blockDim.x) {
    const int t = idx / packets, pk = idx % packets;
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (t < nt) {
      const uint4 raw = *reinterpret_cast<const uint4*>(A + (size_t)(m0 + t) * lda + (size_t)b * batch_a + 8 * pk);
      const T* v = reinterpret_cast<const T*>(&raw);
      lo = make_float4(to_f32(v[0]), to_f32(v[1]), to_f32(v[2]), to_f32(v[3]));
      hi = make_float4(to_f32(v[4]), to_f32(v[5]), to_f32(v[6]), to_f32(v[7]));
    }
    float4* dst = reinterpret_cast<float4*>(hf_x + (size_t)t * K + 8 * pk);
    dst[0] = lo;
    dst[1] = hi;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int o = blockIdx.x * kHfWarps + warp;
  if (o >= N) return;
  const T* wr = W + ((size_t)b * N + o) * K;
  float acc[kHfTok];
#pragma unroll
  for (int t = 0; t < kHfTok; ++t) acc[t] = 0.f;
  for (int i = lane * 8; i < K; i += 256) {
    const uint4 raw = *reinterpret_cast<const uint4*>(wr + i);
    const T* v = reinterpret_cast<const T*>(&raw);
    float w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e] = to_f32(v[e]);
#pragma unroll
    for (int t = 0; t < kHfTok; ++t) {
      const float4* xp = reinterpret_cast<const float4*>(hf_x + (size_t)t * K + i);
      const float4 x0 = xp[0], x1 = xp[1];
      float a = acc[t];
      a = fmaf(w[0], x0.x, a); a = fmaf(w[1], x0.y, a); a = fmaf(w[2], x0.z, a); a = fmaf(w[3], x0.w, a);
      a = fmaf(w[4], x1.x, a); a = fmaf(w[5], x1.y, a); a = fmaf(w[6], x1.z, a); a = fmaf(w[7], x1.w, a);
      acc[t] = a;
    }
  }
#pragma unroll
  for (int t = 0; t < kHfTok; ++t) {
    const float v = warp_sum(acc[t]);
    if (lane == t && t < nt) {
      const size_t m = (size_t)(m0 + t);
      const float g = gate ? 1.0f / (1.0f + expf(-to_f32(gate[m * gate_ld + b]))) : 1.0f;
      out[m * ldo + (size_t)b * batch_o + o] = from_f32<T>(v * g);
    }
  }
}

template <typename T>
int head_linear_few(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldo, int heads, int batch_a,
                    int batch_o, const void* gate, int gate_ld, void* stream) {
  PTL_REQUIRE(M >= 0 && N > 0 && K > 0 && heads >= 1 && heads <= 65535, "head_linear_few: bad sizes M=%d N=%d K=%d", M, N, K);
  PTL_REQUIRE(sizeof(T) == 2 && K % 8 == 0 && lda % 8 == 0 && batch_a % 8 == 0 && aligned16(A) && aligned16(W) &&
                  (size_t)kHfTok * K * sizeof(float) <= 48 * 1024,
              "head_linear_few: 16-bit rows of whole packets of 16 bytes on 16-byte boundaries, K=%d at most 1536", K);
  if (M == 0) return 0;
  const dim3 grid((N + kHfWarps - 1) / kHfWarps, heads, (M + kHfTok - 1) / kHfTok);
  PTL_REQUIRE(grid.z <= 65535, "head_linear_few: M=%d too large", M);
  return launch_kernel("head_linear_few", head_linear_few_kernel<T>, grid, dim3(kHfWarps * 32), (size_t)kHfTok * K * sizeof(float),
                       as_stream(stream), (T*)out, (const T*)A, (const T*)W, M, N, K, lda, ldo, batch_a, batch_o, (const T*)gate,
                       gate_ld);
}

}  // namespace ptl

// The tile shape that a float32 product of many rows takes, as 10 * rows + columns of a thread.
PTL_EXPORT int ptl_gemm_simt_tile(int M, int N, int batch) { return ptl::simt_tile(M, N, batch); }

PTL_EXPORT int ptl_gemm_simt_f32(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldo, int accumulate, void* stream) {
  return ptl::gemm_simt<float, float>(out, A, W, M, N, K, lda, ldw, ldo, accumulate, stream);
}
PTL_EXPORT int ptl_gemm_simt_bf16(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldo, int accumulate, void* stream) {
  return ptl::gemm_simt<__nv_bfloat16, __nv_bfloat16>(out, A, W, M, N, K, lda, ldw, ldo, accumulate, stream);
}
PTL_EXPORT int ptl_gemm_simt_bf16_f32out(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldw, int ldo, int accumulate, void* stream) {
  return ptl::gemm_simt<__nv_bfloat16, float>(out, A, W, M, N, K, lda, ldw, ldo, accumulate, stream);
}

// The heads of an activation against per-head weights: for b < heads,
//   out[m, b * batch_o + n] = sum_k A[m, b * batch_a + k] * W[b, n, k]   (times sigmoid(gate[m * gate_ld + b]) with a gate).
PTL_EXPORT int ptl_head_linear_f32(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldo, int heads,
                                   int batch_a, int batch_o, const void* gate, int gate_ld, void* stream) {
  return ptl::gemm_simt<float, float>(out, A, W, M, N, K, lda, K, ldo, 0, stream, heads, batch_a, (long long)N * K, batch_o, gate, gate_ld);
}
PTL_EXPORT int ptl_head_linear_bf16(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldo, int heads,
                                    int batch_a, int batch_o, const void* gate, int gate_ld, void* stream) {
  return ptl::gemm_simt<__nv_bfloat16, __nv_bfloat16>(out, A, W, M, N, K, lda, K, ldo, 0, stream, heads, batch_a, (long long)N * K,
                                                      batch_o, gate, gate_ld);
}
PTL_EXPORT int ptl_head_linear_few_bf16(void* out, const void* A, const void* W, int M, int N, int K, int lda, int ldo, int heads,
                                        int batch_a, int batch_o, const void* gate, int gate_ld, void* stream) {
  return ptl::head_linear_few<__nv_bfloat16>(out, A, W, M, N, K, lda, ldo, heads, batch_a, batch_o, gate, gate_ld, stream);
}
