// True 32-bit matrix product on the CUDA cores:  C[M,N] (+)= A[M,K] . W[N,K]^T.
//
// 32-bit fused multiply-adds only: no tensor cores, no TF32, no reduced-precision mode of any kind.  An output element is
// summed in one fixed order whatever M is and whichever kernel runs: k is cut into chunks of F32_CHUNK, a
// chunk is one chain of fused multiply-adds in ascending k from zero, and the chunks' sums are added in
// ascending order.  A row's result therefore does not depend on which other rows share the launch: a
// token gives the same bits in a prompt, alone, or in a batch.  The cut lets warps work on several chunks
// of one element at a time, and its error against 64 bits is smaller than that of one chain over K.  (The
// reference's all-float path is its CPU forward, src/dense.rs:94-102, one dot product per output row.)
//
// Weights are [N,K] row-major as in the reference (src/dense.rs:96).  With group_offsets the
// rows of A and C are grouped by expert: group e owns rows [off[e], off[e+1]) and the weight
// matrix W + e * w_group_stride.
#include "stream_common.cuh"

#define F32_CHUNK 128

// ---- up to 16 rows: the weights are streamed ---------------------------------------------------------
// A decode step's product is bound by reading W once.  A block owns 16 weight rows at a time; a warp owns
// two chunks of k of all 16 (a lane is one weight row in one chunk and holds the sums of every row of A), so
// eight warps cover 2,048 k per round, and after a round 16 x M threads add the round's 16 chunk sums to
// their element in order.  W and the same k of A come through a ring of cp.async stages per warp (32 k: 4 KB of
// W), which runs on across rounds and tiles; segments of 32 floats lie 36 apart, so the lanes' 16-byte loads
// of different rows meet no bank twice.  K = 2,048: 17.5 us for 2 rows x 11,264 (92 MB: 0.8 of the copy rate) where
// the tiles of 64 x 64 took 209; from 8 rows on the multiply-adds and the loads of A (one per row of A and 4 k) weigh in:
// 25 us for 8 rows, 45 for 16, against 54 for 16 rows in tiles.
#define F32S_SEG 36
#define F32S_ROWS 16
template <int MT> struct F32Stream {
  static constexpr int STAGE = (32 + 2 * MT) * F32S_SEG;          // floats of a warp's stage: W, then A
  static constexpr int STAGES = MT <= 4 ? 4 : (MT <= 8 ? 3 : 2);
  static constexpr int SMEM = (8 * STAGES * STAGE + 2 * 16 * MT * F32S_ROWS) * 4;
};

template <int MT>
__global__ void __launch_bounds__(256, 1)
gemm_f32_stream_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                       int M, int N, int K, int lda, int ldc, int accumulate, int tiles) {
  constexpr int STAGES = F32Stream<MT>::STAGES, STAGE = F32Stream<MT>::STAGE;
  extern __shared__ __align__(16) float smem[];
  float* part = smem + 8 * STAGES * STAGE;                         // [2][chunk of the round][row of A][weight row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* ring = smem + warp * STAGES * STAGE;
  const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
  const int chunks = (K + F32_CHUNK - 1) / F32_CHUNK, rounds = (chunks + 15) / 16;
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int steps = mine * rounds * 4;

  auto k_of = [&](int s, int half) { return ((((s >> 2) % rounds) * 16 + warp * 2 + half) * F32_CHUNK) + (s & 3) * 32; };
  auto issue_w = [&](int s) {
    const int n0 = (blockIdx.x + (s / (4 * rounds)) * gridDim.x) * F32S_ROWS;
    const uint32_t dst = ring_s + (s % STAGES) * STAGE * 4;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int p = lane + 32 * j, seg = p >> 3, k = k_of(s, seg >> 4) + (p & 7) * 4, n = n0 + (seg & 15);
      const bool in = n < N && k < K;
      st_cp16(dst + (seg * F32S_SEG + (p & 7) * 4) * 4, in ? W + (size_t)n * K + k : W, in ? 16 : 0);
    }
  };
  auto issue_a = [&](int s) {
    const uint32_t dst = ring_s + ((s % STAGES) * STAGE + 32 * F32S_SEG) * 4;
#pragma unroll
    for (int j = 0; j < (MT + 1) / 2; j++) {
      const int p = lane + 32 * j, seg = p >> 3, m = seg >> 1, k = k_of(s, seg & 1) + (p & 7) * 4;
      if (m >= MT) break;
      const bool in = m < M && k < K;
      st_cp16(dst + (seg * F32S_SEG + (p & 7) * 4) * 4, in ? A + (size_t)m * lda + k : A, in ? 16 : 0);
    }
  };

  for (int s = 0; s < STAGES - 1; s++)
    if (s < steps) issue_w(s);      // the weights do not depend on the kernel before this one
  pdl_wait();
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < steps) issue_a(s);
    st_commit();
  }
  float acc[MT], total = 0.f;
#pragma unroll
  for (int m = 0; m < MT; m++) acc[m] = 0.f;
  int buf = 0;
  for (int s = 0; s < steps; s++) {
    const int ahead = s + STAGES - 1;
    if (ahead < steps) {
      issue_w(ahead);
      issue_a(ahead);
    }
    st_commit();
    st_wait<STAGES - 1>();
    __syncwarp();
    const float* w = ring + (s % STAGES) * STAGE + lane * F32S_SEG;
    const float* a = ring + (s % STAGES) * STAGE + (32 + (lane >> 4)) * F32S_SEG;
#pragma unroll
    for (int kk = 0; kk < 8; kk++) {
      const float4 wv = load4(w + kk * 4);
#pragma unroll
      for (int m = 0; m < MT; m++) {
        const float4 av = load4(a + m * 2 * F32S_SEG + kk * 4);
        acc[m] = fmaf(av.x, wv.x, acc[m]);
        acc[m] = fmaf(av.y, wv.y, acc[m]);
        acc[m] = fmaf(av.z, wv.z, acc[m]);
        acc[m] = fmaf(av.w, wv.w, acc[m]);
      }
    }
    __syncwarp();
    if ((s & 3) == 3) {
      const int round = (s >> 2) % rounds;
      float* p = part + buf * 16 * MT * F32S_ROWS;
#pragma unroll
      for (int m = 0; m < MT; m++) {
        p[((warp * 2 + (lane >> 4)) * MT + m) * F32S_ROWS + (lane & 15)] = acc[m];
        acc[m] = 0.f;
      }
      __syncthreads();
      // the sums of a round are read before the barrier of the next, and written over after it
      if (tid < F32S_ROWS * MT) {
        const int m = tid >> 4, r = tid & 15, c1 = min(16, chunks - round * 16);
        for (int c = 0; c < c1; c++) total += p[(c * MT + m) * F32S_ROWS + r];
        if (round == rounds - 1) {
          const int n = (blockIdx.x + (s / (4 * rounds)) * gridDim.x) * F32S_ROWS + r;
          if (m < M && n < N) {
            float* c = C + (size_t)m * ldc + n;
            *c = accumulate ? *c + total : total;
          }
          total = 0.f;
        }
      }
      buf ^= 1;
    }
  }
}

// ---- a few dozen rows: small tiles over many chunks ---------------------------------------------------------
// 256 threads; a block's tile is BM x BN, and its eight warps are WM x WN x WK: WM x WN parts of the tile, and WK chunks
// of k at a time (a small tile over eight chunks gives a few dozen rows as many blocks as a stream of the weights has).  A
// lane of a warp's 8 x 4 holds TM x TN sums, rows 8 apart and columns side by side.  Both operands lie in shared memory as
// rows of 32 k at a pitch of 36 floats, where the 16-byte loads of eight lanes meet no bank twice, and come through a ring of
// cp.async stages that runs on across chunks and tiles, so only a block's first loads are waited for.
template <int BM, int BN, int WK>
struct F32Tile {
  static constexpr int ROWS = WK * (BM + BN);                       // rows of 32 k in a stage
  static constexpr int STAGE = ROWS * F32S_SEG;
  static constexpr int PART = WK * BM * (BN + 4);                   // chunk sums on their way to being added up
  static constexpr int STAGES = (3 * STAGE + PART) * 4 <= 220 * 1024 ? 3 : 2;
  static constexpr int SMEM = (STAGES * STAGE + PART) * 4;
};

__device__ __forceinline__ void f32_cp4(uint32_t dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}

template <int BM, int BN, int WM, int WN, int WK, bool VEC>
__global__ void __launch_bounds__(32 * WM * WN * WK, 1)
gemm_f32_tile_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                     int M, int N, int K, int lda, int ldc, int accumulate,
                     const int* __restrict__ group_offsets, size_t w_group_stride) {
  using T = F32Tile<BM, BN, WK>;
  constexpr int TM = BM / WM / 8, TN = BN / WN / 4, STAGES = T::STAGES, THREADS = 32 * WM * WN * WK;
  constexpr int SUMS = BM * BN / THREADS;
  static_assert(TN % 4 == 0 && BM * BN % THREADS == 0 && T::ROWS * 8 % THREADS == 0, "whole vectors and equal shares");
  extern __shared__ __align__(16) float smem[];
  float* part = smem + STAGES * T::STAGE;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane & 7, ln = lane >> 3;
  const int wk = warp % WK, wn = warp / WK % WN, wm = warp / (WK * WN);
  pdl_wait();
  int row_begin = 0, row_end = M;
  if (group_offsets) {
    row_begin = group_offsets[blockIdx.z];
    row_end = group_offsets[blockIdx.z + 1];
    W += (size_t)blockIdx.z * w_group_stride;
  }
  // tiles in order of their rows first, so that blocks that run together share their weights
  const int tiles_m = (row_end - row_begin + BM - 1) / BM, tiles = tiles_m * ((N + BN - 1) / BN);
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int chunks = (K + F32_CHUNK - 1) / F32_CHUNK, rounds = (chunks + WK - 1) / WK;
  const int steps = mine * rounds * 4;      // stages of 32 k: four to a chunk

  auto issue = [&](int s) {
    const int tile = blockIdx.x + (s / (4 * rounds)) * gridDim.x;
    const int m0 = row_begin + tile % tiles_m * BM, n0 = tile / tiles_m * BN;
    const uint32_t dst = ring + (s % STAGES) * T::STAGE * 4;
    const int k0 = ((s >> 2) % rounds) * WK * F32_CHUNK + (s & 3) * 32;
#pragma unroll
    for (int j = 0; j < T::ROWS * 8 / THREADS; j++) {
      const int p = tid + THREADS * j, row = p >> 3, c = row / (BM + BN), r = row % (BM + BN);
      const int k = k0 + c * F32_CHUNK + (p & 7) * 4;
      const int g = r < BM ? m0 + r : n0 + r - BM;
      const bool in = g < (r < BM ? row_end : N);
      const float* src = r < BM ? A + (size_t)g * lda : W + (size_t)g * K;
      const uint32_t d = dst + (row * F32S_SEG + (p & 7) * 4) * 4;
      if (VEC) {
        st_cp16(d, in && k < K ? src + k : W, in && k < K ? 16 : 0);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++) f32_cp4(d + e * 4, in && k + e < K ? src + k + e : W, in && k + e < K);
      }
    }
  };

  for (int s = 0; s < STAGES - 1; s++) {
    if (s < steps) issue(s);
    st_commit();
  }
  float acc[TM][TN], sum[SUMS];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.f;
#pragma unroll
  for (int i = 0; i < SUMS; i++) sum[i] = 0.f;
  for (int s = 0; s < steps; s++) {
    st_wait<STAGES - 2>();
    __syncthreads();      // stage s has arrived for everyone, and everyone is done with the one before it
    if (s + STAGES - 1 < steps) issue(s + STAGES - 1);
    st_commit();
    const float* a = smem + (s % STAGES) * T::STAGE + (wk * (BM + BN) + wm * (BM / WM) + lm) * F32S_SEG;
    const float* w = smem + (s % STAGES) * T::STAGE + (wk * (BM + BN) + BM + wn * (BN / WN) + ln * TN) * F32S_SEG;
#pragma unroll
    for (int kk = 0; kk < 32; kk += 4) {
      float4 av[TM];
#pragma unroll
      for (int i = 0; i < TM; i++) av[i] = load4(a + i * 8 * F32S_SEG + kk);
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const float4 wv = load4(w + j * F32S_SEG + kk);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(av[i].x, wv.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(av[i].y, wv.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(av[i].z, wv.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; i++) acc[i][j] = fmaf(av[i].w, wv.w, acc[i][j]);
      }
    }
    if ((s & 3) != 3) continue;
    // WK chunks are done
    const int round = (s >> 2) % rounds, tile = blockIdx.x + (s / (4 * rounds)) * gridDim.x;
    const int m0 = row_begin + tile % tiles_m * BM, n0 = tile / tiles_m * BN;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        store4(part + (wk * BM + wm * (BM / WM) + lm + 8 * i) * (BN + 4) + wn * (BN / WN) + ln * TN + j,
               make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]));
        acc[i][j] = acc[i][j + 1] = acc[i][j + 2] = acc[i][j + 3] = 0.f;
      }
    __syncthreads();      // the next write to `part` comes after the barriers of the stages between
    const int c1 = min(WK, chunks - round * WK);
#pragma unroll
    for (int i = 0; i < SUMS; i++) {
      const int e = tid + THREADS * i, m = e / BN, n = e % BN;
      for (int c = 0; c < c1; c++) sum[i] += part[(c * BM + m) * (BN + 4) + n];
      if (round == rounds - 1) {
        if (m0 + m < row_end && n0 + n < N) {
          float* c = C + (size_t)(m0 + m) * ldc + n0 + n;
          *c = accumulate ? *c + sum[i] : sum[i];
        }
        sum[i] = 0.f;
      }
    }
  }
}

// ---- more rows: tiles of pairs --------------------------------------------------------------------------
// 256 threads, a tile of BM x BN, warps dealt as above (WK 1 for many rows; 4 chunks of k at a time where larger tiles would leave SMs
// idle); a lane holds 8 x 8 sums.  Bound by the FMA pipes and what is issued beside them.  Single multiply-adds read three
// registers an instruction, which the register ports do not bear at full rate (37 TFLOP/s of the pipes' 72 with 8 x 8 sums);
// fma.rn.f32x2 does two an instruction and leaves every second issue slot to the loads.  Each half rounds like fmaf and goes
// through its k in the same order, so the bits are the same.  A pair holds two rows of one k, side by side: rows (m, m + 1) times
// columns (n, n + 1) make one pair product as they lie and one with the columns changed over, two moves for eight sums.  So
// operands lie in shared memory by k, rows side by side, and must be turned on their way there: a thread takes 4 k of a row to
// registers a stage ahead and stores them under four k.  (Turned by 4-byte cp.async instead, the copies took a third of
// the time: 2.49 ms for 2,048 x 11,264 x 2,048, and 1.75 with them left out.)  Rows are XORed by their k / 4, so those stores meet
// no bank twice; lanes of one row and of one column alternate, so a 16-byte load takes two passes over the banks and not
// three or four; stores and loads are spread over the stage's products.  2,048 rows x 11,264 x 2,048: 2,530 -> 2,110 us
// (45 TFLOP/s); 523 x 11,264 x 2,048 761 -> 635, x 6,144 480 -> 389; 523 x 2,048 x 5,632 437 -> 355; 1,000 x 1,000 x 1,000 86.5 -> 73.8.
template <int BM, int BN, int WK>
struct F32Pairs {
  static constexpr int PITCH = BM + BN;                             // floats of one k: the tile's rows of A, then of W
  static constexpr int STAGE = WK * 32 * PITCH;
  static constexpr int PART = WK > 1 ? WK * BM * (BN + 4) : 0;
  static constexpr int SMEM = (2 * STAGE + PART) * 4;
};

typedef unsigned long long f32pair;
__device__ __forceinline__ f32pair f32_fma2(f32pair a, f32pair b, f32pair c) {
  f32pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float f32_lo(f32pair p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float f32_hi(f32pair p) { return __uint_as_float((unsigned)(p >> 32)); }
__device__ __forceinline__ f32pair f32_pair(float lo, float hi) {
  return (f32pair)__float_as_uint(hi) << 32 | __float_as_uint(lo);
}

template <int BM, int BN, int WM, int WN, int WK, bool VEC>
__global__ void __launch_bounds__(32 * WM * WN * WK, 1)
gemm_f32_pairs_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                      int M, int N, int K, int lda, int ldc, int accumulate,
                      const int* __restrict__ group_offsets, size_t w_group_stride) {
  using T = F32Pairs<BM, BN, WK>;
  constexpr int PITCH = T::PITCH, THREADS = 32 * WM * WN * WK, LOADS = WK * PITCH / 32;
  constexpr int SUMS = WK > 1 ? BM * BN / THREADS : 1;
  static_assert(BM == WM * 64 && BN == WN * 32 && THREADS == 256 && BM % 32 == 0, "8 x 8 sums a lane, 8 warps");
  extern __shared__ __align__(16) float smem[];
  float* part = smem + 2 * T::STAGE;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lm = (lane >> 1) & 7, ln = (lane & 1) | (lane >> 4) << 1;
  const int wk = warp % WK, wn = warp / WK % WN, wm = warp / (WK * WN);
  pdl_wait();
  int row_begin = 0, row_end = M;
  if (group_offsets) {
    row_begin = group_offsets[blockIdx.z];
    row_end = group_offsets[blockIdx.z + 1];
    W += (size_t)blockIdx.z * w_group_stride;
  }
  // tiles in order of their rows first, so that blocks that run together share their weights
  const int tiles_m = (row_end - row_begin + BM - 1) / BM, tiles = tiles_m * ((N + BN - 1) / BN);
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int chunks = (K + F32_CHUNK - 1) / F32_CHUNK, rounds = (chunks + WK - 1) / WK;
  const int steps = mine * rounds * 4;      // stages of 32 k: four to a chunk
  if (steps <= 0) return;                   // a group without rows

  // a thread brings 4 k of every 32nd row of the stage's operands
  const int cv = lane & 7, cr = warp * 4 + (lane >> 3);
  float4 held[LOADS];
  struct From {
    const float *a, *w;
    int rows, cols, ks;      // how many rows of A, rows of W and k lie from this thread's first ones on
  };
  auto from = [&](int s) {
    const int tile = blockIdx.x + (s / (4 * rounds)) * gridDim.x;
    const int m0 = row_begin + tile % tiles_m * BM + cr, n0 = tile / tiles_m * BN + cr;
    const int k0 = ((s >> 2) % rounds) * WK * F32_CHUNK + (s & 3) * 32 + cv * 4;
    return From{A + (size_t)m0 * lda + k0, W + (size_t)n0 * K + k0, row_end - m0, N - n0, s < steps ? K - k0 : 0};
  };
  auto fetch = [&](const From& f, int l) {
    const int c = l / (PITCH / 32), r = l % (PITCH / 32) * 32, k = f.ks - c * F32_CHUNK;
    const bool in = r < BM ? r < f.rows : r - BM < f.cols;
    const float* src = (r < BM ? f.a + (size_t)r * lda : f.w + (size_t)(r - BM) * K) + c * F32_CHUNK;
    held[l] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC) {
      if (in && k > 0) held[l] = load4(src);
    } else {
      if (in && k > 0) held[l].x = src[0];
      if (in && k > 1) held[l].y = src[1];
      if (in && k > 2) held[l].z = src[2];
      if (in && k > 3) held[l].w = src[3];
    }
  };
  auto put = [&](int s, int l) {
    float* p = smem + (s & 1) * T::STAGE + (l / (PITCH / 32) * 32 + cv * 4) * PITCH + l % (PITCH / 32) * 32 + (cr ^ cv * 4);
    p[0] = held[l].x;
    p[PITCH] = held[l].y;
    p[2 * PITCH] = held[l].z;
    p[3 * PITCH] = held[l].w;
  };
  From next = from(0);
#pragma unroll
  for (int l = 0; l < LOADS; l++) fetch(next, l);
#pragma unroll
  for (int l = 0; l < LOADS; l++) put(0, l);
  next = from(1);
#pragma unroll
  for (int l = 0; l < LOADS; l++) fetch(next, l);
  // of rows (m, m + 1) and columns (n, n + 1): `same` holds (m, n) and (m + 1, n + 1), `cross` (m, n + 1) and (m + 1, n)
  f32pair same[4][4], cross[4][4];
  float total[WK > 1 ? 1 : 8][WK > 1 ? 1 : 8], sum[SUMS];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) same[i][j] = cross[i][j] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) total[WK > 1 ? 0 : i][WK > 1 ? 0 : j] = 0.f;
#pragma unroll
  for (int i = 0; i < SUMS; i++) sum[i] = 0.f;
  auto value = [&](int i, int j) {
    const f32pair p = (i ^ j) & 1 ? cross[i >> 1][j >> 1] : same[i >> 1][j >> 1];
    return i & 1 ? f32_hi(p) : f32_lo(p);
  };
  for (int s = 0; s < steps; s++) {
    __syncthreads();      // stage s is there, and everyone is done with the one before it
    next = from(s + 2);
    const float* a = smem + (s & 1) * T::STAGE + wk * 32 * PITCH + wm * 64;
    const float* w = smem + (s & 1) * T::STAGE + wk * 32 * PITCH + BM + wn * 32;
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const int am = (lm ^ v) * 4, w0n = (ln ^ v) * 4, w1n = w0n ^ 16;
#pragma unroll
      for (int k = v * 4; k < v * 4 + 4; k++) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(a + k * PITCH + am), a1 = *reinterpret_cast<const ulonglong2*>(a + k * PITCH + am + 32);
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(w + k * PITCH + w0n), w1 = *reinterpret_cast<const ulonglong2*>(w + k * PITCH + w1n);
        const f32pair av[4] = {a0.x, a0.y, a1.x, a1.y}, wv[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const f32pair wx = f32_pair(f32_hi(wv[j]), f32_lo(wv[j]));
#pragma unroll
          for (int i = 0; i < 4; i++) same[i][j] = f32_fma2(av[i], wv[j], same[i][j]);
#pragma unroll
          for (int i = 0; i < 4; i++) cross[i][j] = f32_fma2(av[i], wx, cross[i][j]);
        }
      }
      // a share of the next stage, and of the loads for the one after it (zeros past the last)
#pragma unroll
      for (int l = v * LOADS / 8; l < (v + 1) * LOADS / 8; l++) {
        put(s + 1, l);
        fetch(next, l);
      }
    }
    if ((s & 3) != 3) continue;
    // a chunk (or WK of them) is done
    const int round = (s >> 2) % rounds, tile = blockIdx.x + (s / (4 * rounds)) * gridDim.x;
    const int m0 = row_begin + tile % tiles_m * BM, n0 = tile / tiles_m * BN;
    if (WK == 1) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) total[WK > 1 ? 0 : i][WK > 1 ? 0 : j] += value(i, j);
      if (round == rounds - 1) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int r = m0 + wm * 64 + lm * 4 + (i & 3) + 32 * (i >> 2);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int n = n0 + wn * 32 + ln * 4 + (j & 3) + 16 * (j >> 2);
            float& t = total[WK > 1 ? 0 : i][WK > 1 ? 0 : j];
            if (r < row_end && n < N) {
              float* c = C + (size_t)r * ldc + n;
              *c = accumulate ? *c + t : t;
            }
            t = 0.f;
          }
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j += 4)
          store4(part + (wk * BM + wm * 64 + lm * 4 + (i & 3) + 32 * (i >> 2)) * (BN + 4) + wn * 32 + ln * 4 + 16 * (j >> 2),
                 make_float4(value(i, j), value(i, j + 1), value(i, j + 2), value(i, j + 3)));
      __syncthreads();      // the next write to `part` comes after the barriers of the stages between
      const int c1 = min(WK, chunks - round * WK);
#pragma unroll
      for (int i = 0; i < SUMS; i++) {
        const int e = tid + THREADS * i, m = e / BN, n = e % BN;
        for (int c = 0; c < c1; c++) sum[i] += part[(c * BM + m) * (BN + 4) + n];
        if (round == rounds - 1) {
          if (m0 + m < row_end && n0 + n < N) {
            float* c = C + (size_t)(m0 + m) * ldc + n0 + n;
            *c = accumulate ? *c + sum[i] : sum[i];
          }
          sum[i] = 0.f;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) same[i][j] = cross[i][j] = 0;
  }
}

// ---- few k, and operands without whole 16-byte vectors: blocks by the SM --------------------------------
// A block of 256 threads computes 64 x 64 outputs, 4 x 4 a thread, from 16 k at a time that single loads bring to shared memory.
// Nothing overlaps inside a block; four or five of them share an SM and overlap each other.  It takes any alignment, a
// stage is 16 k, and a block costs nothing where it has no rows: where K is a chunk or three it is ahead of the
// tiles above, whose warps share out chunks that are not there (300 rows x 2,048 x 128: 15 us, 59 in tiles of 64 x 64 over four
// chunks; 64 experts of one row, 512 x 512: 87 and 121), and of their 4-byte copies where vectors are broken (300 x 771 x 301:
// 20 and 33 us).  CHUNKS: K is more than one chunk (the sums over chunks take 16 registers, and one of five blocks).  Launched
// plainly: with the programmatic attribute its blocks came to the SMs unevenly (1,100 x 1,024 x 1,024: 103 and 160 us).
#define F32_BM 64
#define F32_BN 64
#define F32_BK 16
template <bool CHUNKS>
__global__ void __launch_bounds__(256)
gemm_f32_plain_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W,
                      int M, int N, int K, int lda, int ldc, int accumulate,
                      const int* __restrict__ group_offsets, size_t w_group_stride) {
  __shared__ float As[F32_BK][F32_BM + 4];
  __shared__ float Ws[F32_BK][F32_BN + 4];
  int row_begin = 0, row_end = M;
  if (group_offsets) {
    row_begin = group_offsets[blockIdx.z];
    row_end = group_offsets[blockIdx.z + 1];
    W += (size_t)blockIdx.z * w_group_stride;
  }
  const int m0 = row_begin + blockIdx.y * F32_BM;
  if (m0 >= row_end) return;
  const int n0 = blockIdx.x * F32_BN;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;  // loader: row of the tile, first of 4 k
  float acc[4][4], total[CHUNKS ? 4 : 1][CHUNKS ? 4 : 1];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = total[CHUNKS ? i : 0][CHUNKS ? j : 0] = 0.f;
  for (int k0 = 0; k0 < K; k0 += F32_BK) {
    {
      const int r = m0 + lrow;
      const float* src = A + (size_t)r * lda + k0 + lk;
#pragma unroll
      for (int e = 0; e < 4; e++) As[lk + e][lrow] = (r < row_end && k0 + lk + e < K) ? src[e] : 0.f;
      const int n = n0 + lrow;
      const float* wsrc = W + (size_t)n * K + k0 + lk;
#pragma unroll
      for (int e = 0; e < 4; e++) Ws[lk + e][lrow] = (n < N && k0 + lk + e < K) ? wsrc[e] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < F32_BK; kk++) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; j++) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
    if (CHUNKS && (k0 + F32_BK) % F32_CHUNK == 0) {      // a chunk is done
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          total[CHUNKS ? i : 0][CHUNKS ? j : 0] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = m0 + ty * 4 + i;
    if (r >= row_end) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float* c = C + (size_t)r * ldc + n;
      const float sum = (CHUNKS ? total[CHUNKS ? i : 0][CHUNKS ? j : 0] : 0.f) + acc[i][j];
      *c = accumulate ? *c + sum : sum;
    }
  }
}

template <int MT>
static int launch_f32_stream(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldc,
                             int accumulate, cudaStream_t st) {
  constexpr int smem = F32Stream<MT>::SMEM;
  const cudaError_t set = leb_allow_smem<gemm_f32_stream_kernel<MT>>();
  LEB_REQUIRE(set == cudaSuccess, "leb_gemm_f32: %s", cudaGetErrorString(set));
  const int tiles = ceil_div(N, F32S_ROWS), sms = sm_count();
  const int blocks = ceil_div(tiles, ceil_div(tiles, sms));        // as many tiles for every block
  leb_launch(gemm_f32_stream_kernel<MT>, dim3(blocks), dim3(256), smem, st, C, A, W, M, N, K, lda, ldc, accumulate, tiles);
  LEB_CHECK_LAUNCH("leb_gemm_f32");
  return 0;
}

template <int BM, int BN, int WM, int WN, int WK, bool VEC>
static int launch_f32_tile(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldc, int accumulate,
                           const int* group_offsets, int groups, size_t w_group_stride, cudaStream_t st) {
  constexpr int smem = F32Tile<BM, BN, WK>::SMEM;
  constexpr auto kernel = gemm_f32_tile_kernel<BM, BN, WM, WN, WK, VEC>;
  const cudaError_t set = leb_allow_smem<kernel>();
  LEB_REQUIRE(set == cudaSuccess, "leb_gemm_f32: %s", cudaGetErrorString(set));
  const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, BN);
  LEB_REQUIRE(tiles < (1ll << 24) && groups <= 65535, "leb_gemm_f32: too many tiles (%lld) or groups (%d)", tiles, groups);
  const int sms = sm_count(), blocks = ceil_div((int)tiles, ceil_div((int)tiles, sms));
  leb_launch(kernel, dim3(blocks, 1, groups), dim3(32 * WM * WN * WK), smem, st, C, A, W, M, N, K, lda, ldc, accumulate, group_offsets,
             w_group_stride);
  LEB_CHECK_LAUNCH("leb_gemm_f32");
  return 0;
}

template <int BM, int BN, int WM, int WN, int WK, bool VEC>
static int launch_f32_pairs(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldc, int accumulate,
                           const int* group_offsets, int groups, size_t w_group_stride, cudaStream_t st) {
  constexpr int smem = F32Pairs<BM, BN, WK>::SMEM;
  constexpr auto kernel = gemm_f32_pairs_kernel<BM, BN, WM, WN, WK, VEC>;
  const cudaError_t set = leb_allow_smem<kernel>();
  LEB_REQUIRE(set == cudaSuccess, "leb_gemm_f32: %s", cudaGetErrorString(set));
  const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, BN);
  LEB_REQUIRE(tiles < (1ll << 24) && groups <= 65535, "leb_gemm_f32: too many tiles (%lld) or groups (%d)", tiles, groups);
  const int sms = sm_count(), blocks = ceil_div((int)tiles, ceil_div((int)tiles, sms));
  leb_launch(kernel, dim3(blocks, 1, groups), dim3(32 * WM * WN * WK), smem, st, C, A, W, M, N, K, lda, ldc, accumulate, group_offsets,
             w_group_stride);
  LEB_CHECK_LAUNCH("leb_gemm_f32");
  return 0;
}

// Which kernel takes a product (0-4: tiles in the order below, F32_PLAIN, F32_STREAM): the one whose blocks take the SM with most of
// them least, in nanoseconds measured on B200 (9 to 2,048 rows, 16 to 11,264 columns, K from 16 to 2,048; 4 to 64 groups): a
// fixed part, and per block of an SM a part of its own and one per round, of `wk` chunks of k (the plain kernel: of 16 k).  Over 967
// such sizes the choice takes 0.46 (up to 16 rows), 0.62 (more; 0.83 with broken vectors) and 0.56 (groups) of the time of blocks of
// 64 x 64 throughout, and above 1.1 of it at ten small sizes (by 0.3 to 2.4 us); the two larger tiles' figures were taken
// again when they came to hold pairs (150 sizes of 17 to 2,048 rows: 0.91 of the time before).  Groups count as many equally large ones as can
// have rows; blocks of groups without any cost their start.
enum { F32_PLAIN = 5, F32_STREAM = 6 };
struct F32Cost {
  int bm, bn, wk, fixed, block, round;
};
static int f32_choice(int M, int N, int K, int groups, bool vec, int sms) {      // groups: 0 for a product that is not grouped
  static const F32Cost whole[5] = {{128, 128, 1, 0, 8800, 12200}, {64, 64, 4, 6000, 600, 15800}, {32, 32, 8, 1350, 0, 12200},
                                   {64, 16, 8, 1400, 0, 12550}, {32, 16, 8, 1500, 0, 7600}};
  static const F32Cost broken[5] = {{128, 128, 1, 0, 4200, 17100}, {64, 64, 4, 0, 1550, 18500}, {32, 32, 8, 1500, 1700, 13400},
                                    {64, 16, 8, 1100, 1900, 14500}, {32, 16, 8, 1500, 2400, 7700}};
  if (groups == 0 && M <= 8 && vec) return F32_STREAM;      // (measured up to 16 rows; up to 8 it is ahead or within 0.4 us everywhere)
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long live = groups > M ? M : groups < 1 ? 1 : groups, rows = up(M, live), chunks = up(K, F32_CHUNK);
  auto per_sm = [&](int bm, int bn) { return up(live * up(rows, bm) * up(N, bn), sms); };
  auto idle = [&](long long blocks, long long busy) { const long long n = up(blocks, sms) - busy; return n > 0 ? n : 0; };
  int pick = F32_PLAIN;
  const long long steps = up(K, F32_BK), per = per_sm(F32_BM, F32_BN), m_tiles = up(M, F32_BM);
  const long long apart = per * (vec ? 230 + 870 * steps : 230 + 775 * steps), alone = up(per, 4) * steps * (vec ? 970 : 890);
  long long best = (vec ? 1850 : 2100) + (apart > alone ? apart : alone) + 370 * idle(m_tiles * up(N, F32_BN) * (groups > 1 ? groups : 1), per);
  if (groups > 1 && rows > F32_BM) best = best * 14 / 10;      // live blocks come to an SM in clusters
  if (m_tiles > 65535) best = 1ll << 60;
  const F32Cost* cost = vec ? whole : broken;
  for (int i = 0; i < 5; i++) {
    if (groups > 1 && (i == 0 || i == 3)) continue;
    const F32Cost& c = cost[i];
    const long long n = per_sm(c.bm, c.bn), all = up(M, c.bm) * up(N, c.bn), blocks = up(all, up(all, sms)) * (groups > 1 ? groups : 1);
    const long long t = c.fixed + n * (c.block + c.round * up(chunks, c.wk)) + 600 * idle(blocks, n);
    if (t < best) best = t, pick = i;
  }
  if (vec && groups == 0 && M <= 16 && 1000 + up(up(N, F32S_ROWS), sms) * 8300 * up(chunks, 16) <= best) pick = F32_STREAM;
  return pick;
}
LEB_API int leb_gemm_f32_choice(int M, int N, int K, int groups, int vec, int sms) {
  return M > 0 && N > 0 && K > 0 && sms > 0 ? f32_choice(M, N, K, groups, vec != 0, sms) : -1;
}

LEB_API int leb_gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda,
                         int ldc, int accumulate, const int* group_offsets, int n_groups,
                         size_t w_group_stride, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  LEB_REQUIRE(K > 0, "leb_gemm_f32: K must be positive");
  // 16-byte loads: rows of both operands begin on 16 bytes and hold whole vectors
  const bool vec = K % 4 == 0 && lda % 4 == 0 && w_group_stride % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
  const int groups = group_offsets ? n_groups : 1;
  const int pick = f32_choice(M, N, K, group_offsets ? (n_groups > 0 ? n_groups : 1) : 0, vec, sm_count());
  if (pick == F32_STREAM) {
    if (M == 1) return launch_f32_stream<1>(C, A, W, M, N, K, lda, ldc, accumulate, st);
    if (M == 2) return launch_f32_stream<2>(C, A, W, M, N, K, lda, ldc, accumulate, st);
    if (M <= 4) return launch_f32_stream<4>(C, A, W, M, N, K, lda, ldc, accumulate, st);
    if (M <= 8) return launch_f32_stream<8>(C, A, W, M, N, K, lda, ldc, accumulate, st);
    return launch_f32_stream<16>(C, A, W, M, N, K, lda, ldc, accumulate, st);
  }
  if (pick == F32_PLAIN) {
    const dim3 grid(ceil_div(N, F32_BN), ceil_div(M, F32_BM), groups);
    LEB_REQUIRE(groups <= 65535, "leb_gemm_f32: too many groups (%d)", groups);
    (K > F32_CHUNK ? gemm_f32_plain_kernel<true> : gemm_f32_plain_kernel<false>)<<<grid, 256, 0, st>>>(
        C, A, W, M, N, K, lda, ldc, accumulate, group_offsets, w_group_stride);
    LEB_CHECK_LAUNCH("leb_gemm_f32");
    return 0;
  }
#define LEB_F32_TILE(KIND, BM, BN, WM, WN, WK)                                                                                \
  return vec ? launch_f32_##KIND<BM, BN, WM, WN, WK, true>(C, A, W, M, N, K, lda, ldc, accumulate, group_offsets, groups, w_group_stride, st) \
             : launch_f32_##KIND<BM, BN, WM, WN, WK, false>(C, A, W, M, N, K, lda, ldc, accumulate, group_offsets, groups, w_group_stride, st)
  if (pick == 0) LEB_F32_TILE(pairs, 128, 128, 2, 4, 1);
  if (pick == 1) LEB_F32_TILE(pairs, 64, 64, 1, 2, 4);
  if (pick == 2) LEB_F32_TILE(tile, 32, 32, 1, 2, 8);
  if (pick == 3) LEB_F32_TILE(tile, 64, 16, 1, 1, 8);
  LEB_F32_TILE(tile, 32, 16, 1, 1, 8);
#undef LEB_F32_TILE
}
