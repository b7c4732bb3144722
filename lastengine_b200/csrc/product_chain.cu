// Consecutive bfloat16 products of a step of 17 to 128 rows as ONE resident kernel:
//   C_i[M,N_i] (+)= A_i[M,K_i] . W_i[N_i,K_i]^T,   i = 0, 1, ...,   A_{i+1} made from C_i
//
// Such a step is bound by reading every W once, and a launch per product stops that stream at each seam: the last
// block's sums, the release of the next kernel's wait, and the activations' trip from L2 leave memory idle for 3 to
// 7 us a product.  Weights do not depend on anything the step computes, so here the blocks stay on their SMs for the
// whole chain and a loading warp per block walks all of its products' weight tiles through one ring of shared
// memory, whatever product the block is at; what stands between two products is a barrier over the grid, and the ring
// fills while it is waited for.
//
// Split: a cluster of 4 blocks takes tiles of up to 128 weight rows; within the cluster block r takes slice r of K.  W is
// the 128-row operand of tcgen05.mma, the activations (padded to MP rows) the narrow one, the accumulator the
// transposed tile C^T[128 n][MP m] in tensor memory.  An accumulator loses in proportion to the products added up in it (2,048 x 5,632
// with a slice of 22 k-blocks in one: 1.4e-6 from 64 bits; the product alone, in slices of ten: 5.9e-7), so it takes no more
// k-blocks than a slice of the product alone, the next ones go to the next accumulator of a ring, and a block adds a tile's
// accumulators up in float (4.4e-7; 0.22 to 1.00 of the error alone over 19 sizes of 64 to 14,336 columns and K from 64 to
// 17,408).  Those before the last are read while that one fills, where the registers hold them for all owners (up to 64 rows).
// A slice's partial tile does not go to memory: the rows of A are dealt to the 4 blocks (MP / 4 each, their owners), and a block
// sends each owner its share of the partial tile into the owner's shared memory (st.async, counted by the owner's mbarrier).  The
// owner adds the slices in slice order and applies the epilogue.  So a result does not depend on timing, nor on the other rows.
//
// Epilogues as in gemm_bf16_stream.cu: 0 store (with an activation), 1 add into float C (leaving the next norm's
// half), 2 gated activation over interleaved weight rows, 3 the one-token gated convolution (a tile is then the B, C
// and x rows of 32 channels), each optionally scaled by a split norm.
//
// What bounds it: the four products of a conv layer of width 2,048, chained and as launches alone, in us, a norm's launch between
// layers:
//   rows              32            64            96            128
//   5,632 wide   39.7 / 42.1   44.0 / 49.2   53.6 / 59.9   58.5 / 67.7     103 MB of weights, 15.7 us at the copy rate
//   7,168 wide   43.6 / 56.7   48.3 / 65.7   59.2 / 83.4   64.8 / 101.3    122 MB, 18.6 us
// The stream runs at the memory's rate while there is room in the ring; the chain of a product (grid barrier 1.3 us, activations
// 0.7, last k-blocks 0.5 to 2, exchange 0.7, sums and stores 1, each once per product) is longer than what the ring holds.  The
// accumulators of shorter runs cost 1 to 4% of these times.
// Variants, each beside the kernel as it was when they were tried (7,168 wide, no norm between; 64 rows where none are named).  A
// cluster of 8 halves a block's k-blocks, but only 15 such clusters fit the chip (120 blocks against 132 in 33 clusters of 4) and 16
// tiles then take two rounds: 57 us, against 47.  Two more weight slots in the place of the second exchange buffer: 50.9 against 47.2, the
// senders wait for their credits.  Epilogues unrolled over all of a thread's outputs (128 KB of instructions) in the place of loops: 47.2
// against 45.8.  A tile exchanged in two parts, so that two buffers fit: 52 against 46, but from 65 rows on, where only one fits
// otherwise, 52 against 55 at 96 rows and 58 against 64 at 128 (5,632 wide), so it is done there.
//
// All blocks wait for one another, so they must all be resident: the launch is cooperative.  Every wait is bounded
// (mbarriers and the grid barrier by their polls): a wait that runs out sets the block's abort flag and the status
// word, and all blocks leave through one cluster barrier, so that none exits while another may still send to it.
#include "stream_common.cuh"
#include "tc_common.cuh"

#define PC_CLUSTER 4
#define PC_THREADS 512
#define PC_SUMMING 256     // threads that add partial tiles up and apply the epilogue
#define PC_MAX_OPS 40
#define PC_SPIN_LIMIT (1u << 20)
#define PC_CONV_CH 32      // channels of a convolution tile
#define PC_SLOT 16384      // bytes of a weight slot: up to 128 rows of one k-block of 64, or up to 64 rows of two
#define PC_STAGES 16       // barriers of the weight ring; a stage is two k-blocks, in one slot or two (never more stages than slots)

// A product as the kernel needs it, beside its tensor maps.
struct ChainOp {
  void* C;
  const float* ssq_in;
  bf16* emit_vals;
  const float* emit_g;
  float* emit_ssq;
  const float* conv_w;
  const float* conv_bias;
  float* conv_state;
  const int* row_seq;
  const int* seq_slot;
  int N, ldc, epilogue, c_dtype, parts_in, d_in;
  float eps;
  int width;               // columns of C
  int Lc, unused[3];
};
static_assert(sizeof(ChainOp) == 128, "copied to shared memory by words");
struct __align__(64) ChainMaps {
  CUtensorMap w, x;
};
// What the warps that issue copies and products take of it: read as parameters, so that it is known to be the same for a
// whole warp and stays in uniform registers.
struct __align__(16) ChainGeo {
  int blocks, n_tiles, rows, conv_width;      // k-blocks of 64 in K; tiles; weight rows of a tile; channels of a convolution (0: none)
  int per, skip, arrivals, run;               // k-blocks of a block's slice; tiles dealt before this product, modulo the clusters; blocks that arrive at its end; k-blocks added up in one accumulator
};
struct __align__(64) ChainArgs {
  ChainMaps map[PC_MAX_OPS];
  ChainOp op[PC_MAX_OPS];
  ChainGeo geo[PC_MAX_OPS];
  int n_ops, M;
  unsigned* sync;          // [2]: arrivals at the grid barrier, blocks that have left; both 0 between launches
  int* status;
};
static_assert(sizeof(ChainArgs) < 32000, "kernel parameters");

__device__ __forceinline__ uint32_t pc_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void pc_send4(uint32_t dst, uint32_t bar, const uint32_t* v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void pc_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void pc_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Waits on mbarriers by their shared addresses.  The usual case, a phase that has passed, is one try and no loop: as a call of
// the loop it took the warp that issues the products 170 cycles instead of 55, twice for every k-block.
template <bool CLUSTER>      // whether other blocks of the cluster arrive on the barrier (their writes are then visible)
__device__ __forceinline__ bool pc_passed(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
template <bool CLUSTER>
__device__ __noinline__ bool pc_wait_long(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < PC_SPIN_LIMIT; i++) {
    if (pc_passed<CLUSTER>(bar, parity)) return true;
    if (*abort_flag) return false;
    if (i > 4096) __nanosleep(64);
  }
  *abort_flag = 1;
  return false;
}
template <bool CLUSTER>
__device__ __forceinline__ bool pc_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return pc_passed<CLUSTER>(bar, parity) || pc_wait_long<CLUSTER>(bar, parity, abort_flag);
}
// N columns of a warp's 32 lanes of tensor memory.
template <int N>
__device__ __forceinline__ void pc_tmem_read(uint32_t* v, uint32_t src) {
  if (N == 16)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8 % N]), "=r"(v[9 % N]), "=r"(v[10 % N]), "=r"(v[11 % N]), "=r"(v[12 % N]), "=r"(v[13 % N]), "=r"(v[14 % N]), "=r"(v[15 % N])
                 : "r"(src));
  else
#pragma unroll
    for (int c = 0; c < N; c += 4)
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(v[c]), "=r"(v[c + 1]), "=r"(v[c + 2]), "=r"(v[c + 3])
                   : "r"(src + c));
}
// What was read is used after the wait, and not moved before it.
template <int N>
__device__ __forceinline__ void pc_tmem_there(uint32_t* v) {
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < N; c++) asm volatile("" : "+r"(v[c]));
}
// By all lanes of a warp.
__device__ __forceinline__ bool pc_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, pc_passed<false>(bar, parity))) return true;
  return __all_sync(0xffffffffu, pc_wait_long<false>(bar, parity, abort_flag)) != 0;
}
__device__ __forceinline__ void pc_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void pc_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void pc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Until `target` blocks in all have arrived at the grid barrier.  The polls are relaxed and the fence follows once: an acquiring
// load at device scope empties the SM's L1, and a thread that polls with it slows every other warp's shared memory accesses.
__device__ __forceinline__ bool pc_wait_grid(const unsigned* count, unsigned target, volatile int* abort_flag) {
  for (uint32_t i = 0; i < PC_SPIN_LIMIT; i++) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
    if ((int)(v - target) >= 0) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      return true;
    }
    if (*abort_flag) return false;
    if (i > 65536) __nanosleep(64);
  }
  *abort_flag = 1;
  return false;
}
// Whether all 256 threads of the summing warps say yes: a wait that ran out in one of them ends all of them together.
__device__ __forceinline__ bool pc_all_summing(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 2, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1u : 0u)
      : "memory");
  return r != 0;
}

// Activations that are not the usual one are calls: their code, inlined for every row, would push the kernel's own out of the
// instruction cache.
__device__ __noinline__ void pc_gate_call(float* g, const float* u, int act, int c_dtype) {
#pragma unroll 1
  for (int e = 0; e < 4; e++) g[e] = c_dtype == LEB_F32 ? gate_mul<float>(g[e], u[e], act) : gate_mul<bf16>(g[e], u[e], act);
}
__device__ __noinline__ void pc_act_call(float* z, int act) {
#pragma unroll 1
  for (int e = 0; e < 4; e++) z[e] = plain_act(z[e], act);
}

// By MP: accumulators in tensor memory, weight slots of 16 KB, stages of two k-blocks of activations (MP x 256 bytes), parts in which a partial tile is exchanged
// (an owner's first rows, then its last), buffers for such a part of the cluster's partial tiles (MP x 512 / parts bytes).
template <int MP> struct ChainRing;
template <> struct ChainRing<32> { static constexpr int NACC = 8, NW = 9, NX = 4, H = 1, RB = 2; };
template <> struct ChainRing<64> { static constexpr int NACC = 8, NW = 7, NX = 2, H = 1, RB = 2; };
template <> struct ChainRing<96> { static constexpr int NACC = 4, NW = 7, NX = 2, H = 2, RB = 2; };
template <> struct ChainRing<128> { static constexpr int NACC = 4, NW = 5, NX = 2, H = 2, RB = 2; };

template <int MP>
static constexpr size_t chain_smem() {
  typedef ChainRing<MP> Ring;
  return (size_t)Ring::NW * PC_SLOT + (size_t)Ring::NX * MP * 256 + (size_t)Ring::RB * MP * 512 / Ring::H + 1024 /* alignment */ +
         sizeof(ChainOp) * PC_MAX_OPS + 8 * (2 * PC_STAGES + 2 * Ring::NX + 2 * Ring::NACC + 3 * Ring::RB) + 4 * (MP / 4) * 2 + 80;
}

template <int MP>
__global__ void __launch_bounds__(PC_THREADS, 1)
product_chain_kernel(const __grid_constant__ ChainArgs args) {
  typedef ChainRing<MP> Ring;
  constexpr int NACC = Ring::NACC, NW = Ring::NW, NX = Ring::NX, H = Ring::H, RB = Ring::RB, R = MP / PC_CLUSTER, RH = R / H;
  constexpr bool EARLY = MP <= 64;
  constexpr int X_BYTES = MP * 128, RECV = MP * 512 / H;     // RECV: 4 slices of [RH / 4][128][4] floats
  constexpr uint32_t ACC_COLS = MP <= 32 ? 32 : (MP <= 64 ? 64 : 128), TMEM_COLS = NACC * ACC_COLS;
  extern __shared__ uint8_t smem_raw[];
  // the same offset in every block of the cluster (addresses of peers' buffers are formed from this block's)
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sw = smem;
  uint8_t* sx = sw + NW * PC_SLOT;
  uint8_t* sr = sx + NX * 2 * X_BYTES;
  ChainOp* ops = (ChainOp*)(sr + RB * RECV);
  uint64_t* wfull = (uint64_t*)(ops + PC_MAX_OPS);
  uint64_t* wempty = wfull + PC_STAGES;
  uint64_t* xfull = wempty + PC_STAGES;
  uint64_t* xempty = xfull + NX;
  uint64_t* acc_full = xempty + NX;
  uint64_t* acc_empty = acc_full + NACC;
  uint64_t* recv_full = acc_empty + NACC;
  uint64_t* credit = recv_full + RB;
  uint64_t* taken = credit + RB;
  float* row_scale = (float*)(((uintptr_t)(taken + RB) + 15) & ~(uintptr_t)15);     // [R]
  int* row_slot = (int*)(row_scale + R);             // [R]
  uint32_t* tmem_slot = (uint32_t*)(row_slot + R);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  // shared addresses of the buffers and barriers
  const uint32_t a_w = smem_u32(sw), a_x = smem_u32(sx), a_r = smem_u32(sr), b_wfull = smem_u32(wfull), b_wempty = smem_u32(wempty),
                 b_xfull = smem_u32(xfull), b_xempty = smem_u32(xempty), b_acc_full = smem_u32(acc_full), b_acc_empty = smem_u32(acc_empty),
                 b_recv = smem_u32(recv_full), b_credit = smem_u32(credit), b_taken = smem_u32(taken);

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = blockIdx.x % PC_CLUSTER, cluster = blockIdx.x / PC_CLUSTER, n_clusters = gridDim.x / PC_CLUSTER;
  const int M = args.M, n_ops = args.n_ops;
  const int n_owners = (M + R - 1) / R;              // blocks of a cluster that own rows
  const bool owner = rank < n_owners;

  if (threadIdx.x == 0) {
    for (int s = 0; s < PC_STAGES; s++) {
      mbar_init(&wfull[s], 1);
      mbar_init(&wempty[s], 1);
    }
    for (int s = 0; s < NX; s++) {
      mbar_init(&xfull[s], 1);
      mbar_init(&xempty[s], 1);
    }
    for (int s = 0; s < NACC; s++) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], 4);
    }
    for (int s = 0; s < RB; s++) {
      mbar_init(&recv_full[s], 1);
      mbar_init(&credit[s], n_owners);
      mbar_init(&taken[s], PC_SUMMING / 32);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // the parameters are used from shared memory: what a product needs of them lies in lines of the constant bank that nobody
  // has touched before, a miss each
  for (int o = warp; o < n_ops; o += PC_THREADS / 32) ((uint32_t*)&ops[o])[lane] = ((const uint32_t*)&args.op[o])[lane];
  if (warp == 3) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  __syncwarp();
  tc_fence_before();
  // no block sends to another before that one's barriers are there
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_acc = *tmem_slot;
  pdl_trigger();

  // A block's slice of K, k-blocks [lo, lo + n) of 64, and its cluster's tiles: first, first + clusters, ...  The deal goes on from
  // one product to the next, so that over a few products every block streams the same number of bytes; its ring evens
  // out what it does not within one.
  struct Share {
    int lo, n, first, n_tiles, rows;
  };
  auto share_of = [&](int o) {
    const ChainGeo& g = args.geo[o];
    Share s;
    s.lo = rank * g.per;
    s.n = max(0, min(g.blocks, s.lo + g.per) - s.lo);
    s.first = cluster - g.skip + (cluster < g.skip ? n_clusters : 0);
    s.n_tiles = g.n_tiles;
    s.rows = g.rows;
    return s;
  };
  // slots that a stage of `blocks` (one or two) k-blocks of a tile of `rows` rows takes
  auto slots_of = [](int rows, int blocks) { return rows > 64 ? blocks : 1; };
  int gave_up = 0;

  if (warp == 0) {
    // weights: every tile of every product of the chain, as fast as the ring empties
    int slot = 0, room = NW;               // the next slot; slots that are free
    unsigned stage = 0, oldest = 0, twos = 0;      // stages asked for; the oldest whose slots are not known to be free; bit i: stage i takes two
    for (int o = 0; o < n_ops && !gave_up; o++) {
      const Share sl = share_of(o);
      const int n_tiles = sl.n_tiles, rows = sl.rows, width = args.geo[o].conv_width;
      const bool conv = width > 0;
      const CUtensorMap* map = &args.map[o].w;
      for (int t = sl.first; t < n_tiles && !gave_up; t += n_clusters)
        for (int kb = 0; kb < sl.n; kb += 2) {
          const int here = min(2, sl.n - kb), need = slots_of(rows, here);
          while (room < need) {
            if (!pc_wait_warp(b_wempty + 8 * (oldest % PC_STAGES), (oldest / PC_STAGES) & 1, abort_flag)) { gave_up = 41; break; }
            room += 1 + ((twos >> (oldest % PC_STAGES)) & 1);
            oldest++;
          }
          if (gave_up) break;
          const uint32_t bar = b_wfull + 8 * (stage % PC_STAGES), bit = 1u << (stage % PC_STAGES);
          if (elect_lane()) {
            pc_expect(bar, here * rows * 128);
            for (int u = 0; u < here; u++) {
              const int k = (sl.lo + kb + u) * TC_BK;
              int at = slot + (rows > 64 ? u : 0);
              if (at >= NW) at -= NW;
              const uint32_t dst = a_w + at * PC_SLOT + (rows > 64 ? 0 : u * rows * 128);
              if (conv) {
                for (int c = 0; c < 3; c++) pc_load(dst + c * PC_CONV_CH * 128, map, bar, k, c * width + t * PC_CONV_CH);
              } else {
                pc_load(dst, map, bar, k, t * rows);
              }
            }
          }
          __syncwarp();
          twos = need > 1 ? twos | bit : twos & ~bit;
          room -= need;
          slot += need;
          if (slot >= NW) slot -= NW;
          stage++;
        }
    }
  } else if (warp == 1) {
    // activations, two k-blocks to a stage.  A slice that fits the ring is fetched once for all tiles of the product.
    pdl_wait();
    int s = 0, ph = 1;
    unsigned target = 0;
    for (int o = 0; o < n_ops && !gave_up; o++) {
      const Share sl = share_of(o);
      const int n_tiles = sl.n_tiles;
      const CUtensorMap* map = &args.map[o].x;
      if (sl.first < n_tiles) {
        if (elect_lane()) asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
        __syncwarp();
        // the activations of product o are there once every block has finished product o - 1; they were written by
        // ordinary stores and are read by the copy unit
        bool ok = true;
        if (lane == 0) ok = pc_wait_grid(args.sync, target, abort_flag);
        if (!__all_sync(0xffffffffu, ok)) { gave_up = 42; break; }
        asm volatile("fence.proxy.async.global;" ::: "memory");
        const bool once = sl.n <= 2 * NX;
        for (int t = sl.first; t < n_tiles && !gave_up; t += n_clusters) {
          for (int kb = 0; kb < sl.n; kb += 2) {
            if (!pc_wait_warp(b_xempty + 8 * s, ph, abort_flag)) { gave_up = 43; break; }
            const int here = min(2, sl.n - kb);
            if (elect_lane()) {
              pc_expect(b_xfull + 8 * s, here * X_BYTES);
              for (int u = 0; u < here; u++) pc_load(a_x + (2 * s + u) * X_BYTES, map, b_xfull + 8 * s, (sl.lo + kb + u) * TC_BK, 0);
            }
            __syncwarp();
            if (++s == NX) s = 0, ph ^= 1;
          }
          if (once) break;
        }
      }
      target += args.geo[o].arrivals;
    }
  } else if (warp == 2) {
    pdl_wait();
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MP >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const uint64_t w_desc = make_desc(a_w), x_desc = make_desc(a_x);
    int slot = 0, x = 0, xph = 0;
    unsigned stage = 0, run = 0;           // run: accumulators filled
    for (int o = 0; o < n_ops && !gave_up; o++) {
      const Share sl = share_of(o);
      const int n_tiles = sl.n_tiles, rows = sl.rows, most = args.geo[o].run;
      if (sl.n == 0) continue;
      const bool once = sl.n <= 2 * NX;
      const int x0 = x, xph0 = xph;
      for (int t = sl.first; t < n_tiles && !gave_up; t += n_clusters) {
        const bool first = !once || t == sl.first, last = !once || t + n_clusters >= n_tiles;    // who waits for, and who frees, a stage
        if (!first) x = x0, xph = xph0;
        int left = 0;                      // k-blocks that the accumulator still takes
        for (int kb = 0; kb < sl.n && !gave_up; kb += 2) {
          const int here = min(2, sl.n - kb);
          const int slot2 = slot + 1 >= NW ? 0 : slot + 1;
          const uint64_t da = w_desc + (uint64_t)(slot * (PC_SLOT / 16)), db = x_desc + (uint64_t)(2 * x * (X_BYTES / 16));
          const uint64_t da2 = rows > 64 ? w_desc + (uint64_t)(slot2 * (PC_SLOT / 16)) : da + (uint64_t)(rows * 8);
          const uint32_t begins = left == 0;
          if (begins) {
            if (!pc_wait_warp(b_acc_empty + 8 * (run % NACC), ((run / NACC) & 1) ^ 1, abort_flag)) { gave_up = 44; break; }
            left = most;
          }
          const bool apart = left < here;      // the accumulator ends between the stage's k-blocks
          const bool ends = left <= here || kb + 2 >= sl.n;
          const uint32_t acc = tmem_acc + (run % NACC) * ACC_COLS, full = b_acc_full + 8 * (run % NACC), empty = b_wempty + 8 * (stage % PC_STAGES);
          if (first && !pc_wait_warp(b_xfull + 8 * x, xph, abort_flag)) { gave_up = 45; break; }
          if (!pc_wait_warp(b_wfull + 8 * (stage % PC_STAGES), (stage / PC_STAGES) & 1, abort_flag)) { gave_up = 45; break; }
          tc_fence_after();
          if (elect_lane()) {
#pragma unroll
            for (int k = 0; k < TC_BK / 16; k++)
              umma_bf16(acc, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, !begins || k != 0);
            if (here == 2 && !apart) {
#pragma unroll
              for (int k = 0; k < TC_BK / 16; k++)
                umma_bf16(acc, da2 + (uint64_t)(k * 2), db + (uint64_t)(X_BYTES / 16 + k * 2), idesc, 1);
            }
            if (!apart) {
              pc_commit(empty);
              if (last) pc_commit(b_xempty + 8 * x);
            }
            if (ends) pc_commit(full);
          }
          __syncwarp();
          left -= here;
          if (ends) left = 0, run++;
          if (apart) {      // the stage's second k-block is the next accumulator's first
            if (!pc_wait_warp(b_acc_empty + 8 * (run % NACC), ((run / NACC) & 1) ^ 1, abort_flag)) { gave_up = 44; break; }
            tc_fence_after();
            const bool whole = most == 1 || kb + 2 >= sl.n;      // it holds no other
            if (elect_lane()) {
#pragma unroll
              for (int k = 0; k < TC_BK / 16; k++)
                umma_bf16(tmem_acc + (run % NACC) * ACC_COLS, da2 + (uint64_t)(k * 2), db + (uint64_t)(X_BYTES / 16 + k * 2), idesc, k != 0);
              pc_commit(empty);
              if (last) pc_commit(b_xempty + 8 * x);
              if (whole) pc_commit(b_acc_full + 8 * (run % NACC));
            }
            __syncwarp();
            left = whole ? 0 : most - 1;
            if (whole) run++;
          }
          slot += slots_of(rows, here);
          if (slot >= NW) slot -= NW;
          stage++;
          if (++x == NX) x = 0, xph ^= 1;
        }
      }
    }
  } else if (warp == 3) {
    // a buffer that all summing warps have read is given back to the cluster's senders (here, since the release they need would
    // hold the summing warps up for half a microsecond)
    int q = 0;
    if (owner)
      for (int o = 0; o < n_ops && !gave_up; o++) {
        const Share sl = share_of(o);
        const int n_tiles = sl.n_tiles;
        for (int i = 0, parts = sl.first < n_tiles ? H * ((n_tiles - sl.first + n_clusters - 1) / n_clusters) : 0; i < parts; i++, q++) {
          const int rb = q % RB;
          if (!pc_wait_warp(b_taken + 8 * rb, (q / RB) & 1, abort_flag)) { gave_up = 49; break; }
          if (lane < PC_CLUSTER) pc_arrive_remote(pc_mapa(b_credit + 8 * rb, lane));
          __syncwarp();
        }
      }
  } else if (warp < 8) {
    // the partial tile from tensor memory to the rows' owners; a thread holds one weight row, all activation rows
    pdl_wait();
    const int quad = warp & 3;
    int q = 0;
    unsigned run = 0;
    for (int o = 0; o < n_ops && !gave_up; o++) {
      const Share sl = share_of(o);
      int runs = 0;                        // accumulators of a tile
      for (int k = 0; k < sl.n; k += args.geo[o].run) runs++;
      for (int t = sl.first; t < sl.n_tiles && !gave_up; t += n_clusters, run += runs) {
        bool ok = true;
        const uint32_t src = tmem_acc + ((uint32_t)(quad * 32) << 16);
        const bool has = sl.n > 0 && quad * 32 < sl.rows;
        // what the accumulators before the last hold is added up while that one is filled, for all owners, where the registers suffice
        uint32_t sum[EARLY ? PC_CLUSTER : 1][RH];
        for (int j = 0; j < runs - 1 && ok; j++) {
          ok = pc_wait<false>(b_acc_full + 8 * ((run + j) % NACC), ((run + j) / NACC) & 1, abort_flag);
          if (EARLY && has) {
            ok = __all_sync(0xffffffffu, ok) != 0;
            if (!ok) break;
            tc_fence_after();
            if (j == 0) {
#pragma unroll
              for (int to = 0; to < (EARLY ? PC_CLUSTER : 1); to++) pc_tmem_read<RH>(sum[to], src + (run % NACC) * ACC_COLS + to * R);
#pragma unroll
              for (int to = 0; to < (EARLY ? PC_CLUSTER : 1); to++) pc_tmem_there<RH>(sum[to]);
            } else {
#pragma unroll
              for (int to = 0; to < (EARLY ? PC_CLUSTER : 1); to++) {
                uint32_t w[RH];
                pc_tmem_read<RH>(w, src + ((run + j) % NACC) * ACC_COLS + to * R);
                pc_tmem_there<RH>(w);
#pragma unroll
                for (int c = 0; c < RH; c++) sum[to][c] = __float_as_uint(__uint_as_float(sum[to][c]) + __uint_as_float(w[c]));
              }
            }
          }
        }
        const uint32_t final = run + max(runs - 1, 0);
        if (runs > 0 && ok) ok = pc_wait<false>(b_acc_full + 8 * (final % NACC), (final / NACC) & 1, abort_flag);
#pragma unroll 1
        for (int h = 0; h < H; h++, q++) {
          const int rb = q % RB;
          // the owners have taken what lay in this buffer (a block without k-blocks waits too and sends nothing: a wait tells only odd
          // phases from even ones, so a phase that is passed by would be taken for the one after the next)
          if (ok && q >= RB) ok = pc_wait<true>(b_credit + 8 * rb, ((q / RB) - 1) & 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok) != 0;
          if (!ok) break;
          tc_fence_after();
          if (has) {
            const uint32_t base = a_r + rb * RECV + (uint32_t)rank * (RH * 512) + (uint32_t)(quad * 32 + lane) * 16, bar = b_recv + 8 * rb;
            auto send = [&](int to, const uint32_t* v) {
              const uint32_t there = pc_mapa(base, to), bar_there = pc_mapa(bar, to);
#pragma unroll
              for (int c = 0; c < RH; c += 4) pc_send4(there + (c / 4) * 2048, bar_there, v + c);
            };
            if (EARLY) {
#pragma unroll
              for (int to = 0; to < PC_CLUSTER; to++)
                if (to < n_owners) {
                  uint32_t v[RH];
                  pc_tmem_read<RH>(v, src + (final % NACC) * ACC_COLS + to * R);
                  pc_tmem_there<RH>(v);
                  if (runs > 1) {
#pragma unroll
                    for (int c = 0; c < RH; c++) v[c] = __float_as_uint(__uint_as_float(sum[EARLY ? to : 0][c]) + __uint_as_float(v[c]));
                  }
                  send(to, v);
                }
            } else {
#pragma unroll 1
              for (int to = 0; to < n_owners; to++) {
                uint32_t v[RH], w[RH];
                pc_tmem_read<RH>(v, src + h * RH + (run % NACC) * ACC_COLS + to * R);
#pragma unroll 1
                for (int j = 1; j < runs; j++) {
                  pc_tmem_read<RH>(w, src + h * RH + ((run + j) % NACC) * ACC_COLS + to * R);
                  pc_tmem_there<RH>(v);
                  pc_tmem_there<RH>(w);
#pragma unroll
                  for (int c = 0; c < RH; c++) v[c] = __float_as_uint(__uint_as_float(v[c]) + __uint_as_float(w[c]));
                }
                pc_tmem_there<RH>(v);
                send(to, v);
              }
            }
          }
        }
        if (!ok) { gave_up = 46; break; }
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          for (int j = 0; j < runs; j++) pc_arrive(b_acc_empty + 8 * ((run + j) % NACC));
      }
    }
  } else if (owner) {
    // The owner of rows [m0, m0 + R) adds the slices in order, applies the epilogue, stores.  A thread takes units of one output
    // column and four rows (16 bytes of every slice).  Loops over units stay loops: all of a chain's epilogues
    // unrolled are 128 KB of instructions, which come from L2 every time.
    const int tid = threadIdx.x - 256, m0 = rank * R, ew = tid >> 5;
    constexpr int G = RH / 4;           // row groups of a part
    pdl_wait();
    int q = 0;
    unsigned target = 0;
    for (int o = 0; o < n_ops && !gave_up; o++) {
      const Share sl = share_of(o);
      const int n_tiles = sl.n_tiles, rows = sl.rows, active = (args.geo[o].blocks + args.geo[o].per - 1) / args.geo[o].per;
      const unsigned arrivals = args.geo[o].arrivals;
      if (sl.first >= n_tiles) {
        target += arrivals;
        continue;
      }
      const ChainOp op = ops[o];       // in registers: a store might change what is read from shared memory
      const int act = op.epilogue >> 8, kind = op.epilogue & 255;
      if (kind == 3)      // the state lies in memory: on its way to L2 while the product before this one ends
        for (int t = sl.first; t < n_tiles; t += n_clusters)
          for (int r = tid; r < R; r += PC_SUMMING) {
            const int slot = m0 + r < M ? op.seq_slot[op.row_seq[m0 + r]] : -1;
            if (slot >= 0)
              for (int b = 0; b < PC_CONV_CH * (op.Lc - 1); b += 32)
                if (t * PC_CONV_CH * (op.Lc - 1) + b < op.width * (op.Lc - 1))
                  asm volatile("prefetch.global.L2 [%0];" ::"l"(op.conv_state + ((size_t)slot * op.width + t * PC_CONV_CH) * (op.Lc - 1) + b));
          }
      bool there = true;
      if (tid == 0) there = pc_wait_grid(args.sync, target, abort_flag);
      __syncwarp();
      if (!pc_all_summing(there)) { gave_up = 47; break; }
      // the rows' factors of a split norm (1 without one): a warp takes rows ew, ew + 8, ...; the convolution's slots
      constexpr int RW = (R + 7) / 8;      // (all loads first: one after the other they would be eight trips to L2)
      float part[RW][4];
#pragma unroll
      for (int i = 0; i < RW; i++)
#pragma unroll
        for (int p = 0; p < 4; p++) {
          const int r = ew + 8 * i;
          part[i][p] = op.ssq_in && r < R && m0 + r < M && lane + 32 * p < op.parts_in
                           ? __ldcg(op.ssq_in + (size_t)(m0 + r) * op.parts_in + lane + 32 * p) : 0.f;
        }
#pragma unroll
      for (int i = 0; i < RW; i++) {
        const int r = ew + 8 * i;
        float s = (part[i][0] + part[i][1]) + (part[i][2] + part[i][3]);
        if (op.ssq_in && r < R && m0 + r < M)
          for (int p = lane + 128; p < op.parts_in; p += 32) s += __ldcg(op.ssq_in + (size_t)(m0 + r) * op.parts_in + p);
        s = warp_sum(s);
        if (lane == 0 && r < R) {
          row_scale[r] = op.ssq_in ? 1.0f / sqrtf(s / (float)op.d_in + op.eps) : 1.f;
          row_slot[r] = kind == 3 && m0 + r < M ? op.seq_slot[op.row_seq[m0 + r]] : -1;
        }
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
      // units of a tile: columns (rounded up to a power of two) x row groups
      const int width = kind == 3 ? PC_CONV_CH : (kind == 2 ? rows / 2 : rows);
      const int ps = width > 64 ? 7 : (width > 32 ? 6 : 5), n_units = G << ps;
      const int end = kind == 3 ? op.width : (kind == 2 ? op.width : op.N);     // columns of the result
#pragma unroll 1
      for (int i_part = 0, parts = H * ((n_tiles - sl.first + n_clusters - 1) / n_clusters); i_part < parts; i_part++, q++) {
        const int t = sl.first + i_part / H * n_clusters, rb = q % RB, r0 = i_part % H * RH;
        if (tid == 0) pc_expect(b_recv + 8 * rb, (uint32_t)active * (RH * 4) * rows);
        const float* recv = (const float*)(sr + rb * RECV);
        // column n, rows 4 g ... 4 g + 3 of the part: the slices' shares, RH * 128 floats apart, added in order
        auto sum = [&](int n, int g) {
          const float4* p = (const float4*)(recv + g * 512 + n * 4);
          float4 a = p[0];
#pragma unroll
          for (int s = 1; s < PC_CLUSTER; s++)
            if (s < active) {
              const float4 b = p[s * (RH * 32)];
              a.x += b.x, a.y += b.y, a.z += b.z, a.w += b.w;
            }
          return a;
        };
        bool waited = false;
#pragma unroll 1
        for (int u = tid; u < n_units; u += PC_SUMMING) {        // (whole warps share u's row group)
          const int i = u & ((1 << ps) - 1), g = u >> ps, col = t * width + i, row0 = r0 + 4 * g, m = m0 + row0;
          const bool in = i < width && col < end;
          // what does not depend on the sums is on its way while they come
          float old[4], st[4][ST_CONV_MAX_LC - 1], tap[ST_CONV_MAX_LC], extra = 0.f;      // extra: the next norm's weight, or the convolution's bias
          if (kind == 3) {
            const float* sp = op.conv_state + (size_t)col * (op.Lc - 1);
            extra = in && op.conv_bias ? op.conv_bias[col] : 0.f;
#pragma unroll
            for (int k = 0; k < ST_CONV_MAX_LC; k++) tap[k] = in && k < op.Lc ? op.conv_w[(size_t)col * op.Lc + k] : 0.f;
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const int slot = row_slot[row0 + e];
              const float* sr_ = sp + (size_t)max(slot, 0) * (op.width * (op.Lc - 1));
#pragma unroll
              for (int k = 0; k < ST_CONV_MAX_LC - 1; k++) st[e][k] = in && slot >= 0 && k < op.Lc - 1 ? __ldcg(sr_ + k) : 0.f;
            }
          } else if (kind == 1) {
            const float* cp = (const float*)op.C + m * op.ldc + col;
            extra = in && op.emit_vals ? op.emit_g[col] : 0.f;
#pragma unroll
            for (int e = 0; e < 4; e++) old[e] = in && m + e < M ? __ldcg(cp + e * op.ldc) : 0.f;
          }
          if (!waited) {
            there = true;
            if (tid == 0) there = pc_wait<true>(b_recv + 8 * rb, (q / RB) & 1, abort_flag);
            __syncwarp();
            there = pc_all_summing(there);
            waited = true;
            if (!there) break;
          }
          const int ng = kind == 2 ? 32 * (i >> 4) + (i & 15) : i;
          const float4 scale = *(const float4*)(row_scale + row0);
          float4 a = in ? sum(ng, g) : make_float4(0.f, 0.f, 0.f, 0.f), b = a, c = a;
          if (kind >= 2 && in) b = sum(ng + (kind == 2 ? 16 : PC_CONV_CH), g);
          if (kind == 3 && in) c = sum(ng + 2 * PC_CONV_CH, g);
          float va[4] = {a.x * scale.x, a.y * scale.y, a.z * scale.z, a.w * scale.w};
          float vb[4] = {b.x * scale.x, b.y * scale.y, b.z * scale.z, b.w * scale.w};
          if (kind == 3) {
            // as shortconv_single_kernel: the projections rounded to bfloat16 as if they had been stored; padding rows give 0
            const float vc[4] = {c.x * scale.x, c.y * scale.y, c.z * scale.z, c.w * scale.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const int slot = row_slot[row0 + e];
              const float bx = to_f32(__float2bfloat16_rn(va[e])) * to_f32(__float2bfloat16_rn(vc[e]));
              float acc = extra, tail = 0.f;
#pragma unroll
              for (int k = 0; k < ST_CONV_MAX_LC - 1; k++)
                if (k < op.Lc - 1) acc += tap[k] * st[e][k];
#pragma unroll
              for (int k = 0; k < ST_CONV_MAX_LC; k++)
                if (k == op.Lc - 1) tail = tap[k];
              acc += tail * bx;
              if (in && slot >= 0) {
                float* sc = op.conv_state + ((size_t)slot * op.width + col) * (op.Lc - 1);
#pragma unroll
                for (int k = 0; k < ST_CONV_MAX_LC - 2; k++)
                  if (k < op.Lc - 2) sc[k] = st[e][k + 1];
                sc[op.Lc - 2] = bx;
              }
              va[e] = slot >= 0 ? to_f32(__float2bfloat16_rn(vb[e])) * acc : 0.f;
            }
          } else if (kind == 2) {
            if (act == 0 && op.c_dtype == LEB_BF16) {
#pragma unroll
              for (int e = 0; e < 4; e++) va[e] = silu_mul<bf16>(va[e], vb[e]);
            } else {
              float z[4] = {va[0], va[1], va[2], va[3]}, z2[4] = {vb[0], vb[1], vb[2], vb[3]};
              pc_gate_call(z, z2, act, op.c_dtype);
#pragma unroll
              for (int e = 0; e < 4; e++) va[e] = z[e];
            }
          } else if (kind == 1) {
#pragma unroll
            for (int e = 0; e < 4; e++) va[e] += old[e];
          } else if (LEB_PLAIN_ACT_OK(act, kind)) {
            float z[4] = {va[0], va[1], va[2], va[3]};
            pc_act_call(z, act);
#pragma unroll
            for (int e = 0; e < 4; e++) va[e] = z[e];
          }
          if (op.c_dtype == LEB_F32) {
            float* cp = (float*)op.C + m * op.ldc + col;
#pragma unroll
            for (int e = 0; e < 4; e++)
              if (in && m + e < M) cp[e * op.ldc] = va[e];
          } else {
            bf16* cp = (bf16*)op.C + m * op.ldc + col;
#pragma unroll
            for (int e = 0; e < 4; e++)
              if (in && m + e < M) cp[e * op.ldc] = __float2bfloat16_rn(va[e]);
          }
          if (op.emit_vals) {                  // the new residual, for the norm that follows
            bf16* ep = op.emit_vals + m * op.N + col;
            const int parts = (op.N + 15) / 16;
            float* qp = op.emit_ssq + m * parts + col / 16;
            float sq[4];
#pragma unroll
            for (int e = 0; e < 4; e++) sq[e] = in ? va[e] * va[e] : 0.f;
#pragma unroll
            for (int sh = 8; sh > 0; sh >>= 1)
#pragma unroll
              for (int e = 0; e < 4; e++) sq[e] += __shfl_xor_sync(0xffffffffu, sq[e], sh);
#pragma unroll
            for (int e = 0; e < 4; e++)
              if (in && m + e < M) {
                ep[e * op.N] = __float2bfloat16_rn(va[e] * extra);
                if ((col & 15) == 0) qp[e * parts] = sq[e];
              }
          }
        }
        if (!waited) {                         // (fewer units than threads: the others wait here)
          there = pc_all_summing(true);
        }
        if (!there) { gave_up = 48; break; }
        // this warp has read the buffer
        __syncwarp();
        if (lane == 0) pc_arrive(b_taken + 8 * rb);
      }
      target += arrivals;
      if (gave_up) break;
      if (o + 1 < n_ops) {
        // this block's part of product o is stored; the copy units of all blocks may read it
        asm volatile("fence.proxy.async.global;" ::: "memory");
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(args.sync) : "memory");
      }
    }
  }
  if (gave_up && lane == 0) {
    *abort_flag = 1;
    atomicExch(args.status, gave_up);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (*abort_flag)      // copies of a chain that was given up may still be on their way: they land within microseconds
    for (int i = 0; i < 64; i++) __nanosleep(20000);
  __syncwarp();
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_acc, TMEM_COLS);
  }
  __syncwarp();
  // nobody leaves while a block of the cluster may still send to it
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (threadIdx.x == 0) {
    // the last block to leave makes the words ready for the next chain
    __threadfence();
    if (atomicInc(args.sync + 1, gridDim.x - 1) == gridDim.x - 1) atomicExch(args.sync, 0u);
  }
}

// ---- host side -------------------------------------------------------------------------------------
// The products of the chain that is being put together, per host thread.
static thread_local ChainArgs g_chain;
static thread_local int g_chain_ops = 0;

// Clusters that are on the device at once, per row padding (0: not asked, -1: the kernel does not fit).
template <int MP>
static int chain_clusters() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n) return n;
  n = -1;
  if (leb_allow_smem<product_chain_kernel<MP>>() == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(PC_CLUSTER);
    cfg.blockDim = dim3(PC_THREADS);
    cfg.dynamicSmemBytes = chain_smem<MP>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = PC_CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, product_chain_kernel<MP>, &cfg) == cudaSuccess && fit > 0)
      n = fit < sm_count() / PC_CLUSTER ? fit : sm_count() / PC_CLUSTER;
  }
  cudaGetLastError();
  known[dev].store(n, std::memory_order_relaxed);
  return n;
}

template <int MP>
static int launch_chain(cudaStream_t st) {
  const int clusters = chain_clusters<MP>();
  if (clusters <= 0) return leb_fail("leb_chain_run: the chain's blocks do not fit the device");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * PC_CLUSTER);
  cfg.blockDim = dim3(PC_THREADS);
  cfg.dynamicSmemBytes = chain_smem<MP>();
  cfg.stream = st;
  cudaLaunchAttribute attr[3];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PC_CLUSTER;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  attr[2].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[2].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_leb_pdl ? 3 : 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, product_chain_kernel<MP>, g_chain);
  if (e != cudaSuccess) return leb_fail("leb_chain_run: %s", cudaGetErrorString(e));
  LEB_CHECK_LAUNCH("leb_chain_run");
  return 0;
}

LEB_API int leb_chain_max_ops() { return PC_MAX_OPS; }

// Clusters of blocks the chain of M rows runs on (0 or less: there is none on this device).
LEB_API int leb_chain_clusters(int M) {
  if (M < 17 || M > 128) return 0;
  return M <= 32 ? chain_clusters<32>() : M <= 64 ? chain_clusters<64>()
         : M <= 96 ? chain_clusters<96>() : chain_clusters<128>();
}

LEB_API int leb_chain_drop() {
  g_chain_ops = 0;
  return 0;
}

extern "C" int leb_gemm_bf16_skinny_slices(int N, int K);

// Accumulators of a block's slice: each takes at most the k-blocks of a slice of the product alone.
static int chain_runs(int N, int K) {
  const int blocks = ceil_div(K, TC_BK);
  return ceil_div(ceil_div(blocks, PC_CLUSTER), ceil_div(blocks, leb_gemm_bf16_skinny_slices(N, K)));
}
// Whether the chain takes a product of M rows: whether there are so many accumulators.
LEB_API int leb_chain_takes(int M, int N, int K) {
  return chain_runs(N, K) <= (M <= 64 ? ChainRing<64>::NACC : ChainRing<128>::NACC);
}

// Adds a product to the chain (nothing is launched).  Arguments as leb_gemm_bf16_stream; with conv_w the product is the conv
// mixer's in_proj [3D, K] of a decode step (N is 3D, C is y [M, D], bfloat16) as in leb_gemm_bf16_stream_conv.
LEB_API int leb_chain_add(void* C, int c_dtype, const void* A, const void* W, int M, int N, int K, int lda, int ldc, int epilogue,
                          const float* ssq_in, int parts_in, int d_in, float eps, void* emit_vals, const float* emit_g, float* emit_ssq,
                          const float* conv_w, const float* bias, float* state, const int* row_seq, const int* seq_slot, int Lc) {
  const int act = epilogue >> 8;
  int kind = epilogue & 255;
  LEB_REQUIRE(M >= 17 && M <= 128 && N > 0 && K > 0 && K % 8 == 0 && lda % 8 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0,
              "leb_chain_add: takes 17..128 rows and operands the copy unit can fetch (M %d, N %d, K %d, lda %d)", M, N, K, lda);
  LEB_REQUIRE(g_chain_ops < PC_MAX_OPS, "leb_chain_add: the chain is full");
  LEB_REQUIRE(g_chain_ops == 0 || g_chain.M == M, "leb_chain_add: %d rows in a chain of %d", M, g_chain.M);
  LEB_REQUIRE(c_dtype == LEB_F32 || c_dtype == LEB_BF16, "leb_chain_add: unknown C dtype %d", c_dtype);
  LEB_REQUIRE(!ssq_in || (parts_in > 0 && d_in > 0), "leb_chain_add: the sums of squares need their count and the row width");
  if (conv_w) {
    LEB_REQUIRE(kind == 0 && act == 0 && c_dtype == LEB_BF16 && N % 3 == 0 && Lc >= 2 && Lc <= ST_CONV_MAX_LC && state && row_seq && seq_slot && !emit_vals,
                "leb_chain_add: a convolution stores bfloat16, of 2..%d taps, with state and the step's tables", ST_CONV_MAX_LC);
    kind = 3;
  } else {
    LEB_REQUIRE(kind >= 0 && kind <= 2 && (LEB_GATE_ACT_OK(act, kind) || (LEB_PLAIN_ACT_OK(act, kind) && c_dtype == LEB_BF16)),
                "leb_chain_add: activation %d does not go with epilogue %d", act, kind);
    LEB_REQUIRE(kind != 1 || c_dtype == LEB_F32, "leb_chain_add: adding needs a float C");
    LEB_REQUIRE(kind != 2 || N % 32 == 0, "leb_chain_add: the gated epilogue needs N (%d) to be a multiple of 32", N);
    LEB_REQUIRE(!emit_vals || (kind == 1 && emit_g && emit_ssq), "leb_chain_add: only an adding product leaves the next norm's input");
  }
  // Weight rows of a tile: those with the fewest bytes in a block's way, a round counted as 45 rows more (what its sums
  // and their exchange take); 96 for the convolution (three times its channels).
  const int clusters = leb_chain_clusters(M);
  int rows = kind == 3 ? 3 * PC_CONV_CH : 128;
  if (kind != 3 && clusters > 0) {
    long best = -1;
    for (int r : {128, 96, 64, 32}) {
      const long cost = (long)ceil_div(ceil_div(N, r), clusters) * (r + 45);
      if (best < 0 || cost < best) best = cost, rows = r;
    }
  }
  LEB_REQUIRE(leb_chain_takes(M, N, K), "leb_chain_add: %d columns of %d numbers need more accumulators than there are at %d rows", N, K, M);
  const int MP = M <= 32 ? 32 : (M <= 64 ? 64 : (M <= 96 ? 96 : 128)), blocks = ceil_div(K, TC_BK), per = ceil_div(blocks, PC_CLUSTER);
  ChainOp& op = g_chain.op[g_chain_ops];
  ChainMaps& map = g_chain.map[g_chain_ops];
  if (tensor_map(&map.w, W, N, K, K, kind == 3 ? PC_CONV_CH : rows)) return 1;
  if (tensor_map(&map.x, A, M, K, lda, MP)) return 1;
  op.C = C;
  op.ssq_in = ssq_in;
  op.emit_vals = (bf16*)emit_vals;
  op.emit_g = emit_g;
  op.emit_ssq = emit_ssq;
  op.conv_w = conv_w;
  op.conv_bias = bias;
  op.conv_state = state;
  op.row_seq = row_seq;
  op.seq_slot = seq_slot;
  op.Lc = Lc;
  op.N = N;
  op.ldc = ldc;
  op.epilogue = kind | (act << 8);
  op.c_dtype = c_dtype;
  op.width = kind == 3 ? N / 3 : (kind == 2 ? N / 2 : N);
  const int n_tiles = kind == 3 ? ceil_div(N / 3, PC_CONV_CH) : ceil_div(N, rows), dealt = max(clusters, 1);
  const ChainGeo* before = g_chain_ops ? &g_chain.geo[g_chain_ops - 1] : nullptr;
  g_chain.geo[g_chain_ops] = ChainGeo{blocks, n_tiles, rows, kind == 3 ? N / 3 : 0, per,
                                      before ? (before->skip + before->n_tiles) % dealt : 0, min(dealt, n_tiles) * ceil_div(M, MP / PC_CLUSTER), ceil_div(per, chain_runs(N, K))};
  op.parts_in = parts_in;
  op.d_in = d_in;
  op.eps = eps;
  g_chain.M = M;
  g_chain_ops++;
  return 0;
}

// Launches the products that were added, in their order, as one kernel.  sync: two words, 0 before the first chain that
// uses them and left at 0 by every chain; chains that may run at the same time need their own.
LEB_API int leb_chain_run(void* sync, int* status, cudaStream_t st) {
  const int n = g_chain_ops, M = g_chain.M;
  g_chain_ops = 0;
  if (n == 0) return 0;
  LEB_REQUIRE(sync && status, "leb_chain_run: the barrier's words and a status word are required");
  g_chain.n_ops = n;
  g_chain.sync = (unsigned*)sync;
  g_chain.status = status;
  return M <= 32 ? launch_chain<32>(st) : M <= 64 ? launch_chain<64>(st)
         : M <= 96 ? launch_chain<96>(st) : launch_chain<128>(st);
}
