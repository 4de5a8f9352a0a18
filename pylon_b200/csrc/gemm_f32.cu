// y[M, N] = x[M, K] * W[N, K]^T in true float32: plain FMA on the CUDA cores (fma.rn.f32x2: two of
// them to an instruction, each rounded like any other), float32 accumulation, no tensor cores and no
// reduced-precision matrix mode.  This is the matrix product of the engine's 32-bit path
// (raun6k/Pylon runs its float32 model through nn.Linear, src/pylon/model/layers.py:17-23,95-106).
//
// The order of a sum depends on K alone, so a row's result does not depend on which other rows share
// the launch, nor on which of the kernels below computed it.  K is cut into LEAVES leaves of
// equal length (a multiple of 32).  A leaf is two chains in ascending k, one over its even and one
// over its odd places, added at its end; four neighbouring leaves are added up in order to a quarter,
// and the quarters in order to the result.  Short chains also keep the rounding error below that of one
// chain over the whole of k (3.2e-7 against 1.8e-6 of the result at K = 9,728).
//
//   rows   up to 16 rows of x (decode steps, the head): bound by the bytes of W up to some 8 rows, above by the FMA units and
//          the reads of x from shared memory, which do not overlap on them.  A lane owns two rows of W (with 9 to 16 rows of x, eight rows of W and four of x), a warp one leaf
//          or quarter of 64 rows, which it streams through a ring of its own with cp.async; no warp waits for another before
//          its part is done.  Lanes read the rows of x that they share from shared memory as broadcasts.  W [19456, 2560]: 48 us for one row of x (199 MB:
//          4.2 TB/s), 74 us for 16; W [151936, 2560]: 243 and 369 us (6.4 TB/s and 34 TFLOP/s).
//   tile   more rows: bound by the FMA units (2.2 to 2.5 cycles an instruction and scheduler, whatever the order of the
//          operands) and by the reads from shared memory, which add to them.  256 threads take 16 TM x 16 TN results, each thread TM x TN
//          of them with two accumulators apiece; pairs of neighbouring k are the packed operands, so both operands stay
//          in shared memory the way they lie in memory.  Two blocks to an SM (7 x 5: only in clusters of four, whose parking place is one tile): with
//          one of 8 x 8 results a thread, 740 us for [224, 2560] x [19456, 2560]; with 7 x 4 or 7 x 5, 626 us, and with stages of 32 k, which halve the
//          barriers, 544 (41 TFLOP/s).  One multiply-add
//          to an instruction: the same.
//
//   short  k up to 128 and more than a few rows: a start of microseconds, not the sums, is what is left, and neither a ring of copies nor a
//          cluster pays.  256 threads take 64 x 64 results a leaf at a time.  12 rows of [6144, 64]: 5.0 us, the
//          streaming kernel 7.5 alone and 16 in clusters, the tile kernel 6.9.
//
// In the first two, the blocks of a thread-block cluster take different leaves of the same results where there are too
// few results to fill the GPU, and add them up through each other's shared memory.
//
// What went before, 64 x 64 results to a block and a chain over the whole of k to each: 354 us for 16 rows and 1,093 us for 224 rows of
// [19456, 2560], 307 us for 16 rows of [2560, 4096] (now 29).
#include "common.cuh"

#include <algorithm>
#include <cooperative_groups.h>

namespace pylon {

namespace cg = cooperative_groups;

constexpr int LEAVES = 16, LEAVES_PER_QUARTER = 4, BK = 16;

__host__ __device__ __forceinline__ int leaf_length(int K) { return ((K + LEAVES - 1) / LEAVES + 31) / 32 * 32; }

struct GemmArgs {
  const float *x, *w;
  float* y;
  int M, N, K;
  long long ldx, ldw, ldy, batch_x, batch_w, batch_y;
  int w_static;   // nothing queued on the stream writes w: its first stages are asked for while the kernel ahead still runs
};

typedef unsigned long long Pair;   // two float32: the element of an even k and that of the next
__device__ __forceinline__ void fma_pair(Pair& c, Pair a, Pair b) { asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ float add_pair(Pair c) {
  float even, odd;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(c));
  return even + odd;
}

// Copies VEC floats (16 or 4 bytes) to shared memory, or zeros when !inside.  `src` is a valid address in either case.
template <int VEC>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool inside) {
  const unsigned address = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = inside ? 4 * VEC : 0;
  if (VEC == 4)
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;\n" ::"r"(address), "l"(src), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(address), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory"); }

// Copies columns [k0, k0 + COLUMNS) of ROWS rows, from row0 on, into a stage whose rows lie ROW floats apart.  Rows past the last one
// are copies of it (what is computed from them is not written), columns past K zeros.  SWIZZLE: the 16-byte unit u of row r goes to
// unit u ^ ((r / 2) % 4), so that eight neighbouring rows of 64 bytes give the same unit from all 32 banks.  A thread's copies
// lie in one column of units, a fixed number of rows apart: one address computation each.
template <int VEC, int ROWS, int THREADS, int ROW, bool SWIZZLE, int COLUMNS = BK>
__device__ __forceinline__ void stage_copy(float* dst, const float* __restrict__ src, long long ld, int row0, int last, int k0, int K, int t) {
  constexpr int UNITS = COLUMNS / VEC, APART = THREADS / UNITS;
  const int r0 = t / UNITS, c = (t % UNITS) * VEC;
  const bool inside = k0 + c < K;
  src += inside ? k0 + c : 0;
  dst += r0 * ROW + (SWIZZLE ? ((((c >> 2) ^ (r0 >> 1)) & 3) << 2) + (c & 3) : c);
  static_assert(!SWIZZLE || VEC == 1 || APART % 8 == 0, "the unit's place must be the same for all of a thread's rows");
#pragma unroll
  for (int i = 0; i < (ROWS + APART - 1) / APART; ++i) {
    const int r = r0 + i * APART;
    if (ROWS % APART != 0 && r >= ROWS) continue;
    float* place = dst + i * APART * ROW;
    if (SWIZZLE && VEC == 1) place = dst - r0 * ROW - (((((c >> 2) ^ (r0 >> 1)) & 3) << 2) + (c & 3)) + r * ROW + ((((c >> 2) ^ (r >> 1)) & 3) << 2) + (c & 3);
    copy_async<VEC>(place, src + (size_t)min(row0 + r, last) * ld, inside);
  }
}

// stage_copy of a warp's lanes with the swizzle, 16 bytes at a time, with the lane's first row looked up once: a copy then costs an addition of
// addresses instead of a product: 8 rows of [2560, 9728] 30.9 to 28.6 us, of [2560, 4096] 15.5 to 14.5.
template <int ROWS>
struct RowsCopy {
  static constexpr int UNITS = BK / 4, APART = 32 / UNITS, COPIES = (ROWS + APART - 1) / APART;
  static_assert(APART % 8 == 0, "the unit's place must be the same for all of a lane's rows");
  const float* src;
  __device__ __forceinline__ RowsCopy(const float* matrix, long long ld, int row0, int last, int lane) { src = matrix + (size_t)min(row0 + lane / UNITS, last) * ld; }
  __device__ __forceinline__ void operator()(float* stage, long long ld, int row0, int last, int k0, int K, int lane) const {
    const int r0 = lane / UNITS, c = (lane % UNITS) * 4;
    const bool inside = k0 + c < K, all = row0 + ROWS - 1 <= last;
    const float* from = src + (inside ? k0 + c : 0);
    float* to = stage + r0 * BK + ((((c >> 2) ^ (r0 >> 1)) & 3) << 2);
#pragma unroll
    for (int i = 0; i < COPIES; ++i) {
      const int r = r0 + i * APART;
      if (ROWS % APART != 0 && r >= ROWS) continue;
      const bool there = all || row0 + r <= last;   // else zeros, and what is computed from them is not written
      copy_async<4>(to + i * APART * BK, there ? from + i * (APART * ld) : src, there && inside);
    }
  }
};

// ---------------------------------------------------------------------------------------------
// few rows
// ---------------------------------------------------------------------------------------------
// A stage is BK columns: NR * 32 rows of W, MT rows of x.  Rows are 64 bytes; the 16-byte unit u of row r lies at unit
// u ^ ((r / 2) % 4), so that eight neighbouring rows read the same unit from all 32 banks.
template <int MT, int NR, int STAGES_>
struct RowsRing {
  static constexpr int STAGES = STAGES_, W_FLOATS = NR * 32 * BK, X_FLOATS = MT * BK, STAGE = W_FLOATS + X_FLOATS;
};

// Grid (slabs of NR * 32 rows of W x cluster size, MT rows of x each, products); blocks of `warps` warps.  With 16 warps in a
// cluster each takes a leaf, with 4 a quarter.
template <int MT, int NR, int VEC, int STAGES>
__global__ void __launch_bounds__(128, 3) gemm_f32_rows_kernel(const GemmArgs a) {
  using Ring = RowsRing<MT, NR, STAGES>;
  constexpr int TILE = MT * NR * 32;
  extern __shared__ __align__(16) float smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int blocks = cluster.num_blocks(), rank = cluster.block_rank();
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = blocks * warps, unit = rank * warps + warp;   // 16 or 4
  const int n0 = (int)(blockIdx.x / blocks) * NR * 32, m0 = blockIdx.y * MT;
  const float* x = a.x + (size_t)blockIdx.z * a.batch_x;
  const float* w = a.w + (size_t)blockIdx.z * a.batch_w;
  float* y = a.y + (size_t)blockIdx.z * a.batch_y;
  const int share = TILE / blocks;                  // results this block adds up
  float* gathered = smem;                           // [units][share]
  float* ring = smem + (size_t)units * share + (size_t)warp * Ring::STAGES * Ring::STAGE;

  const int leaf = leaf_length(a.K), leaves = LEAVES / units;
  const int k_begin = unit * leaves * leaf, k_end = min(a.K, k_begin + leaves * leaf);
  const int steps = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;

  const RowsCopy<NR * 32> rows_of_w(w, a.ldw, n0, a.N - 1, lane);
  const RowsCopy<MT> rows_of_x(x, a.ldx, m0, a.M - 1, lane);
  auto copy_w = [&](float* dst, int k0) {
    if (VEC == 4) rows_of_w(dst, a.ldw, n0, a.N - 1, k0, a.K, lane);
    else stage_copy<VEC, NR * 32, 32, BK, true>(dst, w, a.ldw, n0, a.N - 1, k0, a.K, lane);
  };
  auto copy_x = [&](float* dst, int k0) {
    if (VEC == 4) rows_of_x(dst, a.ldx, m0, a.M - 1, k0, a.K, lane);
    else stage_copy<VEC, MT, 32, BK, true>(dst, x, a.ldx, m0, a.M - 1, k0, a.K, lane);
  };
  if (!a.w_static) grid_dependency_wait();
#pragma unroll
  for (int s = 0; s < Ring::STAGES - 1; ++s)
    if (s < steps) copy_w(ring + s * Ring::STAGE, k_begin + s * BK);
  grid_dependency_wait();
  allow_dependents();
  if (blocks > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");   // this block runs: its shared memory may be written
#pragma unroll
  for (int s = 0; s < Ring::STAGES - 1; ++s) {
    if (s < steps) copy_x(ring + s * Ring::STAGE + Ring::W_FLOATS, k_begin + s * BK);
    copies_commit();
  }

  // A lane's results.  Up to 8 rows of x: all of them, of rows lane, lane + 32 of W.  16 rows: a read of x serves all lanes alike but takes as long as one of W, so
  // the lanes share them 4 x 8: rows tm + 4 i of x, tn + 8 j of W (12 reads for 64 multiply-adds instead of 18, and from the bits of the lane
  // that take two passes): 16 rows of [2560, 9728] 53.0 to 49.6 us, of [151936, 2560] 378 to 369.
  constexpr bool SHARED = MT == 16 && NR == 2;
  constexpr int MI = SHARED ? 4 : MT, NJ = SHARED ? 8 : NR;
  const int tm = SHARED ? (lane >> 1) & 3 : 0, tn = SHARED ? ((lane >> 2) & 6) + (lane & 1) : lane;
  auto result = [&](int i, int j) { return SHARED ? (tm + 4 * i) * (NR * 32) + tn + 8 * j : (i * NR + j) * 32 + lane; };
  Pair acc[MI][NJ];
#pragma unroll
  for (int m = 0; m < MI; ++m)
#pragma unroll
    for (int r = 0; r < NJ; ++r) acc[m][r] = 0;
  const int leaf_steps = leaf / BK, w_xor = (tn >> 1) & 3;
  bool first = true;   // the first leaf of a quarter is its sum so far
  int until_fold = leaf_steps;
  for (int step = 0; step < steps; ++step) {
    copies_wait<Ring::STAGES - 2>();
    __syncwarp();
    {
      const int ahead = step + Ring::STAGES - 1;
      if (ahead < steps) {
        float* dst = ring + (ahead % Ring::STAGES) * Ring::STAGE;
        copy_w(dst, k_begin + ahead * BK);
        copy_x(dst + Ring::W_FLOATS, k_begin + ahead * BK);
      }
      copies_commit();
    }
    const float* stage = ring + (step % Ring::STAGES) * Ring::STAGE;
#pragma unroll
    for (int u = 0; u < BK / 4; ++u) {
      constexpr int GROUP = MI < 4 ? MI : 4;   // rows whose chains take turns, so that no multiply-add waits for the one before it
      ulonglong2 wv[NJ];
#pragma unroll
      for (int r = 0; r < NJ; ++r) wv[r] = *reinterpret_cast<const ulonglong2*>(stage + (r * (SHARED ? 8 : 32) + tn) * BK + ((u ^ w_xor) << 2));
#pragma unroll
      for (int g = 0; g < MI; g += GROUP) {
        ulonglong2 xv[GROUP];
#pragma unroll
        for (int m = 0; m < GROUP; ++m) {
          const int row = SHARED ? 4 * m : g + m;   // and tm; its swizzle is that of row + tm
          const int unit = SHARED ? (u ^ (2 * (m & 1)) ^ (tm >> 1)) : u ^ ((row >> 1) & 3);
          xv[m] = *reinterpret_cast<const ulonglong2*>(stage + Ring::W_FLOATS + (row + tm) * BK + (unit << 2));
        }
#pragma unroll
        for (int m = 0; m < GROUP; ++m)
#pragma unroll
          for (int r = 0; r < NJ; ++r) fma_pair(acc[g + m][r], xv[m].x, wv[r].x);
#pragma unroll
        for (int m = 0; m < GROUP; ++m)
#pragma unroll
          for (int r = 0; r < NJ; ++r) fma_pair(acc[g + m][r], xv[m].y, wv[r].y);
      }
    }
    if (--until_fold == 0 && step != steps - 1) {   // a leaf of a quarter: a lone block's warp, which keeps the sum in its own place
#pragma unroll
      for (int m = 0; m < MI; ++m)
#pragma unroll
        for (int r = 0; r < NJ; ++r) {
          float* place = gathered + (size_t)unit * share + result(m, r);
          const float value = add_pair(acc[m][r]);
          *place = first ? value : *place + value;
          acc[m][r] = 0;
        }
      first = false;
      until_fold = leaf_steps;
    }
  }

  if (blocks > 1) asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  if (steps > 0) {
#pragma unroll
    for (int m = 0; m < MI; ++m)
#pragma unroll
      for (int r = 0; r < NJ; ++r) {
        const int e = result(m, r);
        float* place = gathered + (size_t)unit * share + e % share;
        if (blocks > 1) place = cluster.map_shared_rank(place, e / share);
        const float value = add_pair(acc[m][r]);
        *place = first ? value : *place + value;
      }
  }
  if (blocks > 1) cluster.sync(); else __syncthreads();

  const int present = (a.K + leaves * leaf - 1) / (leaves * leaf);   // units that have any k
  const int in_order = LEAVES_PER_QUARTER / leaves;                  // units to a quarter
  for (int i = threadIdx.x; i < share; i += blockDim.x) {
    const int e = rank * share + i, m = m0 + e / (NR * 32), n = n0 + e % (NR * 32);
    if (m >= a.M || n >= a.N) continue;
    float total = 0.f;
    for (int q = 0; q < present; q += in_order) {
      float quarter = gathered[(size_t)q * share + i];
      for (int j = 1; j < in_order && q + j < present; ++j) quarter += gathered[(size_t)(q + j) * share + i];
      total = q == 0 ? quarter : total + quarter;
    }
    y[(size_t)m * a.ldy + n] = total;
  }
}

// ---------------------------------------------------------------------------------------------
// many rows
// ---------------------------------------------------------------------------------------------
template <int TM, int TN>
struct TileShape {
  static constexpr int BM = 16 * TM, BN = 16 * TN;
  static constexpr int BK = 32, STAGES = 2;                // a barrier every 32 k (193 rows of [19456, 2560] 543 us; every 16 k, three stages, 621)
  static constexpr int ROW = BK + 4;                       // floats from row to row of a stage: eight rows' units lie in all 32 banks
  static constexpr int STAGE = (BM + BN) * ROW;
  static constexpr int PARK_ROW = BN + 4, PARK = BM * PARK_ROW;
  static constexpr size_t smem(int blocks) { return ((size_t)STAGES * STAGE + (size_t)(blocks == 4 ? 1 : 2) * PARK) * sizeof(float); }
};

// Grid (tiles of 16 TN rows of W x cluster size, tiles of 16 TM rows of x, products), 256 threads.  A cluster of 1, 2, 4 or 8 blocks
// shares the leaves of a tile; a block lays down what it has summed in one or two parking places (one float per result):
//   8 blocks  each of its two leaves        4 blocks  its quarter        2 blocks  each of its two quarters
//   1 block   the quarter it is in, and the quarters before it
template <int TM, int TN, int VEC, bool HALVES>
__global__ void __launch_bounds__(256, 2) gemm_f32_tile_kernel(const GemmArgs a) {
  using Shape = TileShape<TM, TN>;
  constexpr int BK = Shape::BK;
  extern __shared__ __align__(16) float smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int blocks = cluster.num_blocks(), rank = cluster.block_rank();
  const int n0 = (int)(blockIdx.x / blocks) * Shape::BN, m0 = blockIdx.y * Shape::BM;
  const float* x = a.x + (size_t)blockIdx.z * a.batch_x;
  const float* w = a.w + (size_t)blockIdx.z * a.batch_w;
  float* y = a.y + (size_t)blockIdx.z * a.batch_y;
  float* stages = smem;
  float* park = smem + (size_t)Shape::STAGES * Shape::STAGE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // This thread's rows: tm + 16 i of x, tn + 16 j of W.  Which bits of the lane choose which row decides how many passes a 16-byte
  // read from shared memory takes: two where the rows hang on bits {1, 2} or {0, 3, 4}, four on {0, 1, 2} (3.9 against 2.1 cycles).
  const int tm = (warp >> 1) * 4 + ((lane >> 1) & 3), tn = (warp & 1) * 8 + ((lane >> 2) & 6) + (lane & 1);

  const int leaf = leaf_length(a.K), leaf_begin = rank * (LEAVES / blocks);
  const int k_begin = leaf_begin * leaf, k_end = min(a.K, (leaf_begin + LEAVES / blocks) * leaf);
  const int steps = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;

  if (!a.w_static) grid_dependency_wait();
#pragma unroll
  for (int s = 0; s < Shape::STAGES - 1; ++s)
    if (s < steps) stage_copy<VEC, Shape::BN, 256, Shape::ROW, false, BK>(stages + s * Shape::STAGE + Shape::BM * Shape::ROW, w, a.ldw, n0, a.N - 1, k_begin + s * BK, a.K, threadIdx.x);
  grid_dependency_wait();
  allow_dependents();
#pragma unroll
  for (int s = 0; s < Shape::STAGES - 1; ++s) {
    if (s < steps) stage_copy<VEC, Shape::BM, 256, Shape::ROW, false, BK>(stages + s * Shape::STAGE, x, a.ldx, m0, a.M - 1, k_begin + s * BK, a.K, threadIdx.x);
    copies_commit();
  }

  Pair acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0;
  const int leaf_steps = leaf / BK;
  int until_fold = leaf_steps, at = leaf_begin;
  for (int step = 0; step < steps; ++step) {
    copies_wait<Shape::STAGES - 2>();
    __syncthreads();
    {
      const int ahead = step + Shape::STAGES - 1;
      if (ahead < steps) {
        float* dst = stages + (ahead % Shape::STAGES) * Shape::STAGE;
        stage_copy<VEC, Shape::BM, 256, Shape::ROW, false, BK>(dst, x, a.ldx, m0, a.M - 1, k_begin + ahead * BK, a.K, threadIdx.x);
        stage_copy<VEC, Shape::BN, 256, Shape::ROW, false, BK>(dst + Shape::BM * Shape::ROW, w, a.ldw, n0, a.N - 1, k_begin + ahead * BK, a.K, threadIdx.x);
      }
      copies_commit();
    }
    const float* xs = stages + (step % Shape::STAGES) * Shape::STAGE + tm * Shape::ROW;
    const float* ws = stages + (step % Shape::STAGES) * Shape::STAGE + (Shape::BM + tn) * Shape::ROW;
    constexpr int UNITS = HALVES ? BK / 8 : BK / 4;   // of four k
    const int parts = HALVES && k_begin + step * BK + BK / 2 < a.K ? 2 : 1;
#pragma unroll 1
    for (int part = 0; part < parts; ++part, xs += BK / 2, ws += BK / 2) {
      ulonglong2 wv[TN], xv[2];
      xv[0] = *reinterpret_cast<const ulonglong2*>(xs);
#pragma unroll
      for (int u = 0; u < UNITS; ++u) {
#pragma unroll
        for (int j = 0; j < TN; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(ws + j * 16 * Shape::ROW + 4 * u);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const int next = u * TM + i + 1;   // the row of x after this one is on its way while this one is multiplied
          if (next < TM * UNITS) xv[next & 1] = *reinterpret_cast<const ulonglong2*>(xs + (next % TM) * 16 * Shape::ROW + 4 * (next / TM));
          const ulonglong2 x4 = xv[(next - 1) & 1];
#pragma unroll
          for (int j = 0; j < TN; ++j) fma_pair(acc[i][j], x4.x, wv[j].x);   // the chains take turns: no multiply-add waits for the one before it
#pragma unroll
          for (int j = 0; j < TN; ++j) fma_pair(acc[i][j], x4.y, wv[j].y);
        }
      }
    }
    if (--until_fold == 0 || step == steps - 1) {
      const int quarter = at / LEAVES_PER_QUARTER;
      const bool store = blocks == 8 || at % LEAVES_PER_QUARTER == 0;   // else: added to the quarter's leaves before it
      float* place = park + (size_t)(blocks == 8 ? (at & 1) : blocks == 2 ? (quarter & 1) : 0) * Shape::PARK;
      // a lone block keeps its quarters' sum in the second place: the quarter joins it with its last leaf
      const bool join = blocks == 1 && (at % LEAVES_PER_QUARTER == LEAVES_PER_QUARTER - 1 || step == steps - 1);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const int e = (tm + 16 * i) * Shape::PARK_ROW + tn + 16 * j;
          float value = add_pair(acc[i][j]);
          if (!store) value = place[e] + value;
          if (!join) place[e] = value;
          else if (quarter == 0) place[Shape::PARK + e] = value;
          else place[Shape::PARK + e] += value;
          acc[i][j] = 0;
        }
      ++at;
      until_fold = leaf_steps;
    }
  }
  if (blocks > 1) cluster.sync(); else __syncthreads();

  // Each block of the cluster adds up its share of the tile's rows.
  const int rows = Shape::BM / blocks, present = (a.K + leaf - 1) / leaf;
  const bool wide = a.N % 4 == 0 && a.ldy % 4 == 0 && a.batch_y % 4 == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
  for (int index = threadIdx.x; index < rows * (Shape::BN / 4); index += 256) {
    const int row = rank * rows + index / (Shape::BN / 4), col = (index % (Shape::BN / 4)) * 4;
    const int m = m0 + row, n = n0 + col;
    if (m >= a.M || n >= a.N) continue;
    const size_t e = (size_t)row * Shape::PARK_ROW + col;
    float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [](float4 p, float4 q) { return make_float4(p.x + q.x, p.y + q.y, p.z + q.z, p.w + q.w); };
    if (blocks == 1) {
      total = *reinterpret_cast<const float4*>(park + Shape::PARK + e);
    } else if (blocks == 8) {
      float4 value[LEAVES];
#pragma unroll
      for (int l = 0; l < LEAVES; ++l)
        if (l < present) value[l] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(park + (size_t)(l & 1) * Shape::PARK + e, l >> 1));
#pragma unroll
      for (int q = 0; q < LEAVES / LEAVES_PER_QUARTER; ++q) {
        if (q * LEAVES_PER_QUARTER >= present) continue;
        float4 quarter = value[q * LEAVES_PER_QUARTER];
#pragma unroll
        for (int l = 1; l < LEAVES_PER_QUARTER; ++l)
          if (q * LEAVES_PER_QUARTER + l < present) quarter = add(quarter, value[q * LEAVES_PER_QUARTER + l]);
        total = q == 0 ? quarter : add(total, quarter);
      }
    } else {
#pragma unroll
      for (int q = 0; q < LEAVES / LEAVES_PER_QUARTER; ++q) {
        if (q * LEAVES_PER_QUARTER >= present) continue;
        const float* place = blocks == 2 ? park + (size_t)(q & 1) * Shape::PARK + e : park + e;
        const float4 quarter = *reinterpret_cast<const float4*>(cluster.map_shared_rank(place, blocks == 2 ? q >> 1 : q));
        total = q == 0 ? quarter : add(total, quarter);
      }
    }
    float* out = y + (size_t)m * a.ldy + n;
    if (wide) {
      *reinterpret_cast<float4*>(out) = total;
    } else {
      const float values[4] = {total.x, total.y, total.z, total.w};
      for (int c = 0; c < 4 && n + c < a.N; ++c) out[c] = values[c];
    }
  }
  if (blocks > 1) cluster.sync();   // no block leaves while another reads what it has parked
}

// ---------------------------------------------------------------------------------------------
// short k
// ---------------------------------------------------------------------------------------------
// Grid (64 rows of W, 64 rows of x, products), 256 threads of 4 x 4 results.  A stage is a leaf of 32 k, and all of k one quarter; operands are
// read element by element, whatever their alignment.
constexpr int SHORT_MOST = 32 * LEAVES_PER_QUARTER;
__global__ void __launch_bounds__(256) gemm_f32_short_kernel(const GemmArgs a) {
  constexpr int ROWS = 64, T = 4, LEAF = 32;
  __shared__ __align__(16) float xs[LEAF][ROWS + 4], ws[LEAF][ROWS + 4];
  const float* x = a.x + (size_t)blockIdx.z * a.batch_x;
  const float* w = a.w + (size_t)blockIdx.z * a.batch_w;
  float* y = a.y + (size_t)blockIdx.z * a.batch_y;
  const int m0 = blockIdx.y * ROWS, n0 = blockIdx.x * ROWS, tm = (threadIdx.x / 16) * T, tn = (threadIdx.x % 16) * T;
  const int row = threadIdx.x / 4, column = threadIdx.x % 4;   // what this thread copies: every fourth k of a row of each
  const bool has_x = m0 + row < a.M, has_w = n0 + row < a.N;
  x += (size_t)(has_x ? m0 + row : 0) * a.ldx + column;
  w += (size_t)(has_w ? n0 + row : 0) * a.ldw + column;
  float total[T][T];
#pragma unroll
  for (int i = 0; i < T; ++i)
#pragma unroll
    for (int j = 0; j < T; ++j) total[i][j] = 0.f;
  grid_dependency_wait();
  allow_dependents();
  for (int k0 = 0; k0 < a.K; k0 += LEAF) {
    const int here = a.K - k0 - column;   // from this thread's first k on
    float xr[LEAF / 4], wr[LEAF / 4];
#pragma unroll
    for (int j = 0; j < LEAF / 4; ++j) {
      xr[j] = has_x && 4 * j < here ? x[k0 + 4 * j] : 0.f;
      wr[j] = has_w && 4 * j < here ? w[k0 + 4 * j] : 0.f;
    }
    if (k0 > 0) __syncthreads();   // the leaf before has been read
#pragma unroll
    for (int j = 0; j < LEAF / 4; ++j) {
      xs[column + 4 * j][row] = xr[j];
      ws[column + 4 * j][row] = wr[j];
    }
    __syncthreads();
    float even[T][T], odd[T][T];
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) even[i][j] = odd[i][j] = 0.f;
    const int halves = k0 + LEAF / 2 < a.K ? 2 : 1;
#pragma unroll 1
    for (int half = 0; half < halves; ++half)
#pragma unroll
      for (int k = 0; k < LEAF / 2; ++k) {
        const float4 x4 = *reinterpret_cast<const float4*>(&xs[half * (LEAF / 2) + k][tm]), w4 = *reinterpret_cast<const float4*>(&ws[half * (LEAF / 2) + k][tn]);
        const float xv[T] = {x4.x, x4.y, x4.z, x4.w}, wv[T] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int i = 0; i < T; ++i)
#pragma unroll
          for (int j = 0; j < T; ++j) {
            if (k % 2 == 0) even[i][j] = fmaf(xv[i], wv[j], even[i][j]);
            else odd[i][j] = fmaf(xv[i], wv[j], odd[i][j]);
          }
      }
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j) total[i][j] = k0 == 0 ? even[i][j] + odd[i][j] : total[i][j] + (even[i][j] + odd[i][j]);
  }
  const bool wide = n0 + tn + T <= a.N && a.ldy % 4 == 0 && a.batch_y % 4 == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
#pragma unroll
  for (int i = 0; i < T; ++i) {
    if (m0 + tm + i >= a.M) continue;
    float* out = y + (size_t)(m0 + tm + i) * a.ldy + n0 + tn;
    if (wide) {
      *reinterpret_cast<float4*>(out) = make_float4(total[i][0], total[i][1], total[i][2], total[i][3]);
    } else {
#pragma unroll
      for (int j = 0; j < T; ++j)
        if (n0 + tn + j < a.N) out[j] = total[i][j];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef void (*GemmKernel)(const GemmArgs);

// Function attributes and the number of clusters that run at once are asked for once per kernel and device.
struct KernelState {
  bool configured = false;
  int clusters[9] = {};
};

static int clusters_at_once(GemmKernel kernel, KernelState& state, int blocks, int threads, size_t smem) {
  if (state.clusters[blocks] == 0) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = blocks;
    attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    int count = 0;
    if (cudaOccupancyMaxActiveClusters(&count, (const void*)kernel, &config) != cudaSuccess || count < 1) {
      cudaGetLastError();
      count = multiprocessors() / blocks > 0 ? multiprocessors() / blocks : 1;
    }
    state.clusters[blocks] = count;
  }
  return state.clusters[blocks];
}

static cudaError_t configure(GemmKernel kernel, KernelState& state, size_t smem) {
  if (state.configured) return cudaSuccess;
  const cudaError_t err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  state.configured = err == cudaSuccess;
  return err;
}

// Rows kernel: 16 warps of a cluster (eight blocks of two) take a leaf each, so that 40 slabs (a matrix of 2,560 rows) are 640 warps.
// With enough slabs, four warps of a lone block take a quarter each: no cluster to place and no shared memory to cross, and a warp's ring runs four
// times as long.  With four rows of x or fewer the loads bound it and more, smaller blocks keep more of them in flight (one row, 2,374 slabs: 243
// against 268 us).  With a short k most of a cluster's warps have nothing to do (one row of [2560, 64]: 2.9 us alone, 3.9 in clusters; 12 of [9728, 300] 14.7
// and 26.7; but one of [512, 128] 3.7 and 3.4).  5 to 8 rows: from 96 slabs on up to a k of 2,560 (8 of [6144, 2560] 20.9 and 22.1 us, of [24576, 512] 16 and
// 33; but of [5120, 2560] 20.6 and 15.6, of [19456, 4096] 77 and 70), whatever k is from LONE_WORK results in groups of 64 on.  9 to 16 rows: by an estimate of
// both forms fitted to their times over 16 to 640 slabs and k of 512 to 9,728, and where it is 7 % ahead (9 rows alone and in clusters: [6144, 2560] 32 and
// 35 us, [16384, 2560] 50 and 72, [19456, 2560] 72 and 85; but [5120, 4096] 48.7 and 41, [19456, 9728] 253 and 225).
constexpr long long LONE_WORK = 4096;

static bool rows_alone(const GemmArgs& a, long long slabs) {
  if (a.K <= 64 || (a.K < 512 && slabs >= (a.K <= 256 ? 32 : 64))) return true;
  if (a.M <= 4 || a.K < 512) return false;
  if (slabs * a.M >= LONE_WORK) return true;
  if (a.M <= 8) return slabs >= 96 && a.K <= 2560;
  const long long rounds = (slabs + multiprocessors() - 1) / multiprocessors();
  return slabs >= 80 && 1.07 * (6.0 + a.K * (0.0018 + 0.0083 * rounds)) < 4.5 + 0.003 * a.K + slabs * (0.105 + 5.1e-5 * a.K);   // us
}

template <int MT, int NR, int VEC>
static int launch_rows(const GemmArgs& a, int batch, int force, cudaStream_t stream) {
  // A third lone block fits an SM with two stages of 16 rows instead of four, which pays where there is one for it: 16 rows of [151936, 2560] 394 to 378 us, of
  // [19456, 2560] 75 to 72; but [16384, 2560], two blocks an SM either way, 53 us with four stages and 70 with two.
  constexpr int SHORT = MT == 16 ? 2 : 4;
  const long long slabs = (a.N + NR * 32 - 1) / (NR * 32);
  const long long all = slabs * batch;
  const bool lone = force ? (force & 2) : rows_alone(a, all);
  const bool brief = lone && SHORT != 4 && all > 2LL * multiprocessors();
  GemmKernel kernel = brief ? gemm_f32_rows_kernel<MT, NR, VEC, SHORT> : gemm_f32_rows_kernel<MT, NR, VEC, 4>;
  static KernelState states[2][MAX_DEVICES];
  KernelState& state = states[brief][current_device_slot()];
  const int blocks = lone ? 1 : 8, warps = lone ? 4 : 2;
  const auto bytes = [](int places, int warps_, int stage_floats) { return ((size_t)places * MT * NR * 32 + (size_t)warps_ * stage_floats) * sizeof(float); };
  const int ring = RowsRing<MT, NR, 4>::STAGES * RowsRing<MT, NR, 4>::STAGE, brief_ring = RowsRing<MT, NR, SHORT>::STAGES * RowsRing<MT, NR, SHORT>::STAGE;
  const size_t lone_bytes = bytes(4, 4, brief ? brief_ring : ring), cluster_bytes = bytes(2, 2, ring);
  cudaError_t err = configure(kernel, state, brief ? lone_bytes : std::max(lone_bytes, cluster_bytes));
  if (err != cudaSuccess) PYLON_REFUSE("gemm_f32: %s", cudaGetErrorString(err));
  launch_dependent_cluster<LAUNCH_GEMM>(kernel, dim3((unsigned)(slabs * blocks), (a.M + MT - 1) / MT, batch), dim3(32 * warps), lone ? lone_bytes : cluster_bytes, stream,
                                        (unsigned)blocks, a);
  PYLON_CHECK_LAUNCH("gemm_f32");
}

template <int VEC>
static int dispatch_rows(const GemmArgs& a, int batch, int force, cudaStream_t stream) {
  if (a.M <= 1) return launch_rows<1, 2, VEC>(a, batch, force, stream);
  if (a.M <= 2) return launch_rows<2, 2, VEC>(a, batch, force, stream);
  if (a.M <= 4) return launch_rows<4, 2, VEC>(a, batch, force, stream);
  if (a.M <= 8) return launch_rows<8, 2, VEC>(a, batch, force, stream);
  return launch_rows<16, 2, VEC>(a, batch, force, stream);
}

// With `cost`: the estimated time of the launch in us instead of the launch.
template <int TM, int TN, int VEC>
static int tile_kernel(const GemmArgs& a, int batch, int blocks, cudaStream_t stream, double* cost) {
  using Shape = TileShape<TM, TN>;
  // Where the last stage of a short k is half empty or emptier, stages are multiplied by halves and an empty one is passed over: 300 rows of [6144, 80] 19.5
  // us, whole stages 21.7; 2,048 of [6144, 208] 174 and 184.  Elsewhere the seam between the halves costs 3 to 5 %.
  const bool halves = a.K <= 240 && a.K % 32 != 0 && a.K % 32 <= 16;
  GemmKernel kernel = halves ? gemm_f32_tile_kernel<TM, TN, VEC, true> : gemm_f32_tile_kernel<TM, TN, VEC, false>;
  static KernelState states[2][MAX_DEVICES];
  KernelState& state = states[halves][current_device_slot()];
  cudaError_t err = configure(kernel, state, Shape::smem(1));
  if (err != cudaSuccess) PYLON_REFUSE("gemm_f32: %s", cudaGetErrorString(err));
  const long long tiles_n = (a.N + Shape::BN - 1) / Shape::BN, tiles_m = (a.M + Shape::BM - 1) / Shape::BM;
  if (cost) {
    const int sms = multiprocessors();
    const long long tiles = tiles_n * tiles_m * batch, at_once = clusters_at_once(kernel, state, blocks, 256, Shape::smem(blocks));
    const long long resident = at_once * blocks > sms ? 2 : 1, full = tiles / at_once, rest = (tiles % at_once) * blocks;   // blocks to an SM; rounds; blocks of the last, partial one
    const long long last = rest == 0 ? 0 : rest > sms * (resident - 1) ? resident : 1;
    const double k = std::min(a.K, leaf_length(a.K) * (LEAVES / blocks)) / 1000.0, results = TM * TN;   // a short k is not shared by all blocks
    *cost = (double)(full * resident + last) * (1.4 * results + 0.78 * (TM + TN) + 5.9) * k + (double)(full + (rest ? 1 : 0)) * (0.31 * results - 2.7) +
            (last == 1 ? 0.25 * results * k : 0.0) + 7.3;
    return 0;
  }
  launch_dependent_cluster<LAUNCH_GEMM>(kernel, dim3((unsigned)(tiles_n * blocks), (unsigned)tiles_m, batch), dim3(256), Shape::smem(blocks), stream,
                                        (unsigned)blocks, a);
  PYLON_CHECK_LAUNCH("gemm_f32");
}

// The estimate is a least-squares fit to 580 launches of stages of 16 k (32 to 320 rows of the four matrices of the Qwen3-4B shape, all tiles and
// cluster sizes).  With stages of 32 all tiles became faster alike: it is 14 % too long on average, but of 48 such sizes (17 to 320 rows, all tiles timed again)
// the tile it picks is within 1.1 % of the fastest on average, 19 % at worst ([256, 9728] x [2560, 9728]), and of 160 others (17 to 2,048 rows, 64 to 32,000 weight rows,
// k from 16 to 2,556) 7 % behind it on average.  A fit to all of these launches picks 1.5 % better on average and up to 40 % worse (960 rows of [249, 424]).  What it weighs: results
// and reads per four k, rounds of blocks (a lone block in the last round runs faster than two that share an SM), the sum across blocks.
typedef int (*TileEntry)(const GemmArgs&, int, int, cudaStream_t, double*);

static int launch_tile(const GemmArgs& a, int batch, bool aligned, int force, cudaStream_t stream) {
  static const struct { int tm, tn; TileEntry entry; } wide[] = {
      {2, 8, tile_kernel<2, 8, 4>}, {3, 5, tile_kernel<3, 5, 4>}, {3, 6, tile_kernel<3, 6, 4>}, {4, 5, tile_kernel<4, 5, 4>}, {4, 6, tile_kernel<4, 6, 4>},
      {4, 7, tile_kernel<4, 7, 4>}, {5, 5, tile_kernel<5, 5, 4>}, {6, 5, tile_kernel<6, 5, 4>}, {7, 4, tile_kernel<7, 4, 4>}, {7, 5, tile_kernel<7, 5, 4>}},
                      narrow[] = {{4, 4, tile_kernel<4, 4, 1>}};   // rows that 16-byte copies do not reach
  const auto* best = aligned ? wide : narrow;
  const auto* end = aligned ? wide + sizeof(wide) / sizeof(wide[0]) : narrow + 1;
  int best_blocks = 1;
  double least = -1.0;
  for (const auto* candidate = best; candidate != end; ++candidate)
    for (int blocks = 1; blocks <= 8; blocks *= 2) {
      double cost = 0.0;
      const int code = candidate->entry(a, batch, blocks, stream, &cost);
      if (code != 0) return code;
      if (force && force != candidate->tm * 100 + candidate->tn * 10 + blocks) continue;
      if ((a.M + 16 * candidate->tm - 1) / (16 * candidate->tm) > 65535) continue;
      if (least < 0.0 || cost < least) { least = cost; best = candidate; best_blocks = blocks; }
    }
  if (least < 0.0) PYLON_REFUSE("gemm_f32: no tile %d for these operands", force);
  return best->entry(a, batch, best_blocks, stream, nullptr);
}

constexpr int ROWS_MOST = 16;

static int launch_short(const GemmArgs& a, int batch, cudaStream_t stream) {
  launch_dependent<LAUNCH_GEMM>(gemm_f32_short_kernel, dim3((a.N + 63) / 64, (a.M + 63) / 64, batch), dim3(256), 0, stream, a);
  PYLON_CHECK_LAUNCH("gemm_f32");
}

static int gemm_f32(const GemmArgs& a, int batch, int force, cudaStream_t stream) {
  const bool aligned = a.K % 4 == 0 && a.ldx % 4 == 0 && a.ldw % 4 == 0 && a.batch_x % 4 == 0 && a.batch_w % 4 == 0 &&
                       (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.w) & 15) == 0;
  if (force == -4 && a.K <= SHORT_MOST) return launch_short(a, batch, stream);
  if (force < -2) PYLON_REFUSE("gemm_f32: no form %d", force);
  if (force > 0) return launch_tile(a, batch, aligned, force, stream);
  if (force == 0) {
    const long long slabs = (long long)((a.N + 63) / 64) * batch;
    // Few rows stream the weights whatever k is (one row of [6144, 128]: 4.0 us, the short kernel 8.2), up to 8 of them, or 4 where k is so
    // short or so placed that a lane's copies are more than its sums (5 rows of [512, 32]: 3.7 and 3.1; of [512, 64]: 4.5 and 4.6).
    const bool few = a.M <= (aligned && a.K > 32 ? 8 : 4);
    // Short k: always up to 64 (64 rows of [6144, 64] 5.7 us, tile kernel 6.2; 16 of [1000, 64] 4.9 and 5.7); up to 128 where 16-byte copies do not reach
    // (300 rows of [1000, 65] 6.3 and 6.9) or a grid of few rows is many blocks (64 rows of [2560, 128] level at 9.2, but of [512, 128] 9.2 and 6.7).
    if (!few && (a.K <= 64 || (a.K <= SHORT_MOST && (!aligned || (a.M <= 64 && slabs >= 64))))) return launch_short(a, batch, stream);
    // 9 to 16 rows stream the weights where there are enough of them for lone blocks (12 rows of [9728, 300] 15.2 us, tile kernel 19.7) or a long
    // k over a large matrix (12 of [2560, 2560] 20.0 and 24.8); else the tile kernel's clusters end sooner (16 of [1000, 512] 9.0 and 6.5).
    const bool streams = a.M <= ROWS_MOST && (slabs * a.M >= LONE_WORK || (aligned && a.K < 512 && slabs >= 64) || (a.K >= 512 && slabs * 64 * a.K >= 1 << 20));
    if (!few && !streams) return launch_tile(a, batch, aligned, 0, stream);
  }
  return aligned ? dispatch_rows<4>(a, batch, force < 0 ? -force : 0, stream) : dispatch_rows<1>(a, batch, force < 0 ? -force : 0, stream);
}

}  // namespace pylon

// w_static: 1 where nothing queued on the stream writes w; its first columns are then asked for while the kernel ahead is still running.
extern "C" int pylon_gemm_f32_nt(const float* x, const float* w, float* y, int M, int N, int K, long long ldx,
                                 long long ldw, long long ldy, int w_static, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) PYLON_REFUSE("gemm_f32: K = %d", K);
  if (ldx < K || ldw < K || ldy < N) PYLON_REFUSE("gemm_f32: a leading dimension is shorter than its row");
  if ((M + 63) / 64 > 65535) PYLON_REFUSE("gemm_f32: M = %d is too large", M);
  return pylon::gemm_f32({x, w, y, M, N, K, ldx, ldw, ldy, 0, 0, 0, w_static}, 1, 0, stream);
}

// `batch` products of one shape in one launch: y_b[M, N] = x_b[M, K] * W_b[N, K]^T, the operands of product b lying
// b * batch_x / batch_w / batch_y elements behind the first (a head's slice of a row, say: batch_x = the head's width, ldx = the row's).
extern "C" int pylon_gemm_f32_nt_batched(const float* x, const float* w, float* y, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                                         int batch, long long batch_x, long long batch_w, long long batch_y, int w_static, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K <= 0) PYLON_REFUSE("gemm_f32_batched: K = %d", K);
  if (ldx < K || ldw < K || ldy < N) PYLON_REFUSE("gemm_f32_batched: a leading dimension is shorter than its row");
  if ((M + 63) / 64 > 65535 || batch > 65535) PYLON_REFUSE("gemm_f32_batched: M = %d, batch = %d", M, batch);
  return pylon::gemm_f32({x, w, y, M, N, K, ldx, ldw, ldy, batch_x, batch_w, batch_y, w_static}, batch, 0, stream);
}

// For measurements and tests: the kernel for few rows (force = -1: clusters of eight blocks, -2: lone blocks) or a tile kernel
// (100 TM + 10 TN + cluster size; 0: the choice by size).  What is not there for the operands is refused.
extern "C" int pylon_gemm_f32_nt_forced(const float* x, const float* w, float* y, int M, int N, int K, long long ldx,
                                        long long ldw, long long ldy, int force, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || ldx < K || ldw < K || ldy < N || (M + 15) / 16 > 65535 || (force < 0 && force != -4 && M > pylon::ROWS_MOST)) PYLON_REFUSE("gemm_f32_forced: M = %d, K = %d", M, K);
  return pylon::gemm_f32({x, w, y, M, N, K, ldx, ldw, ldy, 0, 0, 0, 0}, 1, force, stream);
}
