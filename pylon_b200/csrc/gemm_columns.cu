// The gated unit of a feed-forward in bfloat16 for a few rows of x on the fifth-generation tensor cores, with the weights on the wide side of the tile:
// 128 interleaved rows of gate and up are the M of a tcgen05.mma and the rows of x, rounded up to 16, its N.
//
// Bound by the bytes of W: 16 rows of [34816, 5120] and the norm ahead of them 62.2 us (356 MB: 5.7 TB/s and more), where the kernel that multiplies with mma.sync
// from registers (gemm_stream.cu) takes 66.6 us, its warps busy with fragments; 32 rows 62.9 and 77.7 us.  The products' dispatch sends it 9 to 32 rows; it takes up to 256,
// those above 32 with one set of accumulators.  A block takes 128 rows of W over the whole of k; two share an
// SM, so that one's epilogue overlaps the other's loads.  Six warps: one lane of the fifth asks for boxes of W and x (TMA, 128-byte
// swizzle) into a ring of stages - the boxes of W that nothing queued writes before it waits for the kernel ahead - one lane of the next issues the
// products, and the first four read the accumulators back, each its 32 lanes, a lane being a row of W.
//
// Measured and dropped: partial sums over slices of k for the products into the stream and the rotation (33 to 200 rows: 6.4 us for the 4B shape's output
// projection of 64 rows where the library takes 8.4, 10.6 and 14.9 for the down projection; but the norm that adds 14 parts up lost what they gained: steps of
// 64 to 190 tokens 2 % faster to 10 % slower); slices added up in a cluster (2.5 to 4 us more than partial sums) or by the last block of a tile (9 to 60 us).
//
// The tensor core cuts off what a sum drops instead of rounding it, so a long chain's error grows with k.  The steps of 16 k take turns on several
// accumulators beside each other in tensor memory, and up to 32 rows of x two sets of them take turns, 512 k each (1,024 up to 16 rows): while one is filled the readers add the
// other up in float32, so that no chain is longer than eight steps whatever k is.  Elements that are not the rounded 64-bit result: 32 rows of [34816, 5120] 2.3e-4
// of them, with one set of chains over the whole of k 7.1e-4, gemm_stream.cu 3.8e-4; 24 of [37888, 8192] 2.8e-4, 12.3e-4 and 3.8e-4.  It costs 0.2 % of the time up to 16 rows, 1 % above.
//
// All waits on mbarriers are bounded: one that runs out sets an error word, the block waits for its own copies, frees its tensor memory and returns.
// No TMA load here uses cluster multicast.
//
// Stands in for the first half of raun6k/Pylon's feed-forward (src/pylon/model/layers.py:13-27).
#include "common.cuh"

#include <cuda.h>

#include <algorithm>
#include <functional>
#include <mutex>
#include <unordered_map>

namespace pylon {

constexpr int GC_ROWS = 128, GC_BK = 64, GC_THREADS = 192, GC_MOST_STAGES = 8;   // weight rows and k of a box
constexpr int GC_COLUMNS = 256;                                                             // of tensor memory: two blocks to an SM
constexpr int GC_SETS_MOST = 32, GC_SEGMENT = 8;                                  // columns up to which two sets of accumulators take turns; boxes to a turn of so many
constexpr unsigned GC_WAIT_LIMIT = 1u << 22;                                                 // try_wait calls before a wait gives up

__device__ __forceinline__ uint32_t gc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gc_mbar_init(uint64_t* bar, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(gc_smem(bar)), "r"(count)); }
__device__ __forceinline__ void gc_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(gc_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gc_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(gc_smem(bar)) : "memory"); }
__device__ __forceinline__ bool gc_wait(uint64_t* bar, uint32_t parity) {
  for (unsigned tries = 0; tries < GC_WAIT_LIMIT; ++tries) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(gc_smem(bar)), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void gc_load(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(gc_smem(dst)), "l"((uint64_t)map), "r"(gc_smem(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void gc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(gc_smem(bar)) : "memory");
}
__device__ __forceinline__ void gc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// 16 consecutive float32 columns of this thread's lane of tensor memory; valid after gc_read_done().
__device__ __forceinline__ void gc_read(uint32_t address, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                 "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(address));
}
__device__ __forceinline__ void gc_read_done() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// A K-major tile whose rows are 128 bytes in the 128-byte swizzle: start address, 1024 bytes between groups of 8 rows, version 1, swizzle 128B.
__device__ __forceinline__ uint64_t gc_desc(const void* tile) {
  return (uint64_t)((gc_smem(tile) & 0x3FFFF) >> 4) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ float gc_unit(float gate, float up, float limit, float alpha) {
  float gain = 1.f;
  if (limit > 0.f) {   // the clamped unit: min(gate, limit) * sigmoid(alpha * gate) * (clamp(up, -limit, limit) + 1)
    gate = fminf(gate, limit);
    up = fminf(fmaxf(up, -limit), limit) + 1.f;
    gain = alpha;
  }
  return __fdividef(gate, 1.f + __expf(-gain * gate)) * up;   // approximate division: ample for bfloat16, no slow path
}
struct GcArgs {
  __nv_bfloat16* y;
  long long ldy;
  int M, N, K, columns, stages, chains, segment, tmem_columns;   // columns: M rounded up to 16; chains of a set: a power of two; segment: boxes to a set's turn
  float unit_limit, unit_alpha;
  int w_static;
  int* error;   // 1: the copies, 2: the products, 3: the accumulator did not come in time
};

// Grid (tiles of 128 weight rows).
__global__ void __launch_bounds__(GC_THREADS) gemm_columns_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const GcArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[GC_MOST_STAGES], empty[GC_MOST_STAGES], filled[2], freed[2];   // freed: a set has been read
  __shared__ uint32_t tmem_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int columns = a.columns, stages = a.stages, w_bytes = GC_ROWS * GC_BK * 2, x_bytes = columns * GC_BK * 2;
  unsigned char* w_tiles = smem;
  unsigned char* x_tiles = smem + stages * w_bytes;
  const int boxes = (a.K + GC_BK - 1) / GC_BK, row0 = blockIdx.x * GC_ROWS;
  const int chains = a.chains, segment = a.segment, segments = (boxes + segment - 1) / segment;   // more than one only where there are two sets

  const int ahead = a.w_static ? min(stages, boxes) : 0;
  if (warp == 4 && lane == 0) {
    for (int s = 0; s < stages; ++s) { gc_mbar_init(&full[s], 1); gc_mbar_init(&empty[s], 1); }
    for (int set = 0; set < 2; ++set) { gc_mbar_init(&filled[set], 1); gc_mbar_init(&freed[set], 4); }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    for (int s = 0; s < ahead; ++s) {
      gc_expect(&full[s], w_bytes + x_bytes);
      gc_load(w_tiles + s * w_bytes, &map_w, &full[s], s * GC_BK, row0);
    }
  }
  if (warp == 5) {   // the whole warp allocates
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(gc_smem(&tmem_slot)), "r"(a.tmem_columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;
  grid_dependency_wait();
  allow_dependents();

  if (warp == 4) {
    if (lane == 0) {
      int issued = 0;   // boxes asked for
      for (int s = 0, round = 0; issued < boxes; ++issued) {
        if (issued >= ahead) {
          if (round > 0 && !gc_wait(&empty[s], (round - 1) & 1)) { atomicExch(a.error, 1); break; }
          gc_expect(&full[s], w_bytes + x_bytes);
          gc_load(w_tiles + s * w_bytes, &map_w, &full[s], issued * GC_BK, row0);
        }
        gc_load(x_tiles + s * x_bytes, &map_x, &full[s], issued * GC_BK, 0);
        if (++s == stages) { s = 0; ++round; }
      }
      for (int box = max(0, issued - stages); box < issued; ++box) gc_wait(&full[box % stages], (box / stages) & 1);   // no copy outlives the block
    }
    __syncwarp();
  } else if (warp == 5) {
    if (lane == 0) {
      // Instruction descriptor of kind::f16: bfloat16 A and B, float32 D, both K-major.
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(columns >> 3) << 17) | ((uint32_t)(GC_ROWS >> 4) << 24);
      const uint64_t w_first = gc_desc(w_tiles), x_first = gc_desc(x_tiles);
      int s = 0, phase = 0, box = 0;
      for (int turn = 0; turn < segments; ++turn) {
        const int set = turn & 1, end = min(boxes, box + segment);
        const uint32_t d = tmem + set * chains * columns;
        if (turn >= 2 && !gc_wait(&freed[set], ((turn >> 1) - 1) & 1)) { atomicExch(a.error, 2); break; }
        bool alive = true;
        for (int step = 0, offset = 0; box < end; ++box) {
          if (!gc_wait(&full[s], phase)) { atomicExch(a.error, 2); alive = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint64_t w_desc = w_first + (uint64_t)(s * (w_bytes >> 4)), x_desc = x_first + (uint64_t)(s * (x_bytes >> 4));
#pragma unroll
          for (int k = 0; k < GC_BK / 16; ++k) {   // 16 k are 32 bytes further along the swizzled row: +2 in 16-byte units
            gc_mma(d + offset, w_desc + 2 * k, x_desc + 2 * k, idesc, step >= chains);
            ++step;
            offset += columns;
            if (offset == chains * columns) offset = 0;
          }
          gc_commit(&empty[s]);
          if (++s == stages) { s = 0; phase ^= 1; }
        }
        if (!alive) break;
        gc_commit(&filled[set]);
      }
    }
    __syncwarp();
  } else {
    // This thread's row of W and, 16 rows of x at a time, its sums: the chains' in order.  Rows of gate and up alternate in groups of 8: lanes 8 apart exchange,
    // the gate's lane then makes the even rows of x, the up's the odd ones.
    const int n = row0 + threadIdx.x, is_up = (lane >> 3) & 1;
    const uint32_t lane_address = tmem + ((uint32_t)(warp * 32) << 16);
    auto add_up = [&](float (&v)[16], int turn, int c0) {
      const int count = min(chains, 4 * min(segment, boxes - turn * segment));   // a last turn of few steps fills the first chains only
      for (int c = 0; c < count; ++c) {
        uint32_t raw[16];
        gc_read(lane_address + ((turn & 1) * chains + c) * columns + c0, raw);
        gc_read_done();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(raw[j]);
      }
    };
    auto finish = [&](const float (&v)[16], int c0) {
      __nv_bfloat16* dst = a.y + (size_t)(c0 + is_up) * a.ldy + (n >> 4) * 8 + (n & 7);
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, is_up ? v[j] : v[j + 1], 8);
        const float unit = is_up ? gc_unit(other, v[j + 1], a.unit_limit, a.unit_alpha) : gc_unit(v[j], other, a.unit_limit, a.unit_alpha);
        if (n < a.N && c0 + j + is_up < a.M) dst[(size_t)j * a.ldy] = __float2bfloat16_rn(unit);
      }
    };
    bool complete = true;
    if (columns <= GC_SETS_MOST) {
      float sums[GC_SETS_MOST / 16][16] = {};
      for (int turn = 0; complete && turn < segments; ++turn) {
        complete = __all_sync(0xffffffffu, gc_wait(&filled[turn & 1], (turn >> 1) & 1));
        if (!complete) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
        for (int t = 0; t < GC_SETS_MOST / 16; ++t)
          if (16 * t < columns) add_up(sums[t], turn, 16 * t);
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) gc_arrive(&freed[turn & 1]);
      }
#pragma unroll
      for (int t = 0; t < GC_SETS_MOST / 16; ++t)
        if (complete && 16 * t < columns) finish(sums[t], 16 * t);
    } else {
      complete = __all_sync(0xffffffffu, gc_wait(&filled[0], 0));
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      for (int c0 = 0; complete && c0 < columns; c0 += 16) {
        float sums[16] = {};
        add_up(sums, 0, c0);
        finish(sums, c0);
      }
    }
    if (!complete && lane == 0) atomicExch(a.error, 3);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(a.tmem_columns));
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Tensor map of a row-major bfloat16 matrix [rows, cols] (row stride ld elements) with boxes of box_rows x 64 columns in the 128-byte
// swizzle.  Maps are kept by all their arguments (they are a function of them): a model multiplies by the same matrices at every step.
static bool matrix_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
  struct Key {
    const void* base; long long rows, cols, ld; int box_rows;
    bool operator==(const Key& o) const { return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows; }
  };
  struct Hash {
    size_t operator()(const Key& k) const { return std::hash<const void*>()(k.base) ^ (size_t)(k.rows * 1315423911LL) ^ (size_t)(k.cols * 2654435761LL) ^ (size_t)k.box_rows; }
  };
  static std::unordered_map<Key, CUtensorMap, Hash> known;
  static std::mutex mutex;
  static EncodeTiled encode = nullptr;
  std::lock_guard<std::mutex> guard(mutex);
  if (!encode) {
    void* symbol = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &symbol, cudaEnableDefault, &result) != cudaSuccess || result != cudaDriverEntryPointSuccess) return false;
    encode = (EncodeTiled)symbol;
  }
  const Key key{base, rows, cols, ld, box_rows};
  auto found = known.find(key);
  if (found != known.end()) { *map = found->second; return true; }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)GC_BK, (cuuint32_t)box_rows};
  cuuint32_t element_strides[2] = {1, 1};
  if (encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (known.size() >= 4096) known.clear();   // activations come and go; the weights' maps are made again on demand
  known.emplace(key, *map);
  return true;
}

constexpr int GC_SMEM = 112 * 1024;   // two blocks to an SM: the next kernel's move in beside the last of this one's and ask for their weights

}  // namespace pylon

// The gated unit of x gate^T and x up^T: x bfloat16 [M, K] (row stride ldx), M <= 256; w bfloat16 [N, K] (row stride ldw), its rows interleaved in groups of
// 8 (rows 16b..16b+7 gate rows 8b..8b+7, rows 16b+8..16b+15 the matching up rows; N a multiple of 16); y bfloat16 [M, N / 2], row stride ldy.  limit 0:
// silu(gate) * up; limit > 0: the clamped unit, min(gate, limit) * sigmoid(alpha * min(gate, limit)) * (clamp(up, -limit, limit) + 1).  K and the
// operands' row strides multiples of 8, x and w 16-byte aligned.  error: one int in device memory that the kernel sets non-zero if one of its waits ran
// out (the result is then void).  w_static: 1 where nothing queued on the stream writes w; its first boxes are then asked for while the kernel ahead is
// still running.
extern "C" int pylon_gemm_columns_gated(const void* x, const void* w, void* y, int M, int N, int K, long long ldx, long long ldw, long long ldy, float limit,
                                        float alpha, int* error, int w_static, cudaStream_t stream) {
  using namespace pylon;
  if (M <= 0 || N <= 0) return 0;
  if (M > 256) PYLON_REFUSE("gemm_columns_gated: M = %d is more than 256 rows", M);
  if (N % 16 || ldy < N / 2) PYLON_REFUSE("gemm_columns_gated: N = %d must be a multiple of 16 and the result N / 2 columns wide", N);
  if (!(limit >= 0.f)) PYLON_REFUSE("gemm_columns_gated: the limit must be positive, or 0 for none");
  if (K <= 0 || K % 8 || ldx % 8 || ldw % 8) PYLON_REFUSE("gemm_columns_gated: K = %d and the row strides must be multiples of 8", K);
  if (((uintptr_t)x % 16) || ((uintptr_t)w % 16) || ((uintptr_t)y % 2)) PYLON_REFUSE("gemm_columns_gated: x and w must be 16-byte aligned");
  if (ldx < K || ldw < K) PYLON_REFUSE("gemm_columns_gated: a row stride is shorter than its row");
  if (!error) PYLON_REFUSE("gemm_columns_gated: an error word is needed");
  static bool configured_on[MAX_DEVICES] = {};   // function attributes belong to a device
  bool& configured = configured_on[current_device_slot()];
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(gemm_columns_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GC_SMEM);
    if (err != cudaSuccess) PYLON_REFUSE("gemm_columns_gated: %s", cudaGetErrorString(err));
    configured = true;
  }
  GcArgs a;
  a.y = (__nv_bfloat16*)y; a.ldy = ldy; a.M = M; a.N = N; a.K = K;
  a.columns = (M + 15) / 16 * 16;
  const int boxes = (K + GC_BK - 1) / GC_BK, stage_bytes = (GC_ROWS + a.columns) * GC_BK * 2;
  a.stages = std::min({(GC_SMEM - 1024) / stage_bytes, GC_MOST_STAGES, boxes});
  const int sets = a.columns <= GC_SETS_MOST ? 2 : 1;
  a.segment = sets == 2 ? GC_SEGMENT * (GC_SETS_MOST / a.columns) : boxes;
  a.chains = 1;
  while (2 * a.chains * sets * a.columns <= GC_COLUMNS && 2 * a.chains <= std::min(a.segment, boxes) * (GC_BK / 16)) a.chains *= 2;
  a.tmem_columns = 32;
  while (a.tmem_columns < sets * a.chains * a.columns) a.tmem_columns *= 2;
  a.unit_limit = limit; a.unit_alpha = alpha; a.w_static = w_static; a.error = error;
  CUtensorMap map_w, map_x;
  if (!matrix_map(&map_w, w, N, K, ldw, GC_ROWS) || !matrix_map(&map_x, x, M, K, ldx, a.columns)) PYLON_REFUSE("gemm_columns_gated: the tensor maps could not be made");
  launch_dependent<LAUNCH_GEMM>(gemm_columns_kernel, dim3((N + GC_ROWS - 1) / GC_ROWS), dim3(GC_THREADS), (size_t)a.stages * stage_bytes + 1024, stream, map_w, map_x, a);
  PYLON_CHECK_LAUNCH("gemm_columns_gated");
}
