// The experts' grouped matrix products in bfloat16 on the fifth-generation tensor cores (float32 sums): the tiles of the
// plan that expert_plan_kernel makes (csrc/experts.cu), up to 16, 32, 64, 128 or 256 sorted rows of one expert each.
//   mode 0: x rows are gathered from h by token; gate and up rows of the expert's matrix;
//           out[row, f] = silu(gate) * up (glu_limit > 0: the clamped unit, gated_unit), bfloat16.
//   mode 1: x rows are the sorted rows themselves; out[row, n] float32.
//   mode 2: x rows gathered as in mode 0, plain matrix rows; out[row, n] = act(row_scale[pair] * sum), bfloat16
//           (an expert without a gate; with row_scale its input is the token's row times the pair's weight).
// A row's sums do not depend on its place in a tile or on the other rows.
//
// What bounds it: the experts' matrices are read once from memory, and what crosses from L2 into an SM for a tile (a block's
// matrix rows and its x rows). So the product is formed transposed: 128 matrix rows (mode 0: 128 gate rows and the 128 up
// rows of the same columns) are the M side of tcgen05.mma, the tile's x rows, rounded up to 16, are the N side, and a tile
// holds all rows of an expert where it can: the matrix crosses once, whatever the number of rows, and nothing is
// computed for padding beyond 15 rows. Accumulators [128 x rows] (two in mode 0) live in tensor memory.
//   warp 0       one thread: per 64 values of k the boxes of 128 matrix rows by TMA (128-byte swizzle) into a ring of stages
//   warp 1       one thread: per stage four (mode 0: eight) matrix instructions of 16 k, tcgen05.commit on the "empty" barrier
//   warps 2 - 9  the x rows: cp.async of 16-byte chunks from rows found through the plan, to their swizzled places, each
//                thread's arrival at the "full" barrier made by the copies themselves when they have landed. Then the
//                epilogue: a warp reads its quarter of the lanes (a lane is a matrix row), every other group of eight x rows.
// Every wait on a barrier is bounded: when one runs out, the error flag is raised and the block carries on to its end without
// waiting again.
//
// One B200, 64 experts of 1,408, width 2,048: 12,288 rows (about 192 an expert, tiles of 256) gate and up 491 -> 204 us
// (695 TFLOP/s), down 263 -> 114 us; 48 rows (tiles of 16) 88 -> 70 and 45 -> 35 us (5.7 TB/s of the matrices of the experts
// in use); before, 64 x 128 tiles on mma.sync. With many rows nothing is saturated (tensor pipe 38 %, memory 52 %): the rings hold too
// little of the way from memory (192 rows: three stages of 56 KB for gate and up; two of 40 KB in each of two blocks for down). Boxes asked into L2 eight stages ahead changed nothing there
// and cost a third with few rows (67 -> 90 us).
#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int XM = 128;                    // matrix rows of a box = M of the matrix instruction
constexpr int XK = 64;                     // k per stage: 128 bytes, one swizzle row
constexpr int X_BOX_BYTES = XM * XK * 2;   // 16 KB
constexpr int X_MAX_STAGES = 6;
constexpr int X_GATHER = 256;              // threads of warps 2 - 9

__device__ __forceinline__ void copy16_or_zero(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0));
}
// an arrival of this thread at `bar` (counted in its initial count) once all its copies so far have landed
__device__ __forceinline__ void arrive_when_copied(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

struct ExpertTcParams {
  const __nv_bfloat16* x;
  void* out;
  const int* plan;
  const float* row_scale;
  int* error_flag;
  int pairs, max_tiles, top, N, K, act;
  int tile_rows;            // most rows of a tile
  int ring_bytes, acc2;     // shared memory for stages; tensor-memory column of the second accumulator
  int tmem_cols;
  float glu_limit, glu_alpha;
};

template <int MODE>
__global__ void __launch_bounds__(64 + X_GATHER)
expert_linear_tc_kernel(const __grid_constant__ CUtensorMap w_map, const ExpertTcParams p) {
  pdl_entry();
  const int tile = blockIdx.y;
  if (tile >= p.plan[0]) return;
  constexpr int BOXES = MODE == 0 ? 2 : 1;
  const int expert = p.plan[1 + tile], row0 = p.plan[1 + p.max_tiles + tile], rows = p.plan[1 + 2 * p.max_tiles + tile];
  const int* pair_of_row = p.plan + 1 + 3 * p.max_tiles + p.pairs;
  const int n16 = (rows + 15) / 16 * 16;
  extern __shared__ unsigned char smem_dyn[];
  // 1024-byte alignment: the swizzle pattern is a function of address bits 4..9
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  // the ring is cut by this tile's rows: fewer rows, more stages in flight
  const int stage_bytes = BOXES * X_BOX_BYTES + n16 * XK * 2;   // a multiple of 1024
  const int stages = min(X_MAX_STAGES, p.ring_bytes / stage_bytes);
  __shared__ uint64_t bars[2 * X_MAX_STAGES + 1];   // full[stages], empty[stages], accumulators complete
  __shared__ uint32_t tmem_slot;
  __shared__ int alive_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * XM;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[X_MAX_STAGES]), bar_done = smem_u32(&bars[2 * X_MAX_STAGES]);
  const uint32_t ring0 = smem_u32(ring);
  const int n_iter = (p.K + XK - 1) / XK;
  if (tid == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full0 + 8 * s, 1 + X_GATHER);     // the TMA thread's arrival and each gathering thread's
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(bar_done, 1);
    alive_s = 1;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "r"(p.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      const int wrow = expert * BOXES * p.N + m0;      // rows past an expert's own come along and are not stored
      uint32_t st = 0, parity = 1;                     // parity of the round before
      int i = 0;
      for (; i < n_iter; ++i) {
        const uint32_t full = full0 + 8 * st, base = ring0 + st * stage_bytes;
        if (i >= stages && !mbar_wait(empty0 + 8 * st, parity, p.error_flag, 31)) break;
        mbar_expect_tx(full, uint32_t(BOXES * X_BOX_BYTES));   // a box delivers all its bytes, zeros where out of range
        tma_load_2d(base, &w_map, i * XK, wrow, full);
        if (MODE == 0) tma_load_2d(base + X_BOX_BYTES, &w_map, i * XK, wrow + p.N, full);
        if (++st == uint32_t(stages)) { st = 0; parity ^= 1; }
      }
      // the copies in flight land before the block ends, also where a wait ran out (bounded waits again)
      for (int j = max(0, i - stages); j < i; ++j) mbar_wait(full0 + 8 * (j % stages), (j / stages) & 1, p.error_flag, 31);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(XM, n16, false);
      const uint64_t desc0 = smem_desc(ring0, 16, 1024);
      const uint64_t step = uint64_t(stage_bytes >> 4), x_off = uint64_t((BOXES * X_BOX_BYTES) >> 4), up_off = uint64_t(X_BOX_BYTES >> 4);
      uint32_t st = 0, parity = 0;
      bool alive = true;
      for (int i = 0; i < n_iter; ++i) {
        alive = mbar_wait(full0 + 8 * st, parity, p.error_flag, 32);
        if (!alive) break;
        proxy_fence_async();      // the x rows came by ordinary copies; the matrix instructions read them through the other proxy
        tc_fence_after();
        const uint64_t d = desc0 + st * step;
        tc_mma4(tmem_base, d, d + x_off, idesc, i > 0 ? 1u : 0u);
        if (MODE == 0) tc_mma4(tmem_base + p.acc2, d + up_off, d + x_off, idesc, i > 0 ? 1u : 0u);
        tc_commit(empty0 + 8 * st);
        if (++st == uint32_t(stages)) { st = 0; parity ^= 1; }
      }
      if (alive) {
        tc_commit(bar_done);
        alive = mbar_wait(bar_done, 0, p.error_flag, 33);
      }
      if (!alive) alive_s = 0;
    }
    __syncwarp();
  } else {
    const int gt = tid - 64, c = gt % 8;      // chunk c (8 values) of rows gt / 8 + 32 j
    const __nv_bfloat16* src[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = gt / 8 + 32 * j;
      src[j] = nullptr;
      if (r < rows) src[j] = p.x + size_t(MODE == 1 ? row0 + r : pair_of_row[row0 + r] / p.top) * p.K + c * 8;
    }
    const uint32_t dst0 = ring0 + BOXES * X_BOX_BYTES + (gt / 8) * 128 + ((c ^ ((gt / 8) & 7)) << 4);
    uint32_t st = 0, parity = 1;
    for (int i = 0; i < n_iter; ++i) {
      if (i >= stages && !mbar_wait(empty0 + 8 * st, parity, p.error_flag, 34)) break;
      const bool k_ok = i * XK + c * 8 < p.K;
      const uint32_t dst = dst0 + st * stage_bytes;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (gt / 8 + 32 * j < n16)
          copy16_or_zero(dst + j * 4096, src[j] && k_ok ? src[j] + i * XK : p.x, src[j] && k_ok);
      arrive_when_copied(full0 + 8 * st);
      if (++st == uint32_t(stages)) { st = 0; parity ^= 1; }
    }
    cp_async_wait_all();
  }
  __syncthreads();
  tc_fence_after();

  // -------------------------------------------------------------------- epilogue
  if (warp >= 2 && alive_s) {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int f = m0 + quarter * 32 + lane;      // output column = lane of tensor memory
    const uint32_t lane_addr = tmem_base + (uint32_t(quarter * 32) << 16);
    for (int g = half; g * 8 < n16; g += 2) {
      float v[8];
      tmem_ld8(lane_addr + g * 8, v);
      if (MODE == 1) {
        float* o = reinterpret_cast<float*>(p.out) + size_t(row0 + g * 8) * p.N + f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (g * 8 + j < rows && f < p.N) o[size_t(j) * p.N] = v[j];
        continue;
      }
      if (MODE == 0) {
        float u[8];
        tmem_ld8(lane_addr + p.acc2 + g * 8, u);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = gated_unit(v[j], u[j], p.glu_limit, p.glu_alpha);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int r = g * 8 + j;
          const float rs = (p.row_scale && r < rows) ? p.row_scale[pair_of_row[row0 + r]] : 1.f;
          v[j] = apply_activation(v[j] * rs, p.act);
        }
      }
      // two rows at a time: an even lane stores columns f, f + 1 of the first, the odd lane above it those of the second
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + size_t(row0 + g * 8 + (lane & 1)) * p.N + (f & ~1);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? v[j] : v[j + 1], 1);
        const uint32_t word = (lane & 1) ? pack_bf16(other, v[j + 1]) : pack_bf16(v[j], other);
        if (g * 8 + j + (lane & 1) < rows && f < p.N) *reinterpret_cast<uint32_t*>(o + size_t(j) * p.N) = word;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(p.tmem_cols));
}

// a [rows, K] bfloat16 row-major matrix in boxes of 128 rows x 64 k, written with the 128-byte swizzle
bool make_expert_map(CUtensorMap* map, const void* base, long long rows, int K) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  if (!encode) return false;
  const cuuint64_t dims[2] = {cuuint64_t(K), cuuint64_t(rows)};
  const cuuint64_t strides[1] = {cuuint64_t(K) * 2};
  const cuuint32_t box[2] = {cuuint32_t(XK), cuuint32_t(XM)};
  const cuuint32_t elem[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE>
int launch_expert_tc(const CUtensorMap& map, ExpertTcParams p, cudaStream_t stream) {
  constexpr int BOXES = MODE == 0 ? 2 : 1;
  p.acc2 = p.tile_rows < 32 ? 32 : p.tile_rows;
  p.tmem_cols = BOXES * p.acc2;
  const int most = BOXES * X_BOX_BYTES + p.tile_rows * XK * 2;     // a stage of the largest tile
  // two blocks an SM where tensor memory holds both and two stages fit into half of its shared memory (one's start and
  // epilogue under the other's products: down, tiles of 256, 142 -> 114 us), else one block with what the SM has
  p.ring_bytes = (p.tmem_cols <= 256 && 2 * most <= 110 * 1024) ? 110 * 1024 : 222 * 1024;
  const size_t smem = 1024 + size_t(p.ring_bytes);
  static SharedLimit limit;
  if (!limit.allows(expert_linear_tc_kernel<MODE>, smem)) return PTB_ERR_LAUNCH;
  launch_pdl(expert_linear_tc_kernel<MODE>, dim3((p.N + XM - 1) / XM, p.max_tiles), 64 + X_GATHER, smem, stream, map, p);
  return launch_status();
}

}  // namespace

// `tile_rows`: 16, 32, 64, 128 or 256, the most rows of the plan's tiles; K and N multiples of 8. `error_flag`: a device int
// that stays 0 unless a bounded wait inside the kernel ran out.
PTB_API int ptb_expert_linear_tc(int mode, const void* x, const void* w, void* out, const int* plan, int pairs, int max_tiles,
                                 int top, int n_experts, int N, int K, int tile_rows, const float* row_scale, int act,
                                 float glu_limit, float glu_alpha, int* error_flag, cudaStream_t stream) {
  if (pairs <= 0 || max_tiles <= 0) return PTB_OK;
  if (N <= 0 || K <= 0 || K % 8 != 0 || N % 8 != 0 || max_tiles > 65535 || top <= 0 || n_experts <= 0 || mode < 0 || mode > 2 ||
      (tile_rows != 16 && tile_rows != 32 && tile_rows != 64 && tile_rows != 128 && tile_rows != 256) ||
      !activation_known(act) || error_flag == nullptr)
    return PTB_ERR_SIZE;
  if (!aligned16(x) || !aligned16(w) || !aligned16(out)) return PTB_ERR_ALIGN;
  CUtensorMap map;
  if (!make_expert_map(&map, w, (long long)n_experts * (mode == 0 ? 2 : 1) * N, K)) return PTB_ERR_LAUNCH;
  ExpertTcParams p = {};
  p.x = (const __nv_bfloat16*)x; p.out = out; p.plan = plan; p.row_scale = row_scale; p.error_flag = error_flag;
  p.pairs = pairs; p.max_tiles = max_tiles; p.top = top; p.N = N; p.K = K; p.act = act; p.tile_rows = tile_rows;
  p.glu_limit = glu_limit; p.glu_alpha = glu_alpha;
  return mode == 0 ? launch_expert_tc<0>(map, p, stream) : mode == 1 ? launch_expert_tc<1>(map, p, stream)
                                                                     : launch_expert_tc<2>(map, p, stream);
}
