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
// A block stays and walks every (blocks)-th tile, matrix columns first, so that the matrix boxes of its next tile are on their way while
// this one's results leave. What it has in flight is two rings, since the boxes come from memory and the rows from L2:
//   warp 0       one thread: per 64 values of k the boxes of 128 matrix rows by TMA (128-byte swizzle) into the ring of matrices
//   warps 1, 2   one thread each, a box and its accumulator: per stage four matrix instructions of 16 k, tcgen05.commit on both rings' "empty"
//                barriers. (A thread's two waits, two commits and four instructions take 625 clocks, two boxes' 805: a stage of
//                few rows would wait for it.)
//   then         the x rows: cp.async of 16-byte chunks from rows found through the plan, to their swizzled places, each
//                thread's arrival at the "full" barrier made by the copies themselves when they have landed; the next tile's rows are
//                looked up meanwhile
//   then         results: a warp reads its quarter of the lanes (a lane is a matrix row), sixteen x rows at a time. Accumulators of two tiles take
//                turns where tensor memory holds them (tiles of up to 128 rows); in tiles of 256 the matrix instructions wait for the gated
//                units (17,500 clocks a tile of 192 rows with a true division for each).
// Every wait on a barrier is bounded: when one runs out, the error flag is raised and the block carries on to its end without
// waiting again.
//
// One B200, 64 experts of 1,408, width 2,048, chosen evenly, plan and both products: 12,288 rows (about 192 an expert, tiles of 256) 322 -> 281 us
// (790 TFLOP/s without the plan), 21,000 rows 487 -> 434, 4,200 rows 223 -> 206, 48 rows 108 -> 102;
// before, a block a tile and one ring of three stages. A router that chooses unevenly leaves a last round of few tiles: 328 -> 318 of such 12,288 rows.
// With many rows shared memory's bandwidth bounds it (a stage of 192 rows: 56 KB in, 80 KB
// read by the matrix instructions, 1,090 of its clocks), then the results of a tile and a last round of few tiles. Boxes asked into L2 eight
// stages ahead cost a third with few rows (67 -> 90 us).
#include <cudaTypedefs.h>

#include <mutex>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int XM = 128;                    // matrix rows of a box = M of the matrix instruction
constexpr int XK = 64;                     // k per stage: 128 bytes, one swizzle row
constexpr int X_BOX_BYTES = XM * XK * 2;   // 16 KB
constexpr int X_MAX_W = 7, X_MAX_X = 4;   // stages of the rings of matrix boxes and of x rows
constexpr int MAX_BOXES = 2;               // boxes of a tile, each with an accumulator and a thread that issues for it
// TWO: two blocks an SM, for tiles of few rows (the first product's units leave registers for four storing warps then)
template <int MODE, bool TWO>
struct ExpertThreads {
  static constexpr int GATHER = TWO ? 64 : 256, STORE = TWO && MODE == 0 ? 128 : 256, ALL = 32 * (1 + MAX_BOXES) + GATHER + STORE;
  static constexpr int RING = (TWO ? 111 : 225) * 1024;
};

__device__ __forceinline__ void copy16_or_zero(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0));
}
// an arrival of this thread at `bar` (counted in its initial count) once all its copies so far have landed
__device__ __forceinline__ void arrive_when_copied(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// gated_unit (common.cuh) without a branch: a division is a call for odd operands at every value, and in tiles of 256 rows the matrix instructions
// wait for the units. Zero where e^-g leaves float32, as there. Layer of 64 experts on 2,048 tokens: 435 us with the division, 430 with a
// branch around the sigmoid for the zero, 416 so.
__device__ __forceinline__ float gated_unit_fast(float gate, float up, float limit, float alpha) {
  float a = 1.f;
  if (limit > 0.f) {
    gate = fminf(gate, limit), up = fminf(fmaxf(up, -limit), limit) + 1.f;
    a = alpha;
  }
  const float x = a * gate, s = sigmoid_of(x);
  return gate * (x < -88.72283f ? 0.f : s) * up;
}

struct ExpertTcParams {
  const __nv_bfloat16* x;
  void* out;
  const int* plan;
  const float* row_scale;
  int* error_flag;
  int pairs, max_tiles, top, N, K, act;
  int w_stages, x_stages, x_stage_bytes;      // the two rings
  int acc2, sets;           // tensor-memory columns from one accumulator to the next; tiles whose accumulators fit side by side
  float glu_limit, glu_alpha;
};

// PER: rows of a tile that a gathering thread copies a chunk of
template <int MODE, bool TWO, int PER>
__global__ void __launch_bounds__(ExpertThreads<MODE, TWO>::ALL, TWO ? 2 : 1)
expert_linear_tc_kernel(const __grid_constant__ CUtensorMap w_map, const ExpertTcParams p) {
  pdl_entry();
  constexpr int X_GATHER = ExpertThreads<MODE, TWO>::GATHER, X_STORE = ExpertThreads<MODE, TWO>::STORE;
  constexpr int TMEM_COLS = TWO ? 256 : 512;
  constexpr int BOXES = MODE != 0 && TWO ? 1 : 2;
  constexpr int COLS = MODE == 0 ? XM : BOXES * XM;      // output columns of a tile
  const int m_tiles = (p.N + COLS - 1) / COLS;
  const int *tile_expert = p.plan + 1, *tile_row0 = tile_expert + p.max_tiles, *tile_n = tile_row0 + p.max_tiles;
  // the first tile is asked for with the number of tiles (a way from memory less before the first box), whether there is one or not: no block lies past
  // the plan's room
  const int tile0 = blockIdx.x / m_tiles, expert0 = tile_expert[tile0], first0 = tile_row0[tile0], rows0 = tile_n[tile0];
  const int total = p.plan[0] * m_tiles;
  if (int(blockIdx.x) >= total) return;
  const int* pair_of_row = tile_n + p.max_tiles + p.pairs;
  extern __shared__ unsigned char smem_dyn[];
  // 1024-byte alignment: the swizzle pattern is a function of address bits 4..9
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  constexpr int W_BYTES = BOXES * X_BOX_BYTES;
  __shared__ uint64_t bars[2 * X_MAX_W + 2 * X_MAX_X + 4];   // full and empty of both rings; accumulators complete, accumulators read
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t wfull0 = smem_u32(&bars[0]), wempty0 = smem_u32(&bars[X_MAX_W]);
  const uint32_t xfull0 = smem_u32(&bars[2 * X_MAX_W]), xempty0 = smem_u32(&bars[2 * X_MAX_W + X_MAX_X]);
  const uint32_t done0 = smem_u32(&bars[2 * X_MAX_W + 2 * X_MAX_X]), read0 = done0 + 16;
  const uint32_t wring = smem_u32(ring), xring = wring + p.w_stages * W_BYTES;
  const int n_iter = (p.K + XK - 1) / XK;
  if (tid == 0) {
    for (int s = 0; s < p.w_stages; ++s) {
      mbar_init(wfull0 + 8 * s, 1);
      mbar_init(wempty0 + 8 * s, BOXES);
    }
    for (int s = 0; s < p.x_stages; ++s) {
      mbar_init(xfull0 + 8 * s, X_GATHER);
      mbar_init(xempty0 + 8 * s, BOXES);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(done0 + 8 * s, BOXES);
      mbar_init(read0 + 8 * s, X_STORE / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "n"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t st = 0, parity = 1;                     // parity of the round before
      int filled = 0;
      bool alive = true;
      int expert = expert0;
      for (int t = blockIdx.x; t < total && alive; t += gridDim.x) {
        const int m0 = t % m_tiles * COLS, wrow = expert * (MODE == 0 ? 2 : 1) * p.N + m0;      // rows past an expert's own come along and are not stored
        if (t + int(gridDim.x) < total) expert = tile_expert[(t + gridDim.x) / m_tiles];
        for (int i = 0; i < n_iter; ++i, ++filled) {
          const uint32_t full = wfull0 + 8 * st, base = wring + st * W_BYTES;
          if (filled >= p.w_stages && !mbar_wait(wempty0 + 8 * st, parity, p.error_flag, 31)) {
            alive = false;
            break;
          }
          mbar_expect_tx(full, uint32_t(W_BYTES));     // a box delivers all its bytes, zeros where out of range
          tma_load_2d(base, &w_map, i * XK, wrow, full);
          if (BOXES == 2) tma_load_2d(base + X_BOX_BYTES, &w_map, i * XK, wrow + (MODE == 0 ? p.N : XM), full);
          if (++st == uint32_t(p.w_stages)) { st = 0; parity ^= 1; }
        }
      }
      // the copies in flight land before the block ends, also where a wait ran out (bounded waits again)
      for (int j = max(0, filled - p.w_stages); j < filled; ++j)
        mbar_wait(wfull0 + 8 * (j % p.w_stages), (j / p.w_stages) & 1, p.error_flag, 31);
    }
  } else if (warp < 1 + MAX_BOXES) {
    if (lane == 0 && warp < 1 + BOXES) {
      const uint32_t box = warp - 1;
      const uint64_t wdesc0 = smem_desc(wring + box * X_BOX_BYTES, 16, 1024), xdesc0 = smem_desc(xring, 16, 1024);
      uint32_t ws = 0, wpar = 0, xs = 0, xpar = 0, n = 0;      // n: tiles so far
      bool alive = true;
      int rows = rows0;
      for (int t = blockIdx.x; t < total && alive; t += gridDim.x, ++n) {
        const uint32_t set = p.sets == 2 ? n & 1 : 0, round = p.sets == 2 ? n >> 1 : n;
        const uint32_t idesc = idesc_bf16(XM, (rows + 15) / 16 * 16, false), acc = tmem_base + (set * BOXES + box) * p.acc2;
        if (t + int(gridDim.x) < total) rows = tile_n[(t + gridDim.x) / m_tiles];
        if (round > 0) alive = mbar_wait(read0 + 8 * set, (round - 1) & 1, p.error_flag, 35);
        tc_fence_after();
        for (int i = 0; i < n_iter && alive; ++i) {
          alive = mbar_wait(xfull0 + 8 * xs, xpar, p.error_flag, 32) && mbar_wait(wfull0 + 8 * ws, wpar, p.error_flag, 32);
          if (!alive) break;
          proxy_fence_async();      // the x rows came by ordinary copies; the matrix instructions read them through the other proxy
          tc_fence_after();
          const uint64_t dw = wdesc0 + uint64_t(ws * (W_BYTES >> 4)), dx = xdesc0 + uint64_t(xs * (uint32_t(p.x_stage_bytes) >> 4));
          tc_mma4(acc, dw, dx, idesc, i > 0 ? 1u : 0u);
          tc_commit(xempty0 + 8 * xs);
          tc_commit(wempty0 + 8 * ws);
          if (++ws == uint32_t(p.w_stages)) { ws = 0; wpar ^= 1; }
          if (++xs == uint32_t(p.x_stages)) { xs = 0; xpar ^= 1; }
        }
        if (alive) tc_commit(done0 + 8 * set);
      }
    }
    __syncwarp();
  } else if (warp < 1 + MAX_BOXES + X_GATHER / 32) {
    const int gt = tid - 32 * (1 + MAX_BOXES), c = gt % 8;      // chunk c (8 values) of rows gt / 8 + X_GATHER / 8 j
    // a tile's rows; those of the block's next tile are looked up while this one's are copied
    int row[PER], next[PER], rows = 0, next_rows = 0;
    auto look_up = [&](int row0, int n, int (&to)[PER]) {
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int r = gt / 8 + X_GATHER / 8 * j;
        to[j] = r < n ? (MODE == 1 ? row0 + r : pair_of_row[row0 + r]) : -1;
      }
    };
    rows = rows0;
    look_up(first0, rows, row);
    const uint32_t dst0 = xring + (gt / 8) * 128 + ((c ^ ((gt / 8) & 7)) << 4);
    uint32_t st = 0, parity = 1;
    int filled = 0;
    bool alive = true;
    for (int t = blockIdx.x; t < total && alive; t += gridDim.x) {
      const bool more = t + int(gridDim.x) < total;
      if (more) {
        const int tile = (t + gridDim.x) / m_tiles;
        next_rows = tile_n[tile];
        look_up(tile_row0[tile], next_rows, next);
      }
      const int n16 = (rows + 15) / 16 * 16;
      const __nv_bfloat16* src[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j) src[j] = row[j] >= 0 ? p.x + size_t(MODE == 1 ? row[j] : row[j] / p.top) * p.K + c * 8 : nullptr;
      for (int i = 0; i < n_iter; ++i, ++filled) {
        if (filled >= p.x_stages && !mbar_wait(xempty0 + 8 * st, parity, p.error_flag, 34)) {
          alive = false;
          break;
        }
        const bool k_ok = i * XK + c * 8 < p.K;
        const uint32_t dst = dst0 + st * p.x_stage_bytes;
#pragma unroll
        for (int j = 0; j < PER; ++j)
          if (gt / 8 + X_GATHER / 8 * j < n16)
            copy16_or_zero(dst + j * (X_GATHER * 16), src[j] && k_ok ? src[j] + i * XK : p.x, src[j] && k_ok);
        arrive_when_copied(xfull0 + 8 * st);
        if (++st == uint32_t(p.x_stages)) { st = 0; parity ^= 1; }
      }
#pragma unroll
      for (int j = 0; j < PER; ++j) row[j] = next[j];
      rows = next_rows;
    }
    cp_async_wait_all();
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3, half = (warp - 1 - MAX_BOXES - X_GATHER / 32) >> 2;
    const uint32_t lane_addr = tmem_base + (uint32_t(quarter * 32) << 16);
    uint32_t n = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, ++n) {
      const uint32_t set = p.sets == 2 ? n & 1 : 0, round = p.sets == 2 ? n >> 1 : n;
      const int tile = t / m_tiles, row0 = n == 0 ? first0 : tile_row0[tile], rows = n == 0 ? rows0 : tile_n[tile];
      const int f0 = t % m_tiles * COLS + quarter * 32 + lane;      // output column = lane of tensor memory
      if (!mbar_wait(done0 + 8 * set, round & 1, p.error_flag, 33)) break;
      tc_fence_after();
      const uint32_t acc = lane_addr + set * BOXES * p.acc2;
      for (int g = 2 * half; g * 8 < rows; g += X_STORE / 64) {      // sixteen rows at a time
        uint32_t r[BOXES][16];
#pragma unroll
        for (int b = 0; b < BOXES; ++b) tmem_ld16_nowait(acc + b * p.acc2 + g * 8, r[b]);
        tmem_ld_wait();
        if constexpr (MODE == 1) {
#pragma unroll
          for (int b = 0; b < BOXES; ++b) {
            const int f = f0 + b * XM;
            float* o = reinterpret_cast<float*>(p.out) + size_t(row0 + g * 8) * p.N + f;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (g * 8 + j < rows && f < p.N) o[size_t(j) * p.N] = __uint_as_float(r[b][j]);
          }
        } else {
#pragma unroll
          for (int b = 0; b < (MODE == 0 ? 1 : BOXES); ++b) {
            const int f = f0 + b * XM;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              v[j] = __uint_as_float(r[b][j]);
              if (MODE == 0) {
                v[j] = gated_unit_fast(v[j], __uint_as_float(r[BOXES - 1][j]), p.glu_limit, p.glu_alpha);
              } else {
                const int at = g * 8 + j;
                const float rs = (p.row_scale && at < rows) ? p.row_scale[pair_of_row[row0 + at]] : 1.f;
                v[j] = apply_activation(v[j] * rs, p.act);
              }
            }
            // two rows at a time: an even lane stores columns f, f + 1 of the first, the odd lane above it those of the second
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + size_t(row0 + g * 8 + (lane & 1)) * p.N + (f & ~1);
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
              const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? v[j] : v[j + 1], 1);
              const uint32_t word = (lane & 1) ? pack_bf16(other, v[j + 1]) : pack_bf16(v[j], other);
              if (g * 8 + j + (lane & 1) < rows && f < p.N) *reinterpret_cast<uint32_t*>(o + size_t(j) * p.N) = word;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(read0 + 8 * set);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "n"(TMEM_COLS));
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

template <int MODE, bool TWO, int PER>
int launch_expert_tc(const CUtensorMap& map, ExpertTcParams p, int tile_rows, cudaStream_t stream) {
  constexpr int RING = ExpertThreads<MODE, TWO>::RING, BOXES = MODE != 0 && TWO ? 1 : 2, COLS = MODE == 0 ? XM : BOXES * XM;
  p.acc2 = tile_rows < 32 ? 32 : tile_rows;
  p.sets = 2 * BOXES * p.acc2 <= (TWO ? 256 : 512) ? 2 : 1;
  p.x_stage_bytes = tile_rows * XK * 2;
  p.x_stages = TWO && MODE == 0 && tile_rows == 128 ? 2 : tile_rows >= 128 ? 3 : TWO && tile_rows == 32 ? 3 : X_MAX_X;
  p.w_stages = min(X_MAX_W, (RING - p.x_stages * p.x_stage_bytes) / (BOXES * X_BOX_BYTES));
  const size_t smem = 1024 + size_t(RING);
  static SharedLimit limit;
  if (!limit.allows(expert_linear_tc_kernel<MODE, TWO, PER>, smem)) return PTB_ERR_LAUNCH;
  const long long most = (long long)p.max_tiles * ((p.N + COLS - 1) / COLS), slots = (long long)sm_count() * (TWO ? 2 : 1);
  launch_pdl(expert_linear_tc_kernel<MODE, TWO, PER>, int(most < slots ? most : slots), ExpertThreads<MODE, TWO>::ALL, smem, stream, map, p);
  return launch_status();
}

template <int MODE>
int launch_expert_tc(const CUtensorMap& map, const ExpertTcParams& p, int n_experts, int tile_rows, cudaStream_t stream) {
  // Two blocks an SM, each with half of its shared memory and, in the second product, with tiles of half the columns, where what counts are blocks
  // and the matrices' stream: tiles of up to 32 rows; of 64 in the second product; of 64 and 128 in the first where a block an SM would leave a last
  // round of few tiles, and of 64 where tiles are few at all. Else the first product's deeper rings win. Tiles counted as one an expert. us
  // with one and with two: first product, tiles of 64 rows, 64 tiles 13.3 / 12.8, 88 22.3 / 30.3, 128 48.2 / 58.4, 176 45.1 / 37.9, 256 48.8 / 50.9, 704 115 /
  // 122 (768 of less K 134 / 129); tiles of 128, 176 tiles 48.9 / 41.9, 256 52.8 / 53.0; tiles of 16, 88 to 768 tiles 20.0 / 17.4, 42.3 / 30.1, 113 / 112, 127 / 123. Second
  // product, tiles of 64, 32 tiles of 128 columns 19.9 / 17.0, 128 15.9 / 14.1, 512 29.3 / 27.3, 1,024 65.0 / 62.9; tiles of 128, 32 tiles 21.4 / 24.1, 256 21.7 / 22.1,
  // 512 30.8 / 29.5 (not taken).
  const int sms = sm_count();
  const long long tiles = (long long)min(p.pairs, n_experts) * ((p.N + XM - 1) / XM);
  const bool last_round = tiles > sms && tiles <= 3 * sms / 2;
  if (tile_rows <= 32 || (tile_rows == 64 && (MODE != 0 || tiles <= sms / 2 || last_round)))
    return launch_expert_tc<MODE, true, 8>(map, p, tile_rows, stream);
  if constexpr (MODE == 0)
    if (tile_rows == 128 && last_round) return launch_expert_tc<MODE, true, 16>(map, p, tile_rows, stream);
  return launch_expert_tc<MODE, false, 8>(map, p, tile_rows, stream);
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
  p.pairs = pairs; p.max_tiles = max_tiles; p.top = top; p.N = N; p.K = K; p.act = act;
  p.glu_limit = glu_limit; p.glu_alpha = glu_alpha;
  return mode == 0 ? launch_expert_tc<0>(map, p, n_experts, tile_rows, stream) : mode == 1 ? launch_expert_tc<1>(map, p, n_experts, tile_rows, stream)
                                                                                : launch_expert_tc<2>(map, p, n_experts, tile_rows, stream);
}
