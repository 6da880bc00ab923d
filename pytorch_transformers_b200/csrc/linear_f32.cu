// Float32 linear layer: y[m, n] = act(sum_k x[m, k] * w[n, k] + bias[n]). Matrices of some size go to linear_f32_tc.cu; here what is
// small or laid out oddly, on the CUDA cores: every product and sum is an IEEE float32 FMA.
//
// The sums of one output element: the k of a step of 32 are summed in two chains (even and odd k, 16 products each, ascending),
// the two chains join and go into a running total; a K of 2,048 or more is cut into four stretches whose totals are added in
// order, a K of 1,024 to 2,047 beside fewer than 2,048 outputs into two, any other into none. All of this follows from N and K alone, so a
// row's result depends neither on how many other rows are in the launch nor on the tile, and the rounding error stays small for K in the tens of thousands.
//
// What bounds it is the FMA pipe (128 lanes an SM). A block owns 8 TM rows x 64 outputs, a thread TM x 4 of them: of every
// 16 bytes that it reads from shared memory (operands stay in [row][k] order, so cp.async brings them without a
// transposition, and rows lie 36 floats apart, which lets eight rows' 16-byte words meet no bank twice) it makes
// 2 TM x 4 / (TM + 4) two-wide FMAs (fma.rn.f32x2: the two k chains in one 64-bit register). A three-stage ring keeps two
// steps of copies in flight. Few rows or few outputs would leave SMs idle: K is cut among a thread-block cluster whose blocks
// join their tiles through distributed shared memory.
// One B200, 700 rows: 40 x 4,096 165 us without stretches, 50 with four; 1,000 x 2,050 132 us; 9,001 x 4,545 1.95 ms (29 TFLOP/s of 72; rows that
// are no whole 16-byte words come in 4-byte copies). What linear_f32_tc.cu takes now ran here at 39 TFLOP/s (700 x 1,024 x 4,096:
// 152 us): two-wide FMAs of three blocks an SM leave half of the issue slots empty, registers (168 a thread) allow no more
// warps, and tiles of 8 x 8 a thread, which read less, were as fast at 2,048 rows and slower below.
#include <cooperative_groups.h>

#include "f32x2.cuh"
#include "linear_f32.cuh"
#include "mma_common.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int TN = 4, LBN = 16 * TN, LBK = 32, LPITCH = LBK + 4, LSTAGES = 3, LTHREADS = 128;

// copies that leave zeros where `bytes` is 0 (a row or a k past the end; the address is then any valid one)
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

// rows [row0, row0 + ROWS) x k [k0, k0 + 32) of a matrix with rows ld apart; k_end: the end of this block's stretch
template <int ROWS, bool VEC>
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int row0, int n_rows, size_t ld, int k0, int k_end) {
  constexpr int W = VEC ? 4 : 1, PER_ROW = LBK / W;
#pragma unroll
  for (int i = threadIdx.x; i < ROWS * PER_ROW; i += LTHREADS) {
    const int r = i / PER_ROW, k = k0 + (i % PER_ROW) * W;
    const bool ok = row0 + r < n_rows && k < k_end;
    const float* from = ok ? src + size_t(row0 + r) * ld + k : src;
    const uint32_t to = smem_u32(dst + r * LPITCH + (i % PER_ROW) * W);
    if (VEC) copy16(to, from, ok ? 16 : 0);
    else copy4(to, from, ok ? 4 : 0);
  }
}

template <int TM, bool VEC>
__global__ void __launch_bounds__(LTHREADS, 3)
linear_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                  float* __restrict__ y, int M, int N, int K, int ldx, int act, int stretch) {
  constexpr int BM = 8 * TM, STAGE = (BM + LBN) * LPITCH;
  extern __shared__ __align__(16) float lsm[];
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;      // rows ty + 8 i, outputs tx + 16 j
  const int n0 = blockIdx.x * LBN, m0 = blockIdx.y * BM;
  const int k_begin = int(blockIdx.z) * stretch, k_end = min(K, k_begin + stretch);
  const int steps = k_end > k_begin ? (k_end - k_begin + LBK - 1) / LBK : 0;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  auto load = [&](int s) {
    float* st = lsm + (s % LSTAGES) * STAGE;
    stage_rows<BM, VEC>(st, x, m0, M, size_t(ldx), k_begin + s * LBK, k_end);
    stage_rows<LBN, VEC>(st + BM * LPITCH, w, n0, N, size_t(K), k_begin + s * LBK, k_end);
  };
#pragma unroll
  for (int s = 0; s < LSTAGES - 1; ++s) {
    if (s < steps) load(s);
    cp_async_commit();
  }
  for (int s = 0; s < steps; ++s) {
    cp_async_wait<LSTAGES - 2>();
    __syncthreads();      // step s has landed for everybody, and step s - 1 is no longer read
    if (s + LSTAGES - 1 < steps) load(s + LSTAGES - 1);
    cp_async_commit();
    const float* xs = lsm + (s % LSTAGES) * STAGE + ty * LPITCH;
    const float* ws = lsm + (s % LSTAGES) * STAGE + (BM + tx) * LPITCH;
    unsigned long long part[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) part[i][j] = 0ull;
#pragma unroll
    for (int k = 0; k < LBK; k += 4) {
      ulonglong2 b[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ws + 16 * j * LPITCH + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + 8 * i * LPITCH + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) part[i][j] = fma2(a.x, b[j].x, part[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) part[i][j] = fma2(a.y, b[j].y, part[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float2 p = halves2(part[i][j]);
        acc[i][j] += p.x + p.y;
      }
  }
  cp_async_wait<0>();
  auto store = [&](int gm, int gn, float v) {
    if (gm >= M || gn >= N) return;
    if (bias) v += bias[gn];
    y[size_t(gm) * N + gn] = apply_activation(v, act);
  };
  if (gridDim.z == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) store(m0 + ty + 8 * i, n0 + tx + 16 * j, acc[i][j]);
    return;
  }
  // the stretches' totals join: every block leaves its tile in its shared memory and finishes a share of the rows
  cg::cluster_group cluster = cg::this_cluster();
  __syncthreads();      // the ring is no longer read
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) lsm[(ty + 8 * i) * LBN + tx + 16 * j] = acc[i][j];
  cluster.sync();
  const int rank = int(blockIdx.z), ranks = int(gridDim.z), share = BM / ranks;      // ranks: 2 or 4, BM a multiple of 16
  for (int e = tid; e < share * LBN; e += LTHREADS) {
    const int at = rank * share * LBN + e;
    float v = 0.f;
    for (int r = 0; r < ranks; ++r) v += *cluster.map_shared_rank(lsm + at, r);
    store(m0 + at / LBN, n0 + at % LBN, v);
  }
  cluster.sync();       // no block leaves while its tile is still read
}

template <int TM, bool VEC>
int launch_linear_f32(const float* x, const float* w, const float* bias, float* y, int M, int N, int K, int ldx, int act,
                      int ranks, cudaStream_t stream) {
  const size_t smem = size_t(LSTAGES) * (8 * TM + LBN) * LPITCH * sizeof(float);
  static SharedLimit limit;
  if (!limit.allows(linear_f32_kernel<TM, VEC>, smem)) return PTB_ERR_LAUNCH;
  const int steps = (K + LBK - 1) / LBK, stretch = (steps + ranks - 1) / ranks * LBK;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + LBN - 1) / LBN, (M + 8 * TM - 1) / (8 * TM), ranks);
  cfg.blockDim = dim3(LTHREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ranks;
  cfg.attrs = attr;
  cfg.numAttrs = ranks > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, linear_f32_kernel<TM, VEC>, x, w, bias, y, M, N, K, ldx, act, stretch);
  return launch_status();
}

}  // namespace

// x [M, K] with rows ldx apart
PTB_API int ptb_linear_f32(const float* x, const float* w, const float* bias, float* y, int M, int N, int K, int ldx, int act,
                           int* error_flag, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return PTB_OK;
  if (K <= 0 || ldx < K || !activation_known(act) || error_flag == nullptr) return PTB_ERR_SIZE;
  if ((long(M) + 63) / 64 > 65535) return PTB_ERR_SIZE;
  // The tensor cores (linear_f32_tc.cu) take matrices whose rows are whole 16-byte words, of half a tile's outputs and two stages of k at
  // least: by the matrix alone, so that a row's bits do not follow the batch. us, FMAs against tensor cores, of 64 x 128: 9 and 11 for one row,
  // 14 and 17 for 700; 64 x 1,024: 16 and 12, 33 and 23; 256 x 256: 10 and 12, 18 and 23; 512 x 512: 16 and 13, 29 and 27.
  if (K % 4 == 0 && aligned16(w) && ((N >= 64 && K >= 1024) || (N >= 512 && K >= 256)))
    return linear_f32_tensor(x, w, bias, y, M, N, K, ldx, act, error_flag, stream);
  // Stretches of K, by N and K alone (the order of a row's sums must not follow the number of rows). us for one, two and four, of
  // matrices that stay here: 1 row, 40 x 4,096 78, 43, 25; 1,000 x 1,026 33, 23, 16; 4,097 x 2,050 57, 35, 29; 9,000 x 1,026 33, 29, 37; 9,001 x 4,545
  // 119, 91, 109. 700 rows, 40 x 4,096 165, 92, 50; 1,000 x 1,026 94, 76, 80; 1,000 x 2,050 177, 132, 132; 2,100 x 1,026 126, 121, 139; 4,098 x 1,030
  // 206, 223, 252; 4,097 x 2,050 388, 401, 436; 18,177 x 4,545 3,673, 3,656, 3,893. So long K gains most where rows or outputs are few, and from
  // some 2,048 outputs on the join costs many rows 3 to 12 %, which K of 2,048 and more pays for shorter chains of roundings.
  const int ranks = K >= 2048 ? 4 : (K >= 1024 && N < 2048) ? 2 : 1;
  // 16-byte copies where every row starts at a whole word
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && aligned16(x) && aligned16(w);
#define PTB_LF(TT) (vec ? launch_linear_f32<TT, true>(x, w, bias, y, M, N, K, ldx, act, ranks, stream) \
                        : launch_linear_f32<TT, false>(x, w, bias, y, M, N, K, ldx, act, ranks, stream))
  // rows of a tile: 64, or 16 or 32 for steps of few rows, which would be computed for padding otherwise
  return M <= 16 ? PTB_LF(2) : M <= 32 ? PTB_LF(4) : PTB_LF(8);
#undef PTB_LF
}
