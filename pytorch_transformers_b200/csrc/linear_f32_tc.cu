// The float32 linear layer y[m, n] = act(sum_k x[m, k] w[n, k] + bias[n]) on the fifth-generation tensor cores, to float32.
//
// Every operand value is three bfloat16 terms that hold all its 24 bits, x = x1 + x2 + x3 (each the rounding of what the ones before
// leave), and a product is the six products of terms down to 2^-18 of it: x3 w1, x1 w3, x2 w2, x2 w1, x1 w2, x1 w1. What is left
// out is 2^-27.5 of a product (root mean square) and at most 2^-24. The tensor core cuts its running sums off instead of rounding them, so it
// sums 32 values of k only, from zero, the small products first; these sums are added in float32 registers with rounded additions, a
// stretch of K after the other. A sum is 5.1e-8 of itself too small on average, whatever the values (every cut is towards zero), so that share of
// the result is put back where the last stretch's total joins the others, exactly up to one rounding. The stretches follow from N and K alone and
// join in order, whoever forms them: a row's result depends neither on the other rows nor on the tile. They are as many as the multiply-adds of
// linear_f32.cu take, or more: a stretch is a chain of roundings. 2-norm off 64 bits in 1e-7, multiply-adds in brackets, normal values and ones
// between 0 and 1: 1,024 x 1,024 0.78 (1.13) and 0.43 (0.53), 9,216 x 4,096 1.19 (1.38) and 0.54 (0.55), 1,536 x 6,144 1.39 (1.56) and 0.64 (0.65),
// 65,024 x 4,544 1.24 (1.43) and 0.62 (0.62), 4,544 x 18,176 1.88 (2.35) and 0.74 (0.99). Before, with one or two stretches of a wide
// matrix and nothing put back, 2.13 and 1.59 at 9,216 x 4,096. (Every join exact, with its rest kept: 0.71 and 0.35 at 1,024 x 1,024, but 45 us
// where 700 rows of 3,072 x 1,024 take 43. Both sums of a stage added to each other first: 0.75 and 0.44, 49 us, as nothing is summed meanwhile.)
//
// A block owns 128 outputs (the M side of tcgen05.mma) x BN rows:
//   8 warps      take the operands apart: 32-byte words of both matrices from global memory into registers, a stage of 64 k (two of them
//                for up to 32 rows) ahead, three terms each into swizzled tiles of a ring of stages
//   2 warps      one thread each issues one half of a stage's k: twelve instructions into an accumulator of its own. (One thread for
//                both held the second sum back behind the first one's waits: 340 us for the products of the block below, 259 with two.)
//   4 or 8 warps add the sums to their registers, which gives the accumulator back
// What bounds it with many rows is shared memory: of a stage of 128 x 128, 3,360 clocks, the matrix instructions read 192 KB of operands,
// the terms' stores are 96 KB and the loads through L1 64 KB, 2,816 clocks at 128 bytes; the instructions themselves are 1,536. With few
// rows it is the matrix's way from memory. Results leave through shared memory in a loop, whose activations and re-sum of what is no number
// would else be written out for every register, more than the instruction cache holds (block below 379 -> 330 us).
// One B200: the four products of a block of width 1,024 on 700 rows 517 -> 226 us (700 x 1,024 x 4,096: 152 -> 76), 2,048 rows of
// 4,096 x 2,048 880 -> 266 us (129 TFLOP/s), one row of 65,024 x 4,544 422 -> 285 us; before: float32 FMAs (linear_f32.cu). Pairs of
// blocks on one instruction (two SMs, 256 outputs x 128 or 192 rows, half of the x rows each) were no faster: 344.
#include "common.cuh"
#include "tc_common.cuh"
#include <cooperative_groups.h>

#include "f32x2.cuh"
#include "linear_f32.cuh"

namespace {

namespace cg = cooperative_groups;

constexpr int FM = 128;                       // outputs of a tile: M of the matrix instruction
constexpr int FK = 64;                        // k of a stage: 128 bytes of bfloat16, one swizzle row
constexpr int FSUB = 32;                      // k that the tensor core sums
constexpr int F_CONV = 256, F_ISSUE = FK / FSUB;      // threads that take operands apart, warps that issue
constexpr float F_SCALE = 131072.f;           // 2^17, of both operands
constexpr float F_CUT = 5.1e-8f;              // what a sum of FSUB loses by being cut, of itself, on average (measured: 0.51 to 0.52)
constexpr int F_TERM = FM * FK * 2;           // bytes of one term of a stage's matrix rows

struct LinearF32Params {
  const float *x, *w, *bias;
  float* y;
  int* error_flag;
  int M, N, K, ldx, act;
  int stretches;                              // of K, even but for one stage, divided evenly among a cluster's blocks
  int w_vec, x_vec;                           // floats of a load
};

// eight neighbouring values of a row
__device__ __forceinline__ void load8(float (&f)[8], const float* p, int vec) {
  if (vec == 8) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(p));
  } else if (vec == 4) {
#pragma unroll
    for (int e = 0; e < 8; e += 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + e);
      f[e] = v.x; f[e + 1] = v.y; f[e + 2] = v.z; f[e + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = p[e];
  }
}

// the three terms of two values times F_SCALE, packed
__device__ __forceinline__ void three_terms(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
  auto pair = [](uint64_t v) {
    const float2 f = halves2(v);
    return pack_bf16(f.x, f.y);
  };
  uint64_t v = mul2(pack2(x, y), pack2(F_SCALE, F_SCALE));
  a = pair(v);
  v = minus2(v, wide2(a));
  b = pair(v);
  c = pair(minus2(v, wide2(b)));
}

// ... of eight values, to the same place of three tiles
__device__ __forceinline__ void put_terms(unsigned char* at, int term, const float (&f)[8]) {
  uint4 t1, t2, t3;
  three_terms(f[0], f[1], t1.x, t2.x, t3.x);
  three_terms(f[2], f[3], t1.y, t2.y, t3.y);
  three_terms(f[4], f[5], t1.z, t2.z, t3.z);
  three_terms(f[6], f[7], t1.w, t2.w, t3.w);
  *reinterpret_cast<uint4*>(at) = t1;
  *reinterpret_cast<uint4*>(at + term) = t2;
  *reinterpret_cast<uint4*>(at + 2 * term) = t3;
}
// a stage's eight values of a row from `row` on; zeros from its k_end-th on (WIDE: whole stages in 32-byte words)
template <bool WIDE>
__device__ __forceinline__ void load_step(float (&f)[8], const float* row, int step, int whole, int k_end, int vec) {
  if (WIDE || step < whole) {
    load8(f, row + step * FK, WIDE ? 8 : vec);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = step * FK + e < k_end ? row[step * FK + e] : 0.f;
  }
}
// FSUB values of k of all terms, from zero, the smallest products first; `a`: the matrix's first term, the others and the rows' behind it
template <int X_TERM>
__device__ __forceinline__ void issue_terms(uint32_t acc, uint64_t a, uint32_t idesc) {
  constexpr uint64_t WT = F_TERM >> 4, XT = X_TERM >> 4;
  const uint64_t b = a + 3 * WT;
  uint32_t on = 0;
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const uint64_t at = t == 0 ? 2 : (t == 2 || t == 3) ? 1 : 0, bt = t == 1 ? 2 : (t == 2 || t == 4) ? 1 : 0;
#pragma unroll
    for (int k = 0; k < FSUB / 16; ++k) {
      tc_mma(acc, a + at * WT + 2 * k, b + bt * XT + 2 * k, idesc, on);
      on = 1;
    }
  }
}
// A warp's 32 results of row m, outputs n .. n + 31, from the scaled sums. Infinities, NaN and what leaves float32 by the scale have no three
// terms: a sum that is no number is formed again from the values themselves, by the whole warp.
__device__ __forceinline__ void finish_f32(const LinearF32Params& p, int m, int n, float v, int lane) {
  uint32_t again = __ballot_sync(0xffffffffu, n + lane < p.N && !(fabsf(v) <= 3.402823466e38f));
  v *= 1.f / (F_SCALE * F_SCALE);
  while (again) {
    const int from = __ffs(again) - 1;
    again &= again - 1;
    const float *x = p.x + size_t(m) * p.ldx, *w = p.w + size_t(n + from) * p.K;
    float s = 0.f;
    for (int k0 = lane; k0 < p.K; k0 += 16 * 32) {      // chains of 16
      float t = 0.f;
      for (int k = k0; k < min(p.K, k0 + 16 * 32); k += 32) t = fmaf(x[k], w[k], t);
      s += t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == from) v = s;
  }
  if (n + lane >= p.N) return;
  if (p.bias) v += p.bias[n + lane];
  p.y[size_t(m) * p.N + n + lane] = apply_activation(v, p.act);
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
               ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// The last stretch's total joins the ones before exactly (Knuth's sum of two) and rounds once, with what all sums have lost by being cut.
__device__ __forceinline__ float join_last(float before, float last) {
  const float s = before + last, b = s - before;
  return s + fmaf(s, F_CUT, (before - (s - b)) + (last - b));
}
// v[i] += column i of tensor memory, N a multiple of 8
template <int N>
__device__ __forceinline__ void tmem_add(uint32_t taddr, float (&v)[N]) {
  constexpr int S = N < 32 ? N : 32;
#pragma unroll
  for (int g = 0; g < N; g += S) {
    uint32_t r[S / 8][8];
#pragma unroll
    for (int j = 0; j < S / 8; ++j) tmem_ld8_nowait(taddr + g + 8 * j, r[j]);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < S; ++j) v[g + j] += __uint_as_float(r[j / 8][j % 8]);
  }
}
template <int BN>
struct LinearF32Tile {
  static constexpr int X_TERM = BN * FK * 2, STAGE = 3 * (F_TERM + X_TERM);
  static constexpr int STAGES = BN <= 64 ? 3 : 2;
  static constexpr int SUMS = BN <= 64 ? 128 : 256, THREADS = F_CONV + SUMS + 32 * F_ISSUE;      // up to 16 warps leave 128 registers a thread
  static constexpr int SMEM = 1024 + STAGES * STAGE;
  static constexpr int COLS = 4 * BN;      // two sums in turn, the stretches' total; a power of two
};

template <int BN, bool WIDE>
__global__ void __launch_bounds__(LinearF32Tile<BN>::THREADS, 1)
linear_f32_tc_kernel(const LinearF32Params p) {
  using T = LinearF32Tile<BN>;
  constexpr int STAGES = T::STAGES, X_TERM = T::X_TERM, STAGE = T::STAGE, SUMS = T::SUMS;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t bars[2 * STAGES + 4];     // full[stages], empty[stages], sums complete [2], sums read [2]
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * FM, m0 = blockIdx.y * BN;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[STAGES]);
  const uint32_t done0 = smem_u32(&bars[2 * STAGES]), read0 = smem_u32(&bars[2 * STAGES + 2]);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, F_CONV / 32);
      mbar_init(empty0 + 8 * s, F_ISSUE);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(done0 + 8 * b, 1);
      mbar_init(read0 + 8 * b, SUMS / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == (F_CONV + SUMS) / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)), "n"(T::COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  // this block's stretches and their stages
  const int total = (p.K + FK - 1) / FK, ranks = int(gridDim.z), rank = int(blockIdx.z), own = p.stretches / ranks;
  auto stretch_at = [&](int j) { return int((long long)j * total / p.stretches); };
  const int first = stretch_at(rank * own), last = stretch_at((rank + 1) * own);
  const int steps = last - first, whole = p.K / FK;

  if (warp < F_CONV / 32) {
    // ------------------------------------------------------------------ the operands' terms: eight values of k a thread and pass
    constexpr int AG = FM * 8 / F_CONV, BG = (BN * 8 + F_CONV - 1) / F_CONV;
    const int c = tid & 7, r0 = tid >> 3;             // k c * 8 .. of rows r0 + 32 g
    // values of the next DEPTH stages are on their way: few rows leave registers for two, and then only the matrix's stream counts
    constexpr int DEPTH = BN <= 32 ? 2 : 1;
    float a[DEPTH][AG][8], b[DEPTH][BG][8];
    // rows past the end read the last one: what they sum is not stored
    const float *wrow[AG], *xrow[BG];
#pragma unroll
    for (int g = 0; g < AG; ++g) wrow[g] = p.w + size_t(min(n0 + r0 + 32 * g, p.N - 1)) * p.K + c * 8;
#pragma unroll
    for (int g = 0; g < BG; ++g) xrow[g] = p.x + size_t(min(m0 + r0 + 32 * g, p.M - 1)) * p.ldx + c * 8;
    auto load = [&](float (&f)[8], const float* row, int step, int vec) { load_step<WIDE>(f, row, step, whole, p.K - c * 8, vec); };
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      if (steps <= d) break;
#pragma unroll
      for (int g = 0; g < AG; ++g) load(a[d][g], wrow[g], first + d, p.w_vec);
#pragma unroll
      for (int g = 0; g < BG; ++g) load(b[d][g], xrow[g], first + d, p.x_vec);
    }
    uint32_t st = 0, parity = 1;                      // parity of the round before
    const uint32_t off = r0 * 128 + ((c ^ (r0 & 7)) << 4);
    bool alive = true;
    for (int i0 = 0; i0 < steps && alive; i0 += DEPTH) {
#pragma unroll
      for (int d = 0; d < DEPTH; ++d) {
        const int i = i0 + d;
        if (i >= steps) break;
        if (i >= STAGES && !mbar_wait(empty0 + 8 * st, parity, p.error_flag, 41)) {
          alive = false;
          break;
        }
        unsigned char* base = ring + st * STAGE + off;
        // a group's registers take a later stage's values as soon as it is taken apart (the last stages read the last one's again)
        const int next = first + min(i + DEPTH, steps - 1);
#pragma unroll
        for (int g = 0; g < AG; ++g) {
          put_terms(base + g * 4096, F_TERM, a[d][g]);
          load(a[d][g], wrow[g], next, p.w_vec);
        }
#pragma unroll
        for (int g = 0; g < BG; ++g) {
          if (BN >= 32 || r0 < BN) put_terms(base + 3 * F_TERM + g * 4096, X_TERM, b[d][g]);
          load(b[d][g], xrow[g], next, p.x_vec);
        }
        proxy_fence_async();        // the matrix instructions read what ordinary stores wrote
        __syncwarp();
        if (lane == 0) mbar_arrive(full0 + 8 * st);
        if (++st == STAGES) { st = 0; parity ^= 1; }
      }
    }
  } else if (warp >= (F_CONV + SUMS) / 32) {
    // ------------------------------------------------------------------ issuers: each its share of a stage's k
    if (lane == 0) {
      const uint32_t sub = warp - (F_CONV + SUMS) / 32, acc = tmem_base + sub * BN;
      const uint32_t idesc = idesc_bf16(FM, BN, false);
      const uint64_t desc0 = smem_desc(smem_u32(ring), 16, 1024) + uint64_t(sub * (FSUB / 8));
      uint32_t st = 0, parity = 0;
      for (int i = 0; i < steps; ++i) {
        if (!mbar_wait(full0 + 8 * st, parity, p.error_flag, 42)) break;
        if (i >= 1 && !mbar_wait(read0 + 8 * sub, (i - 1) & 1, p.error_flag, 43)) break;
        tc_fence_after();
        issue_terms<X_TERM>(acc, desc0 + uint64_t(st * (STAGE >> 4)), idesc);
        tc_commit(empty0 + 8 * st);
        tc_commit(done0 + 8 * sub);
        if (++st == STAGES) { st = 0; parity ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ sums: a lane an output, all rows or half of them a warp
    constexpr int SC = BN * 128 / SUMS;
    const int quarter = warp & 3, half = (warp - F_CONV / 32) >> 2;
    const uint32_t lane_addr = tmem_base + (uint32_t(quarter * 32) << 16) + half * SC;
    float acc[SC];
    uint32_t n = 0;
    bool alive = true;
    for (int j = 0; j < own; ++j) {
#pragma unroll
      for (int e = 0; e < SC; ++e) acc[e] = 0.f;
      const int s0 = stretch_at(rank * own + j), s1 = stretch_at(rank * own + j + 1);
      for (int i = s0; i < s1 && alive; ++i, ++n)
#pragma unroll 1
        for (uint32_t buf = 0; buf < F_ISSUE; ++buf) {
          alive = mbar_wait(done0 + 8 * buf, n & 1, p.error_flag, 44);
          if (!alive) break;
          tc_fence_after();
          tmem_add(lane_addr + buf * BN, acc);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(read0 + 8 * buf);
        }
      // the stretches' totals join in order: in one block as they come, waiting in tensor memory for the last one; of a cluster's blocks at the end
      if (j + 1 < own) {
        if (j > 0) tmem_add(lane_addr + 2 * BN, acc);
#pragma unroll
        for (int e = 0; e < SC; e += 8) tmem_st8(lane_addr + 2 * BN + e, acc + e);
        tmem_st_wait();
      }
    }
    // the ring is free: the last sums are complete, so its last stage has been read. Results leave through it, in a loop of all threads: the
    // activations written out for every register of a tile would be more code than the instruction cache holds
    const int row = quarter * 32 + lane, tiles = min(own, 2);
    float* tile = reinterpret_cast<float*>(ring) + (tiles - 1) * BN * FM;
#pragma unroll
    for (int e = 0; e < SC; ++e) tile[(half * SC + e) * FM + row] = acc[e];
    if (tiles == 2) {
#pragma unroll
      for (int e = 0; e < SC; ++e) acc[e] = 0.f;
      tmem_add(lane_addr + 2 * BN, acc);
#pragma unroll
      for (int e = 0; e < SC; ++e) tile[(half * SC + e) * FM + row - BN * FM] = acc[e];
    }
  }
  {
    const cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const float* tile = reinterpret_cast<const float*>(ring);
#pragma unroll 1
    for (int at = rank * T::THREADS + tid; at < BN * FM; at += ranks * T::THREADS) {
      const int m = m0 + at / FM, n = n0 + (at - lane) % FM;      // a warp's are of one row
      if (m >= p.M) continue;
      float v = 0.f;
      if (ranks == 1) {
        v = join_last(tile[at], tile[BN * FM + at]);
      } else {
        for (int s = 0; s < p.stretches; ++s) {
          const float t = *cluster.map_shared_rank(tile + s % own * BN * FM + at, s / own);
          v = s + 1 < p.stretches ? v + t : join_last(v, t);
        }
      }
      finish_f32(p, m, n, v, lane);
    }
    cluster.sync();       // no block leaves while its tile is still read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == (F_CONV + SUMS) / 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "n"(T::COLS));
}

template <int BN, bool WIDE>
int launch_tc(const LinearF32Params& p, int ranks, cudaStream_t stream) {
  using T = LinearF32Tile<BN>;
  static SharedLimit limit;
  if (!limit.allows(linear_f32_tc_kernel<BN, WIDE>, T::SMEM)) return PTB_ERR_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + FM - 1) / FM, (p.M + BN - 1) / BN, ranks);
  cfg.blockDim = dim3(T::THREADS);
  cfg.dynamicSmemBytes = T::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = ranks;
  cfg.attrs = attr;
  cfg.numAttrs = ranks > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, linear_f32_tc_kernel<BN, WIDE>, p);
  return launch_status();
}

}  // namespace

int linear_f32_tensor(const float* x, const float* w, const float* bias, float* y, int M, int N, int K, int ldx, int act,
                      int* error_flag, cudaStream_t stream) {
  LinearF32Params p;
  p.x = x; p.w = w; p.bias = bias; p.y = y; p.error_flag = error_flag;
  p.M = M; p.N = N; p.K = K; p.ldx = ldx; p.act = act;
  auto at32 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31) == 0; };
  p.w_vec = K % 8 == 0 && at32(w) ? 8 : 4;
  p.x_vec = K % 8 == 0 && ldx % 8 == 0 && at32(x) ? 8 : ldx % 4 == 0 && aligned16(x) ? 4 : 1;
  const int total = (K + FK - 1) / FK, tiles = (N + FM - 1) / FM;
  // Stretches of K, by N and K alone: a row's sums must not follow the number of rows. As many as blocks of a cluster may share a
  // matrix of few tiles, each of four stages at least (clusters of four blocks: 33 are resident at a time with a block an SM, of three 44,
  // of two 70 and more; 36 clusters of four are two waves: 4,544 x 18,176 and one row 157 us, in clusters of three 108), and then as many as keep
  // a stretch at 64 stages or fewer, at least two, from K of 2,048 on four, since each of its additions rounds (one cluster's block holds two
  // at most). A stretch more costs a block its totals' way through tensor memory: with one or two and now, 128 rows of 9,216 x 1,024 47 and 49 us,
  // 700 rows of 9,216 x 4,096 365 and 357, one row of 65,024 x 4,544 279 and 285.
  const int shared = tiles <= 33 ? 4 : tiles <= 44 ? 3 : tiles <= 70 ? 2 : 1;
  int most = shared;
  while (most > 1 && total / most < 4) --most;
  const int least = total >= 32 ? 4 : 2;
  const int each = max((total + 64 * most - 1) / (64 * most), (least + most - 1) / most);
  p.stretches = most * (most > 1 && each > 2 ? 2 : each);
  const bool wide = p.w_vec == 8 && p.x_vec == 8 && K % FK == 0;
  // Rows of a tile: as few as hold them all, then 128. Blocks that share a tile: as many as may where all of them are resident, else two
  // (two stretches each) or one. us at 700 rows, one block a tile against what is taken: 1,024 x 4,096 139 and 76, 1,024 x 1,024 67 and 35.
  const int bn = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  const long long blocks = (long long)tiles * ((M + bn - 1) / bn);
  int ranks = 1;
  if (blocks * most <= sm_count() && (most != 4 || blocks <= 33)) ranks = most;
  else if (p.stretches == 4 && blocks <= 70) ranks = 2;
#define PTB_FTC(BN) return wide ? launch_tc<BN, true>(p, ranks, stream) : launch_tc<BN, false>(p, ranks, stream)
  if (bn == 16) PTB_FTC(16);
  if (bn == 32) PTB_FTC(32);
  if (bn == 64) PTB_FTC(64);
  PTB_FTC(128);
#undef PTB_FTC
}
