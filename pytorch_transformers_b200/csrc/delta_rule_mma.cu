// The gated delta rule in chunks of 64 tokens on the tensor cores (bfloat16 projections, mma.m16n8k16 with float32 sums).
//
// Inside a chunk of n <= 64 tokens let c_t be the sum of the decays' logarithms up to and including token t (a vector over
// key channels), S_0 the state before the chunk, and
//     L[t][s] = beta_t sum_d k_t[d] k_s[d] exp(c_t[d] - c_s[d])   for s < t,      P[t][s] = sum_d q_t[d] k_s[d] exp(c_t[d] - c_s[d])   for s <= t.
// The corrections u_t of the chunk's tokens solve (I + L) U = diag(beta) (V - Kc S_0) with Kc_t = k_t exp(c_t). With
// T = (I + L)^-1 diag(beta), W = T Kc and U_0 = T V (so U = U_0 - W S_0), Qc_t = q_t exp(c_t) and Kd_s = k_s exp(c_n - c_s):
//     S_n = diag(exp(c_n)) S_0 + B + M S_0,     B = Kd^T U_0,   M = -Kd^T W,
//     O   = O_0 + Q S_0,                        O_0 = P U_0,    Q = Qc - P W.
// Pass 1 (parallel over chunks and heads) forms M, Q, B, O_0 and exp(c_n); pass 2 walks a sequence's chunks in order with
// the state's float32 values in registers, one product [M; Q] S_0 a chunk, and writes the outputs.
//
// No factor can grow: inside a sub-block of 16 tokens sums of logarithms start at the sub-block, the exponent between two
// sub-blocks is the rest of the earlier one, the whole ones between and the beginning of the later one; a sub-block's halves of 8
// meet in the same way at their border, and inside a half the exponent of every pair of tokens is formed by itself. Float32 operands (the
// state, decayed keys and queries, T, P, W, U_0) enter the products split in two bfloat16 terms, hi hi + hi lo + lo hi, but for
// the scores inside a sub-block, which keep 32 bits; projections are bfloat16 as they are, their unit norms factors of the results.
#include "chunk_mma.cuh"
#include "f32x2.cuh"

namespace {

constexpr float LOG2E_F = 1.4426950408889634f;

// hi and lo terms of two neighbouring values of a row of a swizzled [rows][D] tile
template <int D>
__device__ __forceinline__ void put_split(unsigned char* hi_tile, unsigned char* lo_tile, int row, int col, float x, float y) {
  uint32_t hi, lo;
  split_pack(x, y, hi, lo);
  const uint32_t off = swz<D>(row, col >> 3) + (col & 7) * 2;
  *reinterpret_cast<uint32_t*>(hi_tile + off) = hi;
  *reinterpret_cast<uint32_t*>(lo_tile + off) = lo;
}

template <int N>
struct Count {       // a number that an unrolled loop knows
  __device__ constexpr operator int() const { return N; }
};

template <int DK, int DV, bool PER_HEAD>
struct LocalSmem {
  static constexpr int KP = DK + 8, CP = PER_HEAD ? 1 : DK + 8, TP = CH + 4;
  static constexpr int cb = 0;                                   // [CH][CP] float: sums of logarithms from the sub-block's start
  static constexpr int tot = cb + (CH * CP * 4 + 127) / 128 * 128;   // [4][DK] float: the sub-blocks' totals
  static constexpr int fr = tot + (PER_HEAD ? 128 : 4 * DK * 4); // [4][DK] float: the totals of the sub-blocks before each, summed
  static constexpr int bk = fr + (PER_HEAD ? 128 : 4 * DK * 4);  // [4][DK] float: of those after
  static constexpr int q = bk + (PER_HEAD ? 128 : 4 * DK * 4);   // [CH][KP] bfloat16
  static constexpr int k = q + CH * KP * 2;
  static constexpr int v = k + CH * KP * 2;                      // [CH][DV] swizzled: values, then U_0's hi
  static constexpr int a = v + CH * DV * 2;                      // [CH][TP] float: L, then T diag(beta) hi and lo [CH][CH]
  static constexpr int p = a + CH * TP * 4;                      // P hi and lo [CH][CH]
  static constexpr int t = p + 2 * CH * CH * 2;                  // [CH][TP] float: (I + L)^-1
  static constexpr int x = t + CH * TP * 4;                      // [32][32] float, or two of [16][16]
  static constexpr int kw = x + 4 * 256 * 4;                     // Kc hi and lo [CH][DK], then W
  static constexpr int ulo = kw + 2 * CH * DK * 2;               // [CH][DV]: U_0's lo
  static constexpr int kd = ulo + CH * DV * 2;                   // Kd hi and lo [CH][DK]
  static constexpr int small = kd + 2 * CH * DK * 2;             // rq, rk, beta [CH] float each
  static constexpr int bytes = small + 3 * CH * 4;
};

// One block = one chunk x one head; DK / 8 warps. What bounds it: a block takes 225 KB of shared memory, so an SM holds one, and its
// phases are short chains between barriers (decay per channel, 128 x 128: 42,000 clocks a block, of them scores 12,000, products 14,000,
// loads 5,400, the inverse with the decayed keys 5,000 and its join 4,000; 79,400 before). So the scores' work is divided by count of
// instructions over all warps: a pair of sub-blocks' keys and queries take the same exponentials and the same decayed keys, halves of a sub-block
// meet by a product too (in three terms), which leaves 288 pairs of tokens with exponents of their own of 544; totals before and after a sub-block are
// kept instead of summed at every use; decayed keys are formed four channels a lane (one channel's neighbours in a lane met the
// same bank eight times); the inverse joins 16 below 16, then 32 below 32, from rows in 16-byte words. 2,048 tokens of 16 heads of
// 128 x 128, both passes 222 -> 171 us (this one 153 -> 102).
// mq [chunk][head][DK / 16 + 4 row tiles][DK / 16][hi, lo][32 lanes] 16-byte words: M's rows, then Q's, as mma A fragments.
// bo [chunk][head][DK / 16 + 4 row tiles][DV / 8][32 lanes] float4: B's rows, then O_0's, as mma C fragments.
// dec [chunk][head][DK]: exp(c_n).
template <int DK, int DV, bool PER_HEAD>
__global__ void __launch_bounds__(DK * 4)
delta_chunk_local_kernel(const __nv_bfloat16* __restrict__ act, const float* __restrict__ inv, const float* __restrict__ logd,
                         const float* __restrict__ beta, StepBatch sb, const int* __restrict__ chunk_seq,
                         const int* __restrict__ chunk_q0, uint4* __restrict__ mq, float4* __restrict__ bo,
                         float* __restrict__ dec, int heads, int kv_heads) {
  using L = LocalSmem<DK, DV, PER_HEAD>;
  extern __shared__ __align__(128) unsigned char sm[];
  constexpr int NW = DK / 8, NT = NW * 32, KP = L::KP, CP = L::CP, TP = L::TP, MT = DK / 16 + 4;
  float* cb = reinterpret_cast<float*>(sm + L::cb);
  float *tot = reinterpret_cast<float*>(sm + L::tot), *fr = reinterpret_cast<float*>(sm + L::fr), *bk = reinterpret_cast<float*>(sm + L::bk);
  __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(sm + L::q);
  __nv_bfloat16* ks = reinterpret_cast<__nv_bfloat16*>(sm + L::k);
  float* As = reinterpret_cast<float*>(sm + L::a);
  float* Ts = reinterpret_cast<float*>(sm + L::t);
  float* Xs = reinterpret_cast<float*>(sm + L::x);
  unsigned char *p_hi = sm + L::p, *p_lo = p_hi + CH * CH * 2, *t_hi = sm + L::a, *t_lo = t_hi + CH * CH * 2;
  unsigned char *w_hi = sm + L::kw, *w_lo = w_hi + CH * DK * 2, *u_hi = sm + L::v, *u_lo = sm + L::ulo;
  unsigned char *kd_hi = sm + L::kd, *kd_lo = kd_hi + CH * DK * 2;
  float *rq = reinterpret_cast<float*>(sm + L::small), *rk = rq + CH, *bt = rk + CH;
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g4 = lane >> 2, t4 = lane & 3, m = lane >> 3;
  const int seq = chunk_seq[c], q0 = chunk_q0[c];
  const int start = sb.seq_start[seq] + q0, n = min(CH, sb.seq_new[seq] - q0);
  const int g = h / (heads / kv_heads), C = 2 * kv_heads * DK + heads * DV;

  // ---- the chunk's rows (tokens from n on: zeros, beta 0)
  {
    StagedWords<DK, NT> qw, kw;
    StagedWords<DV, NT> vw;
    const __nv_bfloat16* row0 = act + size_t(start) * C;
    qw.load(row0 + g * DK, C, n, tid);
    kw.load(row0 + kv_heads * DK + g * DK, C, n, tid);
    vw.load(row0 + 2 * kv_heads * DK + h * DV, C, n, tid);
    if constexpr (!PER_HEAD) {
      constexpr int QUADS = DK / 4, PER = CH * QUADS / NT;
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int i = tid + u * NT, row = i / QUADS, d = i % QUADS * 4;
        float4 l = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < n) l = *reinterpret_cast<const float4*>(logd + (size_t(start + row) * heads + h) * DK + d);
        *reinterpret_cast<float4*>(cb + row * CP + d) = make_float4(l.x * LOG2E_F, l.y * LOG2E_F, l.z * LOG2E_F, l.w * LOG2E_F);
      }
    } else {
      if (tid < CH) cb[tid] = tid < n ? logd[size_t(start + tid) * heads + h] * LOG2E_F : 0.f;
    }
    if (tid < CH) {
      const bool on = tid < n;
      rq[tid] = on ? inv[size_t(start + tid) * 2 * kv_heads + g] : 0.f;
      rk[tid] = on ? inv[size_t(start + tid) * 2 * kv_heads + kv_heads + g] : 0.f;
      bt[tid] = on ? beta[size_t(start + tid) * heads + h] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < qw.PER; ++u) {
      const int i = tid + u * NT, row = i / (DK / 8), cc = i % (DK / 8);
      *reinterpret_cast<uint4*>(qs + row * KP + cc * 8) = qw.w[u];
      *reinterpret_cast<uint4*>(ks + row * KP + cc * 8) = kw.w[u];
    }
    vw.store(u_hi, 0, tid);
    for (int i = tid; i < 2 * CH * CH * 2 / 16; i += NT) reinterpret_cast<uint4*>(p_hi)[i] = make_uint4(0, 0, 0, 0);
  }
  __syncthreads();

  // ---- sums of logarithms from each sub-block's start
  if constexpr (PER_HEAD) {
    if (tid < 4) {
      float s = 0.f;
      for (int i = 0; i < 16; ++i) cb[tid * 16 + i] = s += cb[tid * 16 + i];
      tot[tid] = s;
    }
  } else {
    for (int i = tid; i < 4 * DK; i += NT) {
      const int b = i / DK, d = i % DK;
      float s = 0.f;
#pragma unroll
      for (int r = 0; r < 16; ++r) cb[(b * 16 + r) * CP + d] = s += cb[(b * 16 + r) * CP + d];
      tot[b * DK + d] = s;
    }
  }
  __syncthreads();
  // the totals before and after every sub-block (read after the next barrier)
  constexpr int LD = PER_HEAD ? 1 : DK;
  for (int i = tid; i < 4 * LD; i += NT) {
    const int b = i / LD, d = i % LD;
    float f = 0.f, e = 0.f;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const float t = tot[o * LD + d];
      if (o < b) f += t;
      if (o > b) e += t;
    }
    fr[i] = f;
    bk[i] = e;
  }
  // exponents (base 2) of two neighbouring channels from the chunk's start to the token
  auto from_start = [&](int row, int d) {
    if constexpr (PER_HEAD) {
      const float x = fr[row / 16] + cb[row];
      return make_float2(x, x);
    } else {
      const float2 f = *reinterpret_cast<const float2*>(fr + row / 16 * DK + d), c2 = *reinterpret_cast<const float2*>(cb + row * CP + d);
      return make_float2(f.x + c2.x, f.y + c2.y);
    }
  };
  // ---- L and P
  auto put_scores = [&](int i, int j, int nt, const float (&l)[4], const float (&q)[4], auto factor) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int row = i * 16 + g4 + half * 8, col = j * 16 + nt * 8 + t4 * 2;
      float f[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) f[e] = rk[col + e] * factor(row, col + e);
      const float b = rk[row] * bt[row];
      As[row * TP + col] = l[half * 2] * f[0] * b;
      As[row * TP + col + 1] = l[half * 2 + 1] * f[1] * b;
      put_split<CH>(p_hi, p_lo, row, col, q[half * 2] * f[0] * rq[row], q[half * 2 + 1] * f[1] * rq[row]);
    }
  };
  if constexpr (PER_HEAD) {
    // one decay per head: a factor of the product's result, also inside sub-blocks; a warp per (later, earlier)
    for (int pair = warp; pair < 10; pair += NW) {       // (0,0) (1,0) (1,1) (2,0) ...
      const int i = pair < 1 ? 0 : (pair < 3 ? 1 : (pair < 6 ? 2 : 3)), j = pair - i * (i + 1) / 2;
      float l[2][4] = {}, q[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < DK / 16; ++kk) {
        uint32_t ak[4], aq[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const int at = (i * 16 + g4 + (f & 1) * 8) * KP + kk * 16 + t4 * 2 + (f >> 1) * 8;
          ak[f] = *reinterpret_cast<const uint32_t*>(ks + at);
          aq[f] = *reinterpret_cast<const uint32_t*>(qs + at);
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const __nv_bfloat16* b = ks + (j * 16 + nt * 8 + g4) * KP + kk * 16 + t4 * 2;
          const uint32_t b0 = *reinterpret_cast<const uint32_t*>(b), b1 = *reinterpret_cast<const uint32_t*>(b + 8);
          mma_bf16(l[nt], ak, b0, b1);
          mma_bf16(q[nt], aq, b0, b1);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
        put_scores(i, j, nt, l[nt], q[nt], [&](int row, int col) {
          float x = i == j ? cb[row] - cb[col] : tot[j] - cb[col] + cb[row];
          for (int b = j + 1; b < i; ++b) x += tot[b];
          return col <= row ? fast_exp2(x) : 0.f;       // what comes later takes no part
        });
    }
  } else {
    // Between sub-blocks a warp a pair (later, earlier): keys and queries of the later one take the same exponentials, and L and P the
    // same decayed keys of the earlier one. Inside a sub-block the later half meets the earlier one in the same way, with the sums from
    // the halves' border: keys and queries are the two halves of the matrix instruction's rows. Inside a half every pair of tokens has
    // exponents of its own, four lanes along the channels, eight pairs a warp at a time.
    // KSPLIT warps share a pair's channels; the second one's sums wait where the decayed keys will stand.
    constexpr int KSPLIT = NW == 16 ? 2 : 1;
    if (warp < 6 * KSPLIT) {
      const int pair = warp / KSPLIT, part = warp % KSPLIT;          // (1,0) (2,0) (2,1) (3,0) ...
      const int i = pair < 1 ? 1 : (pair < 3 ? 2 : 3), j = pair - i * (i - 1) / 2;
      float l[2][4] = {}, q[2][4] = {};
#pragma unroll 2
      for (int kk = part * (DK / 16 / KSPLIT); kk < (part + 1) * (DK / 16 / KSPLIT); ++kk) {
        uint32_t kh[4], kl[4], qh[4], ql[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const int row = i * 16 + g4 + (f & 1) * 8, d = kk * 16 + t4 * 2 + (f >> 1) * 8;
          const uint32_t wk = *reinterpret_cast<const uint32_t*>(ks + row * KP + d), wq = *reinterpret_cast<const uint32_t*>(qs + row * KP + d);
          float2 e = *reinterpret_cast<const float2*>(cb + row * CP + d);
          e.x = fast_exp2(e.x), e.y = fast_exp2(e.y);
          split_pack(__uint_as_float(wk << 16) * e.x, __uint_as_float(wk & 0xffff0000u) * e.y, kh[f], kl[f]);
          split_pack(__uint_as_float(wq << 16) * e.x, __uint_as_float(wq & 0xffff0000u) * e.y, qh[f], ql[f]);
        }
        float2 mid[2];      // the whole sub-blocks between
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          const int d = kk * 16 + t4 * 2 + f * 8;
          mid[f] = *reinterpret_cast<const float2*>(tot + j * DK + d);
#pragma unroll
          for (int b = 1; b < 3; ++b) {
            if (b <= j || b >= i) continue;
            const float2 o = *reinterpret_cast<const float2*>(tot + b * DK + d);
            mid[f].x += o.x;
            mid[f].y += o.y;
          }
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          uint32_t bh[2], bl[2];
#pragma unroll
          for (int f = 0; f < 2; ++f) {
            const int row = j * 16 + nt * 8 + g4, d = kk * 16 + t4 * 2 + f * 8;
            const uint32_t w = *reinterpret_cast<const uint32_t*>(ks + row * KP + d);
            const float2 e = *reinterpret_cast<const float2*>(cb + row * CP + d);
            split_pack(__uint_as_float(w << 16) * fast_exp2(mid[f].x - e.x), __uint_as_float(w & 0xffff0000u) * fast_exp2(mid[f].y - e.y), bh[f], bl[f]);
          }
          mma_bf16(l[nt], kh, bh[0], bh[1]);
          mma_bf16(q[nt], qh, bh[0], bh[1]);
          mma_bf16(l[nt], kh, bl[0], bl[1]);
          mma_bf16(q[nt], qh, bl[0], bl[1]);
          mma_bf16(l[nt], kl, bh[0], bh[1]);
          mma_bf16(q[nt], ql, bh[0], bh[1]);
        }
      }
      if constexpr (KSPLIT == 2) {
        float4* wait = reinterpret_cast<float4*>(kd_hi) + pair * 4 * 32 + lane;
        if (part == 1) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            wait[nt * 32] = make_float4(l[nt][0], l[nt][1], l[nt][2], l[nt][3]);
            wait[(2 + nt) * 32] = make_float4(q[nt][0], q[nt][1], q[nt][2], q[nt][3]);
          }
        }
        asm volatile("bar.sync %0, 64;\n" ::"r"(pair + 1) : "memory");      // the pair's two warps
        if (part == 0) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const float4 x = wait[nt * 32], y = wait[(2 + nt) * 32];
            l[nt][0] += x.x, l[nt][1] += x.y, l[nt][2] += x.z, l[nt][3] += x.w;
            q[nt][0] += y.x, q[nt][1] += y.y, q[nt][2] += y.z, q[nt][3] += y.w;
          }
        }
      }
      if (part == 0) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) put_scores(i, j, nt, l[nt], q[nt], [](int, int) { return 1.f; });
      }
    }
    // The nearest tokens' scores keep 32 bits, as inside a half: operands of three terms, the six products of 16 channels from zero, the
    // small ones first (a matrix instruction cuts its sum off), and rounded additions of these. With two terms a score was 4.5e-6 off 64
    // bits, and a sub-block's outputs 5.9e-6 where they are 5.2e-6 (the products after the scores); the layer took 296.7 us, now 298.2.
    auto halves_meet = [&](int b) {
      float acc[4] = {};      // rows 0 - 7: L, rows 8 - 15: P
      const int row = b * 16 + 8 + g4, col = b * 16 + g4, edge = b * 16 + 7;
#pragma unroll 1
      for (int kk = 0; kk < DK / 16; ++kk) {
        uint32_t a1[4], a2[4], a3[4], b1[2], b2[2], b3[2];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          const int d = kk * 16 + t4 * 2 + f * 8;
          const float2 m = *reinterpret_cast<const float2*>(cb + edge * CP + d);
          float2 e = *reinterpret_cast<const float2*>(cb + row * CP + d);
          e.x = fast_exp2(e.x - m.x), e.y = fast_exp2(e.y - m.y);
          const uint32_t wk = *reinterpret_cast<const uint32_t*>(ks + row * KP + d), wq = *reinterpret_cast<const uint32_t*>(qs + row * KP + d);
          split3_pack(__uint_as_float(wk << 16) * e.x, __uint_as_float(wk & 0xffff0000u) * e.y, a1[2 * f], a2[2 * f], a3[2 * f]);
          split3_pack(__uint_as_float(wq << 16) * e.x, __uint_as_float(wq & 0xffff0000u) * e.y, a1[2 * f + 1], a2[2 * f + 1], a3[2 * f + 1]);
          const uint32_t w = *reinterpret_cast<const uint32_t*>(ks + col * KP + d);
          const float2 o = *reinterpret_cast<const float2*>(cb + col * CP + d);
          split3_pack(__uint_as_float(w << 16) * fast_exp2(m.x - o.x), __uint_as_float(w & 0xffff0000u) * fast_exp2(m.y - o.y), b1[f], b2[f], b3[f]);
        }
        float x[4] = {};
        mma_bf16(x, a3, b1[0], b1[1]);
        mma_bf16(x, a1, b3[0], b3[1]);
        mma_bf16(x, a2, b2[0], b2[1]);
        mma_bf16(x, a2, b1[0], b1[1]);
        mma_bf16(x, a1, b2[0], b2[1]);
        mma_bf16(x, a1, b1[0], b1[1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] += x[e];
      }
      const int c0 = b * 16 + t4 * 2;
      const float w = rk[row] * bt[row];
      As[row * TP + c0] = acc[0] * rk[c0] * w;
      As[row * TP + c0 + 1] = acc[1] * rk[c0 + 1] * w;
      put_split<CH>(p_hi, p_lo, row, c0, acc[2] * rk[c0] * rq[row], acc[3] * rk[c0 + 1] * rq[row]);
    };
    // shares by count of instructions: a pair's half of the channels costs what two halves of a sub-block do, or two and a half eights
    constexpr int EIGHTS = 8 * 36 / 8;
    int eight, step, last;
    if constexpr (NW == 16) {
      if (warp >= 12) halves_meet(warp - 12);
      eight = warp < 12 ? warp : 24 + warp - 12;
      step = warp < 12 ? 12 : 4;
      last = warp < 12 ? 24 : EIGHTS;
    } else {
      if (warp >= 6) {
        halves_meet(2 * (warp - 6));
        halves_meet(2 * (warp - 6) + 1);
      }
      eight = warp < 6 ? 8 + warp : warp - 6;
      step = warp < 6 ? 6 : 2;
      last = warp < 6 ? EIGHTS : 8;
    }
    const int sub = lane & 3;
    for (; eight < last; eight += step) {
      const int task = eight * 8 + (lane >> 2), b = task / 36, pr = task % 36, ra = pr / 9, rb = pr % 9;
      const int r = rb <= ra ? ra : 7 - ra, s = rb <= ra ? rb : rb - ra - 1;     // s <= r
      const int row = b * 8 + r, col = b * 8 + s;
      uint64_t a2 = 0ull, p2 = 0ull;      // the even and the odd channels' sums
#pragma unroll 4
      for (int d = sub * 4; d < DK; d += 16) {
        const ulonglong2 ct = *reinterpret_cast<const ulonglong2*>(cb + row * CP + d);
        const ulonglong2 cs = *reinterpret_cast<const ulonglong2*>(cb + col * CP + d);
        const uint2 kt = *reinterpret_cast<const uint2*>(ks + row * KP + d);
        const uint2 k2 = *reinterpret_cast<const uint2*>(ks + col * KP + d);
        const uint2 qt = *reinterpret_cast<const uint2*>(qs + row * KP + d);
        const float2 x = halves2(minus2(ct.x, cs.x)), y = halves2(minus2(ct.y, cs.y));
        const uint64_t e0 = mul2(wide2(k2.x), pack2(fast_exp2(x.x), fast_exp2(x.y)));
        const uint64_t e1 = mul2(wide2(k2.y), pack2(fast_exp2(y.x), fast_exp2(y.y)));
        a2 = fma2(wide2(kt.x), e0, a2);
        a2 = fma2(wide2(kt.y), e1, a2);
        p2 = fma2(wide2(qt.x), e0, p2);
        p2 = fma2(wide2(qt.y), e1, p2);
      }
      float a = halves2(a2).x + halves2(a2).y, p = halves2(p2).x + halves2(p2).y;
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      p += __shfl_xor_sync(0xffffffffu, p, 1);
      a += __shfl_xor_sync(0xffffffffu, a, 2);
      p += __shfl_xor_sync(0xffffffffu, p, 2);
      if (sub == 0) {
        As[row * TP + col] = a * rk[col] * rk[row] * bt[row];      // the diagonal is not read
        const float v = p * rk[col] * rq[row];
        const __nv_bfloat16 hi = __float2bfloat16_rn(v), lo = __float2bfloat16_rn(v - __bfloat162float(hi));
        const uint32_t off = swz<CH>(row, col >> 3) + (col & 7) * 2;
        *reinterpret_cast<__nv_bfloat16*>(p_hi + off) = hi;
        *reinterpret_cast<__nv_bfloat16*>(p_lo + off) = lo;
      }
    }
  }
  __syncthreads();

  // ---- (I + L)^-1 by sub-blocks: the four on the diagonal by substitution, a thread per column of the first two warps
  if (tid < 64) {
    const int b = tid / 16, cc = tid % 16;
    const float* Lb = As + b * 16 * TP + b * 16;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      float s = r == cc ? 1.f : 0.f;
#pragma unroll
      for (int i = 0; i < r; i += 4) {
        const float4 l = *reinterpret_cast<const float4*>(Lb + r * TP + i);
        const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (i + e < r) s = fmaf(-lv[e], x[i + e], s);
      }
      x[r] = s;
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) Ts[(b * 16 + r) * TP + b * 16 + cc] = x[r];
  }
  // decayed keys meanwhile, four channels a thread (neighbouring lanes' words then meet no bank twice): both as they stand at the
  // token and as they reach the chunk's end
  for (int i = tid - 64; i >= 0 && i < CH * (DK / 4); i += NT - 64) {
    const int row = i / (DK / 4), d = i % (DK / 4) * 4;
    const uint2 w = *reinterpret_cast<const uint2*>(ks + row * KP + d);
    const float r = rk[row];
    const float x[4] = {__uint_as_float(w.x << 16) * r, __uint_as_float(w.x & 0xffff0000u) * r, __uint_as_float(w.y << 16) * r,
                        __uint_as_float(w.y & 0xffff0000u) * r};
    float up[4], down[4];
    if constexpr (PER_HEAD) {
      const float u = fast_exp2(fr[row / 16] + cb[row]), v = fast_exp2((tot[row / 16] - cb[row]) + bk[row / 16]);
#pragma unroll
      for (int e = 0; e < 4; ++e) up[e] = u, down[e] = v;
    } else {
      const float4 f = *reinterpret_cast<const float4*>(fr + row / 16 * DK + d), t = *reinterpret_cast<const float4*>(tot + row / 16 * DK + d);
      const float4 z = *reinterpret_cast<const float4*>(bk + row / 16 * DK + d), y = *reinterpret_cast<const float4*>(cb + row * CP + d);
      up[0] = fast_exp2(f.x + y.x), up[1] = fast_exp2(f.y + y.y), up[2] = fast_exp2(f.z + y.z), up[3] = fast_exp2(f.w + y.w);
      down[0] = fast_exp2((t.x - y.x) + z.x), down[1] = fast_exp2((t.y - y.y) + z.y);
      down[2] = fast_exp2((t.z - y.z) + z.z), down[3] = fast_exp2((t.w - y.w) + z.w);
    }
    uint2 hi, lo, hi2, lo2;
    split_pack(x[0] * up[0], x[1] * up[1], hi.x, lo.x);
    split_pack(x[2] * up[2], x[3] * up[3], hi.y, lo.y);
    split_pack(x[0] * down[0], x[1] * down[1], hi2.x, lo2.x);
    split_pack(x[2] * down[2], x[3] * down[3], hi2.y, lo2.y);
    const uint32_t off = swz<DK>(row, d >> 3) + (d & 4) * 2;
    *reinterpret_cast<uint2*>(w_hi + off) = hi;
    *reinterpret_cast<uint2*>(w_lo + off) = lo;
    *reinterpret_cast<uint2*>(kd_hi + off) = hi2;
    *reinterpret_cast<uint2*>(kd_lo + off) = lo2;
  }
  for (int d = tid; d < DK; d += NT)
    dec[(size_t(c) * heads + h) * DK + d] = fast_exp2(fr[3 * LD + (PER_HEAD ? 0 : d)] + tot[3 * LD + (PER_HEAD ? 0 : d)]);
  __syncthreads();
  // ... and the others, T_21 = -T_22 (L_21 T_11): first of 16 rows below 16, then of 32 below 32; four columns a thread
  auto row_times = [&](const float* left, const float* right, int pitch, int from, auto to, float4& s) {     // += sum_x left[x] right[x][0..3]
#pragma unroll
    for (int x = 0; x < to; x += 4) {
      if (x < from) continue;
      const float4 l = *reinterpret_cast<const float4*>(left + x);
      const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 t = *reinterpret_cast<const float4*>(right + (x + e) * pitch);
        s.x = fmaf(lv[e], t.x, s.x), s.y = fmaf(lv[e], t.y, s.y), s.z = fmaf(lv[e], t.z, s.z), s.w = fmaf(lv[e], t.w, s.w);
      }
    }
  };
  {
    const int i = tid / 64 * 2 + 1, j = i - 1, r = tid % 64 / 4, cc = tid % 4 * 4;
    const bool on = tid < 128;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
      row_times(As + (i * 16 + r) * TP + j * 16, Ts + j * 16 * TP + j * 16 + cc, TP, 0, Count<16>(), s);
      *reinterpret_cast<float4*>(Xs + (tid / 64) * 256 + r * 16 + cc) = s;
    }
    __syncthreads();
    if (on) {
      s = make_float4(0.f, 0.f, 0.f, 0.f);
      row_times(Ts + (i * 16 + r) * TP + i * 16, Xs + (tid / 64) * 256 + cc, 16, 0, Count<16>(), s);
      *reinterpret_cast<float4*>(Ts + (i * 16 + r) * TP + j * 16 + cc) = make_float4(-s.x, -s.y, -s.z, -s.w);
    }
    __syncthreads();
  }
  {
    const int r = tid / 8, cc = tid % 8 * 4;      // a row and four columns of 32 x 32
    const bool on = tid < 256;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
      row_times(As + (32 + r) * TP, Ts + cc, TP, cc & 16, Count<32>(), s);      // above the diagonal T_11 is zero
      *reinterpret_cast<float4*>(Xs + r * 32 + cc) = s;
    }
    __syncthreads();
    if (on) {
      s = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < 16) row_times(Ts + (32 + r) * TP + 32, Xs + cc, 32, 0, Count<16>(), s);
      else row_times(Ts + (32 + r) * TP + 32, Xs + cc, 32, 0, Count<32>(), s);
      *reinterpret_cast<float4*>(Ts + (32 + r) * TP + cc) = make_float4(-s.x, -s.y, -s.z, -s.w);
    }
    __syncthreads();
  }
  for (int i = tid; i < CH * (CH / 8); i += NT) {      // T diag(beta), over L
    const int row = i / (CH / 8), cc = i % (CH / 8);
    uint4 hi, lo;
    uint32_t *H = &hi.x, *Lo = &lo.x;
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const int s = cc * 8 + e;
      split_pack(s <= row ? Ts[row * TP + s] * bt[s] : 0.f, s + 1 <= row ? Ts[row * TP + s + 1] * bt[s + 1] : 0.f, H[e / 2], Lo[e / 2]);
    }
    *reinterpret_cast<uint4*>(t_hi + swz<CH>(row, cc)) = hi;
    *reinterpret_cast<uint4*>(t_lo + swz<CH>(row, cc)) = lo;
  }
  __syncthreads();

  // ---- W = T Kc and U_0 = T V: row tile mi, a stretch of columns; sub-blocks after the row tile's are zero
  constexpr int GROUPS = NW / 4, WN = DK / GROUPS / 8, UN = DV / GROUPS / 8;     // column tiles of a warp
  const int mi = warp & 3, ng = warp >> 2;
  const uint32_t th = smem_u32(t_hi), tl = smem_u32(t_lo), wh = smem_u32(w_hi), wl = smem_u32(w_lo), uh = smem_u32(u_hi), ul = smem_u32(u_lo);
  float wa[WN][4] = {}, ua[UN][4] = {};
  for (int kk = 0; kk <= mi; ++kk) {
    uint32_t ah[4], al[4];
    const uint32_t off = swz<CH>(mi * 16 + (lane & 15), kk * 2 + (lane >> 4));
    ldmatrix_x4(ah[0], ah[1], ah[2], ah[3], th + off);
    ldmatrix_x4(al[0], al[1], al[2], al[3], tl + off);
#pragma unroll
    for (int j = 0; j < WN; j += 2) {
      uint32_t b[4], bl[4];
      const uint32_t bo_ = swz<DK>(kk * 16 + (m & 1) * 8 + (lane & 7), ng * WN + j + (m >> 1));
      ldmatrix_x4_trans(b[0], b[1], b[2], b[3], wh + bo_);
      ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], wl + bo_);
      mma_bf16(wa[j], ah, b[0], b[1]);
      mma_bf16(wa[j + 1], ah, b[2], b[3]);
      mma_bf16(wa[j], ah, bl[0], bl[1]);
      mma_bf16(wa[j + 1], ah, bl[2], bl[3]);
      mma_bf16(wa[j], al, b[0], b[1]);
      mma_bf16(wa[j + 1], al, b[2], b[3]);
    }
#pragma unroll
    for (int j = 0; j < UN; j += 2) {
      uint32_t b[4];
      ldmatrix_x4_trans(b[0], b[1], b[2], b[3], uh + swz<DV>(kk * 16 + (m & 1) * 8 + (lane & 7), ng * UN + j + (m >> 1)));
      mma_bf16(ua[j], ah, b[0], b[1]);
      mma_bf16(ua[j + 1], ah, b[2], b[3]);
      mma_bf16(ua[j], al, b[0], b[1]);
      mma_bf16(ua[j + 1], al, b[2], b[3]);
    }
  }
  __syncthreads();      // Kc and V have been read by everybody: W and U_0 take their places
#pragma unroll
  for (int j = 0; j < WN; ++j) {
    const int col = (ng * WN + j) * 8 + t4 * 2;
    put_split<DK>(w_hi, w_lo, mi * 16 + g4, col, wa[j][0], wa[j][1]);
    put_split<DK>(w_hi, w_lo, mi * 16 + g4 + 8, col, wa[j][2], wa[j][3]);
  }
#pragma unroll
  for (int j = 0; j < UN; ++j) {
    const int col = (ng * UN + j) * 8 + t4 * 2;
    put_split<DV>(u_hi, u_lo, mi * 16 + g4, col, ua[j][0], ua[j][1]);
    put_split<DV>(u_hi, u_lo, mi * 16 + g4 + 8, col, ua[j][2], ua[j][3]);
  }
  __syncthreads();

  uint4* mq_c = mq + (size_t(c) * heads + h) * MT * (DK / 16) * 2 * 32;
  float4* bo_c = bo + (size_t(c) * heads + h) * MT * (DV / 8) * 32;
  // ---- Q = Qc - P W and O_0 = P U_0
  {
    const uint32_t ph = smem_u32(p_hi), pl = smem_u32(p_lo);
#pragma unroll
    for (int j = 0; j < WN; ++j) wa[j][0] = wa[j][1] = wa[j][2] = wa[j][3] = 0.f;
#pragma unroll
    for (int j = 0; j < UN; ++j) ua[j][0] = ua[j][1] = ua[j][2] = ua[j][3] = 0.f;
    for (int kk = 0; kk <= mi; ++kk) {
      uint32_t ah[4], al[4];
      const uint32_t off = swz<CH>(mi * 16 + (lane & 15), kk * 2 + (lane >> 4));
      ldmatrix_x4(ah[0], ah[1], ah[2], ah[3], ph + off);
      ldmatrix_x4(al[0], al[1], al[2], al[3], pl + off);
      auto three = [&](float (&acc0)[4], float (&acc1)[4], uint32_t hi_at, uint32_t lo_at) {
        uint32_t b[4], bl[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], hi_at);
        ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], lo_at);
        mma_bf16(acc0, ah, b[0], b[1]);
        mma_bf16(acc1, ah, b[2], b[3]);
        mma_bf16(acc0, ah, bl[0], bl[1]);
        mma_bf16(acc1, ah, bl[2], bl[3]);
        mma_bf16(acc0, al, b[0], b[1]);
        mma_bf16(acc1, al, b[2], b[3]);
      };
#pragma unroll
      for (int j = 0; j < WN; j += 2) {
        const uint32_t o = swz<DK>(kk * 16 + (m & 1) * 8 + (lane & 7), ng * WN + j + (m >> 1));
        three(wa[j], wa[j + 1], wh + o, wl + o);
      }
#pragma unroll
      for (int j = 0; j < UN; j += 2) {
        const uint32_t o = swz<DV>(kk * 16 + (m & 1) * 8 + (lane & 7), ng * UN + j + (m >> 1));
        three(ua[j], ua[j + 1], uh + o, ul + o);
      }
    }
#pragma unroll
    for (int j = 0; j < WN; j += 2) {     // two column tiles of C fragments are one A fragment of 16 columns
      uint4 hi, lo;
      uint32_t *H = &hi.x, *Lo = &lo.x;
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const int row = mi * 16 + g4 + (f & 1) * 8, d = (ng * WN + j + (f >> 1)) * 8 + t4 * 2;
        const uint32_t w = *reinterpret_cast<const uint32_t*>(qs + row * KP + d);
        const float2 e = from_start(row, d);
        const float x = __uint_as_float(w << 16) * rq[row] * fast_exp2(e.x);
        const float y = __uint_as_float(w & 0xffff0000u) * rq[row] * fast_exp2(e.y);
        split_pack(x - wa[j + (f >> 1)][(f & 1) * 2], y - wa[j + (f >> 1)][(f & 1) * 2 + 1], H[f], Lo[f]);
      }
      uint4* dst = mq_c + ((size_t(DK / 16 + mi) * (DK / 16) + (ng * WN + j) / 2) * 2) * 32 + lane;
      dst[0] = hi;
      dst[32] = lo;
    }
#pragma unroll
    for (int j = 0; j < UN; ++j)
      bo_c[(size_t(DK / 16 + mi) * (DV / 8) + ng * UN + j) * 32 + lane] = make_float4(ua[j][0], ua[j][1], ua[j][2], ua[j][3]);
  }
  // ---- M = -Kd^T W and B = Kd^T U_0: row tile mt of the key channels, half of the columns
  {
    constexpr int MN = DK / 16, BN = DV / 16;      // column tiles of half the columns
    const int mt = warp % (DK / 16), half = warp / (DK / 16);
    const uint32_t kh = smem_u32(kd_hi), kl = smem_u32(kd_lo);
    float ma[MN][4] = {}, ba[BN][4] = {};
#pragma unroll
    for (int kk = 0; kk < CH / 16; ++kk) {
      uint32_t ah[4], al[4];
      const uint32_t off = swz<DK>(kk * 16 + (m >> 1) * 8 + (lane & 7), mt * 2 + (m & 1));
      ldmatrix_x4_trans(ah[0], ah[1], ah[2], ah[3], kh + off);
      ldmatrix_x4_trans(al[0], al[1], al[2], al[3], kl + off);
      auto three = [&](float (&acc0)[4], float (&acc1)[4], uint32_t hi_at, uint32_t lo_at) {
        uint32_t b[4], bl[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], hi_at);
        ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], lo_at);
        mma_bf16(acc0, ah, b[0], b[1]);
        mma_bf16(acc1, ah, b[2], b[3]);
        mma_bf16(acc0, ah, bl[0], bl[1]);
        mma_bf16(acc1, ah, bl[2], bl[3]);
        mma_bf16(acc0, al, b[0], b[1]);
        mma_bf16(acc1, al, b[2], b[3]);
      };
#pragma unroll
      for (int j = 0; j < MN; j += 2) {
        const uint32_t o = swz<DK>(kk * 16 + (m & 1) * 8 + (lane & 7), half * MN + j + (m >> 1));
        three(ma[j], ma[j + 1], wh + o, wl + o);
      }
#pragma unroll
      for (int j = 0; j < BN; j += 2) {
        const uint32_t o = swz<DV>(kk * 16 + (m & 1) * 8 + (lane & 7), half * BN + j + (m >> 1));
        three(ba[j], ba[j + 1], uh + o, ul + o);
      }
    }
#pragma unroll
    for (int j = 0; j < MN; j += 2) {
      uint4 hi, lo;
      split_pack(-ma[j][0], -ma[j][1], hi.x, lo.x);
      split_pack(-ma[j][2], -ma[j][3], hi.y, lo.y);
      split_pack(-ma[j + 1][0], -ma[j + 1][1], hi.z, lo.z);
      split_pack(-ma[j + 1][2], -ma[j + 1][3], hi.w, lo.w);
      uint4* dst = mq_c + ((size_t(mt) * (DK / 16) + (half * MN + j) / 2) * 2) * 32 + lane;
      dst[0] = hi;
      dst[32] = lo;
    }
#pragma unroll
    for (int j = 0; j < BN; ++j)
      bo_c[(size_t(mt) * (DV / 8) + half * BN + j) * 32 + lane] = make_float4(ba[j][0], ba[j][1], ba[j][2], ba[j][3]);
  }
}

// One block = one sequence x one head x 8 NTILE value columns; a warp per row tile of [M; Q]. The chunks in order: the
// warps of M hold the state's float32 values and leave them split in shared memory for all; a chunk's fragments are read
// from memory while the chunk before is multiplied.
template <int DK, int DV, int NTILE>
__global__ void __launch_bounds__((DK / 16 + 4) * 32)
delta_chunk_join_kernel(const uint4* __restrict__ mq, const float4* __restrict__ bo, const float* __restrict__ dec,
                        float* __restrict__ state, int state_stride, int state_off, const int* __restrict__ slots, StepBatch sb,
                        const int* __restrict__ seq_chunk0, float* __restrict__ out, int heads) {
  constexpr int MT = DK / 16 + 4, KS = DK / 16, PITCH = NTILE * 16 + 16;       // bytes of a state row: 16 more than its values
  __shared__ __align__(128) unsigned char s_sm[2][2][DK * PITCH];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g4 = lane >> 2, t4 = lane & 3, m = lane >> 3;
  const int seq = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * NTILE * 8;
  const int n_new = sb.seq_new[seq], c0 = seq_chunk0[seq], start = sb.seq_start[seq];
  const int n_chunks = (n_new + CH - 1) / CH;
  if (n_chunks <= 0) return;
  const bool is_state = warp < KS;
  float* st = state + size_t(slots[seq]) * state_stride + state_off + (size_t(h) * DV + j0) * DK;
  float S[NTILE][4];
  const int d0 = warp * 16 + g4;
#pragma unroll
  for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      S[nt][e] = is_state ? st[size_t(nt * 8 + t4 * 2 + (e & 1)) * DK + d0 + (e >> 1) * 8] : 0.f;
  uint4 a[KS][2];
  float4 init[NTILE];
  float dc0 = 1.f, dc1 = 1.f;
  auto frag = [&](int chunk) { return mq + (((size_t(chunk) * heads + h) * MT + warp) * KS * 2) * 32 + lane; };
  auto rest = [&](int chunk) { return bo + ((size_t(chunk) * heads + h) * MT + warp) * (DV / 8) * 32 + (j0 / 8) * 32 + lane; };
  {
    const uint4* f = frag(c0);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      a[ks][0] = f[(ks * 2) * 32];
      a[ks][1] = f[(ks * 2 + 1) * 32];
    }
    const float4* r = rest(c0);
#pragma unroll
    for (int nt = 0; nt < NTILE; ++nt) init[nt] = r[nt * 32];
    if (is_state) {
      dc0 = dec[(size_t(c0) * heads + h) * DK + d0];
      dc1 = dec[(size_t(c0) * heads + h) * DK + d0 + 8];
    }
  }
  for (int i = 0; i < n_chunks; ++i) {
    unsigned char* hi_s = s_sm[i & 1][0];
    unsigned char* lo_s = s_sm[i & 1][1];
    if (is_state) {
#pragma unroll
      for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t hi, lo;
          split_pack(S[nt][half * 2], S[nt][half * 2 + 1], hi, lo);
          const int at = (d0 + half * 8) * PITCH + nt * 16 + t4 * 4;
          *reinterpret_cast<uint32_t*>(hi_s + at) = hi;
          *reinterpret_cast<uint32_t*>(lo_s + at) = lo;
        }
    }
    // one barrier a chunk: the buffer written next was last read before this barrier
    __syncthreads();
    float acc[NTILE][4], low[NTILE][4] = {};      // the products with a second term apart: half as long a chain of matrix instructions
#pragma unroll
    for (int nt = 0; nt < NTILE; ++nt) {
      acc[nt][0] = init[nt].x; acc[nt][1] = init[nt].y; acc[nt][2] = init[nt].z; acc[nt][3] = init[nt].w;
    }
    const float e0 = dc0, e1 = dc1;
    const bool more = i + 1 < n_chunks;
    const int nxt = c0 + (more ? i + 1 : i);       // after the last chunk its own fragments are read once more and not used
    const uint4* f = frag(nxt);
    {
      const float4* r = rest(nxt);
#pragma unroll
      for (int nt = 0; nt < NTILE; ++nt) init[nt] = r[nt * 32];
      if (is_state) {
        dc0 = dec[(size_t(nxt) * heads + h) * DK + d0];
        dc1 = dec[(size_t(nxt) * heads + h) * DK + d0 + 8];
      }
    }
    const uint32_t hb = smem_u32(hi_s), lb = smem_u32(lo_s);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const uint32_t ah[4] = {a[ks][0].x, a[ks][0].y, a[ks][0].z, a[ks][0].w};
      const uint32_t al[4] = {a[ks][1].x, a[ks][1].y, a[ks][1].z, a[ks][1].w};
      a[ks][0] = f[(ks * 2) * 32];
      a[ks][1] = f[(ks * 2 + 1) * 32];
      const uint32_t row = uint32_t(ks * 16 + (m & 1) * 8 + (lane & 7)) * PITCH + (m >> 1) * 16;
#pragma unroll
      for (int j = 0; j < NTILE; j += 2) {
        uint32_t b[4], bl[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], hb + row + j * 16);
        ldmatrix_x4_trans(bl[0], bl[1], bl[2], bl[3], lb + row + j * 16);
        mma_bf16(acc[j], ah, b[0], b[1]);
        mma_bf16(acc[j + 1], ah, b[2], b[3]);
        mma_bf16(low[j], ah, bl[0], bl[1]);
        mma_bf16(low[j + 1], ah, bl[2], bl[3]);
        mma_bf16(low[j], al, b[0], b[1]);
        mma_bf16(low[j + 1], al, b[2], b[3]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[nt][e] += low[nt][e];
    if (is_state) {
#pragma unroll
      for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[nt][e] = fmaf(e < 2 ? e0 : e1, S[nt][e], acc[nt][e]);
    } else {
      const int t0 = (warp - KS) * 16 + g4;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int t = i * CH + t0 + half * 8;
        if (t < n_new) {
          float* o = out + (size_t(start + t) * heads + h) * DV + j0 + t4 * 2;
#pragma unroll
          for (int nt = 0; nt < NTILE; ++nt) *reinterpret_cast<float2*>(o + nt * 8) = make_float2(acc[nt][half * 2], acc[nt][half * 2 + 1]);
        }
      }
    }
  }
  if (is_state) {
#pragma unroll
    for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) st[size_t(nt * 8 + t4 * 2 + (e & 1)) * DK + d0 + (e >> 1) * 8] = S[nt][e];
  }
}

size_t scratch_part(int n_chunks, int heads, int dk, int dv, int which) {
  const size_t ch = size_t(n_chunks) * heads, mt = dk / 16 + 4;
  const size_t mq = ch * mt * (dk / 16) * 2 * 32 * sizeof(uint4), bo = ch * mt * (dv / 8) * 32 * sizeof(float4);
  return which == 0 ? mq : (which == 1 ? bo : ch * dk * sizeof(float));
}

template <int DK, int DV, bool PER_HEAD>
int launch_local(const void* act, const float* inv, const float* logd, const float* beta, const StepBatch& sb,
                 const int* chunk_seq, const int* chunk_q0, int n_chunks, void* mq, void* bo, float* dec, int heads, int kv_heads,
                 cudaStream_t stream) {
  constexpr int smem = LocalSmem<DK, DV, PER_HEAD>::bytes;
  static SharedLimit limit;
  if (!limit.allows(delta_chunk_local_kernel<DK, DV, PER_HEAD>, smem)) return PTB_ERR_LAUNCH;
  delta_chunk_local_kernel<DK, DV, PER_HEAD><<<dim3(n_chunks, heads), DK * 4, smem, stream>>>(
      (const __nv_bfloat16*)act, inv, logd, beta, sb, chunk_seq, chunk_q0, (uint4*)mq, (float4*)bo, dec, heads, kv_heads);
  return launch_status();
}

template <int DK, int DV>
int launch_chunks(const void* act, const float* inv, const float* logd, const float* beta, float* state, int state_stride,
                  const int* slots, const StepBatch& sb, const int* chunk_seq, const int* chunk_q0, const int* seq_chunk0,
                  int n_chunks, unsigned char* scratch, float* out, int heads, int kv_heads, int taps, int per_head,
                  cudaStream_t stream) {
  unsigned char* mq = scratch;
  unsigned char* bo = mq + scratch_part(n_chunks, heads, DK, DV, 0);
  float* dec = reinterpret_cast<float*>(bo + scratch_part(n_chunks, heads, DK, DV, 1));
  const int rc = per_head ? launch_local<DK, DV, true>(act, inv, logd, beta, sb, chunk_seq, chunk_q0, n_chunks, mq, bo, dec, heads, kv_heads, stream)
                          : launch_local<DK, DV, false>(act, inv, logd, beta, sb, chunk_seq, chunk_q0, n_chunks, mq, bo, dec, heads, kv_heads, stream);
  if (rc != PTB_OK) return rc;
  const int state_off = (taps - 1) * (2 * kv_heads * DK + heads * DV);
  // 32 value columns a block, or 16 where that many blocks would leave half of the device idle (2,048 tokens of 16 heads of
  // 128 x 128: 245 -> 222 us both passes; of 32 heads 16 columns were slower, 362 -> 406). A column's sums are the same.
#define PTB_JOIN(NTILE)                                                                                                        \
  delta_chunk_join_kernel<DK, DV, NTILE><<<dim3(DV / (8 * NTILE), heads, sb.n_seqs), (DK / 16 + 4) * 32, 0, stream>>>(         \
      (const uint4*)mq, (const float4*)bo, dec, state, state_stride, state_off, slots, sb, seq_chunk0, out, heads)
  if ((long long)(DV / 32) * heads * sb.n_seqs * 2 <= sm_count()) PTB_JOIN(2);
  else PTB_JOIN(4);
#undef PTB_JOIN
  return launch_status();
}

}  // namespace

PTB_API int ptb_delta_chunk_tokens() { return CH; }
PTB_API int ptb_delta_chunks_supports(int dim, int v_dim) { return (dim == 64 || dim == 128) && (v_dim == 64 || v_dim == 128); }
PTB_API long long ptb_delta_chunks_scratch_bytes(int n_chunks, int heads, int dim, int v_dim) {
  long long total = 0;
  for (int w = 0; w < 3; ++w) total += (long long)scratch_part(n_chunks, heads, dim, v_dim, w);
  return total;
}

// The step's tokens in chunks: arguments as ptb_delta_walk takes them (bfloat16), and the step's chunks: chunk_seq, chunk_q0
// (sequence and first of its new tokens of every chunk), seq_chunk0 (a sequence's first chunk). scratch: as many bytes as
// ptb_delta_chunks_scratch_bytes says, on a 16-byte boundary.
PTB_API int ptb_delta_chunks(const void* act, const float* inv, const float* logd, const float* beta, float* state,
                             int state_stride, const int* slots, const StepBatch* sb, const int* chunk_seq, const int* chunk_q0,
                             const int* seq_chunk0, int n_chunks, void* scratch, float* out, int heads, int kv_heads, int dim,
                             int v_dim, int taps, int per_head, cudaStream_t stream) {
  if (sb->n_tokens <= 0 || n_chunks <= 0) return PTB_OK;
  if (!ptb_delta_chunks_supports(dim, v_dim) || heads <= 0 || heads > 65535 || kv_heads <= 0 || heads % kv_heads != 0 || taps < 1 ||
      sb->n_seqs > 65535 || state_stride < (taps - 1) * (2 * kv_heads * dim + heads * v_dim) + heads * dim * v_dim)
    return PTB_ERR_SIZE;
  if (!aligned16(act) || !aligned16(scratch) || !aligned16(logd)) return PTB_ERR_ALIGN;
#define PTB_DC(DK, DV)                                                                                                       \
  return launch_chunks<DK, DV>(act, inv, logd, beta, state, state_stride, slots, *sb, chunk_seq, chunk_q0, seq_chunk0, n_chunks, \
                               (unsigned char*)scratch, out, heads, kv_heads, taps, per_head, stream)
  if (dim == 64 && v_dim == 64) PTB_DC(64, 64);
  if (dim == 64 && v_dim == 128) PTB_DC(64, 128);
  if (dim == 128 && v_dim == 64) PTB_DC(128, 64);
  PTB_DC(128, 128);
#undef PTB_DC
}
