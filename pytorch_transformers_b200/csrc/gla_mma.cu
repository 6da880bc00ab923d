// Gated linear attention, passes 1 and 3 of the chunked form on the tensor cores (bfloat16 projections, mma.m16n8k16 with
// float32 sums). Pass 1: a chunk's own sum from a zero state.
//
// A chunk holds n <= 64 tokens j = 0..n-1 with the logarithms l_j [dim] of their decays (float32). Token j's outer
// product k_j v_j^T reaches the chunk's end decayed by the tokens after it, channel by channel:
//     B = sum_j diag(w_j) k_j v_j^T,      w_j[c] = exp(l_(j+1)[c] + .. + l_(n-1)[c])  (<= 1: no factor can grow),
//     total[c] = l_0[c] + .. + l_(n-1)[c]                  the chunk's total decay, for the join
// so B = Kw^T V with Kw[j][c] = w_j[c] k_j[c], a product of [dim, n] by [n, v_dim]. Kw is float32 (the decays and what
// they meet are 32-bit): it enters the product split into two bfloat16 terms, hi + lo; V is a rounded projection.
// The result has the layout of the walk's pass 1 (csrc/gla.cu): sums [chunks][heads][dim][v_dim], chunk_decay
// [chunks][heads][dim].
#include "chunk_mma.cuh"
#include "f32x2.cuh"

namespace {

// One block = one chunk x one head; DK / 16 warps, warp w owns rows 16 w .. 16 w + 15 of B [DK, DV].
template <int DK, int DV>
__global__ void __launch_bounds__(DK * 2)
gla_chunk_sum_mma_kernel(const __nv_bfloat16* __restrict__ proj, int stride, const float* __restrict__ log_decay, StepBatch sb,
                         const int* __restrict__ chunk_seq, const int* __restrict__ chunk_q0, float* __restrict__ sums,
                         float* __restrict__ chunk_decay, int heads) {
  pdl_entry();
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* k_hi = sm;                       // [CH][DK] weighted keys, hi
  unsigned char* k_lo = k_hi + CH * DK * 2;       // lo
  unsigned char* v_s = k_lo + CH * DK * 2;        // [CH][DV]
  float* w_s = reinterpret_cast<float*>(v_s + CH * DV * 2);   // [CH][DK]: the logarithms, then the weights w_j[c]
  constexpr int NT = DK * 2;
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int seq = chunk_seq[c], q0 = chunk_q0[c];
  const int start = sb.seq_start[seq] + q0, n = min(CH, sb.seq_new[seq] - q0);
  const __nv_bfloat16* row0 = proj + size_t(start) * stride;
  StagedWords<DK, NT> kw;
  StagedWords<DV, NT> vw;
  kw.load(row0 + heads * DK + h * DK, stride, n, tid);
  vw.load(row0 + 2 * heads * DK + h * DV, stride, n, tid);
  {   // the chunk's logarithms, four channels a load (rows from n on: zero)
    constexpr int QUADS = DK / 4, PER = CH * QUADS / NT;
    const float* l0 = log_decay + size_t(start) * heads * DK + h * DK;
    float4 l[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid + u * NT, row = i / QUADS, q = i % QUADS;
      l[u] = row < n ? *reinterpret_cast<const float4*>(l0 + size_t(row) * heads * DK + q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid + u * NT, row = i / QUADS, q = i % QUADS;
      *reinterpret_cast<float4*>(w_s + row * DK + q * 4) = l[u];
    }
  }
  __syncthreads();
  if (tid < DK) {     // channel tid from the chunk's last token to its first: what comes after token j, then with it
    float after = 0.f;
#pragma unroll 8
    for (int j = CH - 1; j >= 0; --j) {
      const float l = w_s[j * DK + tid];
      w_s[j * DK + tid] = expf(after);
      after += l;
    }
    chunk_decay[(size_t(c) * heads + h) * DK + tid] = after;
  }
  __syncthreads();
  {
    constexpr int CHUNKS = DK / 8;
#pragma unroll
    for (int u = 0; u < kw.PER; ++u) {
      const int i = tid + u * NT, row = i / CHUNKS, cc = i % CHUNKS;
      float f[8];
      unpack_bf16x8(kw.w[u], f);      // rows from n on were loaded as zeros and their weights are exp(0)
      const float4 wa = *reinterpret_cast<const float4*>(w_s + row * DK + cc * 8);
      const float4 wb = *reinterpret_cast<const float4*>(w_s + row * DK + cc * 8 + 4);
      uint4 hi, lo;
      split_pack(f[0] * wa.x, f[1] * wa.y, hi.x, lo.x);
      split_pack(f[2] * wa.z, f[3] * wa.w, hi.y, lo.y);
      split_pack(f[4] * wb.x, f[5] * wb.y, hi.z, lo.z);
      split_pack(f[6] * wb.z, f[7] * wb.w, hi.w, lo.w);
      *reinterpret_cast<uint4*>(k_hi + swz<DK>(row, cc)) = hi;
      *reinterpret_cast<uint4*>(k_lo + swz<DK>(row, cc)) = lo;
    }
  }
  vw.store(v_s, 0, tid);
  __syncthreads();

  float acc[DV / 8][4];
#pragma unroll
  for (int j = 0; j < DV / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  const uint32_t khi = smem_u32(k_hi), klo = smem_u32(k_lo), vs = smem_u32(v_s);
  const int m = lane >> 3;
#pragma unroll
  for (int kk = 0; kk < CH / 16; ++kk) {
    // A[m = d][k = s] from the [s][d] tiles: transposed 8x8 matrices (d 0-7 | 8-15) x (s 0-7 | 8-15)
    uint32_t ah[4], al[4];
    const uint32_t off = swz<DK>(kk * 16 + (m >> 1) * 8 + (lane & 7), warp * 2 + (m & 1));
    ldmatrix_x4_trans(ah[0], ah[1], ah[2], ah[3], khi + off);
    ldmatrix_x4_trans(al[0], al[1], al[2], al[3], klo + off);
#pragma unroll
    for (int j = 0; j < DV / 8; j += 2) {
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4_trans(b0, b1, b2, b3, vs + swz<DV>(kk * 16 + (m & 1) * 8 + (lane & 7), j + (m >> 1)));
      mma_bf16(acc[j], ah, b0, b1);
      mma_bf16(acc[j], al, b0, b1);
      mma_bf16(acc[j + 1], ah, b2, b3);
      mma_bf16(acc[j + 1], al, b2, b3);
    }
  }
  float* dst = sums + (size_t(c) * heads + h) * DK * DV;
  const int g4 = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int j = 0; j < DV / 8; ++j) {
    *reinterpret_cast<float2*>(dst + size_t(warp * 16 + g4) * DV + j * 8 + t4 * 2) = make_float2(acc[j][0], acc[j][1]);
    *reinterpret_cast<float2*>(dst + size_t(warp * 16 + g4 + 8) * DV + j * 8 + t4 * 2) = make_float2(acc[j][2], acc[j][3]);
  }
}

template <int DK, int DV>
int launch_sum(const void* proj, int stride, const float* log_decay, const StepBatch& sb, const int* chunk_seq,
               const int* chunk_q0, int n_chunks, float* sums, float* chunk_decay, int heads, cudaStream_t stream) {
  const size_t smem = size_t(2) * CH * DK * 2 + size_t(CH) * DV * 2 + size_t(CH) * DK * sizeof(float);
  static SharedLimit limit;
  if (!limit.allows(gla_chunk_sum_mma_kernel<DK, DV>, smem)) return PTB_ERR_LAUNCH;
  launch_pdl(gla_chunk_sum_mma_kernel<DK, DV>, dim3(n_chunks, heads), DK * 2, smem, stream, (const __nv_bfloat16*)proj, stride, log_decay, sb,
                                                                                   chunk_seq, chunk_q0, sums, chunk_decay, heads);
  return launch_status();
}

// ------------------------------------------------------------------------------------------------
// Pass 3 on the tensor cores: a chunk's outputs from the state before it,
//     o_t = q_scale * ( sum_c q_t[c] exp(l_0 + .. + l_t)[c] S0[c]  +  sum_(i <= t) s_ti v_i ),
//     s_ti = sum_c q_t[c] k_i[c] exp(l_(i+1) + .. + l_t)[c].
// The decay differs per key channel, so the scores are no plain product of q and k. The chunk is cut into four sub-blocks of
// 16 tokens. Between sub-blocks u < w the exponent is a sum of three sums of logarithms of one sign, the rest of u after i,
// the whole sub-blocks between, and w up to t: the first goes into the keys, the others into the queries, all factors are at
// most 1, nothing is subtracted, and the scores are a product. Inside a sub-block every (t, i, channel) has an exponent of its
// own: a warp takes four keys and walks the tokens, its lanes' channels' sums for each key in registers; no branch on the keys' places, so that
// the loads run ahead (117 -> 109 us). What bounds this part is the exponential unit: 160 (t, i) pairs a sub-block and channel (ten squares of
// four by four; 24 of them lie before their key and count as zero), 82,000 exponentials a block against 16 a clock and SM. Decaying the four keys to their last one's token, and one exponential for all four from there
// on, took 100 us, but two roundings and an exponential more a term: 1.48e-7 off 64 bits (one chunk, 2-norm) instead of 1.43e-7. 2,900
// tokens of 16 heads of 128 x 128; with operands of two terms 94 (before), the walk on the CUDA cores 175.
// Operands of a product that are float32 (scaled queries and keys, scores, the state) enter it as three bfloat16 terms, 24 bits: what
// a product leaves out (second x third, third x third) is 2^-27.5 of it (root mean square; 2^-24 at most), below the rounding of its float32 sum. A matrix instruction
// cuts its sum off instead of rounding it, so the six products of 16 entries are summed from zero, the small ones first, and
// join the running sum by a rounded addition. With two terms the outputs of one chunk from a given state were 4e-6 off 64
// bits, with three into one running sum 1e-6, where the walk in float32 is 2e-7 off.
// One block = one chunk x one head, 8 warps; 112.5 KB of shared memory, two blocks an SM:
//     tiles of q, k (then the keys' first terms, then two terms of the state's quarters), the keys' second terms (then v), the
//     third terms of the keys of the first three sub-blocks (nothing reads the last one's scaled; then the state's), the
//     logarithms (then their sums inside a sub-block up to t), the scores.
constexpr int SUB = 16, SUBS = CH / SUB, SPITCH = CH + 4;     // tokens of a sub-block; pitch of the scores' rows
constexpr float LOG2E = 1.4426950408889634f;

template <int DK, int DV>
struct OutShape {
  static constexpr int LP = DK + 8;                            // floats from one token's logarithms to the next's
  static constexpr int A_BYTES = CH * (DK > DV ? DK : DV) * 2; // a tile, also of v or of a quarter of the state (two terms)
  static constexpr int C_BYTES = (CH - SUB) * DK * 2;          // third terms: of 48 keys, or of a quarter of the state
  static constexpr size_t SMEM =
      size_t(CH) * DK * 2 + 2 * size_t(A_BYTES) + C_BYTES + size_t(CH) * LP * 4 + size_t(SUBS - 1) * DK * 4 + size_t(CH) * SPITCH * 4;
};

__device__ __forceinline__ float2 pair_f(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

template <int DK, int DV>
__global__ void __launch_bounds__(256, 2)
gla_chunk_out_mma_kernel(const __nv_bfloat16* __restrict__ proj, int stride, const float* __restrict__ log_decay, StepBatch sb,
                         const int* __restrict__ chunk_seq, const int* __restrict__ chunk_q0, const float* __restrict__ before,
                         float* __restrict__ out, int heads, float q_scale) {
  pdl_entry();
  using Shape = OutShape<DK, DV>;
  constexpr int LP = Shape::LP, NT = DV / 16;      // NT: n-tiles of 8 value columns that a warp owns
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* q_s = sm;                                  // [CH][DK]
  unsigned char* k_s = q_s + CH * DK * 2;                   // [CH][DK] k, then the scaled keys' hi terms, then quarters of the state
  unsigned char* b_s = k_s + Shape::A_BYTES;                // [CH][DK] the scaled keys' second terms, then [CH][DV] v
  unsigned char* c_s = b_s + Shape::A_BYTES;                // [CH - SUB][DK] their third terms, then a quarter of the state's
  float* l_s = reinterpret_cast<float*>(c_s + Shape::C_BYTES);   // [CH][LP] logarithms (powers of two), then sums up to t
  float* t_s = l_s + CH * LP;                               // [SUBS - 1][DK] a sub-block's sum (nothing follows the last)
  float* s_s = t_s + (SUBS - 1) * DK;                             // [CH][SPITCH] scores
  const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp8 = tid >> 5, warp = warp8 & 3, half = warp8 >> 2;
  const int seq = chunk_seq[c], q0 = chunk_q0[c];
  const int start = sb.seq_start[seq] + q0, n = min(CH, sb.seq_new[seq] - q0);
  const __nv_bfloat16* row0 = proj + size_t(start) * stride;
  {
    StagedWords<DK, 256> qw, kw;
    qw.load(row0 + h * DK, stride, n, tid);
    kw.load(row0 + heads * DK + h * DK, stride, n, tid);
    constexpr int QUADS = DK / 4, PER = CH * QUADS / 256;
    const float* l0 = log_decay + size_t(start) * heads * DK + h * DK;
    float4 l[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid + u * 256, row = i / QUADS, q = i % QUADS;
      l[u] = row < n ? *reinterpret_cast<const float4*>(l0 + size_t(row) * heads * DK + q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    qw.store(q_s, 0, tid);
    kw.store(k_s, 0, tid);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid + u * 256, row = i / QUADS, q = i % QUADS;
      *reinterpret_cast<float4*>(l_s + row * LP + q * 4) = make_float4(l[u].x * LOG2E, l[u].y * LOG2E, l[u].z * LOG2E, l[u].w * LOG2E);
    }
  }
  __syncthreads();
  {   // scores inside sub-block `warp`, in groups of four keys
    constexpr int PAIRS = DK / 64;      // a lane's channels, two in a register pair: half the multiply-adds
    const int c0 = lane * 2 * PAIRS;
    auto load_row = [&](const unsigned char* tile, int row, uint64_t (&f)[PAIRS]) {
      const unsigned char* p = tile + swz<DK>(row, c0 / 8) + (c0 % 8) * 2;
      if constexpr (PAIRS == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        f[0] = wide2(v.x), f[1] = wide2(v.y);
      } else {
        f[0] = wide2(*reinterpret_cast<const uint32_t*>(p));
      }
    };
    const int r0 = warp * SUB;
    // a lane's part of sum_c q[c] k[c] exp2(e[c])
    auto score = [&](const uint64_t (&q)[PAIRS], const uint64_t (&k)[PAIRS], const uint64_t (&e)[PAIRS]) {
      uint64_t sum = 0ull;
#pragma unroll
      for (int u = 0; u < PAIRS; ++u) {
        const float2 x = halves2(e[u]);
        sum = fma2(mul2(q[u], k[u]), pack2(fast_exp2(x.x), fast_exp2(x.y)), sum);
      }
      const float2 v = halves2(sum);
      return v.x + v.y;
    };
    auto load_logs = [&](int row, uint64_t (&l)[PAIRS]) {
      const uint64_t* from = reinterpret_cast<const uint64_t*>(l_s + row * LP + c0);
      if constexpr (PAIRS == 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(from);
        l[0] = v.x, l[1] = v.y;
      } else {
        l[0] = from[0];
      }
    };
    // the lanes' sums of sixteen scores (4 tokens of group T x 4 keys of group g) and their place: at every step a lane hands half of its
    // values on
    auto put16 = [&](int T, int g, float (&p)[16]) {
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) {
        const bool up = (lane & (2 * w)) != 0;
#pragma unroll
        for (int t = 0; t < w; ++t) {
          const float give = up ? p[t] : p[t + w], keep = up ? p[t + w] : p[t];
          p[t] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * w);
        }
      }
      p[0] += __shfl_xor_sync(0xffffffffu, p[0], 1);
      const int v = lane >> 1;
      if ((lane & 1) == 0) s_s[(r0 + 4 * T + (v >> 2)) * SPITCH + r0 + 4 * g + (v & 3)] = p[0];
    };
#pragma unroll 1
    for (int gi = 0; gi < 2; ++gi) {
      const int g = half ? 1 + gi : 3 * gi;      // 20 tokens a warp: groups 0 and 3, or 1 and 2
      uint64_t k[4][PAIRS], e[4][PAIRS], q[PAIRS], l[PAIRS];      // e: a key's logarithms after it, up to the token
      float p[16];
#pragma unroll
      for (int a = 0; a < 4; ++a) load_row(k_s, r0 + 4 * g + a, k[a]);
#pragma unroll 1
      for (int T = g; T < 4; ++T) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          load_row(q_s, r0 + 4 * T + t, q);
          load_logs(r0 + 4 * T + t, l);
#pragma unroll
          for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int u = 0; u < PAIRS; ++u) e[a][u] = T == g && a >= t ? 0ull : add2(e[a][u], l[u]);
            p[4 * t + a] = score(q, k[a], e[a]);
            if (T == g && a > t) p[4 * t + a] = 0.f;      // before the key
          }
        }
        put16(T, g, p);
      }
    }
    // keys of later groups take no part: six squares of four, three a warp
    for (int x = lane + 48 * half; x < 48 + 48 * half; x += 32) {
      const int sq = x >> 4, T = sq < 3 ? 0 : sq < 5 ? 1 : 2, g = sq < 3 ? 1 + sq : sq < 5 ? sq - 1 : 3;      // (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
      s_s[(r0 + 4 * T + ((x >> 2) & 3)) * SPITCH + r0 + 4 * g + (x & 3)] = 0.f;
    }
  }
  __syncthreads();
  // the sums inside sub-blocks: up to t in place of the logarithms, and what follows i into the keys (three terms; no later
  // sub-block meets the last one's keys)
  for (int u = tid; u < SUBS * DK; u += 256) {
    const int sub = u / DK, ch = u % DK;
    float l[SUB], up = 0.f;
#pragma unroll
    for (int t = 0; t < SUB; ++t) l[t] = l_s[(sub * SUB + t) * LP + ch];
#pragma unroll
    for (int t = 0; t < SUB; ++t) {
      up += l[t];
      l_s[(sub * SUB + t) * LP + ch] = up;
    }
    if (sub == SUBS - 1) continue;
    t_s[sub * DK + ch] = up;
    float rest = 0.f;
#pragma unroll
    for (int t = SUB - 1; t >= 0; --t) {
      const uint32_t at = swz<DK>(sub * SUB + t, ch / 8) + (ch % 8) * 2;
      const float k = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(k_s + at)) * fast_exp2(rest);
      const __nv_bfloat16 first = __float2bfloat16_rn(k);
      const float left = k - __bfloat162float(first);
      const __nv_bfloat16 second = __float2bfloat16_rn(left);
      *reinterpret_cast<__nv_bfloat16*>(k_s + at) = first;
      *reinterpret_cast<__nv_bfloat16*>(b_s + at) = second;
      *reinterpret_cast<__nv_bfloat16*>(c_s + at) = __float2bfloat16_rn(left - __bfloat162float(second));
      rest += l[t];
    }
  }
  StagedWords<DV, 256> vw;      // on their way under the scores between sub-blocks
  vw.load(row0 + 2 * heads * DK + h * DV, stride, n, tid);
  __syncthreads();
  const uint32_t ks = smem_u32(k_s), bs = smem_u32(b_s), cs = smem_u32(c_s);
  const int g4 = lane >> 2, t4 = lane & 3, m = lane >> 3;
  // two neighbouring channels (ch, ch + 1) of query row r, times exp2(sum up to r in its sub-block + extra)
  auto scaled_q = [&](int r, int ch, float2 extra, uint32_t& q1, uint32_t& q2, uint32_t& q3) {
    const float2 q = pair_f(*reinterpret_cast<const uint32_t*>(q_s + swz<DK>(r, ch / 8) + (ch % 8) * 2));
    const float2 e = *reinterpret_cast<const float2*>(l_s + r * LP + ch);
    split3_pack(q.x * fast_exp2(e.x + extra.x), q.y * fast_exp2(e.y + extra.y), q1, q2, q3);
  };
  if (warp8 < 6) {      // scores of sub-block w with the keys of sub-block u < w: a pair a warp
    const int w = warp8 == 0 ? 1 : warp8 < 3 ? 2 : 3, u = warp8 == 0 ? 0 : warp8 < 3 ? warp8 - 1 : warp8 - 3;
    const int r_lo = w * SUB + g4, r_hi = r_lo + 8;
    float s[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
    for (int kk = 0; kk < DK / 16; ++kk) {
      uint32_t q1[4], q2[4], q3[4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int ch = kk * 16 + 8 * x + 2 * t4;
        float2 mid = make_float2(0.f, 0.f);
        for (int y = u + 1; y < w; ++y) {
          const float2 t = *reinterpret_cast<const float2*>(t_s + y * DK + ch);
          mid.x += t.x;
          mid.y += t.y;
        }
        scaled_q(r_lo, ch, mid, q1[2 * x], q2[2 * x], q3[2 * x]);
        scaled_q(r_hi, ch, mid, q1[2 * x + 1], q2[2 * x + 1], q3[2 * x + 1]);
      }
      uint32_t b0, b1, b2, b3, d0, d1, d2, d3;      // keys 0..7 and 8..15 of the sub-block, 16 channels each
      const uint32_t off = swz<DK>(u * SUB + (m >> 1) * 8 + (lane & 7), kk * 2 + (m & 1));
      float x0[4] = {0.f, 0.f, 0.f, 0.f}, x1[4] = {0.f, 0.f, 0.f, 0.f};
      ldmatrix_x4(b0, b1, b2, b3, cs + off);
      mma_bf16(x0, q1, b0, b1);
      mma_bf16(x1, q1, b2, b3);
      ldmatrix_x4(b0, b1, b2, b3, bs + off);
      mma_bf16(x0, q2, b0, b1);
      mma_bf16(x1, q2, b2, b3);
      ldmatrix_x4(d0, d1, d2, d3, ks + off);
      mma_bf16(x0, q3, d0, d1);
      mma_bf16(x1, q3, d2, d3);
      mma_bf16(x0, q1, b0, b1);
      mma_bf16(x1, q1, b2, b3);
      mma_bf16(x0, q2, d0, d1);
      mma_bf16(x1, q2, d2, d3);
      mma_bf16(x0, q1, d0, d1);
      mma_bf16(x1, q1, d2, d3);
#pragma unroll
      for (int e = 0; e < 4; ++e) s[0][e] += x0[e], s[1][e] += x1[e];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      *reinterpret_cast<float2*>(s_s + r_lo * SPITCH + u * SUB + j * 8 + 2 * t4) = make_float2(s[j][0], s[j][1]);
      *reinterpret_cast<float2*>(s_s + r_hi * SPITCH + u * SUB + j * 8 + 2 * t4) = make_float2(s[j][2], s[j][3]);
    }
  }
  __syncthreads();      // the scores are complete; the keys are no longer read
  // the state before the chunk comes a quarter of its rows at a time, the next one's loads under this one's products
  constexpr int QR = DK / 4, CHUNKS = DV / 8, PER = QR * CHUNKS / 256 > 0 ? QR * CHUNKS / 256 : 1;
  const float* S0 = before + (size_t(c) * heads + h) * DK * DV;
  float4 sx[PER], sy[PER];
  auto load_state = [&](int quarter) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid + u * 256, row = i / CHUNKS, cc = i % CHUNKS;
      if (i < QR * CHUNKS) {
        sx[u] = *reinterpret_cast<const float4*>(S0 + size_t(quarter * QR + row) * DV + cc * 8);
        sy[u] = *reinterpret_cast<const float4*>(S0 + size_t(quarter * QR + row) * DV + cc * 8 + 4);
      }
    }
  };
  load_state(0);
  vw.store(b_s, 0, tid);
  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  const int r_lo = warp * SUB + g4, r_hi = r_lo + 8, j0 = half * NT;      // this thread's two tokens; the warp's first n-tile
  unsigned char* s_1 = k_s;                       // [QR][DV], the three terms
  unsigned char* s_2 = k_s + QR * DV * 2;
  unsigned char* s_3 = c_s;
  const uint32_t ss1 = smem_u32(s_1), ss2 = smem_u32(s_2), ss3 = smem_u32(s_3);
#pragma unroll 1
  for (int quarter = 0; quarter < 4; ++quarter) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid + u * 256, row = i / CHUNKS, cc = i % CHUNKS;
      if (i < QR * CHUNKS) {
        uint4 a, b, d;
        split3_pack(sx[u].x, sx[u].y, a.x, b.x, d.x);
        split3_pack(sx[u].z, sx[u].w, a.y, b.y, d.y);
        split3_pack(sy[u].x, sy[u].y, a.z, b.z, d.z);
        split3_pack(sy[u].z, sy[u].w, a.w, b.w, d.w);
        *reinterpret_cast<uint4*>(s_1 + swz<DV>(row, cc)) = a;
        *reinterpret_cast<uint4*>(s_2 + swz<DV>(row, cc)) = b;
        *reinterpret_cast<uint4*>(s_3 + swz<DV>(row, cc)) = d;
      }
    }
    __syncthreads();      // this quarter (and v) is staged
    if (quarter < 3) load_state(quarter + 1);
#pragma unroll
    for (int kk = 0; kk < QR / 16; ++kk) {
      uint32_t q1[4], q2[4], q3[4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int ch = quarter * QR + kk * 16 + 8 * x + 2 * t4;
        float2 front = make_float2(0.f, 0.f);
        for (int y = 0; y < warp; ++y) {
          const float2 t = *reinterpret_cast<const float2*>(t_s + y * DK + ch);
          front.x += t.x;
          front.y += t.y;
        }
        scaled_q(r_lo, ch, front, q1[2 * x], q2[2 * x], q3[2 * x]);
        scaled_q(r_hi, ch, front, q1[2 * x + 1], q2[2 * x + 1], q3[2 * x + 1]);
      }
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        uint32_t b0, b1, b2, b3, d0, d1, d2, d3;
        float x0[4] = {0.f, 0.f, 0.f, 0.f}, x1[4] = {0.f, 0.f, 0.f, 0.f};
        const uint32_t off = swz<DV>(kk * 16 + (m & 1) * 8 + (lane & 7), j0 + j + (m >> 1));
        ldmatrix_x4_trans(b0, b1, b2, b3, ss3 + off);
        mma_bf16(x0, q1, b0, b1);
        mma_bf16(x1, q1, b2, b3);
        ldmatrix_x4_trans(b0, b1, b2, b3, ss2 + off);
        mma_bf16(x0, q2, b0, b1);
        mma_bf16(x1, q2, b2, b3);
        ldmatrix_x4_trans(d0, d1, d2, d3, ss1 + off);
        mma_bf16(x0, q3, d0, d1);
        mma_bf16(x1, q3, d2, d3);
        mma_bf16(x0, q1, b0, b1);
        mma_bf16(x1, q1, b2, b3);
        mma_bf16(x0, q2, d0, d1);
        mma_bf16(x1, q2, d2, d3);
        mma_bf16(x0, q1, d0, d1);
        mma_bf16(x1, q1, d2, d3);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] += x0[e], o[j + 1][e] += x1[e];
      }
    }
    __syncthreads();      // the quarter is no longer read
  }
#pragma unroll
  for (int kb = 0; kb < SUBS; ++kb) {
    if (kb > warp) break;
    uint32_t p1[4], p2[4], p3[4];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const float2 a = *reinterpret_cast<const float2*>(s_s + r_lo * SPITCH + kb * 16 + 8 * x + 2 * t4);
      const float2 b = *reinterpret_cast<const float2*>(s_s + r_hi * SPITCH + kb * 16 + 8 * x + 2 * t4);
      split3_pack(a.x, a.y, p1[2 * x], p2[2 * x], p3[2 * x]);
      split3_pack(b.x, b.y, p1[2 * x + 1], p2[2 * x + 1], p3[2 * x + 1]);
    }
#pragma unroll
    for (int j = 0; j < NT; j += 2) {
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4_trans(b0, b1, b2, b3, bs + swz<DV>(kb * 16 + (m & 1) * 8 + (lane & 7), j0 + j + (m >> 1)));
      float x0[4] = {0.f, 0.f, 0.f, 0.f}, x1[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16(x0, p3, b0, b1);
      mma_bf16(x1, p3, b2, b3);
      mma_bf16(x0, p2, b0, b1);
      mma_bf16(x1, p2, b2, b3);
      mma_bf16(x0, p1, b0, b1);
      mma_bf16(x1, p1, b2, b3);
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] += x0[e], o[j + 1][e] += x1[e];
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = i ? r_hi : r_lo;
    if (r >= n) continue;
    float* dst = out + (size_t(start + r) * heads + h) * DV + j0 * 8 + t4 * 2;
#pragma unroll
    for (int j = 0; j < NT; ++j) *reinterpret_cast<float2*>(dst + j * 8) = make_float2(o[j][2 * i] * q_scale, o[j][2 * i + 1] * q_scale);
  }
}

template <int DK, int DV>
int launch_out(const void* proj, int stride, const float* log_decay, const StepBatch& sb, const int* chunk_seq, const int* chunk_q0,
               int n_chunks, const float* before, float* out, int heads, float q_scale, cudaStream_t stream) {
  constexpr size_t smem = OutShape<DK, DV>::SMEM;
  static SharedLimit limit;
  if (!limit.allows(gla_chunk_out_mma_kernel<DK, DV>, smem)) return PTB_ERR_LAUNCH;
  launch_pdl(gla_chunk_out_mma_kernel<DK, DV>, dim3(n_chunks, heads), 256, smem, stream, (const __nv_bfloat16*)proj, stride, log_decay, sb,
                                                                                chunk_seq, chunk_q0, before, out, heads, q_scale);
  return launch_status();
}

}  // namespace

// Sizes and layouts that these passes take: bfloat16 projections, keys and values of 64 or 128 entries, rows that start
// at whole 16-byte words (then q, k, v and the logarithms' rows do too).
PTB_API int ptb_gla_chunk_sum_mma_supports(int dtype, const void* proj, int stride, const float* log_decay, int dim, int v_dim) {
  return (dtype == PTB_BF16 && (dim == 64 || dim == 128) && (v_dim == 64 || v_dim == 128) && stride % 8 == 0 &&
          reinterpret_cast<size_t>(proj) % 16 == 0 && reinterpret_cast<size_t>(log_decay) % 16 == 0) ? 1 : 0;
}

// Every chunk's own sum and total decay (the caller has checked ptb_gla_chunk_sum_mma_supports and the sizes).
PTB_API int ptb_gla_chunk_sum_mma(const void* proj, int stride, const float* log_decay, const StepBatch* sb, const int* chunk_seq,
                                  const int* chunk_q0, int n_chunks, float* sums, float* chunk_decay, int heads, int dim,
                                  int v_dim, cudaStream_t stream) {
  if (n_chunks <= 0) return PTB_OK;
#define PTB_GLA_SUM(DK, DV) \
  return launch_sum<DK, DV>(proj, stride, log_decay, *sb, chunk_seq, chunk_q0, n_chunks, sums, chunk_decay, heads, stream)
  if (dim == 64 && v_dim == 64) PTB_GLA_SUM(64, 64);
  if (dim == 64 && v_dim == 128) PTB_GLA_SUM(64, 128);
  if (dim == 128 && v_dim == 64) PTB_GLA_SUM(128, 64);
  if (dim == 128 && v_dim == 128) PTB_GLA_SUM(128, 128);
#undef PTB_GLA_SUM
  return PTB_ERR_SIZE;
}

// Every chunk's outputs from the state before it (`before`: what the join left of the chunks' sums; the same sizes and layouts).
PTB_API int ptb_gla_chunk_out_mma(const void* proj, int stride, const float* log_decay, const StepBatch* sb, const int* chunk_seq,
                                  const int* chunk_q0, int n_chunks, const float* before, float* out, int heads, int dim, int v_dim,
                                  float q_scale, cudaStream_t stream) {
  if (n_chunks <= 0) return PTB_OK;
#define PTB_GLA_OUT(DK, DV) \
  return launch_out<DK, DV>(proj, stride, log_decay, *sb, chunk_seq, chunk_q0, n_chunks, before, out, heads, q_scale, stream)
  if (dim == 64 && v_dim == 64) PTB_GLA_OUT(64, 64);
  if (dim == 64 && v_dim == 128) PTB_GLA_OUT(64, 128);
  if (dim == 128 && v_dim == 64) PTB_GLA_OUT(128, 64);
  if (dim == 128 && v_dim == 128) PTB_GLA_OUT(128, 128);
#undef PTB_GLA_OUT
  return PTB_ERR_SIZE;
}
