// Attention over the paged cache, general form (CUDA cores, float32 arithmetic), and the kernel
// that splits a fused projection into rotated queries and cache entries.
//
// The general attention kernel takes every head size up to 256, any number of heads and groups,
// float32 or bfloat16 tensors, rotary or ALiBi models, an optional window, prompts and single
// tokens alike. It is the kernel of the float32 path and the fallback of the bfloat16 path for
// sizes that the tensor-core kernels refuse. Every query row is reduced over its keys in blocks
// of 64 aligned to absolute positions, in ascending order, whatever else is in the launch: the
// result of a position does not depend on how tokens were cut into steps or batched.
#include "mma_common.cuh"

namespace {

constexpr int BQ = 16;        // query rows of a tile
constexpr int THREADS = 128;  // 16 threads per pair of query rows
constexpr int MAX_D = 256;    // head sizes up to this
constexpr int PPITCH = PTB_PAGE + 4;

// floats from one row of `n` values to the next: whole 16-byte words, an odd number of them
__host__ __device__ constexpr int odd_words(int n) { return 4 * ((n + 3) / 4 + ((n + 3) / 4 % 2 == 0 ? 1 : 0)); }

// a page's rows of `d` values into shared rows `pitch` apart, zeros in rows from `valid` on and beyond d; `whole`: the rows are
// whole 16-byte words, which go by cp.async in float32 and through registers, a word a load, in bfloat16. (A value a load, a
// head size of 256 in bfloat16 was slower than the kernel before this one where sequences are many, an SM holding one block:
// 64 sequences of 1,000 keys 3,198 us against 2,940; a word a load 1,667 us.)
template <typename T>
__device__ __forceinline__ void load_rows(float* dst, const T* src, int d, int pitch, int valid, int whole) {
  const int words = (d + 3) / 4;
  if (sizeof(T) == 2 && whole) {
    const int per_row = d / 8;
#pragma unroll 4
    for (int i = threadIdx.x; i < PTB_PAGE * per_row; i += THREADS) {
      const int j = i / per_row, c = (i - j * per_row) * 8;
      const uint4 w = j < valid ? *reinterpret_cast<const uint4*>(src + size_t(j) * d + c) : make_uint4(0, 0, 0, 0);
      float f[8];
      unpack_bf16x8(w, f);
      *reinterpret_cast<float4*>(dst + j * pitch + c) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(dst + j * pitch + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
    return;
  }
  if (sizeof(T) == 4 && whole) {
    for (int i = threadIdx.x; i < PTB_PAGE * words; i += THREADS) {
      const int j = i / words, c = (i - j * words) * 4;
      if (j < valid) cp_async16(smem_u32(dst + j * pitch + c), src + size_t(j) * d + c);
      else *reinterpret_cast<float4*>(dst + j * pitch + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  for (int i = threadIdx.x; i < PTB_PAGE * words * 4; i += THREADS) {
    const int j = i / (words * 4), e = i - j * (words * 4);
    dst[j * pitch + e] = (j < valid && e < d) ? to_f(src[size_t(j) * d + e]) : 0.f;
  }
}

// a float as the tensors' type holds it
template <typename T> __device__ __forceinline__ float round_store(float v) { return to_f(from_f<T>(v)); }

// ------------------------------------------------------------------------------------------------
// Fused projection [n_tokens, kv_heads * (q_per_kv + 2) * head_dim], rows grouped per K/V head as
// (q_per_kv query heads, K, V), to: q_out [n_tokens, heads, head_dim] (query head = group *
// q_per_kv + index in group) and the K and V pools of one layer. With inv_freq != nullptr the
// first 2 * rot_pairs dims of every query and key head are rotated: pairs (i, i + rot_pairs), or with
// `interleaved` pairs (2 i, 2 i + 1);
// angle = position * inv_freq[i] in float32, x' = x cos - y sin, y' = y cos + x sin. With a table
// (rope_cos, rope_sin: [n_tokens, rot_pairs], made by rope_table_kernel from the same product) the
// cosines and sines are read instead of computed. One block per token.
template <typename T>
__global__ void split_rotate_store_kernel(const T* __restrict__ fused, T* __restrict__ q_out, T* __restrict__ k_pool,
                                          T* __restrict__ v_pool, StepBatch sb, const float* __restrict__ inv_freq,
                                          const float* __restrict__ rope_cos, const float* __restrict__ rope_sin,
                                          int rot_pairs, int kv_heads, int q_per_kv, int head_dim, int write_cache,
                                          int interleaved) {
  pdl_entry();
  const int t = blockIdx.x;
  const int pos = sb.tok_pos[t];
  const int seq = sb.tok_seq[t];
  const int page = sb.pages[size_t(seq) * sb.pages_stride + pos / PTB_PAGE];
  const int in_page = pos % PTB_PAGE;
  const int rows = q_per_kv + 2;
  const int fused_width = kv_heads * rows * head_dim;
  const T* src_tok = fused + size_t(t) * fused_width;
  const int heads = kv_heads * q_per_kv;
  // work items: (group g, row r in group, pair or plain element)
  const int rot_dims = 2 * rot_pairs;
  // bfloat16 with head sizes and rotation widths in multiples of 8 and a table of cosines: 16-byte words
  if (sizeof(T) == 2 && head_dim % 8 == 0 && rot_pairs % 8 == 0 && (rot_pairs == 0 || (rope_cos != nullptr && !interleaved)) &&
      aligned16(fused) && aligned16(q_out) && (!write_cache || (aligned16(k_pool) && aligned16(v_pool)))) {
    const int chunks = head_dim / 8, rot_chunks = rot_pairs / 8;
    const int total_v = kv_heads * rows * chunks;
    for (int w = threadIdx.x; w < total_v; w += blockDim.x) {
      const int c = w % chunks;
      const int gr = w / chunks;
      const int r = gr % rows, g = gr / rows;
      const T* src = src_tok + size_t(g * rows + r) * head_dim;
      T* dst;
      if (r < q_per_kv) {
        dst = q_out + (size_t(t) * heads + (g * q_per_kv + r)) * head_dim;
      } else {
        if (!write_cache) continue;
        dst = ((r == q_per_kv) ? k_pool : v_pool) + kv_offset(page, g, in_page, kv_heads, head_dim);
      }
      const bool rotated_row = (r <= q_per_kv) && rot_chunks > 0;
      if (rotated_row && c < rot_chunks) {
        float a[8], b[8], cs[8], sn[8];
        unpack_bf16x8(*reinterpret_cast<const uint4*>(src + c * 8), a);
        unpack_bf16x8(*reinterpret_cast<const uint4*>(src + rot_pairs + c * 8), b);
        const float4* cp = reinterpret_cast<const float4*>(rope_cos + size_t(t) * rot_pairs + c * 8);
        const float4* sp = reinterpret_cast<const float4*>(rope_sin + size_t(t) * rot_pairs + c * 8);
        *reinterpret_cast<float4*>(cs) = cp[0];
        *reinterpret_cast<float4*>(cs + 4) = cp[1];
        *reinterpret_cast<float4*>(sn) = sp[0];
        *reinterpret_cast<float4*>(sn + 4) = sp[1];
#pragma unroll
        for (int e = 0; e < 8; ++e) rotate_pair(a[e], b[e], cs[e], sn[e], a[e], b[e]);
        *reinterpret_cast<uint4*>(dst + c * 8) = pack_bf16x8(a);
        *reinterpret_cast<uint4*>(dst + rot_pairs + c * 8) = pack_bf16x8(b);
      } else if (rotated_row && c < 2 * rot_chunks) {
        // the upper half of a rotated pair: written by the thread that holds the lower half
      } else {
        *reinterpret_cast<uint4*>(dst + c * 8) = *reinterpret_cast<const uint4*>(src + c * 8);
      }
    }
    return;
  }
  const int per_row = rot_pairs + (head_dim - rot_dims);  // rotated pairs, then untouched dims
  const int total = kv_heads * rows * per_row;
  for (int w = threadIdx.x; w < total; w += blockDim.x) {
    const int e = w % per_row;
    const int gr = w / per_row;
    const int r = gr % rows;
    const int g = gr / rows;
    const T* src = src_tok + size_t(g * rows + r) * head_dim;
    T* dst;
    if (r < q_per_kv) {
      dst = q_out + (size_t(t) * heads + (g * q_per_kv + r)) * head_dim;
    } else {
      if (!write_cache) continue;
      T* pool = (r == q_per_kv) ? k_pool : v_pool;
      dst = pool + kv_offset(page, g, in_page, kv_heads, head_dim);
    }
    const bool rotated_row = (r <= q_per_kv) && (inv_freq != nullptr || rope_cos != nullptr);  // queries and K, not V
    if (e < rot_pairs) {
      const int ia = interleaved ? 2 * e : e, ib = interleaved ? 2 * e + 1 : e + rot_pairs;   // the pair's two dims
      const float a = to_f(src[ia]);
      const float b = to_f(src[ib]);
      if (rotated_row) {
        float s, c, ra, rb;
        if (rope_cos) {
          c = rope_cos[size_t(t) * rot_pairs + e];
          s = rope_sin[size_t(t) * rot_pairs + e];
        } else {
          sincosf(float(pos) * inv_freq[e], &s, &c);
        }
        rotate_pair(a, b, c, s, ra, rb);
        dst[ia] = from_f<T>(ra);
        dst[ib] = from_f<T>(rb);
      } else {
        dst[ia] = src[ia];
        dst[ib] = src[ib];
      }
    } else {
      const int i = rot_dims + (e - rot_pairs);
      dst[i] = src[i];
    }
  }
}

// ------------------------------------------------------------------------------------------------
// One block = one tile of BQ consecutive new tokens of one sequence x one query head.
//   tile_seq[i], tile_q0[i]: sequence index and first token (within the sequence's new tokens)
// q [n_tokens, heads, head_dim]; out [n_tokens, heads * head_dim].
// score(q at position p, key at position j) = (q . k_j + alibi_h(j)) * scale for j <= p
// (and j > p - window when window > 0); softmax over those keys in float32; out = sum p_j v_j.
// Values may have a size of their own (v_dim; the V pool is [pages][kv_heads][PTB_PAGE][v_dim]).
// With `sinks` [heads] every row's softmax denominator holds one more term, exp(sink_h), taken as stored
// (`scale` is not applied to it); no key or value is read for it. With `gate` (row t, head h at gate[t * gate_stride + h]) the head's
// output is multiplied by sigmoid(gate); with `gate_wide` the gate has a number per output entry instead (row t, head h,
// entry e at gate[t * gate_stride + h * v_dim + e]); `out_scale` multiplies everything. Output row t, head h starts
// at out[t * out_stride + h * v_dim]. `softcap` > 0: score <- softcap * tanh(score / softcap) after the scale.
//
// What bounds it on prompts is the FMA pipe behind shared memory, so operands are read as 16-byte words into register
// tiles: a block is 8 pairs of rows x 16 lanes; a thread forms 2 rows x 4 keys of the scores (6 words for 32 FMAs, the k
// ascending in one chain a score) and 2 rows x 4 columns of the output a group of 64 columns (2 + 4 words for 32 FMAs).
// Shared rows lie an odd number of words apart: eight lanes' words meet no bank twice. float32 pages come by cp.async:
// a page's values while its scores are formed, the next page's keys while the output takes the values.
// 16 heads of 64 on prompts of 233 and 467 tokens, float32: 516 -> 69 us (before: scalar loads, two a product).
template <typename T, int COLS>     // COLS: groups of 64 output columns (v_dim <= 64 COLS)
__global__ void __launch_bounds__(THREADS)
attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                         T* __restrict__ out, StepBatch sb, const int* __restrict__ tile_seq,
                         const int* __restrict__ tile_q0, const float* __restrict__ alibi_slopes, int heads,
                         int kv_heads, int head_dim, float scale, int window, int v_dim,
                         const float* __restrict__ sinks, const T* __restrict__ gate, int gate_stride, float out_scale,
                         int out_stride, int keep_first, float* __restrict__ out_wide, float softcap, int gate_wide, int whole) {
  pdl_entry();
  extern __shared__ __align__(16) float smem[];
  const int kpitch = odd_words(head_dim), vpitch = odd_words(v_dim), kwords = (head_dim + 3) / 4;
  float* qs = smem;                                 // [BQ][kpitch], zeros beyond head_dim
  float* ks = qs + BQ * kpitch;                     // [PTB_PAGE][kpitch], likewise
  float* vs = ks + PTB_PAGE * kpitch;               // [PTB_PAGE][vpitch]
  float* ps = vs + PTB_PAGE * vpitch;               // [BQ][PPITCH]

  const int tile = blockIdx.x, h = blockIdx.y;
  const int seq = tile_seq[tile], q0 = tile_q0[tile];
  const int n_new = sb.seq_new[seq], past = sb.seq_past[seq], start = sb.seq_start[seq];
  const int rows = min(BQ, n_new - q0);
  const int g = h / (heads / kv_heads);
  // with out_wide the grid's third dimension names the K/V head whose values this block reads (the scores are
  // head h's own): every head's weights meet every K/V head's values, for a mixing of the heads' weights afterwards
  const int gv = out_wide ? int(blockIdx.z) : g;
  const int tid = threadIdx.x;
  const int r0 = (tid / 16) * 2, lane = tid % 16;   // rows r0 and r0 + 1; keys lane + 16 jj; columns 4 lane + 64 c
  const float slope = alibi_slopes ? alibi_slopes[h] : 0.f;

  for (int i = tid; i < BQ * kpitch; i += THREADS) {
    const int rr = i / kpitch, e = i % kpitch;
    qs[i] = (rr < rows && e < head_dim) ? to_f(q[(size_t(start + q0 + rr) * heads + h) * head_dim + e]) : 0.f;
  }
  float acc[2][4 * COLS];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int i = 0; i < 4 * COLS; ++i) acc[u][i] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};

  const int last_pos = past + q0 + rows - 1;
  const int first_pos = past + q0;
  int kb_lo = 0;
  if (window > 0) kb_lo = max(0, first_pos - window + 1) / PTB_PAGE;
  const int kb_hi = last_pos / PTB_PAGE;
  const int* pages = sb.pages + size_t(seq) * sb.pages_stride;
  // the first keep_first positions stay visible left of the window: their pages are walked first
  const int kept_pages = (window > 0 && keep_first > 0) ? min((keep_first + PTB_PAGE - 1) / PTB_PAGE, kb_lo) : 0;
  auto after = [&](int kb) { return (kb + 1 == kept_pages && kb + 1 < kb_lo) ? kb_lo : kb + 1; };
  auto load_keys = [&](int kb) {
    const T* src = k_pool + kv_offset(pages[kb], g, 0, kv_heads, head_dim);
    load_rows(ks, src, head_dim, kpitch, min(PTB_PAGE, last_pos + 1 - kb * PTB_PAGE), whole);
  };

  int kb = kept_pages > 0 ? 0 : kb_lo;
  load_keys(kb);
  cp_async_commit();
  while (kb <= kb_hi) {
    const int next = after(kb);
    load_rows(vs, v_pool + kv_offset(pages[kb], gv, 0, kv_heads, v_dim), v_dim, vpitch,
              min(PTB_PAGE, last_pos + 1 - kb * PTB_PAGE), whole);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();  // this page's keys are here
    float s[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) s[u][jj] = 0.f;
    for (int e = 0; e < kwords; ++e) {
      float4 a[2], b[4];
#pragma unroll
      for (int u = 0; u < 2; ++u) a[u] = *reinterpret_cast<const float4*>(qs + (r0 + u) * kpitch + 4 * e);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) b[jj] = *reinterpret_cast<const float4*>(ks + (lane + 16 * jj) * kpitch + 4 * e);
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          s[u][jj] = fmaf(a[u].w, b[jj].w, fmaf(a[u].z, b[jj].z, fmaf(a[u].y, b[jj].y, fmaf(a[u].x, b[jj].x, s[u][jj]))));
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int my_pos = (r0 + u < rows) ? first_pos + r0 + u : -1;  // -1: no key is visible, nothing is stored
      float m_blk = -INFINITY;
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int key_pos = kb * PTB_PAGE + lane + 16 * jj;
        bool visible = key_pos <= my_pos;
        if (window > 0) visible = visible && (key_pos > my_pos - window || key_pos < keep_first);
        float sc = -INFINITY;
        if (visible) {
          sc = s[u][jj];
          if (alibi_slopes) sc += alibi_bias(slope, key_pos);
          sc *= scale;
          if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
        }
        s[u][jj] = sc;
        m_blk = fmaxf(m_blk, sc);
      }
      // row maximum and sum over the 16 lanes of the row
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m_blk = fmaxf(m_blk, __shfl_xor_sync(0xffffffffu, m_blk, o));
      const float m_new = fmaxf(m_run[u], m_blk);
      float corr = 1.f, l_blk = 0.f;
      float* prow = ps + (r0 + u) * PPITCH + lane;
      if (m_new == -INFINITY) {
        // nothing visible so far (rows beyond the tile, or keys left of a window)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) prow[16 * jj] = 0.f;
      } else {
        corr = (m_run[u] == -INFINITY) ? 0.f : expf(m_run[u] - m_new);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const float p = (s[u][jj] == -INFINITY) ? 0.f : expf(s[u][jj] - m_new);
          prow[16 * jj] = p;
          l_blk += p;
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) l_blk += __shfl_xor_sync(0xffffffffu, l_blk, o);
      l_run[u] = l_run[u] * corr + l_blk;
      m_run[u] = m_new;
#pragma unroll
      for (int i = 0; i < 4 * COLS; ++i) acc[u][i] *= corr;
    }
    __syncthreads();  // all scores of this page are written, its keys are no longer read
    if (next <= kb_hi) load_keys(next);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();  // this page's values are here
    for (int j = 0; j < PTB_PAGE; j += 4) {
      float4 p[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) p[u] = *reinterpret_cast<const float4*>(ps + (r0 + u) * PPITCH + j);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          const int e = 4 * lane + 64 * c;
          if (e < v_dim) {
            const float4 v = *reinterpret_cast<const float4*>(vs + (j + jj) * vpitch + e);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const float w = jj == 0 ? p[u].x : jj == 1 ? p[u].y : jj == 2 ? p[u].z : p[u].w;
              acc[u][4 * c] = fmaf(w, v.x, acc[u][4 * c]);
              acc[u][4 * c + 1] = fmaf(w, v.y, acc[u][4 * c + 1]);
              acc[u][4 * c + 2] = fmaf(w, v.z, acc[u][4 * c + 2]);
              acc[u][4 * c + 3] = fmaf(w, v.w, acc[u][4 * c + 3]);
            }
          }
        }
      }
    }
    __syncthreads();  // the values and the scores are no longer read
    kb = next;
  }
  cp_async_wait<0>();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = r0 + u;
    if (r >= rows) continue;
    float keep = 1.f, l = l_run[u];      // keep: what the keys' share of the denominator shrinks by when the sink raises the reference
    if (sinks) {
      const float sink = sinks[h], m_all = fmaxf(m_run[u], sink);
      keep = (m_run[u] == -INFINITY) ? 0.f : expf(m_run[u] - m_all);
      l = l * keep + expf(sink - m_all);
    }
    float inv = (l > 0.f ? 1.f / l : 0.f) * keep * out_scale;
    if (gate && !gate_wide) inv *= 1.f / (1.f + expf(-to_f(gate[size_t(start + q0 + r) * gate_stride + h])));
    // out_wide: float32 [token][head][K/V head][v_dim]
    float* ow = out_wide ? out_wide + ((size_t(start + q0 + r) * heads + h) * kv_heads + gv) * v_dim : nullptr;
    T* o = out_wide ? nullptr : out + size_t(start + q0 + r) * out_stride + size_t(h) * v_dim;
    const T* ge = (gate && gate_wide) ? gate + size_t(start + q0 + r) * gate_stride + size_t(h) * v_dim : nullptr;
#pragma unroll
    for (int i = 0; i < 4 * COLS; ++i) {
      const int e = 4 * lane + 64 * (i / 4) + i % 4;
      if (e >= v_dim) continue;
      if (ow) ow[e] = acc[u][i] * inv;
      else o[e] = from_f<T>(acc[u][i] * inv * (ge ? 1.f / (1.f + expf(-to_f(ge[e]))) : 1.f));
    }
  }
}

// two neighbouring entries in one access (the address a whole pair)
__device__ __forceinline__ float2 load_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load_pair(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}
__device__ __forceinline__ void store_pair(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void store_pair(__nv_bfloat16* p, float a, float b) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}

// four neighbouring entries in one access (the address a whole quad)
__device__ __forceinline__ float4 load_quad(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_quad(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store_quad(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store_quad(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<const uint32_t*>(&a);
  u.y = *reinterpret_cast<const uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// ------------------------------------------------------------------------------------------------
// Separate projections q | k | v side by side in a row of `proj` (rows `stride` apart), an optional bias on all of
// them (float32, added here in float32), then for every query and key head: rotation of the first 2 rot_pairs
// entries (pairs (i, i + rot_pairs); the table holds cos and sin of the token's angles, with whatever factor the
// position part puts on them), then, with `unit_norm`, division by the head's root mean square (eps inside the
// root, no gain). Values: v <- (1 - lam) v + lam v_first with the values of the same token that an earlier layer
// kept (`v_first`, rows v_first_stride apart; lam one float32 on the device); `v_keep` receives this layer's own
// values (with bias, before any mixing) for later layers. Keys and values go into the paged pools at the tokens'
// positions, queries to q_out [tokens, heads, dim]. With `norm_first` the norm comes before the rotation and takes
// gains (`q_gain`, `k_gain` [dim] float32, null: none). With temp_every > 0 a query at position p is multiplied by
// 1 + temp_coef ln(floor((p + 1) / temp_every) + 1) at the end, in float32. A warp per (token, head): query heads, then key heads, then the
// K/V heads' values; the warps of a block share nothing, so a head's chain of loads, rotation, sum and stores waits
// for no other. What rope_norm_store_vec_kernel (below) does not take.
template <typename T>
__global__ void rope_norm_store_kernel(const T* __restrict__ proj, int stride, const float* __restrict__ bias,
                                       T* __restrict__ q_out, T* __restrict__ k_pool, T* __restrict__ v_pool, StepBatch sb,
                                       const float* __restrict__ rope_cos, const float* __restrict__ rope_sin, int rot_pairs,
                                       int heads, int kv_heads, int dim, int v_dim, float eps, int unit_norm,
                                       const T* __restrict__ v_first, int v_first_stride, const float* __restrict__ lam,
                                       T* __restrict__ v_keep, int write_cache, int pairs,
                                       const float* __restrict__ q_gain, const float* __restrict__ k_gain, int norm_first,
                                       float temp_coef, int temp_every) {
  pdl_entry();
  extern __shared__ float rows[];   // per warp: a row of `dim` floats, then cos and sin of the rotated pairs
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int t = blockIdx.x, hh = blockIdx.y * (blockDim.x / 32) + warp;      // grid (tokens, groups of a block's warps)
  if (hh >= heads + 2 * kv_heads) return;
  const T* row = proj + size_t(t) * stride;
  if (hh >= heads + kv_heads) {     // the values of one K/V head
    const int g = hh - heads - kv_heads;
    const T* vsrc = row + size_t(heads + kv_heads) * dim + size_t(g) * v_dim;
    const float* vb = bias ? bias + size_t(heads + kv_heads) * dim + size_t(g) * v_dim : nullptr;
    const float l = (v_first != nullptr) ? lam[0] : 0.f;
    T* dst = nullptr;
    if (write_cache) {
      const int pos = sb.tok_pos[t], seq = sb.tok_seq[t];
      const int page = sb.pages[size_t(seq) * sb.pages_stride + pos / PTB_PAGE];
      dst = v_pool + kv_offset(page, g, pos % PTB_PAGE, kv_heads, v_dim);
    }
    for (int e = lane; e < v_dim; e += 32) {
      float v = to_f(vsrc[e]) + (vb ? vb[e] : 0.f);
      if (v_keep) v_keep[(size_t(t) * kv_heads + g) * v_dim + e] = from_f<T>(v);
      if (v_first != nullptr) v = (1.f - l) * round_store<T>(v) + l * to_f(v_first[size_t(t) * v_first_stride + size_t(g) * v_dim + e]);
      if (dst) dst[e] = from_f<T>(v);
    }
    return;
  }
  const bool is_q = hh < heads;
  if (!is_q && !write_cache) return;
  float* buf = rows + size_t(warp) * (dim + 2 * rot_pairs);
  float* cs = buf + dim;
  const T* src = row + size_t(hh) * dim;
  const float* bsrc = bias ? bias + size_t(hh) * dim : nullptr;
  T* dst;
  const float* gain = is_q ? q_gain : k_gain;     // null: the norm has no gains
  float last = 1.f;     // what the finished row is multiplied by: the query temperature of the token's position
  if (is_q) {
    dst = q_out + (size_t(t) * heads + hh) * dim;
    if (temp_every > 0) last = 1.f + temp_coef * logf(float((sb.tok_pos[t] + 1) / temp_every) + 1.f);
  } else {
    const int pos = sb.tok_pos[t], seq = sb.tok_seq[t];
    const int page = sb.pages[size_t(seq) * sb.pages_stride + pos / PTB_PAGE];
    dst = k_pool + kv_offset(page, hh - heads, pos % PTB_PAGE, kv_heads, dim);
  }
  for (int i = lane; i < rot_pairs; i += 32) {       // issued with the row's loads
    cs[i] = rope_cos[size_t(t) * rot_pairs + i];
    cs[rot_pairs + i] = rope_sin[size_t(t) * rot_pairs + i];
  }
  if (pairs) {      // two entries a load (dim even, rows at whole pairs)
    for (int e = 2 * lane; e < dim; e += 64) {
      const float2 x = load_pair(src + e);
      buf[e] = x.x + (bsrc ? bsrc[e] : 0.f);
      buf[e + 1] = x.y + (bsrc ? bsrc[e + 1] : 0.f);
    }
  } else {
    for (int e = lane; e < dim; e += 32) buf[e] = to_f(src[e]) + (bsrc ? bsrc[e] : 0.f);
  }
  __syncwarp();
  if (unit_norm && norm_first) {
    float ss = 0.f;
    for (int e = lane; e < dim; e += 32) ss = fmaf(buf[e], buf[e], ss);
    const float r = 1.0f / sqrtf(warp_sum(ss) / float(dim) + eps);
    for (int e = lane; e < dim; e += 32) buf[e] = buf[e] * r * (gain ? gain[e] : 1.f);
    __syncwarp();
  }
  for (int i = lane; i < rot_pairs; i += 32) {
    float a, b;
    rotate_pair(buf[i], buf[i + rot_pairs], cs[i], cs[rot_pairs + i], a, b);
    buf[i] = a;
    buf[i + rot_pairs] = b;
  }
  __syncwarp();
  float rstd = last;
  if (unit_norm && !norm_first) {
    float ss = 0.f;
    for (int e = lane; e < dim; e += 32) ss = fmaf(buf[e], buf[e], ss);
    rstd = last / sqrtf(warp_sum(ss) / float(dim) + eps);
  }
  if (pairs) {
    for (int e = 2 * lane; e < dim; e += 64) store_pair(dst + e, buf[e] * rstd, buf[e + 1] * rstd);
  } else {
    for (int e = lane; e < dim; e += 32) dst[e] = from_f<T>(buf[e] * rstd);
  }
}

// The same for heads of whole quads (sizes and rotated parts multiples of 4, heads of up to 8 GROUP entries): GROUP lanes a
// (token, head), each with eight entries in registers. What bounds the work is instructions, not bytes (a warp a head and
// four entries a lane issued 110 instructions a head: 17.0 us for 2,048 tokens of 24 heads of 128, a fifth of the copy
// rate), so a lane holds both entries of four rotated pairs: no shuffles for the rotation, one read of the angles for both
// halves, two to four heads a warp for every address, root and division; blocks of `per` heads of one token, of at most 256
// threads (blocks of 384 at 48 registers left half of an SM's warps unused: 12.3 us; as here 10.2 us). Sums run over a lane's
// eight entries, then a tree over the group's lanes.
template <typename T, int GROUP>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 6 : 5) rope_norm_store_vec_kernel(const T* __restrict__ proj, int stride, const float* __restrict__ bias,
                                           T* __restrict__ q_out, T* __restrict__ k_pool, T* __restrict__ v_pool, StepBatch sb,
                                           const float* __restrict__ rope_cos, const float* __restrict__ rope_sin, int rot_pairs,
                                           int heads, int kv_heads, int dim, int v_dim, float eps, int unit_norm,
                                           const T* __restrict__ v_first, int v_first_stride, const float* __restrict__ lam,
                                           T* __restrict__ v_keep, int write_cache, int v_quads,
                                           const float* __restrict__ q_gain, const float* __restrict__ k_gain, int norm_first,
                                           float temp_coef, int temp_every, int per) {
  pdl_entry();
  const int lane = threadIdx.x % GROUP, t = blockIdx.x;
  const unsigned mask = (GROUP == 32 ? 0xffffffffu : ((1u << (GROUP % 32)) - 1u)) << (threadIdx.x % 32 / GROUP * GROUP);
  const T* row = proj + size_t(t) * stride;
  const int hh = blockIdx.y * per + threadIdx.x / GROUP;      // one path for all lanes of a group
  if (threadIdx.x / GROUP >= per || hh >= heads + 2 * kv_heads) return;
  const bool is_q = hh < heads, is_v = hh >= heads + kv_heads;
  if (!is_q && !write_cache && !(is_v && v_keep)) return;
  T* dst = nullptr;
  const int g = is_v ? hh - heads - kv_heads : hh - heads;
  if (is_q) {
    dst = q_out + (size_t(t) * heads + hh) * dim;
  } else if (write_cache) {
    const int pos = sb.tok_pos[t], seq = sb.tok_seq[t];
    const int page = sb.pages[size_t(seq) * sb.pages_stride + pos / PTB_PAGE];
    dst = is_v ? v_pool + kv_offset(page, g, pos % PTB_PAGE, kv_heads, v_dim) : k_pool + kv_offset(page, g, pos % PTB_PAGE, kv_heads, dim);
  }
  if (is_v) {
    const size_t at = size_t(heads + kv_heads) * dim + size_t(g) * v_dim;
    const float l = (v_first != nullptr) ? lam[0] : 0.f;
    T* keep = v_keep ? v_keep + (size_t(t) * kv_heads + g) * v_dim : nullptr;
    const T* vf = v_first ? v_first + size_t(t) * v_first_stride + size_t(g) * v_dim : nullptr;
    auto mixed = [&](float v, float f) { return (1.f - l) * round_store<T>(v) + l * f; };
    if (v_quads) {
      for (int e = 4 * lane; e < v_dim; e += 4 * GROUP) {
        float4 v = load_quad(row + at + e);
        if (bias) {
          const float4 b = *reinterpret_cast<const float4*>(bias + at + e);
          v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
        }
        if (keep) store_quad(keep + e, v);
        if (vf) {
          const float4 f = load_quad(vf + e);
          v = make_float4(mixed(v.x, f.x), mixed(v.y, f.y), mixed(v.z, f.z), mixed(v.w, f.w));
        }
        if (dst) store_quad(dst + e, v);
      }
    } else {
      for (int e = lane; e < v_dim; e += GROUP) {
        float v = to_f(row[at + e]) + (bias ? bias[at + e] : 0.f);
        if (keep) keep[e] = from_f<T>(v);
        if (vf) v = mixed(v, to_f(vf[e]));
        if (dst) dst[e] = from_f<T>(v);
      }
    }
    return;
  }
  // lanes below P: the pairs (4 lane + i, rot_pairs + 4 lane + i); the others: eight entries behind the rotated part
  const int P = rot_pairs / 4;
  const bool rotated = lane < P;
  const int ea = rotated ? 4 * lane : 2 * rot_pairs + 8 * (lane - P), eb = rotated ? rot_pairs + ea : ea + 4;
  const bool on_a = ea < dim, on_b = eb < dim;
  const T* src = row + size_t(hh) * dim;
  float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float4 c = make_float4(0.f, 0.f, 0.f, 0.f), sn = c;
  if (rotated) {
    c = *reinterpret_cast<const float4*>(rope_cos + size_t(t) * rot_pairs + 4 * lane);
    sn = *reinterpret_cast<const float4*>(rope_sin + size_t(t) * rot_pairs + 4 * lane);
  }
  auto put = [](float* d, float4 v) { d[0] = v.x, d[1] = v.y, d[2] = v.z, d[3] = v.w; };
  if (on_a) put(x, load_quad(src + ea));
  if (on_b) put(x + 4, load_quad(src + eb));
  auto each = [&](const float* w, auto op) {      // op(x, w) with a row of float32 as long as the head
    float y[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (on_a) put(y, *reinterpret_cast<const float4*>(w + ea));
    if (on_b) put(y + 4, *reinterpret_cast<const float4*>(w + eb));
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = op(x[i], y[i]);
  };
  auto root = [&](float over) {      // over / the head's root mean square
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = fmaf(x[i], x[i], ss);
#pragma unroll
    for (int o = GROUP / 2; o > 0; o /= 2) ss += __shfl_xor_sync(mask, ss, o);
    return over / sqrtf(ss / float(dim) + eps);
  };
  if (bias) each(bias + size_t(hh) * dim, [](float a, float b) { return a + b; });
  if (unit_norm && norm_first) {      // the norm (with its gains) comes before the rotation
    const float r = root(1.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] *= r;
    const float* gain = is_q ? q_gain : k_gain;
    if (gain) each(gain, [](float a, float b) { return a * b; });
  }
  if (rotated) {
    rotate_pair(x[0], x[4], c.x, sn.x, x[0], x[4]);
    rotate_pair(x[1], x[5], c.y, sn.y, x[1], x[5]);
    rotate_pair(x[2], x[6], c.z, sn.z, x[2], x[6]);
    rotate_pair(x[3], x[7], c.w, sn.w, x[3], x[7]);
  }
  // what the finished row is multiplied by: the query temperature of the token's position, the norm
  float last = 1.f;
  if (is_q && temp_every > 0) last = 1.f + temp_coef * logf(float((sb.tok_pos[t] + 1) / temp_every) + 1.f);
  if (unit_norm && !norm_first) last = root(last);
  if (on_a) store_quad(dst + ea, make_float4(x[0] * last, x[1] * last, x[2] * last, x[3] * last));
  if (on_b) store_quad(dst + eb, make_float4(x[4] * last, x[5] * last, x[6] * last, x[7] * last));
}

// out[t][h][:] = sum_g talk[h][g] * wide[t][g][kv head of h][:]: the heads' softmax weights mixed after the softmax,
// applied to head h's own values, written as the sum over g of what every head's weights gave on those values.
// wide float32 [tokens][heads][kv_heads][v_dim]; talk float32 [heads][heads]; ascending g, float32.
template <typename T>
__global__ void talk_mix_kernel(const float* __restrict__ wide, const float* __restrict__ talk, T* __restrict__ out,
                                int out_stride, long long total, int heads, int kv_heads, int v_dim) {
  pdl_entry();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int e = int(i % v_dim), h = int((i / v_dim) % heads);
  const long long t = i / (v_dim * (long long)heads);
  const int c = h / (heads / kv_heads);
  const float* src = wide + (size_t(t) * heads * kv_heads + c) * v_dim + e;
  float acc = 0.f;
#pragma unroll 8
  for (int g = 0; g < heads; ++g) acc = fmaf(talk[size_t(h) * heads + g], src[size_t(g) * kv_heads * v_dim], acc);
  out[size_t(t) * out_stride + size_t(h) * v_dim + e] = from_f<T>(acc);
}

// The same with four value columns a thread and all heads of a K/V group in it: what every head's weights gave on the
// group's values is read once (16-byte loads) and meets the group's rows of `talk` in registers, eight heads at a time.
template <typename T>
__global__ void talk_mix_vec_kernel(const float* __restrict__ wide, const float* __restrict__ talk, T* __restrict__ out,
                                    int out_stride, long long total, int heads, int kv_heads, int v_dim) {
  pdl_entry();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int quads = v_dim / 4, qpk = heads / kv_heads;
  const int e = int(i % quads) * 4, c = int((i / quads) % kv_heads);
  const long long t = i / (quads * (long long)kv_heads);
  const float* src = wide + (size_t(t) * heads * kv_heads + c) * v_dim + e;
  for (int h0 = 0; h0 < qpk; h0 += 8) {
    float4 acc[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* trow = talk + size_t(c * qpk + h0) * heads;
    for (int g = 0; g < heads; ++g) {
      const float4 v = *reinterpret_cast<const float4*>(src + size_t(g) * kv_heads * v_dim);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (h0 + u < qpk) {
          const float w = trow[size_t(u) * heads + g];
          acc[u].x = fmaf(w, v.x, acc[u].x);
          acc[u].y = fmaf(w, v.y, acc[u].y);
          acc[u].z = fmaf(w, v.z, acc[u].z);
          acc[u].w = fmaf(w, v.w, acc[u].w);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (h0 + u < qpk) {
        T* dst = out + size_t(t) * out_stride + size_t(c * qpk + h0 + u) * v_dim + e;
        dst[0] = from_f<T>(acc[u].x);
        dst[1] = from_f<T>(acc[u].y);
        dst[2] = from_f<T>(acc[u].z);
        dst[3] = from_f<T>(acc[u].w);
      }
    }
  }
}

template <typename T>
int launch_attention(const void* q, const void* k_pool, const void* v_pool, void* out, const StepBatch& sb,
                     const int* tile_seq, const int* tile_q0, int n_tiles, const float* slopes, int heads,
                     int kv_heads, int head_dim, float scale, int window, int v_dim, const float* sinks, const void* gate,
                     int gate_stride, float out_scale, int out_stride, int keep_first, float* out_wide, float softcap,
                     int gate_wide, cudaStream_t stream) {
  const size_t smem = sizeof(float) * (size_t(BQ + PTB_PAGE) * odd_words(head_dim) + size_t(PTB_PAGE) * odd_words(v_dim) + BQ * PPITCH);
  constexpr int PER = 16 / sizeof(T);
  const int whole = head_dim % PER == 0 && v_dim % PER == 0 && aligned16(k_pool) && aligned16(v_pool);
  dim3 grid(n_tiles, heads, out_wide ? kv_heads : 1);
#define PTB_AG(CC)                                                                                                              \
  do {                                                                                                                          \
    static SharedLimit limit;                                                                                                   \
    if (!limit.allows(attention_generic_kernel<T, CC>, smem)) return PTB_ERR_LAUNCH;                                            \
    launch_pdl(attention_generic_kernel<T, CC>, grid, THREADS, smem, stream,                                                            \
        (const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, sb, tile_seq, tile_q0, slopes, heads, kv_heads, head_dim,     \
        scale, window, v_dim, sinks, (const T*)gate, gate_stride, out_scale, out_stride, keep_first, out_wide, softcap,         \
        gate_wide, whole);                                                                                                      \
  } while (0)
  if (v_dim <= 64) PTB_AG(1);
  else if (v_dim <= 128) PTB_AG(2);
  else PTB_AG(4);
#undef PTB_AG
  return launch_status();
}

}  // namespace

// cos and sin of position * inv_freq[i] for every token of the step, each times `factor` (a product in float32; 1 for a
// plain rotation): [n_tokens, pairs] each, float32.
__global__ void rope_table_kernel(const int* __restrict__ tok_pos, const float* __restrict__ inv_freq,
                                  float* __restrict__ cos_out, float* __restrict__ sin_out, int n_tokens, int pairs,
                                  float factor) {
  pdl_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_tokens * pairs) return;
  float s, c;
  sincosf(float(tok_pos[i / pairs]) * inv_freq[i % pairs], &s, &c);
  cos_out[i] = factor == 1.f ? c : c * factor;
  sin_out[i] = factor == 1.f ? s : s * factor;
}

PTB_API int ptb_rope_table(const int* tok_pos, const float* inv_freq, float* cos_out, float* sin_out, int n_tokens,
                           int pairs, float factor, cudaStream_t stream) {
  if (n_tokens <= 0 || pairs <= 0) return PTB_OK;
  const int total = n_tokens * pairs;
  launch_pdl(rope_table_kernel, (total + 255) / 256, 256, 0, stream, tok_pos, inv_freq, cos_out, sin_out, n_tokens, pairs, factor);
  return launch_status();
}

PTB_API int ptb_split_rotate_store(int dtype, const void* fused, void* q_out, void* k_pool, void* v_pool,
                                   const StepBatch* sb, const float* inv_freq, const float* rope_cos,
                                   const float* rope_sin, int rot_pairs, int kv_heads, int q_per_kv, int head_dim,
                                   int write_cache, int interleaved, cudaStream_t stream) {
  if (sb->n_tokens <= 0) return PTB_OK;
  if (kv_heads <= 0 || q_per_kv <= 0 || head_dim <= 0 || rot_pairs < 0 || 2 * rot_pairs > head_dim)
    return PTB_ERR_SIZE;
  if (inv_freq == nullptr && rope_cos == nullptr) rot_pairs = 0;
  if ((rope_cos == nullptr) != (rope_sin == nullptr)) return PTB_ERR_SIZE;
  const int threads = 256;
  if (dtype == PTB_F32)
    launch_pdl(split_rotate_store_kernel<float>, sb->n_tokens, threads, 0, stream, 
        (const float*)fused, (float*)q_out, (float*)k_pool, (float*)v_pool, *sb, inv_freq, rope_cos, rope_sin,
        rot_pairs, kv_heads, q_per_kv, head_dim, write_cache, interleaved);
  else if (dtype == PTB_BF16)
    launch_pdl(split_rotate_store_kernel<__nv_bfloat16>, sb->n_tokens, threads, 0, stream, 
        (const __nv_bfloat16*)fused, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, *sb,
        inv_freq, rope_cos, rope_sin, rot_pairs, kv_heads, q_per_kv, head_dim, write_cache, interleaved);
  else
    return PTB_ERR_DTYPE;
  return launch_status();
}

PTB_API int ptb_attention_generic_capped(int dtype, const void* q, const void* k_pool, const void* v_pool, void* out,
                                  const StepBatch* sb, const int* tile_seq, const int* tile_q0, int n_tiles,
                                  const float* alibi_slopes, int heads, int kv_heads, int head_dim, float scale,
                                  int window, int v_dim, const float* sinks, const void* gate, int gate_stride,
                                  float out_scale, int out_stride, int keep_first, float* out_wide, float softcap, int gate_wide,
                                         cudaStream_t stream) {
  // softcap > 0: scores are soft-capped; gate_wide: the gate has heads * v_dim numbers a token (gate_stride at least that)
  // keep_first: with a window, the sequence's first keep_first positions stay visible too. out_wide (float32
  // [tokens][heads][kv_heads][v_dim], or null): every head's weights on every K/V head's values instead of `out`.
  if (n_tiles <= 0) return PTB_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || head_dim <= 0 || head_dim > MAX_D || heads > 65535 ||
      v_dim <= 0 || v_dim > MAX_D || (out_wide == nullptr && out_stride < heads * v_dim) || keep_first < 0 ||
      (out_wide != nullptr && kv_heads > 65535) || softcap < 0.f ||
      (gate != nullptr && gate_stride < (gate_wide ? heads * v_dim : heads)))
    return PTB_ERR_SIZE;
  if (dtype == PTB_F32)
    return launch_attention<float>(q, k_pool, v_pool, out, *sb, tile_seq, tile_q0, n_tiles, alibi_slopes, heads,
                                   kv_heads, head_dim, scale, window, v_dim, sinks, gate, gate_stride, out_scale, out_stride,
                                   keep_first, out_wide, softcap, gate_wide, stream);
  if (dtype == PTB_BF16)
    return launch_attention<__nv_bfloat16>(q, k_pool, v_pool, out, *sb, tile_seq, tile_q0, n_tiles, alibi_slopes,
                                           heads, kv_heads, head_dim, scale, window, v_dim, sinks, gate, gate_stride,
                                           out_scale, out_stride, keep_first, out_wide, softcap, gate_wide, stream);
  return PTB_ERR_DTYPE;
}

PTB_API int ptb_attention_generic(int dtype, const void* q, const void* k_pool, const void* v_pool, void* out,
                                  const StepBatch* sb, const int* tile_seq, const int* tile_q0, int n_tiles,
                                  const float* alibi_slopes, int heads, int kv_heads, int head_dim, float scale,
                                  int window, int v_dim, const float* sinks, const void* gate, int gate_stride,
                                  float out_scale, int out_stride, int keep_first, float* out_wide, cudaStream_t stream) {
  return ptb_attention_generic_capped(dtype, q, k_pool, v_pool, out, sb, tile_seq, tile_q0, n_tiles, alibi_slopes, heads,
                                      kv_heads, head_dim, scale, window, v_dim, sinks, gate, gate_stride, out_scale, out_stride,
                                      keep_first, out_wide, 0.f, 0, stream);
}

// rows of a tile of the general kernel, for the host that builds the tile lists
PTB_API int ptb_attention_generic_tile_rows() { return BQ; }

// bias: float32 [(heads + kv_heads) dim + kv_heads v_dim] or null; rope_cos / rope_sin: float32 [tokens, rot_pairs] or null;
// v_first (rows v_first_stride apart), lam, v_keep [tokens, kv_heads v_dim]: null where not used.
PTB_API int ptb_qk_prepare_store(int dtype, const void* proj, int stride, const float* bias, void* q_out, void* k_pool,
                                void* v_pool, const StepBatch* sb, const float* rope_cos, const float* rope_sin, int rot_pairs,
                                int heads, int kv_heads, int dim, int v_dim, float eps, int unit_norm, const void* v_first,
                                int v_first_stride, const float* lam, void* v_keep, int write_cache, const float* q_gain,
                                 const float* k_gain, int norm_first, float temp_coef, int temp_every, cudaStream_t stream) {
  if (sb->n_tokens <= 0) return PTB_OK;
  if (heads <= 0 || kv_heads <= 0 || dim <= 0 || v_dim <= 0 || stride < (heads + kv_heads) * dim + kv_heads * v_dim ||
      rot_pairs < 0 || 2 * rot_pairs > dim || (rot_pairs > 0 && (rope_cos == nullptr || rope_sin == nullptr)) ||
      (v_first != nullptr && lam == nullptr) || dim > 4096 || temp_every < 0 ||
      ((q_gain != nullptr || k_gain != nullptr) && !(unit_norm && norm_first)))
    return PTB_ERR_SIZE;
  const int warps = 8, threads = 32 * warps;
  const size_t smem = size_t(warps) * (dim + 2 * size_t(rot_pairs)) * sizeof(float);
  if (smem > 48 * 1024) return PTB_ERR_SIZE;
  const int units = heads + 2 * kv_heads;
  if ((units + warps - 1) / warps > 65535) return PTB_ERR_SIZE;
  const dim3 blocks(sb->n_tokens, (units + warps - 1) / warps);
  const size_t pair_bytes = dtype == PTB_F32 ? 8 : 4;
  const int pairs = (dim % 2 == 0 && stride % 2 == 0 && reinterpret_cast<uintptr_t>(proj) % pair_bytes == 0 &&
                     reinterpret_cast<uintptr_t>(q_out) % pair_bytes == 0 && reinterpret_cast<uintptr_t>(k_pool) % pair_bytes == 0)
                        ? 1 : 0;
  // whole quads at aligned rows; heads of more than 256 entries would leave a warp too few registers' worth of entries
  const size_t quad_bytes = 2 * pair_bytes;
  auto quads = [&](const void* p) { return reinterpret_cast<uintptr_t>(p) % quad_bytes == 0; };
  if (dim % 4 == 0 && dim <= 256 && rot_pairs % 4 == 0 && stride % 4 == 0 && quads(proj) && quads(q_out) && quads(k_pool) &&
      aligned16(bias) && aligned16(q_gain) && aligned16(k_gain) && (rot_pairs == 0 || (aligned16(rope_cos) && aligned16(rope_sin)))) {
    const int v_quads = v_dim % 4 == 0 && quads(v_pool) && quads(v_first) && v_first_stride % 4 == 0 && quads(v_keep) ? 1 : 0;
    const int group = dim <= 64 ? 8 : dim <= 128 ? 16 : 32;
    const int rows = (units * group + 255) / 256, per = (units + rows - 1) / rows;      // blocks of a token; alike, of at most 256 threads
    const int wide = (per * group + 31) / 32 * 32;
#define PTB_RNS(T, G)                                                                                                        \
  launch_pdl(rope_norm_store_vec_kernel<T, G>, dim3(sb->n_tokens, rows), wide, 0, stream, (const T*)proj, stride, bias, (T*)q_out, (T*)k_pool, \
             (T*)v_pool, *sb, rope_cos, rope_sin, rot_pairs, heads, kv_heads, dim, v_dim, eps, unit_norm, (const T*)v_first,  \
             v_first_stride, lam, (T*)v_keep, write_cache, v_quads, q_gain, k_gain, norm_first, temp_coef, temp_every, per)
    if (dtype != PTB_F32 && dtype != PTB_BF16) return PTB_ERR_DTYPE;
    if (group == 8) dtype == PTB_F32 ? PTB_RNS(float, 8) : PTB_RNS(__nv_bfloat16, 8);
    else if (group == 16) dtype == PTB_F32 ? PTB_RNS(float, 16) : PTB_RNS(__nv_bfloat16, 16);
    else dtype == PTB_F32 ? PTB_RNS(float, 32) : PTB_RNS(__nv_bfloat16, 32);
#undef PTB_RNS
    return launch_status();
  }
  if (dtype == PTB_F32)
    launch_pdl(rope_norm_store_kernel<float>, blocks, threads, smem, stream, 
        (const float*)proj, stride, bias, (float*)q_out, (float*)k_pool, (float*)v_pool, *sb, rope_cos, rope_sin, rot_pairs,
        heads, kv_heads, dim, v_dim, eps, unit_norm, (const float*)v_first, v_first_stride, lam, (float*)v_keep, write_cache,
        pairs, q_gain, k_gain, norm_first, temp_coef, temp_every);
  else if (dtype == PTB_BF16)
    launch_pdl(rope_norm_store_kernel<__nv_bfloat16>, blocks, threads, smem, stream, 
        (const __nv_bfloat16*)proj, stride, bias, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, *sb,
        rope_cos, rope_sin, rot_pairs, heads, kv_heads, dim, v_dim, eps, unit_norm, (const __nv_bfloat16*)v_first,
        v_first_stride, lam, (__nv_bfloat16*)v_keep, write_cache, pairs, q_gain, k_gain, norm_first, temp_coef,
        temp_every);
  else
    return PTB_ERR_DTYPE;
  return launch_status();
}

PTB_API int ptb_rope_norm_store(int dtype, const void* proj, int stride, const float* bias, void* q_out, void* k_pool,
                                void* v_pool, const StepBatch* sb, const float* rope_cos, const float* rope_sin, int rot_pairs,
                                int heads, int kv_heads, int dim, int v_dim, float eps, int unit_norm, const void* v_first,
                                int v_first_stride, const float* lam, void* v_keep, int write_cache, cudaStream_t stream) {
  return ptb_qk_prepare_store(dtype, proj, stride, bias, q_out, k_pool, v_pool, sb, rope_cos, rope_sin, rot_pairs, heads,
                              kv_heads, dim, v_dim, eps, unit_norm, v_first, v_first_stride, lam, v_keep, write_cache, nullptr,
                              nullptr, 0, 0.f, 0, stream);
}

// Whether talk_mix takes the form that reads `wide` once (talk_mix_vec_kernel: a thread has four columns and a K/V group's heads,
// eight of them at a time) or a thread an output. The first costs the same whatever the tokens until its threads fill the
// device; the second is shorter while its threads are few, so the line lies at 768 outputs an SM for every eight heads
// of a group. us, once against an output a thread: 16 heads of 128 on 4: 8 tokens 5.7 / 4.1, 48 5.7 / 4.8, 80 5.8 / 5.8, 148
// 5.8 / 8.5, 256 6.5 / 12.2; 8 on 4: 64 3.8 / 3.2, 128 3.9 / 4.0; 32 heads of 128 on one: 96 22.1 / 14.4, 192 22.1 / 25.4.
PTB_API int ptb_talk_mix_reads_once(int n_tokens, int heads, int kv_heads, int v_dim) {
  const long long passes = (heads / kv_heads + 7) / 8;
  return v_dim % 4 == 0 && (long long)n_tokens * heads * v_dim >= 768LL * sm_count() * passes ? 1 : 0;
}

PTB_API int ptb_talk_mix(int dtype, const float* wide, const float* talk, void* out, int out_stride, int n_tokens, int heads,
                         int kv_heads, int v_dim, cudaStream_t stream) {
  if (n_tokens <= 0) return PTB_OK;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || v_dim <= 0 || out_stride < heads * v_dim) return PTB_ERR_SIZE;
  if (aligned16(wide) && ptb_talk_mix_reads_once(n_tokens, heads, kv_heads, v_dim)) {
    const long long total = (long long)n_tokens * kv_heads * (v_dim / 4);
    const unsigned blocks = unsigned((total + 127) / 128);
    if (dtype == PTB_F32)
      launch_pdl(talk_mix_vec_kernel<float>, blocks, 128, 0, stream, wide, talk, (float*)out, out_stride, total, heads, kv_heads, v_dim);
    else if (dtype == PTB_BF16)
      launch_pdl(talk_mix_vec_kernel<__nv_bfloat16>, blocks, 128, 0, stream, wide, talk, (__nv_bfloat16*)out, out_stride, total, heads,
                                                                     kv_heads, v_dim);
    else
      return PTB_ERR_DTYPE;
    return launch_status();
  }
  const long long total = (long long)n_tokens * heads * v_dim;
  const unsigned blocks = unsigned((total + 255) / 256);
  if (dtype == PTB_F32)
    launch_pdl(talk_mix_kernel<float>, blocks, 256, 0, stream, wide, talk, (float*)out, out_stride, total, heads, kv_heads, v_dim);
  else if (dtype == PTB_BF16)
    launch_pdl(talk_mix_kernel<__nv_bfloat16>, blocks, 256, 0, stream, wide, talk, (__nv_bfloat16*)out, out_stride, total, heads,
                                                               kv_heads, v_dim);
  else
    return PTB_ERR_DTYPE;
  return launch_status();
}
