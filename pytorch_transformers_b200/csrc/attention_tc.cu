// Prompt attention on the fifth-generation tensor cores (tcgen05) with the accumulators in tensor
// memory, for head sizes 64 and 128 (and keys of 192 entries beside values of 128), bfloat16, causal, with or
// without per-head score slopes (ALiBi), over the paged cache. The description below
// is for head size 64; with 128 the tiles of Q, K and V are two blocks of 64 dims, S takes two groups
// of matrix instructions, O is 128 columns, and one block fits on an SM (two with TWO, below). Above 64 the matrix
// instructions of S and of O += P V are issued by a warp each (APART), and extras and weights of two terms have two
// softmax threads a row, where walks are not short (SHORT).
//
// One block = 128 consecutive new tokens of one sequence x one query head. 128 softmax threads, one per
// query row (tensor-memory lane t = row t). One more warp's first lane issues every matrix
// instruction, another warp's first lane asks the tensor memory accelerator for the pages. The roles
// meet only at mbarriers (page landed, stage free, S written, P written, O updated): there is no
// block-wide barrier in the loop. Keys are walked one cache page (64 keys) at a time:
//
//   S = Q K^T      tcgen05.mma  M=128 N=64 K=64   A = Q  (shared, K-major, 128-byte swizzle)
//                                                 B = K page (shared, K-major, 128-byte swizzle)
//                                                 D = S in tensor memory, three buffers of 64 columns:
//                                                 the products of the next two pages run under this
//                                                 page's softmax
//   softmax        each thread reads its row of S with tcgen05.ld, masks, keeps the running maximum and
//                  sum in float32, rescales its row of O in tensor memory when the maximum moved (only
//                  then it waits for the previous page's O += P V), and writes P = exp2(S - max) as
//                  bfloat16 pairs back into tensor memory with tcgen05.st, in place of its row of S
//   O += P V       tcgen05.mma  M=128 N=64 K=64   A = P read from tensor memory, B = V page (shared,
//                                                 MN-major: head dims are contiguous), D = O in tensor
//                                                 memory, columns [192, 256)
//
// The page tiles [64 keys][64 dims] bfloat16 come by TMA (cp.async.bulk.tensor.2d over the cache pool
// seen as rows of D values, 128-byte swizzle) into a four-stage ring: exactly the canonical layout that
// the matrix descriptors name (K-major for Q and K; MN-major for V); a stage's mbarrier counts the
// bytes, and tcgen05.commit after the O += P V that read a stage gives it back to the copy thread. The
// softmax threads neither copy nor wait for copies. Completion of the matrix instructions is signalled
// through tcgen05.commit on mbarriers. Every wait on a barrier is bounded: if it runs out, a flag in
// global memory is raised and the block carries on to its end (tensor memory is freed on every path,
// copies in flight are waited for), so a fault in the pipeline shows as an error, never as a hang.
//
// Two blocks fit on an SM (81 KB of shared memory and 256 columns of tensor memory each): while one
// block's threads do softmax, the other's matrix instructions run. Warps of a block may be up to three
// pages apart (S runs that far ahead), which is why "P written" has a barrier per S buffer and "O
// updated" four that take turns (page % 4): a wait names a barrier's phase by its parity, and an
// arrival for a later or an earlier page must not count for page i.
//
// The copy warp sets the barriers up and asks for the first four pages before the block-wide barrier:
// they travel while the other warps fetch Q and tensor memory is allocated.
//
// Decisions that rest on measurements (2,048 tokens, 71 heads on one K/V head; the profile of this kernel
// has the series): one softmax thread per row; O is rescaled only when a row's maximum has grown by more
// than 2^8; three S buffers with P in place of S; P in tensor memory rather than in shared memory; no cap
// on registers; both halves of a row of S asked for before one wait, three-input maxima and packed
// two-value multiply-adds and adds in the softmax (3 %); four page stages. A block is one chain of
// dependent steps per page (about 1,500 clocks with two chains an SM, of which the exponential unit is
// busy 1,024) plus 6 us of set-up and drain; blocks that stay and draw one tile after another from a
// counter saved the set-up but ran their pages 10 to 25 % slower, and were taken out again.
#include "f32x2.cuh"
#include "mma_common.cuh"
#include "tc_common.cuh"

namespace {

__device__ __forceinline__ float max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}
// tanh(x) / x of z = x^2 up to 1: the polynomial of degree 6 whose largest relative error is smallest (5e-8; 1.6e-7 with float32 roundings)
__device__ __forceinline__ uint64_t tanh_ratio2(uint64_t z) {
  constexpr float C[7] = {0.99999995024f, -0.33332839152f, 0.13325204069f, -0.053457029272f, 0.020289979855f, -0.0062033786024f, 0.0010410224670f};
  uint64_t r = pack2(C[6], C[6]);
#pragma unroll
  for (int k = 5; k >= 0; --k) r = fma2(r, z, pack2(C[k], C[k]));
  return r;
}
// of a divisor from 1 on (infinity: 0)
__device__ __forceinline__ float fast_rcp(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
  return r;
}

constexpr int TQ = 128;          // query rows per block
constexpr int STAGES_TC = 4;      // page stages (three are 15 to 30 % slower, five bring nothing)
// Tiles of D = 64 or 128 dims are kept as D / 64 blocks of [rows][64 dims], one after another, each
// block with the 128-byte swizzle: the layout that the matrix descriptors name for K-major operands
// (Q, K: a block per 64 values of the contraction) and for the MN-major V (a block per 64 dims of
// the output). Byte offset of 16-byte chunk `c` of row `row`:
template <int ROWS> __device__ __forceinline__ uint32_t swz_tc(int row, int c) {
  return uint32_t((c >> 3) * (ROWS * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4));
}
struct TcParams {
  int heads, kv_heads;
  float scale;
  const float* slopes;   // per-head score slopes (ALiBi), or null
  // EXTRAS only
  int window, keep_first;            // window > 0: a query sees the last `window` keys and the sequence's first `keep_first`
  float softcap;                     // > 0: score <- softcap * tanh(score / softcap) after the scale
  const float* sinks;                // per head, or null: exp(sink) joins the softmax's denominator
  const __nv_bfloat16* gate;         // or null: token t, head h at gate[t * gate_stride + h], or with gate_wide a number per
  int gate_stride, gate_wide;        // entry at gate[t * gate_stride + h * DV + e]; the result times sigmoid(gate)
  float out_scale;                   // multiplies everything
  int out_stride;                    // from one token's results to the next's
};

// DK, DV: entries of a query or key row and of a value row (64 or 128 alike, or 192 beside 128).
// BIAS: a per-head slope times the key's position is added to the raw scores, formed in bfloat16 as
// the reference forms it.
// WIDE: the softmax weights meet V as two bfloat16 terms (the rounded weight, then what the rounding left: 16
// bits of mantissa). The terms of a page, 32 columns each, together take the place of its S; O += P V is two
// groups of matrix instructions on the same V tile.
// EXTRAS: a window with kept first positions, a soft cap, sinks, an output gate, an output factor and strided results. A walk
// takes the kept pages, then the window's: page i of the walk is not page i of the sequence, and a row may see nothing of a
// page. Nothing else of the pipeline changes. 16 heads of 128 on 4 K/V heads, 2,048 tokens, window 1,024: 31 us (the mma.sync
// kernel 175); prompts of 500, 1,000 and 1,501 tokens, cap and a gate per entry: 66 us against 261.
// Head sizes above 64: what a page costs is a chain of waits and of instructions issued one after another. One thread that issues S and
// O += P V needs 1,810 clocks a page (weights of two terms): a wait costs a hundred and more also where what it waits for is there, a
// commit 44, a request for a page some hundreds; the instructions are 900. So each product has a thread, and keys and values of a page
// have a barrier each. With two threads a softmax row (each takes 32 keys of a page; they exchange their maxima through shared memory
// and share the work on O by columns) the softmax is no longer the longest part: 1,500. us with one of each and with both: full context
// of 2,048 tokens, 16 heads 41 -> 38, latent keys of 192 at 3,000 tokens 99 -> 82, 32 heads of 3,400 tokens (TWO) 165 -> 131, window of
// 1,024 in 2,048 tokens 37 -> 31; two threads a row alone 41 -> 41 and 38 -> 37. Head size 64 is bound by the exponential unit: 3 to 7 % slower with two issuing threads or two barriers a page.
// SHORT: one issuing thread and one softmax thread a row, as at head size 64. Short walks are their first and last pages, which hands from one thread to
// the next only lengthen; and where the softmax has little to do beside its waits, or the exponential unit binds it (a cap), two threads a row
// win nothing. us with one and with two: window of 64 in 2,048 tokens 12.2 / 13.0, of 100 13.4 / 14.8, of 160 15.3 / 16.3, of 200 17.0 / 17.4 (3,000
// tokens: 24.9 / 24.2 at 160, 28.4 / 26.2 at 200); capped, 100 17.1 / 19.1, 300 23.5 / 25.3, 512 30.0 / 30.8, 700 36.6 / 37.1, 1,024 42.1 / 40.9, without
// a window 54 / 50; full context of 300 tokens 9.3 / 9.8 (weights of two terms without extras 8.8 / 9.1, of one 8.5 / 8.8), 512 12.5 / 12.3 (12.2 / 11.3, 11.0 /
// 10.9), 700 14.9 / 15.7 (14.6 / 14.6, 13.3 / 13.8), 1,000 19.7 / 20.2 (19.4 / 18.8, 17.4 / 17.4), 1,024 20.3 / 18.9 (19.8 / 17.4, 17.3 / 16.3). Weights of
// one term with extras at any length: 1,280 tokens 20.5 / 21.2, 2,048 32.5 / 33.6. So windows up to 160, or 512 under a cap, and steps of few tiles,
// whose walks are as short. (Keys of 192: window of 128 19.7 / 20.2, full context of 300 tokens and of 64 9.9 / 9.7 and 6.4 / 6.1, so windows alone.)
// TWO (head size 128 with weights of two terms): two S buffers and two page stages instead of three and four, 99 KB and 256
// columns of tensor memory a block, so that two blocks fit on an SM and one's softmax runs under the other's waits. A stage of keys is
// asked for again when its S is complete, not only when its O += P V is (before, S waited 1,000 of a page's 2,560 clocks for its keys),
// and by the thread that issues from it: a third warp would leave 80 registers a thread (2 to 4 % slower). Taken where
// the blocks make more than two waves, or more than one with a window, whose walks are alike long; with fewer blocks and the
// triangle of a full context the longest chain counts, and a block with an SM of its own runs it faster. us, one an SM
// against two (two softmax threads a row): full context 208 blocks 32 / 36, 256 37 / 42, 288 44 / 47, 320 56 / 49, 864 (32 heads) 167 / 131; capped 240 51 / 54, 304 73 /
// 71, 864 245 / 187; window of 300: 160 20 / 16; of 1,024: 256 (2,048 tokens) 38 / 31. Where most of a prompt fits into its window the
// walks are a triangle again and one an SM would be the faster: 160 blocks of 1,024 in 2,560 tokens 23 / 27 (the rule does not
// look at lengths).
template <int DK, bool WIDE, bool EXTRAS, bool TWO, bool SHORT> struct TcThreads {
  static constexpr int PER = DK > 64 && (WIDE || EXTRAS) && !SHORT ? 2 : 1, SOFTMAX = TQ * PER;
  static constexpr bool APART = DK > 64 && !SHORT;      // S and O += P V by a thread each; and (not TWO) a third for the pages
  static constexpr int BLOCK = SOFTMAX + (APART && !TWO ? 96 : 64);      // not APART: one that issues, one for the pages
};
template <bool TWO> struct TcShape {
  static constexpr int BUFS = TWO ? 2 : 3;                 // S buffers
  static constexpr int STAGES = TWO ? 2 : STAGES_TC;       // page stages
};
template <int DK, int DV, bool BIAS, bool WIDE, bool EXTRAS, bool TWO, bool SHORT>
__global__ void __launch_bounds__(TcThreads<DK, WIDE, EXTRAS, TWO, SHORT>::BLOCK, DK == 64 || TWO ? 2 : 1)
attention_tc_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_pool,
                    const __nv_bfloat16* __restrict__ v_pool, __nv_bfloat16* __restrict__ out, StepBatch sb,
                    const int* __restrict__ tile_seq, const int* __restrict__ tile_q0, TcParams p,
                    const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                    int* __restrict__ error_flag) {
  constexpr bool APART = TcThreads<DK, WIDE, EXTRAS, TWO, SHORT>::APART;
  constexpr int BUFS = TcShape<TWO>::BUFS, STAGES = TcShape<TWO>::STAGES;
  constexpr int PER = TcThreads<DK, WIDE, EXTRAS, TWO, SHORT>::PER, SOFTMAX_THREADS = TcThreads<DK, WIDE, EXTRAS, TWO, SHORT>::SOFTMAX, MINE = KEYS / PER;
  __shared__ float row_words[PER == 2 ? 2 : 1][2][PER == 2 ? TQ : 1];      // what a row's two threads tell each other
  extern __shared__ unsigned char smem_dyn[];
  // 1024-byte alignment: the swizzle pattern is a function of address bits 4..9
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  constexpr int TILE_Q_BYTES = TQ * DK * 2;      // 16, 32 or 48 KB
  constexpr int TILE_K_BYTES = KEYS * DK * 2;    // 8, 16 or 24 KB
  constexpr int TILE_V_BYTES = KEYS * DV * 2;    // 8 or 16 KB
  // tensor memory: BUFS (three, or two) S buffers of 64 columns (page i uses buffer i % BUFS), then O. P of a
  // page (64 keys as bfloat16 pairs, 32 columns) takes the place of its S: a thread has its row of S in
  // registers before it writes its row of P, nobody else touches that row, and the S of three pages later
  // is issued after the O += P V that reads this P (the tensor pipe runs in order). With three buffers S
  // runs two pages ahead of the softmax, so the softmax does not wait for a matrix product that was
  // issued only when the slowest warp finished the page before.
  constexpr uint32_t TMEM_O = BUFS * 64, TMEM_COLS = (TMEM_O + DV <= 256) ? 256 : 512;
  unsigned char* q_tile = smem;
  unsigned char* k_ring = q_tile + TILE_Q_BYTES;                      // STAGES pages
  unsigned char* v_ring = k_ring + STAGES * TILE_K_BYTES;          // STAGES pages
  // barriers: [0..2] S buffer written; [3..6] O updated (page % 4); [7..9] P written (page % 3);
  // then per stage: keys landed, values landed
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_ring + STAGES * TILE_V_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10 + 2 * STAGES);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool score_warp = warp == SOFTMAX_THREADS / 32;
  const bool value_warp = APART && warp == SOFTMAX_THREADS / 32 + 1;
  const bool copy_warp = !(TWO && APART) && warp == SOFTMAX_THREADS / 32 + (APART ? 2 : 1);
  const int row = tid & (TQ - 1);        // query row of a softmax thread (= its tensor-memory lane)
  // heads are the fast index of the grid: the blocks of one tile start together (they read the same
  // pages), and tiles come in the order of the list, which the caller sorts by falling key count so that
  // the longest chains start first and the short ones fill the end
  const int tile = blockIdx.y, h = blockIdx.x;
  const int qpk = p.heads / p.kv_heads;
  const int g = h / qpk;
  const int seq = tile_seq[tile], q0 = tile_q0[tile];
  const int n_new = sb.seq_new[seq], past = sb.seq_past[seq], start = sb.seq_start[seq];
  const int tok_valid = min(TQ, n_new - q0);
  const bool row_ok = row < tok_valid;
  const int row_pos = row_ok ? past + q0 + row : -1;
  const int last_pos = past + q0 + tok_valid - 1;
  const int* pages = sb.pages + size_t(seq) * sb.pages_stride;
  int kb_lo = 0, kept_pages = 0;      // the window's first page for the tile's first token; kept pages left of it
  if (EXTRAS && p.window > 0) {
    kb_lo = max(0, past + q0 - p.window + 1) / KEYS;
    kept_pages = min((p.keep_first + KEYS - 1) / KEYS, kb_lo);
  }
  const int n_blocks = kept_pages + last_pos / KEYS + 1 - kb_lo;
  auto block_of = [&](int i) { return EXTRAS ? (i < kept_pages ? i : kb_lo + i - kept_pages) : i; };   // page i of the walk

  // A warp may be up to three pages ahead of another one (S of page i + 3 is issued after the O += P V of page i, that of page i + 2
  // before P of page i is complete): arrivals for pages i + 1 and i + 2 must not count for page
  // i, hence a "P written" barrier per S buffer. A wait names a barrier's phase by its parity, which is
  // only right if the completion before the awaited one has happened already. A thread that has read S of
  // page i knows that O += P V of page i - 3 has completed (S of page i was issued after that), and so the one
  // of page i - 4: hence four "O updated" barriers that take turns. With two, a warp that reached the end
  // of its walk pages ahead of the others could take the completion of page i - 2 for that of page i and
  // read O before the last products were in it. With two S buffers every distance is one page less.
  const uint32_t bar_s = smem_u32(&bars[0]), bar_o = smem_u32(&bars[3]);
  const uint32_t bar_p = smem_u32(&bars[7]);
  const uint32_t bar_k = smem_u32(&bars[10]), bar_v = smem_u32(&bars[10 + STAGES]);
  // The keys or values of page b of the walk into stage b % STAGES, as boxes [64 keys x 64 dims] in the swizzled layout; a barrier counts
  // the bytes, one for both where one thread waits for both.
  auto ask_keys = [&](int b, int page) {
    const int st = b % STAGES, y = (page * p.kv_heads + g) * KEYS;   // first row of the page in the pool seen as [rows][D]
    const uint32_t full = bar_k + 8 * st;
    mbar_expect_tx(full, TILE_K_BYTES + (APART ? 0 : TILE_V_BYTES));
#pragma unroll
    for (int blk = 0; blk < DK / 64; ++blk)
      tma_load_2d(smem_u32(k_ring + st * TILE_K_BYTES + blk * (KEYS * 128)), &k_map, blk * 64, y, full);
  };
  auto ask_values = [&](int b, int page) {      // after ask_keys of the page
    const int st = b % STAGES, y = (page * p.kv_heads + g) * KEYS;
    const uint32_t full = (APART ? bar_v : bar_k) + 8 * st;
    if (APART) mbar_expect_tx(full, TILE_V_BYTES);
#pragma unroll
    for (int blk = 0; blk < DV / 64; ++blk)
      tma_load_2d(smem_u32(v_ring + st * TILE_V_BYTES + blk * (KEYS * 128)), &v_map, blk * 64, y, full);
  };
  // The first lane of the copy warp (TWO and APART: of the one that issues S) sets the barriers up and asks for the first pages at once (their numbers
  // read by the warp's lanes, one each): they are on their way while the other warps fetch Q and tensor
  // memory is allocated. Nobody else touches a barrier before the block-wide barrier below.
  if (TWO && APART ? score_warp : copy_warp) {
    const int first_pages = lane < n_blocks ? pages[block_of(lane)] : 0;   // lane b: the number of page b
    if (lane == 0) {
      for (int b = 0; b < 3; ++b) {
        mbar_init(bar_s + 8 * b, 1);
        mbar_init(bar_p + 8 * b, SOFTMAX_THREADS);
      }
      for (int b = 0; b < 4; ++b) mbar_init(bar_o + 8 * b, 1);
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(bar_k + 8 * s, 1);      // the asking thread's expect_tx; the bytes complete it
        mbar_init(bar_v + 8 * s, 1);
      }
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    for (int b = 0; b < STAGES && b < n_blocks; ++b) {
      const int page = __shfl_sync(0xffffffffu, first_pages, b);
      if (lane == 0) {
        ask_keys(b, page);
        ask_values(b, page);
      }
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (warp < SOFTMAX_THREADS / 32) {
    // Q tile: rows of the tile, zero beyond the valid tokens
    const uint32_t qs = smem_u32(q_tile);
    for (int i = tid; i < TQ * (DK / 8); i += SOFTMAX_THREADS) {
      const int r = i / (DK / 8), c = i % (DK / 8);
      if (r < tok_valid)
        cp_async16(qs + swz_tc<TQ>(r, c), q + (size_t(start + q0 + r) * p.heads + h) * DK + c * 8);
      else
        *reinterpret_cast<uint4*>(q_tile + swz_tc<TQ>(r, c)) = make_uint4(0, 0, 0, 0);
    }
    cp_async_commit();
    cp_async_wait<0>();
    proxy_fence_async();
  }
  tc_fence_before();
  __syncthreads();        // barriers, tensor memory and Q are ready for everyone
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_o = tmem_base + TMEM_O;
  bool alive = true;  // false after a wait ran out: keep going without waiting, results are void

  // At head sizes above 64 two threads issue matrix instructions, each for its own products: a wait costs a hundred clocks and more
  // also where what it waits for is there, a commit 44, and one thread's waits and instructions in a row were what a page cost (1,810
  // clocks at head size 128, of which the instructions are 900). At 64 one thread issues both (900 clocks of the 1,500 that a page
  // costs; with two threads 3 to 7 % slower).
  constexpr uint32_t IDESC_S = idesc_bf16(TQ, KEYS, false);
  // all DV dims of the output in one instruction: an instruction of M = 128, K = 16 takes 51 clocks at
  // least whatever its N (N / 2 clocks from N = 128 on), so their number is what a page costs
  constexpr uint32_t IDESC_PV = idesc_bf16(TQ, DV, true);
  const uint64_t desc_q = smem_desc(smem_u32(q_tile), 16, 1024), desc_k0 = smem_desc(smem_u32(k_ring), 16, 1024);
  // V is MN-major: blocks of 64 dims lie KEYS * 128 bytes apart (the leading offset), groups of 8 keys
  // 1024 bytes (the stride offset)
  const uint64_t desc_v0 = smem_desc(smem_u32(v_ring), KEYS * 128, 1024);
  constexpr uint64_t K_UNITS = TILE_K_BYTES >> 4, V_UNITS = TILE_V_BYTES >> 4;   // the address field counts 16-byte units
  constexpr uint64_t Q_BLOCK = (TQ * 128) >> 4, KV_BLOCK = (KEYS * 128) >> 4;   // blocks of 64 dims
  // S = Q K^T of page i into S buffer `buf`
  auto issue_s = [&](int i, int buf) {
    tc_fence_after();
#pragma unroll
    for (int blk = 0; blk < DK / 64; ++blk)
      tc_mma4<2, 2>(tmem_base + buf * 64, desc_q + blk * Q_BLOCK, desc_k0 + (i % STAGES) * K_UNITS + blk * KV_BLOCK, IDESC_S,
                    blk > 0 ? 1u : 0u);
    tc_commit(bar_s + buf * 8);
  };
  // P of page i is written and O is rescaled: O += P V (16 keys: 32 bytes along P's rows, 2048 bytes down V's rows)
  auto issue_pv = [&](int i, int buf) {
    tc_fence_after();
    const uint64_t desc_v = desc_v0 + (i % STAGES) * V_UNITS;
    tc_mma4_ts<128>(tmem_o, tmem_base + buf * 64, desc_v, IDESC_PV, i > 0 ? 1u : 0u);
    if (WIDE) tc_mma4_ts<128>(tmem_o, tmem_base + buf * 64 + KEYS / 2, desc_v, IDESC_PV, 1u);
    tc_commit(bar_o + 8 * (i & 3));
  };
  if (copy_warp) {
    // ------------------------------------------------------------ the pages
    // A stage is free again when the O += P V that read it has completed (S of that page completed before it).
    if (lane == 0) {
      int asked = min(n_blocks, STAGES);
      for (int b = STAGES; b < n_blocks; ++b) {
        const int page = pages[block_of(b)];
        alive = mbar_wait(bar_o + 8 * ((b - STAGES) & 3), ((b - STAGES) >> 2) & 1, error_flag, 6);
        if (!alive) break;
        ask_keys(b, page);
        ask_values(b, page);
        asked = b + 1;
      }
      if (!alive)      // a wait ran out: what is in flight lands before the block ends (bounded waits again)
        for (int b = max(0, asked - STAGES); b < asked; ++b) {
          mbar_wait(bar_k + 8 * (b % STAGES), (b / STAGES) & 1, error_flag, 6);
          if (APART) mbar_wait(bar_v + 8 * (b % STAGES), (b / STAGES) & 1, error_flag, 6);
        }
    }
  } else if (score_warp) {
    // ------------------------------------------------------------ S, and at head size 64 O += P V
    if (lane == 0) {
      int buf = 0, phase = 0;   // S buffer of page i (i % BUFS) and the parity of its barriers ((i / BUFS) & 1)
      if constexpr (APART) {
        int asked = min(n_blocks, STAGES), next_page = TWO && asked < n_blocks ? pages[block_of(asked)] : 0;
        for (int i = 0; i < n_blocks; ++i) {
          if (TWO && i > 0 && asked < n_blocks) {      // the stage of page i - 1 is free again when its S is complete
            alive = mbar_wait(bar_s + 8 * ((i - 1) % BUFS), ((i - 1) / BUFS) & 1, error_flag, 6);
            if (!alive) break;
            ask_keys(asked, next_page);
            if (++asked < n_blocks) next_page = pages[block_of(asked)];
          }
          alive = mbar_wait(bar_k + 8 * (i % STAGES), (i / STAGES) & 1, error_flag, 4);
          // S goes where S and P of page i - BUFS were: the O += P V that read that P has completed, and every thread had read
          // that S before it wrote its P
          if (alive && i >= BUFS) alive = mbar_wait(bar_o + 8 * ((i - BUFS) & 3), ((i - BUFS) >> 2) & 1, error_flag, 4);
          if (!alive) break;
          issue_s(i, buf);
          if (++buf == BUFS) buf = 0;
        }
        if (TWO && !alive)      // a wait ran out: what is in flight lands before the block ends (bounded waits again)
          for (int b = max(0, asked - STAGES); b < asked; ++b) mbar_wait(bar_k + 8 * (b % STAGES), (b / STAGES) & 1, error_flag, 6);
      } else {
        for (int b = 0; b < BUFS - 1 && b < n_blocks && alive; ++b) {
          alive = mbar_wait(bar_k + 8 * b, 0, error_flag, 4);
          if (alive) issue_s(b, b);
        }
        for (int i = 0; i < n_blocks && alive; ++i) {
          const int ahead = i + BUFS - 1;
          if (ahead < n_blocks) {
            // S of page `ahead` goes where S_{i-1} and P_{i-1} were: every thread had read that S before it reported
            // P_{i-1}, and the O += P_{i-1} V_{i-1} that reads the P was issued before (the tensor pipe runs in order)
            alive = mbar_wait(bar_k + 8 * (ahead % STAGES), (ahead / STAGES) & 1, error_flag, 4);
            if (alive) issue_s(ahead, buf == 0 ? BUFS - 1 : buf - 1);
          }
          if (alive) alive = mbar_wait(bar_p + buf * 8, phase, error_flag, 5);
          if (alive) issue_pv(i, buf);
          if (++buf == BUFS) { buf = 0; phase ^= 1; }
        }
      }
    }
  } else if (value_warp) {
    // ------------------------------------------------------------ O += P V
    if (lane == 0) {
      int buf = 0, phase = 0, asked = min(n_blocks, STAGES), next_page = TWO && asked < n_blocks ? pages[block_of(asked)] : 0;
      for (int i = 0; i < n_blocks; ++i) {
        alive = mbar_wait(bar_v + 8 * (i % STAGES), (i / STAGES) & 1, error_flag, 5);
        if (alive) alive = mbar_wait(bar_p + buf * 8, phase, error_flag, 5);
        if (!alive) break;
        issue_pv(i, buf);
        if (++buf == BUFS) { buf = 0; phase ^= 1; }
        if (TWO && i > 0 && asked < n_blocks) {      // the stage of page i - 1 is free again when its O += P V is complete
          alive = mbar_wait(bar_o + 8 * ((i - 1) & 3), ((i - 1) >> 2) & 1, error_flag, 6);
          if (!alive) break;
          ask_values(asked, next_page);
          if (++asked < n_blocks) next_page = pages[block_of(asked)];
        }
      }
      if (TWO && !alive)
        for (int b = max(0, asked - STAGES); b < asked; ++b) mbar_wait(bar_v + 8 * (b % STAGES), (b / STAGES) & 1, error_flag, 6);
    }
  } else {
    // ------------------------------------------------------------ softmax threads
    const int part = PER == 2 ? warp >> 2 : 0;      // of the row: keys [MINE part, MINE part + MINE) of a page, DV / PER columns of O
    const uint32_t lane_addr = tmem_base + (uint32_t((warp & 3) * 32) << 16);   // this warp's lanes
    const uint32_t o_addr = lane_addr + TMEM_O + part * (DV / PER);
    // what the row's other thread says to `mine`; `turn`: 0 and 1 in turns, so that nothing is overwritten before it is read
    auto other = [&](float mine, int turn) {
      row_words[turn][part][row] = mine;
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (warp & 3)) : "memory");
      return row_words[turn][part ^ 1][row];
    };
    int buf = 0, phase = 0;   // S buffer of page i (i % BUFS) and the parity of its barriers ((i / BUFS) & 1)
    float m_run = -INFINITY, l_run = 0.f;   // running maximum of the raw scores, the row's sum
    const float slope = BIAS ? p.slopes[h] : 0.f;
    const bool capped = EXTRAS && p.softcap > 0.f;
    const float sl2 = capped ? 1.f : p.scale * 1.4426950408889634f;      // capped scores are in powers of two already
    const uint64_t sl2_2 = pack2(sl2, sl2);
    for (int i = 0; i < n_blocks; ++i) {
      const int page0 = block_of(i) * KEYS, key0 = page0 + part * MINE;
      // (1) this thread's row of S_i: both halves asked for, one wait
      if (alive) alive = mbar_wait(bar_s + buf * 8, phase, error_flag, 1);
      tc_fence_after();
      float s[MINE];
      if constexpr (PER == 2) tmem_ld32(lane_addr + buf * 64 + part * MINE, s);
      else tmem_ld64_once(lane_addr + buf * 64, s);
      if (BIAS) {
#pragma unroll
        for (int j = 0; j < MINE; ++j) s[j] += alibi_bias(slope, key0 + j);
      }
      // only pages that reach past some row's position, or left of some row's window, hide keys: `with` in their places
      auto hide = [&](float with) {
        if (page0 + KEYS - 1 > past + q0 || !row_ok) {   // first part is uniform over the block
          const int visible = row_pos - key0;   // columns j <= visible are seen by this row
#pragma unroll
          for (int j = 0; j < MINE; ++j) s[j] = (j <= visible) ? s[j] : with;
        }
        if (EXTRAS && p.window > 0 && page0 <= last_pos - p.window) {   // uniform over the block
          const int left = row_pos - p.window - key0, kept = p.keep_first - key0;   // columns left < j or j < kept are seen
#pragma unroll
          for (int j = 0; j < MINE; ++j) s[j] = (j > left || j < kept) ? s[j] : with;
        }
      };
      if (capped) {      // cap * tanh(score / cap), in powers of two
        // Where none of the visible ones reaches the cap, by multiply-adds: the exponential unit, with its exponential and its
        // reciprocal here beside the softmax's exponential, is 1,536 clocks of a capped page (32 heads of 3,400 tokens, two blocks an SM 202
        // -> 187 us; one block an SM, 2,048 tokens 52 -> 50, 1,000 tokens 28.9 -> 29.7). Else tanh(x) = 1 - 2 / (1 + exp(2 x)). Which one follows from what the
        // thread's row sees of the page.
        const float to_x = p.scale / p.softcap, out2 = p.softcap * 1.4426950408889634f;
        bool inside = false;
        if constexpr (PER == 2) {
          hide(0.f);
          float most = 0.f;
#pragma unroll
          for (int j = 0; j < MINE; ++j) most = fmaxf(most, fabsf(s[j]));
          inside = most * to_x <= 1.f;
        }
        if (inside) {
          const uint64_t to_x2 = pack2(to_x, to_x), to_out2 = pack2(to_x * out2, to_x * out2);
#pragma unroll
          for (int j = 0; j < MINE; j += 2) {
            const uint64_t v = pack2(s[j], s[j + 1]), x = mul2(v, to_x2);
            unpack2(mul2(mul2(v, to_out2), tanh_ratio2(mul2(x, x))), s[j], s[j + 1]);
          }
        } else {
          const float in = to_x * (2.f * 1.4426950408889634f);
#pragma unroll
          for (int j = 0; j < MINE; ++j) s[j] = fmaf(-2.f * out2, fast_rcp(fast_exp2(s[j] * in) + 1.f), out2);
        }
        __syncwarp();
      }
      // (2) maximum of the visible scores
      hide(-INFINITY);
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < MINE; j += 8) {
        mx[0] = max3(mx[0], s[j], s[j + 1]);
        mx[1] = max3(mx[1], s[j + 2], s[j + 3]);
        mx[2] = max3(mx[2], s[j + 4], s[j + 5]);
        mx[3] = max3(mx[3], s[j + 6], s[j + 7]);
      }
      float m_page = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
      if constexpr (PER == 2) {      // and the other thread has its scores in registers: their places may be written below
        tc_fence_before();
        m_page = fmaxf(m_page, other(m_page, i & 1));
        tc_fence_after();
      }
      float m_new = fmaxf(m_run, m_page);
      if ((m_new - m_run) * sl2 <= RESCALE_LOG2) m_new = m_run;   // (false from -inf: the first scores set it)
      const float corr = (m_run == -INFINITY) ? 0.f : fast_exp2((m_run - m_new) * sl2);
      const bool moved = (m_new != m_run) && (m_run != -INFINITY);
      m_run = m_new;
      const float m_off = (m_run == -INFINITY) ? 0.f : m_run * sl2;   // exp2(s * sl2 - m_off); exp2(-inf) = 0
      // (3) rescale this thread's row of O if any row of the warp moved its maximum; only then this warp
      // waits for the previous page's O += P V
      if (i > 0 && __any_sync(0xffffffffu, moved)) {
        if (alive) alive = mbar_wait(bar_o + 8 * ((i - 1) & 3), ((i - 1) >> 2) & 1, error_flag, 2);
        tc_fence_after();
#pragma unroll (PER == 2 ? 1 : DV / 32)
        for (int c0 = 0; c0 < DV / PER; c0 += 32) {
          float o[32];
          tmem_ld32(o_addr + c0, o);
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] *= corr;
          tmem_st32(o_addr + c0, o);
        }
        tmem_st_wait();
      }
      // (4) P = exp2(S - max) as bfloat16 pairs, two values per packed multiply-add
      const uint64_t moff_2 = pack2(-m_off, -m_off);
      uint64_t acc2[4] = {0ull, 0ull, 0ull, 0ull};
      uint32_t w[MINE / 2];
#pragma unroll
      for (int e = 0; e < MINE / 2; ++e) {
        float x0, x1;
        unpack2(fma2(pack2(s[2 * e], s[2 * e + 1]), sl2_2, moff_2), x0, x1);
        const float a = fast_exp2(x0), b = fast_exp2(x1);
        acc2[e & 3] = add2(acc2[e & 3], pack2(a, b));
        w[e] = pack_bf16(a, b);
        if (WIDE) {      // what the rounding left, in the places of the two scores (a bfloat16's bits are a float32's upper half)
          s[2 * e] = a - __uint_as_float(w[e] << 16);
          s[2 * e + 1] = b - __uint_as_float(w[e] & 0xffff0000u);
        }
      }
      // P in place of this page's S: keys 2c, 2c + 1 in column c of the buffer (this thread's row of S is in
      // registers since the load above)
      tmem_st_u32<MINE / 2>(lane_addr + buf * 64 + part * (MINE / 2), w);
      if (WIDE) {
        uint32_t lo[MINE / 2];
#pragma unroll
        for (int e = 0; e < MINE / 2; ++e) lo[e] = pack_bf16(s[2 * e], s[2 * e + 1]);
        tmem_st_u32<MINE / 2>(lane_addr + buf * 64 + KEYS / 2 + part * (MINE / 2), lo);
      }
      tmem_st_wait();
      float l0, l1, l2, l3;
      unpack2(add2(acc2[0], acc2[1]), l0, l1);
      unpack2(add2(acc2[2], acc2[3]), l2, l3);
      l_run = l_run * corr + ((l0 + l1) + (l2 + l3));
      tc_fence_before();
      mbar_arrive(bar_p + buf * 8);   // (5) the issuing thread starts O += P V when all rows have arrived
      if (++buf == BUFS) { buf = 0; phase ^= 1; }
    }
    // the walk's last O += P V
    if (alive) alive = mbar_wait(bar_o + 8 * ((n_blocks - 1) & 3), ((n_blocks - 1) >> 2) & 1, error_flag, 3);
    tc_fence_after();
    if constexpr (PER == 2) l_run += other(l_run, n_blocks & 1);
    float inv = l_run > 0.f ? 1.f / l_run : 0.f;
    const size_t t = size_t(start + q0 + row);
    __nv_bfloat16* dst = out + (t * p.heads + h) * DV + part * (DV / PER);
    const __nv_bfloat16* ge = nullptr;      // a gate per entry
    if (EXTRAS) {
      if (p.sinks) {
        const float m2 = m_run * sl2, sink2 = p.sinks[h] * 1.4426950408889634f, m_all = fmaxf(m2, sink2);
        const float keep = (m_run == -INFINITY) ? 0.f : exp2f(m2 - m_all);
        const float l = l_run * keep + exp2f(sink2 - m_all);
        inv = (l > 0.f ? 1.f / l : 0.f) * keep;
      }
      inv *= p.out_scale;
      dst = out + t * p.out_stride + size_t(h) * DV + part * (DV / PER);
      if (p.gate && p.gate_wide) ge = p.gate + t * p.gate_stride + size_t(h) * DV + part * (DV / PER);
      else if (p.gate && row_ok) inv *= 1.f / (1.f + expf(-__bfloat162float(p.gate[t * p.gate_stride + h])));
    }
#pragma unroll (PER == 2 ? 1 : DV / 32)
    for (int c0 = 0; c0 < DV / PER; c0 += 32) {
      float o[32];
      tmem_ld32(o_addr + c0, o);
      if (row_ok) {
        if (EXTRAS && ge) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float gv[8];
            unpack_bf16x8(*reinterpret_cast<const uint4*>(ge + c0 + c * 8), gv);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[c * 8 + e] *= 1.f / (1.f + expf(-gv[e]));
          }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) w[e] = pack_bf16(o[c * 8 + 2 * e] * inv, o[c * 8 + 2 * e + 1] * inv);
          *reinterpret_cast<uint4*>(dst + c0 + c * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS));
}


// ------------------------------------------------------------------------------------------------
// Two query heads of one K/V group in a block ("pair"), keys in steps of two pages.
//
// A tcgen05.mma of M = 128, K = 16 takes 51 clocks at least whatever its N, N / 2 clocks from N = 128 on,
// and no less than its operands take to come from shared memory at 128 bytes a clock (4 KB of A, 32 N
// bytes of B); measured by issuing them back to back. With N = 64 half of the pipe's time is that floor,
// and what a page costs is the number of instructions issued for it (one O += P V group with N = 128
// instead of two with N = 64 took a seventh off the kernel above at head size 128). Here S = Q K^T is
// formed for 128 keys at once (N = 128: half the instructions a key) and O += P V with N = D.
//
// A block = 128 tokens x heads (h, h + 1) of one K/V group: two chains that share every K/V stage. 256
// softmax threads (threads 0..127 the first head, 128..255 the second; both groups sit on tensor-memory
// lanes 0..127, the second on columns 256..511), one issuing thread, one copy warp. A group with an odd
// number of heads ends in a block whose second chain is idle. Per chain, in tensor memory: S [128 x 128]
// in columns 0..127, P (128 keys as bfloat16 pairs, 64 columns) in place of it, O in columns 128..128+D.
// S has one buffer: S of step j + 1 is issued right after O += P V of step j (the pipe runs in order),
// and while a chain waits for it the other chain's softmax has the SM. It follows that a thread that has
// read S of step j finds O += P V of step j - 1 completed: rescaling O needs no wait, only the walk's
// last product is waited for.
//
// Stages hold 128 keys: two pages side by side (rows 0..63 and 64..127 of the K-major K tile and of the
// MN-major V tile; with head size 128 two blocks of 64 dims each). K and V stages are given back
// separately (K after both chains' S, V after both chains' O += P V). A walk with an odd number of pages
// takes its last page twice: the second copy's keys lie past every row's position and are masked.
//
// The issuing thread never blocks on one chain while the other could move: it polls (mbarrier.test_wait)
// "stage landed" and "P written" of both chains in turn, parks for a fraction of a microsecond when
// nothing can be issued, and gives up like every wait when that goes on for seconds.
constexpr int PAIR_SOFTMAX = 2 * TQ;
constexpr int PAIR_THREADS = PAIR_SOFTMAX + 64;
constexpr int STEP_KEYS = 2 * KEYS;
constexpr uint32_t POLL_LIMIT = 1u << 24;

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// one try with a time hint: parks the thread for `ns` at most (the result is not used)
__device__ __forceinline__ void mbar_park(uint32_t bar, uint32_t parity, uint32_t ns) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1, %2;\n\t}\n"
      ::"r"(bar), "r"(parity), "r"(ns) : "memory");
}

template <int D> struct PairShape {
  static constexpr int STAGES = D == 64 ? 4 : 2;           // stages of 128 keys, for K and for V
  static constexpr int TILE_Q_BYTES = TQ * D * 2;
  static constexpr int STAGE_BYTES = STEP_KEYS * D * 2;     // 16 or 32 KB
  static constexpr int N_BARS = 8 + 4 * STAGES;
  static constexpr size_t SMEM = 1024 + 2 * size_t(TILE_Q_BYTES) + 2 * size_t(STAGES) * STAGE_BYTES + N_BARS * 8 + 16;
};

template <int D, bool BIAS>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
attention_tc_pair_kernel(const __nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ out, StepBatch sb,
                         const int* __restrict__ tile_seq, const int* __restrict__ tile_q0, TcParams p,
                         const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                         int* __restrict__ error_flag) {
  using Shape = PairShape<D>;
  constexpr int STAGES = Shape::STAGES, TILE_Q_BYTES = Shape::TILE_Q_BYTES, STAGE_BYTES = Shape::STAGE_BYTES;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t CHAIN_COLS = 256, TMEM_O = 128;
  unsigned char* q_tiles = smem;
  unsigned char* k_ring = q_tiles + 2 * TILE_Q_BYTES;
  unsigned char* v_ring = k_ring + STAGES * STAGE_BYTES;
  // barriers: per chain c at 3 c: S written, P written, the walk's last O += P V; [6], [7] unused; then
  // per stage: K landed, V landed, K free, V free
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_ring + STAGES * STAGE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Shape::N_BARS);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool mma_warp = warp == PAIR_SOFTMAX / 32;
  const bool copy_warp = warp == PAIR_SOFTMAX / 32 + 1;
  const int chain = (tid >> 7) & 1;
  const int row = tid & (TQ - 1);
  const int tile = blockIdx.y;
  const int qpk = p.heads / p.kv_heads;
  const int pairs = (qpk + 1) / 2;                 // blocks a K/V group
  const int g = blockIdx.x / pairs;
  const int h0 = g * qpk + 2 * (blockIdx.x % pairs);
  const bool two = h0 + 1 < (g + 1) * qpk;          // the second chain has a head
  const int seq = tile_seq[tile], q0 = tile_q0[tile];
  const int n_new = sb.seq_new[seq], past = sb.seq_past[seq], start = sb.seq_start[seq];
  const int tok_valid = min(TQ, n_new - q0);
  const bool row_ok = row < tok_valid;
  const int row_pos = row_ok ? past + q0 + row : -1;
  const int last_pos = past + q0 + tok_valid - 1;
  const int n_pages = last_pos / KEYS + 1;
  const int n_steps = (n_pages + 1) / 2;
  const int* pages = sb.pages + size_t(seq) * sb.pages_stride;

  const uint32_t bar0 = smem_u32(bars);
  auto bar_s = [&](int c) { return bar0 + 8u * uint32_t(3 * c); };
  auto bar_p = [&](int c) { return bar0 + 8u * uint32_t(3 * c + 1); };
  auto bar_end = [&](int c) { return bar0 + 8u * uint32_t(3 * c + 2); };
  const uint32_t bar_k = bar0 + 8u * 8, bar_v = bar_k + 8u * STAGES, bar_kfree = bar_v + 8u * STAGES,
                 bar_vfree = bar_kfree + 8u * STAGES;
  // step j: pages 2j and 2j + 1 (or 2j again) into stage j % STAGES, per block of 64 dims rows 0..63 and 64..127
  auto ask = [&](unsigned char* ring, const CUtensorMap* map, uint32_t full, int j, int page_a, int page_b) {
    unsigned char* stage = ring + (j % STAGES) * STAGE_BYTES;
    mbar_expect_tx(full, STAGE_BYTES);
#pragma unroll
    for (int blk = 0; blk < D / 64; ++blk) {
      tma_load_2d(smem_u32(stage + blk * (STEP_KEYS * 128)), map, blk * 64, (page_a * p.kv_heads + g) * KEYS, full);
      tma_load_2d(smem_u32(stage + blk * (STEP_KEYS * 128) + KEYS * 128), map, blk * 64, (page_b * p.kv_heads + g) * KEYS, full);
    }
  };
  // page i of the walk; past its end the last page again (an odd number of pages: its keys are masked)
  auto page_of = [&](int i) { return pages[min(i, n_pages - 1)]; };
  if (copy_warp && lane == 0) {
    for (int c = 0; c < 2; ++c) {
      mbar_init(bar_s(c), 1);
      mbar_init(bar_p(c), TQ);
      mbar_init(bar_end(c), 1);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_k + 8 * s, 1);
      mbar_init(bar_v + 8 * s, 1);
      mbar_init(bar_kfree + 8 * s, 1);
      mbar_init(bar_vfree + 8 * s, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    // the first stages are asked for at once: they travel while Q is fetched and tensor memory allocated
    for (int j = 0; j < STAGES && j < n_steps; ++j) {
      const int pa = page_of(2 * j), pb = page_of(2 * j + 1);
      ask(k_ring, &k_map, bar_k + 8 * (j % STAGES), j, pa, pb);
      ask(v_ring, &v_map, bar_v + 8 * (j % STAGES), j, pa, pb);
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  const bool chain_on = chain == 0 || two;
  if (!mma_warp && !copy_warp && chain_on) {
    unsigned char* q_tile = q_tiles + chain * TILE_Q_BYTES;
    const uint32_t qs = smem_u32(q_tile);
    const int h = h0 + chain;
    for (int i = row; i < TQ * (D / 8); i += TQ) {
      const int r = i / (D / 8), c = i % (D / 8);
      if (r < tok_valid)
        cp_async16(qs + swz_tc<TQ>(r, c), q + (size_t(start + q0 + r) * p.heads + h) * D + c * 8);
      else
        *reinterpret_cast<uint4*>(q_tile + swz_tc<TQ>(r, c)) = make_uint4(0, 0, 0, 0);
    }
    cp_async_commit();
    cp_async_wait<0>();
    proxy_fence_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool alive = true;

  if (copy_warp) {
    if (lane == 0) {
      int k_asked = min(n_steps, STAGES), v_asked = k_asked;
      for (int j = STAGES; j < n_steps && alive; ++j) {
        const int pa = page_of(2 * j), pb = page_of(2 * j + 1);
        const uint32_t before = ((j / STAGES) - 1) & 1;
        alive = mbar_wait(bar_kfree + 8 * (j % STAGES), before, error_flag, 6);
        if (!alive) break;
        ask(k_ring, &k_map, bar_k + 8 * (j % STAGES), j, pa, pb);
        k_asked = j + 1;
        alive = mbar_wait(bar_vfree + 8 * (j % STAGES), before, error_flag, 6);
        if (!alive) break;
        ask(v_ring, &v_map, bar_v + 8 * (j % STAGES), j, pa, pb);
        v_asked = j + 1;
      }
      if (!alive) {
        // a wait ran out: what is in flight lands before the block ends (bounded waits again)
        for (int j = max(0, k_asked - STAGES); j < k_asked; ++j) mbar_wait(bar_k + 8 * (j % STAGES), (j / STAGES) & 1, error_flag, 6);
        for (int j = max(0, v_asked - STAGES); j < v_asked; ++j) mbar_wait(bar_v + 8 * (j % STAGES), (j / STAGES) & 1, error_flag, 6);
      }
    }
  } else if (mma_warp) {
    if (lane == 0) {
      constexpr uint32_t IDESC_S = idesc_bf16(TQ, STEP_KEYS, false);
      constexpr uint32_t IDESC_PV = idesc_bf16(TQ, D, true);
      const uint64_t desc_q0 = smem_desc(smem_u32(q_tiles), 16, 1024);
      const uint64_t desc_k0 = smem_desc(smem_u32(k_ring), 16, 1024);
      // V is MN-major: blocks of 64 dims lie STEP_KEYS * 128 bytes apart (the leading offset), groups of 8
      // keys 1024 bytes (the stride offset)
      const uint64_t desc_v0 = smem_desc(smem_u32(v_ring), STEP_KEYS * 128, 1024);
      constexpr uint64_t STAGE_UNITS = STAGE_BYTES >> 4, Q_UNITS = TILE_Q_BYTES >> 4;
      constexpr uint64_t Q_BLOCK = (TQ * 128) >> 4, K_BLOCK = (STEP_KEYS * 128) >> 4;
      const int n_chains = two ? 2 : 1;
      int s_next[2] = {0, 0};   // next step whose S is to be issued, per chain
      int p_next[2] = {0, 0};   // next step whose O += P V is to be issued
      int k_freed = 0, v_freed = 0;
      uint32_t idle = 0;
      auto behind = [&](const int* v) { return n_chains == 2 ? min(v[0], v[1]) : v[0]; };
      while (behind(p_next) < n_steps && alive) {
        bool moved = false;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (c >= n_chains) continue;
          // O += P V of step i when its P is written (O rescaled) and its V has landed
          const int i = p_next[c];
          if (i < s_next[c] && mbar_test(bar_p(c), i & 1) && mbar_test(bar_v + 8 * (i % STAGES), (i / STAGES) & 1)) {
            tc_fence_after();
            const uint32_t o = tmem_base + c * CHAIN_COLS + TMEM_O, pp = tmem_base + c * CHAIN_COLS;
            const uint64_t dv = desc_v0 + (i % STAGES) * STAGE_UNITS;
            tc_mma4_ts<128>(o, pp, dv, IDESC_PV, i > 0 ? 1u : 0u);                       // keys 0..63 of the step
            tc_mma4_ts<128>(o, pp + 32, dv + ((KEYS * 128) >> 4), IDESC_PV, 1u);          // keys 64..127
            if (i + 1 == n_steps) tc_commit(bar_end(c));
            p_next[c] = i + 1;
            moved = true;
            while (v_freed < behind(p_next)) {   // both chains' products of the step have been issued
              tc_commit(bar_vfree + 8 * (v_freed % STAGES));
              ++v_freed;
            }
          }
          // S of step j: the buffer held S and P of step j - 1, whose O += P V must have been issued
          const int j = s_next[c];
          if (j < n_steps && j == p_next[c] && mbar_test(bar_k + 8 * (j % STAGES), (j / STAGES) & 1)) {
            tc_fence_after();
#pragma unroll
            for (int blk = 0; blk < D / 64; ++blk)
              tc_mma4<2, 2>(tmem_base + c * CHAIN_COLS, desc_q0 + c * Q_UNITS + blk * Q_BLOCK,
                            desc_k0 + (j % STAGES) * STAGE_UNITS + blk * K_BLOCK, IDESC_S, blk > 0 ? 1u : 0u);
            tc_commit(bar_s(c));
            s_next[c] = j + 1;
            moved = true;
            while (k_freed < behind(s_next)) {
              tc_commit(bar_kfree + 8 * (k_freed % STAGES));
              ++k_freed;
            }
          }
        }
        if (moved) idle = 0;
        else if (++idle > POLL_LIMIT) {
          atomicExch(error_flag, 13);
          alive = false;
        } else {
          // nothing to issue: park on what the chain further behind waits for (a spinning thread would take
          // issue slots from the softmax warps of its quarter of the SM)
          const bool second = n_chains == 2 && p_next[1] < p_next[0];
          const int i = second ? p_next[1] : p_next[0], sn = second ? s_next[1] : s_next[0];
          if (i < sn) mbar_park(bar_p(second ? 1 : 0), i & 1, 200);
          else mbar_park(bar_k + 8 * (i % STAGES), (i / STAGES) & 1, 200);
        }
      }
    }
  } else if (chain_on) {
    // ------------------------------------------------------------ softmax threads of chain `chain`
    const int h = h0 + chain;
    const uint32_t lane_addr = tmem_base + (uint32_t((warp & 3) * 32) << 16) + chain * CHAIN_COLS;
    const uint32_t o_addr = lane_addr + TMEM_O;
    float m_run = -INFINITY, l_run = 0.f;
    const float slope = BIAS ? p.slopes[h] : 0.f;
    const float sl2 = p.scale * 1.4426950408889634f;
    const uint64_t sl2_2 = pack2(sl2, sl2);
    for (int j = 0; j < n_steps; ++j) {
      if (alive) alive = mbar_wait(bar_s(chain), j & 1, error_flag, 1);
      tc_fence_after();
      const int key0 = j * STEP_KEYS;
      const bool masked = key0 + STEP_KEYS - 1 > past + q0 || !row_ok;   // first part is uniform over the block
      // (1) the row's maximum over the step's 128 scores, a half of 64 at a time
      float m_new = m_run;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float s[KEYS];
        tmem_ld64_once(lane_addr + half * KEYS, s);
        if (BIAS) {
#pragma unroll
          for (int e = 0; e < KEYS; ++e) s[e] += alibi_bias(slope, key0 + half * KEYS + e);
        }
        if (masked) {
          const int visible = row_pos - key0 - half * KEYS;
#pragma unroll
          for (int e = 0; e < KEYS; ++e) s[e] = (e <= visible) ? s[e] : -INFINITY;
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < KEYS; e += 8) {
          mx[0] = max3(mx[0], s[e], s[e + 1]);
          mx[1] = max3(mx[1], s[e + 2], s[e + 3]);
          mx[2] = max3(mx[2], s[e + 4], s[e + 5]);
          mx[3] = max3(mx[3], s[e + 6], s[e + 7]);
        }
        m_new = fmaxf(m_new, fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]));
      }
      if ((m_new - m_run) * sl2 <= RESCALE_LOG2) m_new = m_run;   // (false from -inf: the first scores set it)
      const float corr = (m_run == -INFINITY) ? 0.f : fast_exp2((m_run - m_new) * sl2);
      const bool moved = (m_new != m_run) && (m_run != -INFINITY);
      m_run = m_new;
      const float m_off = (m_run == -INFINITY) ? 0.f : m_run * sl2;
      // (2) O rescaled if any row of the warp moved its maximum: O += P V of the step before has completed
      // (S of this step was issued after it)
      if (j > 0 && __any_sync(0xffffffffu, moved)) {
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 32) {
          float o[32];
          tmem_ld32(o_addr + c0, o);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] *= corr;
          tmem_st32(o_addr + c0, o);
        }
        tmem_st_wait();
      }
      // (3) P = exp2(S - max), a half at a time: the first half's P goes over the first half's S (read for
      // the last time just before), the second half's P over the rest of the first half's S
      const uint64_t moff_2 = pack2(-m_off, -m_off);
      uint64_t acc2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float s[KEYS];
        tmem_ld64_once(lane_addr + half * KEYS, s);
        if (BIAS) {
#pragma unroll
          for (int e = 0; e < KEYS; ++e) s[e] += alibi_bias(slope, key0 + half * KEYS + e);
        }
        if (masked) {
          const int visible = row_pos - key0 - half * KEYS;
#pragma unroll
          for (int e = 0; e < KEYS; ++e) s[e] = (e <= visible) ? s[e] : -INFINITY;
        }
        uint32_t w[KEYS / 2];
#pragma unroll
        for (int e = 0; e < KEYS / 2; ++e) {
          float x0, x1;
          unpack2(fma2(pack2(s[2 * e], s[2 * e + 1]), sl2_2, moff_2), x0, x1);
          const float a = fast_exp2(x0), b = fast_exp2(x1);
          acc2[e & 3] = add2(acc2[e & 3], pack2(a, b));
          w[e] = pack_bf16(a, b);
        }
        tmem_st_u32<KEYS / 2>(lane_addr + half * (KEYS / 2), w);
      }
      tmem_st_wait();
      float l0, l1, l2, l3;
      unpack2(add2(acc2[0], acc2[1]), l0, l1);
      unpack2(add2(acc2[2], acc2[3]), l2, l3);
      l_run = l_run * corr + ((l0 + l1) + (l2 + l3));
      tc_fence_before();
      mbar_arrive(bar_p(chain));
    }
    if (alive) alive = mbar_wait(bar_end(chain), 0, error_flag, 3);
    tc_fence_after();
    const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
    __nv_bfloat16* dst = out + (size_t(start + q0 + row) * p.heads + h) * D;
#pragma unroll
    for (int c0 = 0; c0 < D; c0 += 32) {
      float o[32];
      tmem_ld32(o_addr + c0, o);
      if (row_ok) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) w[e] = pack_bf16(o[c * 8 + 2 * e] * inv, o[c * 8 + 2 * e + 1] * inv);
          *reinterpret_cast<uint4*>(dst + c0 + c * 8) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512));
}

template <int D, bool BIAS>
int launch_tc_pair(const void* q, const void* k_pool, const void* v_pool, int pool_pages, void* out, const StepBatch& sb,
                   const int* tile_seq, const int* tile_q0, int n_tiles, const TcParams& p, int* error_flag,
                   cudaStream_t stream) {
  const CUtensorMap* km = pool_map(k_pool, pool_pages, p.kv_heads, D);
  const CUtensorMap* vm = pool_map(v_pool, pool_pages, p.kv_heads, D);
  if (km == nullptr || vm == nullptr) return PTB_ERR_LAUNCH;
  constexpr size_t smem = PairShape<D>::SMEM;
  static SharedLimit limit;
  if (!limit.allows(attention_tc_pair_kernel<D, BIAS>, smem)) return PTB_ERR_LAUNCH;
  const int qpk = p.heads / p.kv_heads;
  dim3 grid(p.kv_heads * ((qpk + 1) / 2), n_tiles);
  attention_tc_pair_kernel<D, BIAS><<<grid, PAIR_THREADS, smem, stream>>>(
      (const __nv_bfloat16*)q, (__nv_bfloat16*)out, sb, tile_seq, tile_q0, p, *km, *vm, error_flag);
  return launch_status();
}
}  // namespace

static int g_pair_mode = 1;
// for measurements and tests: 0 = every head a block of its own also where pairs would do, 1 = pairs where
// they fill the device (the default), 2 = pairs wherever a K/V group has two heads or more
PTB_API void ptb_attention_tc_pairs(int mode) { g_pair_mode = mode; }
PTB_API int ptb_attention_tc_supports(int head_dim) { return (head_dim == 64 || head_dim == 128) ? 1 : 0; }
// with key rows and value rows of different sizes
PTB_API int ptb_attention_tc_supports_sizes(int head_dim, int v_dim) {
  return ((head_dim == 64 || head_dim == 128) && v_dim == head_dim) || (head_dim == 192 && v_dim == 128) ? 1 : 0;
}
PTB_API int ptb_attention_tc_tile_tokens() { return TQ; }

namespace {
template <int DK, int DV, bool BIAS, bool WIDE, bool EXTRAS = false, bool TWO = false, bool SHORT = false>
int launch_tc(const void* q, const void* k_pool, const void* v_pool, int pool_pages, void* out, const StepBatch& sb,
              const int* tile_seq, const int* tile_q0, int n_tiles, const TcParams& p, int* error_flag,
              cudaStream_t stream) {
  constexpr bool NARROW_EXTRAS = DK == 128 && EXTRAS && !WIDE;
  if constexpr (DK > 64 && !SHORT && !TWO) {      // the rule of SHORT
    const int few = DK > 128 ? 0 : WIDE && !EXTRAS ? 3 : 6;
    if (NARROW_EXTRAS || (p.softcap > 0.f ? DK == 128 && p.window > 0 && p.window <= 512 : (p.window > 0 && p.window <= 160) || n_tiles <= few))
      return launch_tc<DK, DV, BIAS, WIDE, EXTRAS, TWO, true>(q, k_pool, v_pool, pool_pages, out, sb, tile_seq, tile_q0, n_tiles, p,
                                                              error_flag, stream);
  }
  if constexpr (!NARROW_EXTRAS || SHORT) {
    if constexpr (DK == 128 && DV == 128 && WIDE && !TWO) {      // the rule of TWO
      const long long blocks = (long long)p.heads * n_tiles, sms = sm_count();
      if (blocks > 2 * sms || (p.window > 0 && blocks > sms))
        return launch_tc<DK, DV, BIAS, WIDE, EXTRAS, true, SHORT>(q, k_pool, v_pool, pool_pages, out, sb, tile_seq, tile_q0, n_tiles, p,
                                                                  error_flag, stream);
    }
    const CUtensorMap* km = pool_map(k_pool, pool_pages, p.kv_heads, DK);
    const CUtensorMap* vm = pool_map(v_pool, pool_pages, p.kv_heads, DV);
    if (km == nullptr || vm == nullptr) return PTB_ERR_LAUNCH;
    const size_t smem = 1024 + TQ * DK * 2 + TcShape<TWO>::STAGES * KEYS * (DK + DV) * 2 + 192;
    static SharedLimit limit;
    if (!limit.allows(attention_tc_kernel<DK, DV, BIAS, WIDE, EXTRAS, TWO, SHORT>, smem)) return PTB_ERR_LAUNCH;
    dim3 grid(p.heads, n_tiles);
    attention_tc_kernel<DK, DV, BIAS, WIDE, EXTRAS, TWO, SHORT><<<grid, TcThreads<DK, WIDE, EXTRAS, TWO, SHORT>::BLOCK, smem, stream>>>(
        (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, (__nv_bfloat16*)out, sb,
        tile_seq, tile_q0, p, *km, *vm, error_flag);
  }
  return launch_status();
}
}  // namespace

// Causal attention of prompt tiles of 128 tokens (tile_seq / tile_q0 as for the other attention
// kernels, 128 tokens per tile), bfloat16, no window. Keys of head_dim and values of v_dim entries: 64 or 128 alike,
// or 192 beside 128. k_pool / v_pool: the pools of one cache entry, [pool_pages][kv_heads][64][head_dim or v_dim].
// `slopes`: per-head score slopes [heads] float32 (already rounded to bfloat16 values), or null. wide_weights: the
// softmax weights meet the values as two bfloat16 terms. `error_flag` is a device int that stays 0 unless a
// bounded wait inside the kernel ran out.
PTB_API int ptb_attention_tc_sizes(const void* q, const void* k_pool, const void* v_pool, int pool_pages, void* out,
                                   const StepBatch* sb, const int* tile_seq, const int* tile_q0, int n_tiles,
                                   const float* slopes, int heads, int kv_heads, int head_dim, int v_dim, float scale,
                                   int wide_weights, int* error_flag, cudaStream_t stream) {
  if (n_tiles <= 0) return PTB_OK;
  if (pool_pages <= 0 || (reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15) return PTB_ERR_ALIGN;
  if (!ptb_attention_tc_supports_sizes(head_dim, v_dim) || heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 ||
      n_tiles > 65535 || error_flag == nullptr)
    return PTB_ERR_SIZE;
  TcParams p = {};
  p.heads = heads; p.kv_heads = kv_heads; p.scale = scale; p.slopes = slopes;
#define PTB_TC(DK, DV, B, W) \
  launch_tc<DK, DV, B, W>(q, k_pool, v_pool, pool_pages, out, *sb, tile_seq, tile_q0, n_tiles, p, error_flag, stream)
  if (wide_weights) {
    if (slopes) return PTB_ERR_SIZE;      // not built: no model has score slopes beside split weights
    return head_dim == 64 ? PTB_TC(64, 64, false, true) : head_dim == 128 ? PTB_TC(128, 128, false, true) : PTB_TC(192, 128, false, true);
  }
  if (head_dim == 192) return slopes ? PTB_ERR_SIZE : PTB_TC(192, 128, false, false);
  if (head_dim == 64) return slopes ? PTB_TC(64, 64, true, false) : PTB_TC(64, 64, false, false);
  // Head size 128 leaves room for one block an SM: two heads of a K/V group share a block, with keys in
  // steps of two pages, where a group has two heads or more and the pairs fill the device. (With head size
  // 64 two blocks of the kernel above share an SM, each with three S buffers, and are a quarter faster than
  // the pairs with their one S buffer a chain: 833 against 1,067 us at 8,192 tokens and 71 heads.)
  const int qpk = heads / kv_heads;
  const long long pair_blocks = (long long)kv_heads * ((qpk + 1) / 2) * n_tiles;
  if (qpk >= 2 && g_pair_mode != 0 && (pair_blocks >= sm_count() || g_pair_mode == 2))
    return slopes ? launch_tc_pair<128, true>(q, k_pool, v_pool, pool_pages, out, *sb, tile_seq, tile_q0, n_tiles, p, error_flag, stream)
                  : launch_tc_pair<128, false>(q, k_pool, v_pool, pool_pages, out, *sb, tile_seq, tile_q0, n_tiles, p, error_flag, stream);
  return slopes ? PTB_TC(128, 128, true, false) : PTB_TC(128, 128, false, false);
#undef PTB_TC
}

PTB_API int ptb_attention_tc(const void* q, const void* k_pool, const void* v_pool, int pool_pages, void* out,
                             const StepBatch* sb,
                             const int* tile_seq, const int* tile_q0, int n_tiles, const float* slopes, int heads,
                             int kv_heads, int head_dim, float scale, int* error_flag, cudaStream_t stream) {
  if (!ptb_attention_tc_supports(head_dim)) return PTB_ERR_SIZE;
  return ptb_attention_tc_sizes(q, k_pool, v_pool, pool_pages, out, sb, tile_seq, tile_q0, n_tiles, slopes, heads, kv_heads,
                                head_dim, head_dim, scale, 0, error_flag, stream);
}

// The same with what some designs put around the softmax (TcParams), the same sizes; wide_weights as above. out: rows
// out_stride apart and a gate per entry's rows at whole 16-byte words.
PTB_API int ptb_attention_tc_extras(const void* q, const void* k_pool, const void* v_pool, int pool_pages, void* out,
                                    const StepBatch* sb, const int* tile_seq, const int* tile_q0, int n_tiles, int heads,
                                    int kv_heads, int head_dim, int v_dim, float scale, int wide_weights, int window, int keep_first, float softcap,
                                    const float* sinks, const void* gate, int gate_stride, int gate_wide, float out_scale,
                                    int out_stride, int* error_flag, cudaStream_t stream) {
  if (n_tiles <= 0) return PTB_OK;
  if (pool_pages <= 0 || !aligned16(k_pool) || !aligned16(v_pool) || !aligned16(q) || !aligned16(out) || out_stride % 8 != 0 ||
      (gate != nullptr && gate_wide && (!aligned16(gate) || gate_stride % 8 != 0)))
    return PTB_ERR_ALIGN;
  if (!ptb_attention_tc_supports_sizes(head_dim, v_dim) || heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || n_tiles > 65535 ||
      error_flag == nullptr || window < 0 || keep_first < 0 || softcap < 0.f || out_stride < heads * v_dim ||
      (gate != nullptr && gate_stride < (gate_wide ? heads * v_dim : heads)))
    return PTB_ERR_SIZE;
  TcParams p = {};
  p.heads = heads; p.kv_heads = kv_heads; p.scale = scale; p.window = window; p.keep_first = keep_first; p.softcap = softcap;
  p.sinks = sinks; p.gate = (const __nv_bfloat16*)gate; p.gate_stride = gate_stride; p.gate_wide = gate_wide;
  p.out_scale = out_scale; p.out_stride = out_stride;
#define PTB_TCX(DK, DV, W) \
  launch_tc<DK, DV, false, W, true>(q, k_pool, v_pool, pool_pages, out, *sb, tile_seq, tile_q0, n_tiles, p, error_flag, stream)
  if (head_dim == 64) return wide_weights ? PTB_TCX(64, 64, true) : PTB_TCX(64, 64, false);
  if (head_dim == 128) return wide_weights ? PTB_TCX(128, 128, true) : PTB_TCX(128, 128, false);
  return wide_weights ? PTB_TCX(192, 128, true) : PTB_TCX(192, 128, false);
#undef PTB_TCX
}
