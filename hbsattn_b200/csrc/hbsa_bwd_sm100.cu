// Backward of the block-sparse attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA), bf16 / fp16,
// head dimensions up to 128.  The mathematics is that of hbsa_bwd_generic.cu:
//     P = exp(scale * Q K^T - lse)      delta = rowsum(dO * O)      dS = P * (dO V^T - delta)
//     dV = P^T dO                       dQ = scale * dS K           dK = scale * dS^T Q
//
// One kernel template, launched twice, each time with one operand pair stationary and the other streamed past it:
//   dK/dV (KV = true):  K, V of up to 128 keys of one k-block stay; Q, dO of the q-blocks that attend to it are streamed in
//                       tiles of at most 64 rows (tokens x GQA heads).  S^T = K Q^T and dP^T = V dO^T land in TMEM with one
//                       key per lane, dV += P^T dO and dK += dS^T Q take their left operand straight from TMEM.
//   dQ   (KV = false):  Q, dO of one 128-row M tile stay (the forward's work items); K, V of the active k-blocks are
//                       streamed.  S = Q K^T, dP = dO V^T, dQ += dS K.
// Recomputing S and dP in both launches costs two of seven products but leaves every gradient element with exactly one
// writer: no fp32 accumulators in memory, no atomics, no conversion pass, and bit-identical results from run to run.
//
// P and dS enter the second products as the sum of two 16-bit terms (hi + lo), which doubles three of the seven products and is
// what bounds the kernel: per 128x64 tile at d = 128 the tensor pipe is occupied 16 x 47 clocks by the two first products (N = 64
// operands from shared memory) and 32 x 64 (dK/dV) or 16 x 64 (dQ) by the second ones.
//
// Precision of the pair.  bf16: 16 significant bits at any magnitude, against the 8 that the gradients are rounded to.  fp16: 22 bits
// down to 2^-3, and 2^-25 absolutely below (fp16 ends at 2^-24).  So P and dS are scaled by powers of two, of their own for
// every row of the stationary tile (a key in dK/dV, a row of q in dQ; a row of an accumulator can be scaled back exactly):
//   first launch   2^15 P;  dS by 2^13 / (|dO row| max|V|) (dQ) or 2^13 / (max|dO| max|V|) (dK/dV), which keeps it below 2^15.
//                  The largest |P| and |dS| of every row are kept track of on the way.
//   second launch  items in which a row's largest value stayed below 2^-10 sqrt(tiles) (keys that share their queries with an attention sink,
//                  rows whose dO is far below their neighbours') or went above 2^16 are done again with powers of two that
//                  bring every row's largest value to 2^14.  What is lost then is 2^-39 of it: less than the fp32 sums lose.
// The norms and maxima are those of the sample and kv-head alone: a gradient does not depend on the rest of the batch.
// Relative error (2-norm) against float64, CUDA-core kernels with fp32 P and dS -> these: 8 ragged samples, d = 64, fp16: dQ 2.1417e-4 ->
// 2.1410e-4, dK 2.1089e-4 -> 2.1081e-4, dV 2.0751e-4 -> 2.0754e-4; two samples of up to 4096, d = 128, bf16: dQ 1.9083e-3 -> 1.9067e-3,
// dK 1.8955e-3 -> 1.8944e-3, dV 1.6515e-3 -> 1.6515e-3.  dV of fp16 keys beside a sink (CUDA cores / P unscaled / these): sink 16
// above, 8192 keys, dO of 256: 2.08e-4 / 0.17 / 2.09e-4; 20 above, 4096 keys, dO of 1024: 2.26e-4 / 1.0 / 2.26e-4.  Nearly flat fp16
// rows over 16384 keys: 2.21e-4 / 3.50e-4 / 2.25e-4; what is left there comes from the length of the fp32 accumulation (2048 products
// in a row).  The scales and the redo launch take 2 to 3 % of the ragged fp16 training step above.
//
// 320 threads, one persistent CTA per SM (TMEM: two tile buffers of 64 S + 64 dP columns, two accumulators of 128):
//   warps 0-3 / 4-7   elementwise work on the even / odd tiles (thread = TMEM lane), then the epilogue: dV / dK, or the two
//                     halves of dQ's columns
//   warp 8            work fetch, mask scan, TMA, and the {-lse, delta} pairs of the streamed rows
//   warp 9            TMEM allocation and the one thread that issues every tcgen05.mma, in the fixed order
//                     S(0) dP(0) S(1) dP(1) acc(0) S(2) dP(2) acc(1) ...; S(t+2) overwrites the columns of P(t) right behind
//                     acc(t) because the instructions of one thread execute in issue order (HBSA_STRICT_TCGEN05 builds wait
//                     for acc(t) to complete instead).
// The stationary pair is double buffered (the next item's first products overlap this item's epilogue), the streamed pair
// has three stages.
#include <math.h>

#include "sm100_common.cuh"

namespace hbsa {

namespace {

constexpr int kBwdThreads = 320;
constexpr int kBwdEwWarps = 8;
constexpr int kBwdProducer = 8;
constexpr int kBwdMma = 9;
constexpr int kBwdTile = 64;           // rows of a streamed tile, at most
constexpr int kBwdStages = 3;
constexpr uint32_t kBwdBuf = 128u;     // TMEM columns of one S + dP buffer
constexpr uint32_t kBwdAcc = 256u;     // first accumulator column
constexpr float kLog2e = 1.4426950408889634f;

// First words of the gradient workspace: work cursors of dQ, dK/dV and of the items that are done again of each, the CTAs that have
// left each of them, and the number of items that have to be done again (dQ, dK/dV).
struct BwdHeader {
  unsigned long long cursor[4];
  unsigned int left[4];
  unsigned long long redo_count[2];
};

// The gradient workspace; everything from `norm_do` on is used with fp16 only.  A sample's maxima are kept at its first token.
struct BwdSpace {
  BwdHeader* head;
  float2* stats;               // [total_q, nhead_q] {-lse * log2 e (-inf: row without keys), delta}
  unsigned int* max_do;        // [total_q, nhead_k] largest |dO row| of the sample's rows of the group (bits of a non-negative float)
  unsigned int* max_v;         // [total_k, nhead_k] largest |V row|
  float* norm_do;              // [total_q, nhead_q]
  uint16_t *top_q, *top_k;     // [total_q, nhead_q], [total_k, nhead_k]: biased exponents of the row's largest |P| (low byte, dK/dV) and |dS|
  long long *redo_q, *redo_k;  // items to do again: each owns at least one row
};
// Carves the workspace at `base`; returns its size.  `zeroed`: bytes at the front that start as zeros.
size_t carve_space(char* base, long long q_tokens, long long k_tokens, int nhead_q, int nhead_k, BwdSpace* s, size_t* zeroed) {
  char* p = base;
  auto take = [&](size_t bytes) { char* r = p; p += (bytes + 255) / 256 * 256; return r; };
  const size_t rows_q = (size_t)q_tokens * nhead_q, rows_k = (size_t)k_tokens * nhead_k;
  s->head = reinterpret_cast<BwdHeader*>(take(sizeof(BwdHeader)));
  s->max_do = reinterpret_cast<unsigned int*>(take((size_t)q_tokens * nhead_k * 4));
  s->max_v = reinterpret_cast<unsigned int*>(take(rows_k * 4));
  *zeroed = (size_t)(p - base);
  s->stats = reinterpret_cast<float2*>(take(rows_q * sizeof(float2)));
  s->norm_do = reinterpret_cast<float*>(take(rows_q * 4));
  s->top_q = reinterpret_cast<uint16_t*>(take(rows_q * 2));
  s->top_k = reinterpret_cast<uint16_t*>(take(rows_k * 2));
  s->redo_q = reinterpret_cast<long long*>(take(rows_q * 8));
  s->redo_k = reinterpret_cast<long long*>(take(rows_k * 8));
  return (size_t)(p - base);
}

struct BwdParams {
  Problem p;
  Workspace ws;
  BwdSpace sp;
  void *out0, *out1;           // dv, dk (KV) or dq
  int total_q, total_k;
  int gp, gp_shift, n_head_sub;      // q-heads packed into one tile of q rows, tiles of heads per group
  int tt;                      // tokens per tile of q rows
  int nt;                      // rows of a streamed tile (multiple of 16)
  int piece;                   // rows of the pieces that a tile with a block end in it is loaded in
  int m_rows, n_msub;          // KV: keys of one stationary tile, tiles per k-block
  int tiles_per_qblock, items_per_row;  // dQ: as in the forward
  long long total_items;
  float scale_log2;
  long long wait_budget;
  int debug_stall;             // debugging aid: the loader publishes nothing, every wait runs out
};

struct BwdMaps { CUtensorMap a, b, x, y, xp, yp; };      // stationary pair, streamed pair, streamed pair in pieces

struct BwdItem {
  int n_tiles;                 // < 0: no more work
  int row0;                    // first stationary row (token) in the packed tensors
  int end;                     // KV: number of valid keys; dQ: one past the last token of the q-block
  int head;                    // KV: kv-head; dQ: first q-head
  int pos0;                    // in-sample position of the first stationary row
  int k_len, off;
  int first;                   // first token of the sample's queries (KV) or keys (dQ)
  long long index;             // of the item
};

struct __align__(16) BwdControl {
  float neg_lse[kBwdStages][kBwdTile];
  float neg_delta[kBwdStages][kBwdTile];
  unsigned long long item_full[2], item_done[2], stat_full[2], stat_free[2];
  unsigned long long strm_full[kBwdStages], strm_free[kBwdStages];
  unsigned long long s_full[2], dp_full[2], p_ready[2], ds_ready[2];
  unsigned long long acc_full, acc_free, drain;
  unsigned long long top_ready[2];            // the exponents in `top` are there
  unsigned long long ragged_full;             // the copies of a tile with rows to clear (see zero_rows)
  uint32_t tmem_base;
  int abort_flag;
  int fill;                                   // the launch gave up and this is its last CTA: the outputs become NaN
  int redo_mark;                              // fp16: 1 + the last item that was put on the redo list
  uint16_t top[2][128];                       // fp16: exponents of the rows' largest |P| (dQ: keys seen) and |dS| in the tiles of warps 4-7
  int info0[kBwdStages], info1[kBwdStages];   // KV: key limit of the tile's first token; dQ: first key, one past the last key
  BwdItem slot[2];
};

template <bool BF16> __device__ __forceinline__ void unpack16(uint32_t w, float& a, float& b) {
  if (BF16) {
    a = __uint_as_float(w << 16);
    b = __uint_as_float(w & 0xffff0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    a = f.x;
    b = f.y;
  }
}
// x0, x1 = hi + lo, two 16-bit terms each
template <bool BF16> __device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  hi = pack2<BF16>(x0, x1);
  float h0, h1;
  unpack16<BF16>(hi, h0, h1);
  float l0, l1;
  ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(h0, h1), ptx::pack_f32x2(-1.f, -1.f), ptx::pack_f32x2(x0, x1)), l0, l1);
  lo = pack2<BF16>(l0, l1);
}

// The lowest n (0 .. 64) bits.
__device__ __forceinline__ unsigned long long first_bits(int n) { return n >= 64 ? ~0ull : (1ull << n) - 1ull; }

__device__ __forceinline__ float pow2(int e) { return __int_as_float((max(min(e, 127), -126) + 127) << 23); }
__device__ __forceinline__ int exponent_of(float x) { return (int)((__float_as_uint(x) >> 23) & 255u); }     // biased; 255: Inf or NaN
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

constexpr int kPShift = 15;          // fp16: P enters its products as 2^15 P
constexpr int kTopHigh = 127 + 16, kTopGoal = 127 + 14;
// The smallest exponent of a row's largest value that will do.  Every value of the row is off by at most 2^-25, evenly spread (2^-26.8
// in the mean), so a sum over n tiles of 64 by 2^-23.8 sqrt(n): 2^-13 or less of the largest value from 2^-10 sqrt(n) on, no more
// than the rounding of the fp16 result loses, and that only where one value stands alone among very small ones.
__device__ __forceinline__ int top_low(int n_tiles) { return 127 - 10 + (32 - __clz(n_tiles)) / 2; }
// fp16: exponent that keeps |dP - delta|, at most 2 * bound, below 2^15
__device__ __forceinline__ int ds_exponent(float bound) {
  const int e = exponent_of(bound);
  return e == 0 || e == 255 ? 0 : max(min(kTopGoal - 1 - e, 100), -100);
}
// fp16: a row whose largest value has this exponent is done again (zero, Inf and NaN stay what they are)
__device__ __forceinline__ bool out_of_range(int top, int low) { return (top > 0 && top < low) || (top >= kTopHigh && top < 255); }
__device__ __forceinline__ int redo_exponent(int top) { return top > 0 && top < 255 ? kTopGoal - top : 0; }

// Streamed rows that take part in no pair: past the end of the q-block or k-block (they hold whatever follows in the packed
// tensor: the next block or sample, or memory behind the last one) and rows of q that see no key.  Masking gives them a P of zero, but
// 0 x NaN and 0 x Inf would still come out of dP and of the accumulating products, so they have to be zeros in shared memory.
//   * Block ends that fall on a piece (16 rows, or the heads of a token where those are more): the tile is loaded in pieces, those
//     past the end from beyond the tensor, where TMA delivers zeros.  All block ends inside a sample are of this kind.
//   * Otherwise (ends of samples, rows without keys): the loader clears the rows once the tile has landed and hands the tile over
//     afterwards.  (Going on to the next tile meanwhile cost more in every tile than it saved in these: up to 5 %.)
// Isolation is by block: elements that a causal mask cuts out of an active pair are multiplied by an exact zero.
// A training step of 4 samples, bf16, d = 64, tiles that keep the neighbours' rows / all such tiles cleared by the loader / as here:
// 4096 tokens, 128x80 blocks 829 / 936 / 827 us; 300 tokens, 80x48 blocks (a ragged end in most items) 631 / 738 / 660 us.  Clearing by
// the elementwise warps, with selects on S and dP, made every tile 6 % slower.
template <int D>
__device__ __forceinline__ void zero_rows(uint32_t tile, uint32_t y_off, uint32_t panel_bytes, unsigned long long gone, int lane) {
  constexpr int CHUNKS = D / 8;                  // 16-byte pieces of a row
  const int piece = lane % CHUNKS, which = lane / CHUNKS;
  const uint32_t base = tile + (which ? y_off : 0u) + (uint32_t)(piece >> 3) * panel_bytes + (uint32_t)(piece & 7) * 16u;
  for (; gone != 0ull; gone &= gone - 1ull)
    if (which < 2) ptx::st_shared_v4(base + (uint32_t)(__ffsll((long long)gone) - 1) * 128u, 0u, 0u, 0u, 0u);
  ptx::fence_proxy_async();
}

// acc (+)= A[tmem] B over `n` 16-wide k-steps.
__device__ __forceinline__ void issue_ts(uint32_t acc, uint32_t a_tmem, uint64_t b_desc, int n, uint32_t idesc, bool first) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    if (ks < n) {
      if (ks == 0 && first) ptx::mma_ts_c<false>(acc, a_tmem, b_desc, idesc);
      else ptx::mma_ts_c<true>(acc, a_tmem + 8u * ks, b_desc + 128u * ks, idesc);
    }
  }
}

// REDO: the launch that does the items of the redo list again, with the scales that their rows need (fp16).
// `block` of `blocks`: the CTA's place among those of the launch that do this half.
template <int D, bool BF16, bool KV, bool REDO>
__device__ __forceinline__ void bwd_body(const CUtensorMap& tm_a, const CUtensorMap& tm_b, const CUtensorMap& tm_x, const CUtensorMap& tm_y,
                                         const CUtensorMap& tm_xp, const CUtensorMap& tm_yp, const BwdParams& P, unsigned block, unsigned blocks) {
  // a, b: stationary pair (K, V or Q, dO); x, y: streamed pair (Q, dO or K, V)
  using namespace ptx;
  constexpr int PANELS = D / 64;
  constexpr uint32_t STAT = 128u * D * 2u, STRM = (uint32_t)kBwdTile * D * 2u;
  using OutT = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
  const Problem& p = P.p;
  OutT* const out0 = static_cast<OutT*>(P.out0);
  OutT* const out1 = static_cast<OutT*>(P.out1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // tm_xp, tm_yp: the streamed pair in pieces
  const long long total_items = REDO ? (long long)P.sp.head->redo_count[KV ? 1 : 0] : P.total_items;
  if (REDO && total_items == 0) return;
  auto fill_outputs = [&](float x, unsigned part, unsigned parts) {
    const long long n = KV ? (long long)P.total_k * p.nhead_k * p.headdim : (long long)P.total_q * p.nhead_q * p.headdim;
    for (long long i = (long long)part * kBwdThreads + tid; i < n; i += (long long)parts * kBwdThreads) {
      out0[i] = OutT(x);
      if (KV) out1[i] = OutT(x);
    }
  };
  const int status = *(volatile int32_t*)&P.ws.status[0];
  if (status == HBSA_STATUS_BLOCK_COUNT_MISMATCH) {       // zero gradients
    fill_outputs(0.f, block, blocks);
    return;
  }

  extern __shared__ __align__(1024) uint8_t smem[];   // 1024-byte aligned tiles for the 128-byte swizzle
  const uint32_t sStat = smem_u32(smem);              // [2 buffers][a, b]
  const uint32_t sStrm = sStat + 4 * STAT;            // [stages][x, y]
  BwdControl* const ctl = reinterpret_cast<BwdControl*>(smem + 4 * STAT + 2 * kBwdStages * STRM);
  volatile int* const abort_flag = &ctl->abort_flag;
  const long long budget = P.wait_budget;
  // Last thing every CTA does.  A launch that gave up (or found that the one before had) owes outputs: its last CTA, when all
  // others have written theirs, fills them with NaN, so that nobody takes them for gradients.
  auto leave = [&]() {
    if (tid == 0) {
      __threadfence();
      const bool last = atomicAdd(&P.sp.head->left[(KV ? 1 : 0) + (REDO ? 2 : 0)], 1u) == blocks - 1u;
      ctl->fill = last && *(volatile int32_t*)&P.ws.status[0] == HBSA_STATUS_WAIT_LIMIT;
    }
    __syncthreads();
    if (ctl->fill) fill_outputs(NAN, 0, 1);
  };
  if (__syncthreads_or(status != HBSA_STATUS_OK)) {      // (a CTA of the same launch may set it at any time)
    leave();
    return;
  }
  const uint32_t b_item_full = smem_u32(ctl->item_full), b_item_done = smem_u32(ctl->item_done);
  const uint32_t b_stat_full = smem_u32(ctl->stat_full), b_stat_free = smem_u32(ctl->stat_free);
  const uint32_t b_strm_full = smem_u32(ctl->strm_full), b_strm_free = smem_u32(ctl->strm_free);
  const uint32_t b_s_full = smem_u32(ctl->s_full), b_dp_full = smem_u32(ctl->dp_full);
  const uint32_t b_p_ready = smem_u32(ctl->p_ready), b_ds_ready = smem_u32(ctl->ds_ready);
  const uint32_t b_acc_full = smem_u32(&ctl->acc_full), b_acc_free = smem_u32(&ctl->acc_free);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(b_item_full + 8 * i, 1);
      mbar_init(b_item_done + 8 * i, kBwdEwWarps + 1);
      mbar_init(b_stat_full + 8 * i, 1);
      mbar_init(b_stat_free + 8 * i, 1);
      mbar_init(b_s_full + 8 * i, 1);
      mbar_init(b_dp_full + 8 * i, 1);
      mbar_init(b_p_ready + 8 * i, kBwdEwWarps / 2);
      mbar_init(b_ds_ready + 8 * i, kBwdEwWarps / 2);
      mbar_init(smem_u32(&ctl->top_ready[i]), kBwdEwWarps / 2);
    }
    for (int i = 0; i < kBwdStages; ++i) {
      mbar_init(b_strm_full + 8 * i, 1);
      mbar_init(b_strm_free + 8 * i, 1);
    }
    mbar_init(b_acc_full, 1);
    mbar_init(b_acc_free, kBwdEwWarps);
    mbar_init(smem_u32(&ctl->drain), 1);
    mbar_init(smem_u32(&ctl->ragged_full), 1);
    // the tiles need a 1024-byte aligned base; without static shared memory the dynamic part has one
    ctl->redo_mark = 0;
    ctl->abort_flag = (sStat & 1023u) != 0 ? 1 : 0;
    fence_barrier_init();
  }
  if (warp == kBwdMma) {
    tmem_alloc(smem_u32(&ctl->tmem_base), 512u);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;
  const int nt = P.nt;
  const uint32_t strm_panel = (uint32_t)nt * 128u;

  if (warp == kBwdProducer) {
    // =============================== work fetch, mask scan, TMA ===============================
    if (lane == 0) {
      prefetch_tensormap(&tm_a);
      prefetch_tensormap(&tm_b);
      prefetch_tensormap(&tm_x);
      prefetch_tensormap(&tm_y);
    }
    unsigned long long* const cursor = &P.sp.head->cursor[(KV ? 1 : 0) + (REDO ? 2 : 0)];
    int I = 0, Iq = 0, T = 0, stage = 0;
    uint32_t stage_par = 1u;                       // parity of "stage free" for the current round (first round: free)
    uint32_t ragged_par = 0u;                      // parity of the next tile with rows to clear
    bool ok = *abort_flag == 0 && P.debug_stall == 0;
    long long next_idx = 0;
    if (lane == 0) next_idx = (long long)atomicAdd(cursor, 1ull);
    next_idx = __shfl_sync(0xffffffffu, next_idx, 0);

    auto publish = [&](int n_tiles, int row0, int end, int head, int pos0, int k_len, int off, int first, long long index) {
      if (I >= 2) ok = warp_wait(bar_of(b_item_done, I), par_of(I - 2), abort_flag, budget);
      if (!ok) return;
      if (lane == 0) {
        volatile BwdItem* sl = &ctl->slot[I & 1];
        sl->n_tiles = n_tiles; sl->row0 = row0; sl->end = end; sl->head = head;
        sl->pos0 = pos0; sl->k_len = k_len; sl->off = off;
        sl->first = first; sl->index = index;
        __threadfence_block();
        mbar_arrive(bar_of(b_item_full, I));
      }
      ++I;
    };
    // stationary pair of the next item with tiles: rows (tokens) from row0, heads from head0
    auto load_stationary = [&](int row0, int head0) {
      if (Iq >= 2) ok = warp_wait(bar_of(b_stat_free, Iq), par_of(Iq - 2), abort_flag, budget);
      if (!ok) return;
      if (lane == 0) {
        const uint32_t bar = bar_of(b_stat_full, Iq), dst = sStat + (uint32_t)(Iq & 1) * 2u * STAT;
        mbar_arrive_expect_tx(bar, 2u * STAT);
#pragma unroll
        for (int pn = 0; pn < PANELS; ++pn) {
          tma_load_3d(dst + pn * 16384u, &tm_a, bar, pn * 64, head0, row0);
          tma_load_3d(dst + STAT + pn * 16384u, &tm_b, bar, pn * 64, head0, row0);
        }
      }
      ++Iq;
    };
    // one streamed tile; its first `valid` tokens (KV) or keys (dQ) are the block's.  KV: the {-lse, delta} pairs of the rows go along
    auto load_tile = [&](int row0, int head0, int valid, int i0, int i1) {
      float2 st0 = make_float2(-INFINITY, 0.f), st1 = st0;
      if (KV) {
        const int c1 = lane + 32, h = P.gp - 1;
        if ((lane >> P.gp_shift) < valid && lane < nt) st0 = P.sp.stats[(long long)(row0 + (lane >> P.gp_shift)) * p.nhead_q + head0 + (lane & h)];
        if ((c1 >> P.gp_shift) < valid && c1 < nt) st1 = P.sp.stats[(long long)(row0 + (c1 >> P.gp_shift)) * p.nhead_q + head0 + (c1 & h)];
      }
      // what the tile needs is settled before the wait: the loader is on the critical path behind it
      const int rows = KV ? min(valid << P.gp_shift, nt) : min(valid, nt);      // of the tile that are the block's
      unsigned long long gone = 0ull;
      bool late = false;                             // handed over only when rows have been cleared
      if (KV) {
        const uint32_t g0 = __ballot_sync(0xffffffffu, lane < nt && st0.x == -INFINITY);
        const uint32_t g1 = __ballot_sync(0xffffffffu, lane + 32 < nt && st1.x == -INFINITY);
        gone = (unsigned long long)g1 << 32 | g0;
        if (gone != 0ull) late = (rows & (P.piece - 1)) != 0 || gone != (first_bits(nt) & ~first_bits(rows));
      } else if (rows < nt) {
        gone = first_bits(nt) & ~first_bits(rows);
        late = (rows & (P.piece - 1)) != 0;
      }
      const uint32_t dst = sStrm + (uint32_t)stage * 2u * STRM;
      const uint32_t bar = late ? smem_u32(&ctl->ragged_full) : b_strm_full + 8u * stage;
      if (T >= kBwdStages) ok = warp_wait(b_strm_free + 8u * stage, stage_par, abort_flag, budget);
      if (!ok) return;
      if (KV) {
        ctl->neg_lse[stage][lane] = BF16 ? st0.x : st0.x + (float)kPShift;
        ctl->neg_lse[stage][lane + 32] = BF16 ? st1.x : st1.x + (float)kPShift;
        ctl->neg_delta[stage][lane] = -st0.y;
        ctl->neg_delta[stage][lane + 32] = -st1.y;
      }
      __syncwarp();
      if (lane == 0) {
        ctl->info0[stage] = i0;
        ctl->info1[stage] = i1;
        __threadfence_block();
        mbar_arrive_expect_tx(bar, 2u * (uint32_t)nt * D * 2u);
        if (gone == 0ull || late) {
#pragma unroll
          for (int pn = 0; pn < PANELS; ++pn) {
            tma_load_3d(dst + pn * strm_panel, &tm_x, bar, pn * 64, head0, row0);
            tma_load_3d(dst + STRM + pn * strm_panel, &tm_y, bar, pn * 64, head0, row0);
          }
        }
      }
      if (gone != 0ull && !late) {
        __syncwarp();
        const int which = lane & 1, pn = (lane >> 1) % PANELS, r = lane / (2 * PANELS) * P.piece;
        const int tok = r < rows ? row0 + (KV ? r >> P.gp_shift : r) : KV ? P.total_q : P.total_k;
        const uint32_t to = dst + pn * strm_panel + (uint32_t)r * 128u;
        if (r < nt && !which) tma_load_3d(to, &tm_xp, bar, pn * 64, head0, tok);
        if (r < nt && which) tma_load_3d(to + STRM, &tm_yp, bar, pn * 64, head0, tok);
      }
      if (late) {
        ok = warp_wait(bar, ragged_par, abort_flag, budget);
        if (!ok) {                                   // the copy is still in flight: bounded, like the others at the end
          mbar_wait_clock(bar, ragged_par, budget >> 4);
          return;
        }
        ragged_par ^= 1u;
        zero_rows<D>(dst, STRM, strm_panel, gone, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(b_strm_full + 8u * stage);
      }
      ++T;
      if (++stage == kBwdStages) {
        stage = 0;
        stage_par ^= 1u;
      }
    };

    while (ok) {
      long long idx = next_idx;
      if (idx >= total_items) {
        publish(-1, 0, 0, 0, 0, 0, 0, 0, 0);
        break;
      }
      if (REDO) idx = (KV ? P.sp.redo_k : P.sp.redo_q)[idx];
      if (lane == 0) next_idx = (long long)atomicAdd(cursor, 1ull);
      next_idx = __shfl_sync(0xffffffffu, next_idx, 0);
      if (KV) {
        // item = (kv-head, k-block, sub-tile); under a causal mask the first k-blocks of a sample have the most work
        const int msub = (int)(idx % P.n_msub);
        const long long r = idx / P.n_msub;
        const int kb = (int)(r % p.num_k_block), hk = (int)(r / p.num_k_block);
        const int b = sample_of_block(P.ws.cnk, p.batch, kb);
        const int k_begin = p.cu_k[b], k_len = p.cu_k[b + 1] - k_begin, q_begin = p.cu_q[b], q_len = p.cu_q[b + 1] - q_begin;
        const int off = k_len - q_len;
        const int blk0 = (kb - P.ws.cnk[b]) * p.kbs;
        const int k0 = blk0 + msub * P.m_rows, k_end = min(blk0 + p.kbs, k_len);
        if (k0 >= k_end) continue;
        const int qb0 = P.ws.cnq[b], nqb = P.ws.cnq[b + 1] - qb0;
        int i_min = 0;
        if (p.causal) {                             // first q-block whose last row reaches key k0
          const int need = k0 - off + 1 - p.qbs;    // (i + 1) * qbs - 1 + off >= k0
          i_min = need > 0 ? min((need + p.qbs - 1) / p.qbs, nqb - 1) : 0;
        }
        // tiles of q-block i: token sub-tiles [first, last) x head sub-tiles
        auto sub_range = [&](int i, int& first, int& last) {
          const int rows = min(p.qbs, q_len - i * p.qbs);
          last = (rows + P.tt - 1) / P.tt;
          first = 0;
          if (p.causal) {                           // a sub-tile counts when its last token reaches key k0
            const int t = k0 - off - i * p.qbs;     // first in-block token that does
            first = t <= 0 ? 0 : t >= rows ? last : t / P.tt;
          }
        };
        auto active = [&](int i) -> bool {
          if (i >= nqb) return false;
          if (p.csr_ptr != nullptr) {
            const long long row = (long long)hk * p.num_q_block + qb0 + i;
            const int e1 = p.csr_ptr[row + 1];
            const int e = lower_bound_i32(p.csr_idx, p.csr_ptr[row], e1, kb);
            return e < e1 && p.csr_idx[e] == kb;
          }
          return p.mask[hk * p.mask_s0 + (long long)(qb0 + i) * p.mask_s1 + (long long)kb * p.mask_s2] != 0;
        };
        int n_tiles = 0;
        for (int base = i_min; base < nqb; base += 32) {
          const int i = base + lane;
          int first, last;
          if (active(i)) {
            sub_range(i, first, last);
            n_tiles += (last - first) * P.n_head_sub;
          }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) n_tiles += __shfl_xor_sync(0xffffffffu, n_tiles, d);
        publish(n_tiles, k_begin + k0, min(P.m_rows, k_end - k0), hk, k0, k_len, off, q_begin, idx);
        if (!ok || n_tiles == 0) continue;
        load_stationary(k_begin + k0, hk);
        for (int base = i_min; base < nqb && ok; base += 32) {
          uint32_t bal = __ballot_sync(0xffffffffu, active(base + lane));
          while (bal != 0 && ok) {
            const int i = base + __ffs(bal) - 1;
            bal &= bal - 1;
            int first, last;
            sub_range(i, first, last);
            const int rows = min(p.qbs, q_len - i * p.qbs);
            for (int s = first; s < last && ok; ++s)
              for (int hs = 0; hs < P.n_head_sub && ok; ++hs) {
                const int t0 = s * P.tt;
                load_tile(q_begin + i * p.qbs + t0, hk * p.group + hs * P.gp, min(P.tt, rows - t0),
                          p.causal ? i * p.qbs + t0 + off : 0x7fffffff - 4096, 0);
              }
          }
        }
      } else {
        const ItemRecord rec = reinterpret_cast<const ItemRecord*>(P.ws.items)[idx / P.items_per_row];
        const int rem = (int)(idx % P.items_per_row);
        const int hsub = rem / P.tiles_per_qblock, qt = rem % P.tiles_per_qblock;
        const int tok0 = rec.q_begin + qt * P.tt, head0 = rec.hk * p.group + hsub * P.gp;
        if (tok0 >= rec.q_end) continue;
        publish(rec.n_tiles, tok0, rec.q_end, head0, rec.q_in0 + qt * P.tt, rec.k_len, rec.off, rec.k_begin, idx);
        if (!ok || rec.n_tiles <= 0) continue;
        load_stationary(tok0, head0);
        const bool csr = p.csr_ptr != nullptr;
        const int n_src = csr ? rec.count : rec.n_reach;
        const uint8_t* mrow = csr ? nullptr : p.mask + rec.hk * p.mask_s0 + rec.qb * p.mask_s1 + (long long)rec.kb0 * p.mask_s2;
        for (int base = 0; base < n_src && ok; base += 32) {
          const int jn = base + lane;
          int val = jn;
          bool on = jn < n_src;
          if (csr) val = on ? p.csr_idx[rec.csr_begin + jn] - rec.kb0 : 0;
          else on = on && mrow[(long long)jn * p.mask_s2] != 0;
          uint32_t bal = __ballot_sync(0xffffffffu, on);
          while (bal != 0 && ok) {
            const int pos = __ffs(bal) - 1;
            bal &= bal - 1;
            const int blk0 = __shfl_sync(0xffffffffu, val, pos) * p.kbs;
            const int blk_end = min(blk0 + p.kbs, rec.k_len), k_end = min(blk_end, rec.k_stop);
            for (int k0 = blk0; k0 < k_end && ok; k0 += nt) load_tile(rec.k_begin + k0, rec.hk, blk_end - k0, k0, k_end);
          }
        }
      }
    }
    if (!ok) {                                      // gave up: let the copies already issued land (bounded)
      for (int back = 1; back <= kBwdStages && T - back >= 0; ++back) {
        const int c = T - back;
        mbar_wait_clock(b_strm_full + 8u * (uint32_t)(c % kBwdStages), (uint32_t)(c / kBwdStages) & 1u, budget >> 4);
      }
      for (int back = 1; back <= 2 && Iq - back >= 0; ++back)
        mbar_wait_clock(bar_of(b_stat_full, Iq - back), par_of(Iq - back), budget >> 4);
    }
  } else if (warp == kBwdMma) {
    // =============================== MMA issuer ===============================
    if (lane == 0 && *abort_flag == 0) {
      const uint32_t idesc_s = make_idesc(BF16, false, false, 128, nt);
      const uint32_t idesc_acc = make_idesc(BF16, false, true, 128, D);
      const int ksteps = nt >> 4;
      const uint32_t desc_hi = smem_desc_hi(1024u);
      const uint32_t panel_units = strm_panel >> 4;
      bool ok = true, fin = false;
      int sI = 0, sIq = 0, sT = 0, s_left = 0, s_stage = 0;       // S side
      uint32_t s_par = 0u;
      bool s_first = false;
      int aT = 0, aIq = 0, a_stage = 0;                           // accumulator side
      int fl0 = 0, fl1 = 0;                                       // per tile in flight: bit 0 first, bit 1 last of its item

      // S and dP of the next tile; false when there is none (yet).  While a tile waits for its accumulator products nothing here
      // blocks: a later item may only be published once the epilogue of an earlier one, which needs those products, is done.
      auto there = [&](uint32_t bar, uint32_t par) -> bool {
        if (aT < sT) return mbar_test(bar, par);
        return ok = mbar_wait_bounded(bar, par, abort_flag, budget);
      };
      auto issue_s = [&]() -> bool {
        while (s_left == 0) {
          if (fin || !there(bar_of(b_item_full, sI), par_of(sI))) return false;
          const int n = *(volatile int*)&ctl->slot[sI & 1].n_tiles;
          mbar_arrive(bar_of(b_item_done, sI));
          ++sI;
          fin = n < 0;
          s_left = n < 0 ? 0 : n;
          s_first = true;
        }
        if (s_first && !there(bar_of(b_stat_full, sIq), par_of(sIq))) return false;
        if (!there(b_strm_full + 8u * s_stage, s_par)) return false;
#ifdef HBSA_STRICT_TCGEN05
        if (sT >= 2) {                              // the products that read P and dS of tile sT - 2 have completed
          const int c = sT - 2;
          if (!(ok = mbar_wait_bounded(b_strm_free + 8u * (uint32_t)(c % kBwdStages), (uint32_t)(c / kBwdStages) & 1u, abort_flag, budget))) return false;
        }
#endif
        tc_fence_after();
        const uint32_t stat = sStat + (uint32_t)(sIq & 1) * 2u * STAT, strm = sStrm + (uint32_t)s_stage * 2u * STRM;
        const uint32_t tS = tmem + (uint32_t)(sT & 1) * kBwdBuf;
#pragma unroll
        for (int half = 0; half < 2; ++half) {      // S = a x^T, then dP = b y^T
          const uint32_t la = smem_desc_lo(stat + half * STAT, 16u), lx = smem_desc_lo(strm + half * STRM, 16u);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint64_t da = smem_desc_join(la + (uint32_t)(ks >> 2) * 1024u + (uint32_t)(ks & 3) * 2u, desc_hi);
            const uint64_t dx = smem_desc_join(lx + (uint32_t)(ks >> 2) * panel_units + (uint32_t)(ks & 3) * 2u, desc_hi);
            if (ks == 0) mma_ss_c<false>(tS + half * 64u, da, dx, idesc_s);
            else mma_ss_c<true>(tS + half * 64u, da, dx, idesc_s);
          }
          tc_commit(half == 0 ? bar_of(b_s_full, sT) : bar_of(b_dp_full, sT));
        }
        const int fl = (s_first ? 1 : 0) | (s_left == 1 ? 2 : 0);
        if (sT & 1) fl1 = fl; else fl0 = fl;
        s_first = false;
        if (--s_left == 0) {
          tc_commit(bar_of(b_stat_free, sIq));      // the stationary pair is read by S and dP only
          ++sIq;
        }
        ++sT;
        if (++s_stage == kBwdStages) {
          s_stage = 0;
          s_par ^= 1u;
        }
        return true;
      };

      while (ok) {
        if (sT < aT + 2 && issue_s()) continue;
        if (aT == sT) {
          if (fin) break;
          continue;                                 // a wait gave up, or items without tiles went by
        }
        if (!ok) break;
        const int fl = (aT & 1) ? fl1 : fl0;
        const bool first = (fl & 1) != 0;
        const uint32_t tS = tmem + (uint32_t)(aT & 1) * kBwdBuf, strm = sStrm + (uint32_t)a_stage * 2u * STRM;
        const uint64_t dx = smem_desc_join(smem_desc_lo(strm, strm_panel), desc_hi);
        const uint64_t dy = smem_desc_join(smem_desc_lo(strm + STRM, strm_panel), desc_hi);
        // the first product of an item overwrites the accumulators: the previous epilogue must have read them
        if (first && aIq >= 1 && !(ok = mbar_wait_bounded(b_acc_free, (uint32_t)(aIq - 1) & 1u, abort_flag, budget))) break;
        if (KV) {
          if (!(ok = mbar_wait_bounded(bar_of(b_p_ready, aT), par_of(aT), abort_flag, budget))) break;
          tc_fence_after();
          issue_ts(tmem + kBwdAcc, tS, dy, ksteps, idesc_acc, first);
          issue_ts(tmem + kBwdAcc, tS + 32u, dy, ksteps, idesc_acc, false);
        }
        if (!(ok = mbar_wait_bounded(bar_of(b_ds_ready, aT), par_of(aT), abort_flag, budget))) break;
        tc_fence_after();
        const uint32_t acc = tmem + kBwdAcc + (KV ? (uint32_t)D : 0u);
        issue_ts(acc, tS + 64u, dx, ksteps, idesc_acc, first);
        issue_ts(acc, tS + 96u, dx, ksteps, idesc_acc, false);
        tc_commit(b_strm_free + 8u * a_stage);
        if (fl & 2) tc_commit(b_acc_full);
        if (first) ++aIq;
        ++aT;
        if (++a_stage == kBwdStages) a_stage = 0;
      }
      tc_commit(smem_u32(&ctl->drain));             // whatever was issued completes before tensor memory is given back
      mbar_wait_clock(smem_u32(&ctl->drain), 0u, budget);
    }
    __syncwarp();
  } else {
    // =============================== elementwise + epilogue ===============================
    const int wg = warp >> 2, row = tid & 127;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const float scale_log2 = P.scale_log2;
    const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);
    int I = 0, Iq = 0, T = 0, stage = 0;
    uint32_t stage_par = 0u;
    bool ok = *abort_flag == 0;
    while (ok) {
      ok = warp_wait(bar_of(b_item_full, I), par_of(I), abort_flag, budget);
      if (!ok) break;
      volatile BwdItem* sl = &ctl->slot[I & 1];
      const int n_tiles = sl->n_tiles;
      if (n_tiles < 0) break;
      const int row0 = sl->row0, end = sl->end, head = sl->head, pos0 = sl->pos0, k_len = sl->k_len, off = sl->off;
      // this thread's row of the stationary tile: a key (KV) or a (token, head) pair
      const int tok = KV ? row0 + row : row0 + (row >> P.gp_shift);
      const bool valid = KV ? row < end : tok < end;
      const int hq = KV ? 0 : head + (row & (P.gp - 1));
      const int key = pos0 + row;
      float neg_lse = -INFINITY, neg_delta = 0.f;
      bool no_keys = false;                        // dQ: the row's log-sum-exp says that it saw no key
      int limit_row = k_len - 1;
      if (!KV) {
        if (valid && n_tiles > 0) {
          const float2 st = P.sp.stats[(long long)tok * p.nhead_q + hq];
          neg_lse = st.x;
          neg_delta = -st.y;
          no_keys = neg_lse == -INFINITY;
        }
        if (p.causal) limit_row = min(limit_row, pos0 + (row >> P.gp_shift) + off);
      }
      // fp16: P is formed as 2^p_exp P (2^kPShift of it by the loader), dS as 2^ds_exp dS; the largest |P| and |dS| so scaled
      const long long kv_row = (long long)tok * p.nhead_k + head, q_row = (long long)tok * p.nhead_q + hq;
      int p_exp = 0, ds_exp = 0, seen = 0;             // dQ: keys that the row has seen
      float top_p = 0.f, top_ds = 0.f;
      uint64_t p_exp2 = 0ull, ds_mul2 = 0ull;
      if (!BF16) {
        p_exp = KV ? kPShift : 0;
        if (valid && n_tiles > 0) {
          ds_exp = KV ? ds_exponent(__uint_as_float(P.sp.max_do[(long long)sl->first * p.nhead_k + head]) *
                                    __uint_as_float(P.sp.max_v[(long long)(row0 - pos0) * p.nhead_k + head]))
                      : ds_exponent(P.sp.norm_do[q_row] * __uint_as_float(P.sp.max_v[(long long)sl->first * p.nhead_k + hq / p.group]));
          if (REDO) {
            const int top = KV ? P.sp.top_k[kv_row] : P.sp.top_q[q_row];
            if (KV) p_exp = min(p_exp + redo_exponent(top & 255), 110);
            ds_exp = max(min(ds_exp + redo_exponent(top >> 8), 120), -120);
          }
        }
        if (KV && REDO) p_exp2 = pack_f32x2((float)(p_exp - kPShift), (float)(p_exp - kPShift));
        ds_mul2 = pack_f32x2(pow2(ds_exp - p_exp), pow2(ds_exp - p_exp));
      }
      for (int t = 0; t < n_tiles && ok; ++t, ++T) {
        if ((T & 1) == wg) {
          ok = warp_wait(b_strm_full + 8u * stage, stage_par, abort_flag, budget) && warp_wait(bar_of(b_s_full, T), par_of(T), abort_flag, budget);
          if (!ok) break;
          tc_fence_after();
          const uint32_t tS = tmem + (uint32_t)(T & 1) * kBwdBuf + lane_off;
          uint32_t r[64], g[64];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (nt > 16 * j) tmem_ld16(tS + 16 * j, *reinterpret_cast<uint32_t(*)[16]>(&r[16 * j]));
          // columns this row may not see: below `lo_col` (KV: tokens before the key) or above `hi_col` (dQ: keys past the limit)
          int lo_col = 0, hi_col = 63;
          if (KV) {
            const int lim0 = *(volatile int*)&ctl->info0[stage];
            if (key > lim0) lo_col = min(key - lim0, 64) << P.gp_shift;
          } else {
            const int k0 = *(volatile int*)&ctl->info0[stage], k_end = *(volatile int*)&ctl->info1[stage];
            hi_col = min(limit_row, k_end - 1) - k0;
            if (!BF16 && !REDO) seen += max(min(hi_col + 1, 64), 0);
          }
          const bool edge = KV ? lo_col > 0 : hi_col < nt - 1;
          tmem_wait_ld();
          if (__any_sync(0xffffffffu, edge)) {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if (KV ? i < lo_col : i > hi_col) r[i] = 0xff800000u;     // -inf: its P is an exact zero
          }
          const float4* nl4 = reinterpret_cast<const float4*>(ctl->neg_lse[stage]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (nt > 16 * j) {
              uint32_t hi[8], lo[8];
#pragma unroll
              for (int i = 0; i < 16; i += 4) {
                const int c = 16 * j + i;
                float4 nl = make_float4(neg_lse, neg_lse, neg_lse, neg_lse);
                if (KV) nl = nl4[c >> 2];
                uint64_t nl01 = pack_f32x2(nl.x, nl.y), nl23 = pack_f32x2(nl.z, nl.w);
                if (KV && REDO) {
                  nl01 = add_f32x2(nl01, p_exp2);
                  nl23 = add_f32x2(nl23, p_exp2);
                }
                float x0, x1, x2, x3;
                unpack_f32x2(fma_f32x2(pack_b32x2(r[c], r[c + 1]), scale2, nl01), x0, x1);
                unpack_f32x2(fma_f32x2(pack_b32x2(r[c + 2], r[c + 3]), scale2, nl23), x2, x3);
                x0 = ex2_approx(x0); x1 = ex2_approx(x1); x2 = ex2_approx(x2); x3 = ex2_approx(x3);
                if (KV) {
                  if (!BF16 && !REDO) top_p = max3_abs(max3_abs(top_p, x0, x1), x2, x3);
                  split2<BF16>(x0, x1, hi[i >> 1], lo[i >> 1]);
                  split2<BF16>(x2, x3, hi[(i >> 1) + 1], lo[(i >> 1) + 1]);
                }
                r[c] = __float_as_uint(x0); r[c + 1] = __float_as_uint(x1);
                r[c + 2] = __float_as_uint(x2); r[c + 3] = __float_as_uint(x3);
              }
              if (KV) {
                tmem_st8(tS + 8 * j, hi);
                tmem_st8(tS + 32 + 8 * j, lo);
              }
            }
          }
          if (KV) {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_of(b_p_ready, T));
          }
          ok = warp_wait(bar_of(b_dp_full, T), par_of(T), abort_flag, budget);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (nt > 16 * j) tmem_ld16(tS + 64 + 16 * j, *reinterpret_cast<uint32_t(*)[16]>(&g[16 * j]));
          tmem_wait_ld();
          const float4* dl4 = reinterpret_cast<const float4*>(ctl->neg_delta[stage]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (nt > 16 * j) {
              uint32_t hi[8], lo[8];
#pragma unroll
              for (int i = 0; i < 16; i += 4) {
                const int c = 16 * j + i;
                float4 dl = make_float4(neg_delta, neg_delta, neg_delta, neg_delta);
                if (KV) dl = dl4[c >> 2];
                uint64_t d01 = pack_f32x2(dl.x, dl.y), d23 = pack_f32x2(dl.z, dl.w);
                d01 = mul_f32x2(pack_b32x2(r[c], r[c + 1]), add_f32x2(pack_b32x2(g[c], g[c + 1]), d01));
                d23 = mul_f32x2(pack_b32x2(r[c + 2], r[c + 3]), add_f32x2(pack_b32x2(g[c + 2], g[c + 3]), d23));
                if (!BF16) {
                  d01 = mul_f32x2(d01, ds_mul2);
                  d23 = mul_f32x2(d23, ds_mul2);
                }
                float x[4];
                unpack_f32x2(d01, x[0], x[1]);
                unpack_f32x2(d23, x[2], x[3]);
                if (!BF16 && !REDO) top_ds = max3_abs(max3_abs(top_ds, x[0], x[1]), x[2], x[3]);
                split2<BF16>(x[0], x[1], hi[i >> 1], lo[i >> 1]);
                split2<BF16>(x[2], x[3], hi[(i >> 1) + 1], lo[(i >> 1) + 1]);
              }
              tmem_st8(tS + 64 + 8 * j, hi);
              tmem_st8(tS + 96 + 8 * j, lo);
            }
          }
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_of(b_ds_ready, T));
        }
        if (++stage == kBwdStages) {
          stage = 0;
          stage_par ^= 1u;
        }
      }
      if (!ok) break;

      if (!BF16 && !REDO && n_tiles > 0) {
        // The rows' largest values, from both warpgroups; items with a row out of range go on the redo list (once).
        int tp = KV ? exponent_of(top_p) : min(seen, 127), ts = exponent_of(top_ds);
        if (wg == 1) {
          ctl->top[Iq & 1][row] = (uint16_t)(tp | ts << 8);
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_of(smem_u32(ctl->top_ready), Iq));
        } else {
          ok = warp_wait(bar_of(smem_u32(ctl->top_ready), Iq), par_of(Iq), abort_flag, budget);
          if (!ok) break;
          const int other = *(volatile uint16_t*)&ctl->top[Iq & 1][row];
          tp = KV ? max(tp, other & 255) : tp + (other & 255);
          ts = max(ts, other >> 8);
          if (valid) (KV ? P.sp.top_k[kv_row] : P.sp.top_q[q_row]) = (uint16_t)(tp | ts << 8);
          const int low = top_low(n_tiles);
          // (the dS of a row that sees a single key is what the rounding of two equal numbers leaves: small by right)
          const bool again = __any_sync(0xffffffffu, valid && (KV ? out_of_range(tp, low) || out_of_range(ts, low) : tp > 1 && out_of_range(ts, low)));
          if (again && lane == 0 && atomicMax(&ctl->redo_mark, Iq + 1) < Iq + 1)
            (KV ? P.sp.redo_k : P.sp.redo_q)[atomicAdd(&P.sp.head->redo_count[KV ? 1 : 0], 1ull)] = sl->index;
        }
      }

      // ---- epilogue: KV: warpgroup 0 writes dV, 1 writes dK; dQ: each writes half of the columns
      constexpr int NC = KV ? D : D / 2;
      const int c_base = KV ? 0 : wg * NC;
      OutT* const orow = KV ? (wg == 0 ? out0 : out1) + kv_row * p.headdim : out0 + q_row * p.headdim;
      const float mul = KV && wg == 0 ? (BF16 ? 1.f : pow2(-p_exp)) : (BF16 ? p.scale : p.scale * pow2(-ds_exp));
      if (n_tiles > 0) {
        ok = warp_wait(b_acc_full, (uint32_t)Iq & 1u, abort_flag, budget);
        if (!ok) break;
        tc_fence_after();
      }
      const uint32_t tA = tmem + kBwdAcc + (uint32_t)(wg * NC) + lane_off;
#pragma unroll
      for (int cb = 0; cb < NC; cb += 32) {
        uint32_t a[32];
        if (n_tiles > 0) {
          tmem_ld32(tA + cb, a);
          tmem_wait_ld();
          if (cb + 32 >= NC) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(b_acc_free);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) a[i] = 0u;
        }
        if (valid) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            if (c_base + cb + c < p.headdim) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e)
                w[e] = !KV && no_keys ? 0u : pack2<BF16>(__uint_as_float(a[c + 2 * e]) * mul, __uint_as_float(a[c + 2 * e + 1]) * mul);
              *reinterpret_cast<uint4*>(orow + c_base + cb + c) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
      if (n_tiles > 0) ++Iq;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_of(b_item_done, I));
      ++I;
    }
  }

  // ---- teardown: every thread gets here (all waits are bounded)
  tc_fence_before();
  __syncthreads();
  if (warp == kBwdMma) {
    tc_fence_after();
    tmem_dealloc(tmem, 512u);
  }
  if (tid == 0 && ctl->abort_flag) {
    atomicExch(&P.ws.status[0], HBSA_STATUS_WAIT_LIMIT);
    P.ws.status[3] = (int)block;
  }
  leave();
}

template <int D, bool BF16, bool KV>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_sm100_kernel(const __grid_constant__ BwdMaps m, const __grid_constant__ BwdParams P) {
  bwd_body<D, BF16, KV, false>(m.a, m.b, m.x, m.y, m.xp, m.yp, P, blockIdx.x, gridDim.x);
}
// Both redo lists in one launch (usually empty ones, so what counts is one launch less): the first half of the CTAs takes dQ's.
template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
bwd_redo_kernel(const __grid_constant__ BwdMaps q, const __grid_constant__ BwdMaps kv, const __grid_constant__ BwdParams Pq,
                const __grid_constant__ BwdParams Pkv) {
  const unsigned half = gridDim.x / 2;
  if (blockIdx.x < half) bwd_body<D, false, false, true>(q.a, q.b, q.x, q.y, q.xp, q.yp, Pq, blockIdx.x, half);
  else bwd_body<D, false, true, true>(kv.a, kv.b, kv.x, kv.y, kv.xp, kv.yp, Pkv, blockIdx.x - half, half);
}

// Raises one slot to the largest finite x it is given, with an atomic per run of the same slot; non-negative floats order like their bits.
struct MaxRun {
  unsigned int* slot = nullptr;
  float top = 0.f;
  __device__ __forceinline__ void flush() const {
    if (slot != nullptr && top > 0.f) atomicMax(slot, __float_as_uint(top));
  }
  __device__ __forceinline__ void take(unsigned int* s, float x) {
    if (s != slot) {
      flush();
      slot = s;
      top = 0.f;
    }
    if (x < INFINITY) top = fmaxf(top, x);
  }
};
// First token of the sample that holds token `tok`; [lo, hi) is the sample found last.
__device__ __forceinline__ int first_token(const int32_t* __restrict__ cu, int batch, int tok, int& lo, int& hi) {
  if (tok < lo || tok >= hi) {
    const int b = sample_of_block(cu, batch, tok);
    lo = cu[b];
    hi = cu[b + 1];
  }
  return lo;
}

// {-lse * log2 e, delta = rowsum(dO * O)} of every (token, q-head) row; with fp16 also the norms of the rows of dO, and the
// maxima of those of dO and V over every sample and kv-head (rows that see no key and rows with Inf or NaN left out).  16 lanes per row, 16 bytes per lane; bound by the read of O and dO.
// Rows of q / k outside every sample get zero gradients here.
template <bool BF16>
__global__ void __launch_bounds__(256) bwd_prep_kernel(BwdParams P, const uint16_t* __restrict__ o, long long o0, long long o1,
                                                       const uint16_t* __restrict__ d_o, long long g0, long long g1,
                                                       const uint16_t* __restrict__ v, long long v0, long long v1,
                                                       const float* __restrict__ lse, uint16_t* dq, uint16_t* dk, uint16_t* dv) {
  const Problem& p = P.p;
  const int chunk = threadIdx.x & 15, n_chunk = p.headdim >> 3;
  const long long step = (long long)gridDim.x * 16;
  const long long rows = (long long)P.total_q * p.nhead_q, k_rows = (long long)P.total_k * p.nhead_k;
  const int q_lo = p.cu_q[0], q_hi = p.cu_q[p.batch], k_lo = p.cu_k[0], k_hi = p.cu_k[p.batch];
  MaxRun run;
  int lo = 0, hi = 0;
  // uniform per block: the shuffles need whole warps
  for (long long base = (long long)blockIdx.x * 16; base < rows; base += step) {
    const long long row = base + (threadIdx.x >> 4);
    float acc = 0.f, sq = 0.f;
    const long long tok = row / p.nhead_q, h = row % p.nhead_q;
    if (row < rows && chunk < n_chunk) {
      const uint4 a = *reinterpret_cast<const uint4*>(o + tok * o0 + h * o1 + chunk * 8);
      const uint4 b = *reinterpret_cast<const uint4*>(d_o + tok * g0 + h * g1 + chunk * 8);
      const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float x0, x1, y0, y1;
        unpack16<BF16>(wa[i], x0, x1);
        unpack16<BF16>(wb[i], y0, y1);
        acc = fmaf(x0, y0, fmaf(x1, y1, acc));
        if (!BF16) sq = fmaf(y0, y0, fmaf(y1, y1, sq));
      }
    }
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) {
      acc += __shfl_xor_sync(0xffffffffu, acc, s);
      if (!BF16) sq += __shfl_xor_sync(0xffffffffu, sq, s);
    }
    if (row < rows) {
      const bool outside = tok < q_lo || tok >= q_hi;
      if (chunk == 0) {
        const float l = lse[row];
        const bool live = fabsf(l) < INFINITY;
        P.sp.stats[row] = live ? make_float2(-l * kLog2e, acc) : make_float2(-INFINITY, 0.f);
        if (!BF16) {
          const float norm = sqrtf(sq);
          P.sp.norm_do[row] = norm;
          if (!outside && live) run.take(P.sp.max_do + (long long)first_token(p.cu_q, p.batch, (int)tok, lo, hi) * p.nhead_k + h / p.group, norm);
        }
      }
      if (outside && chunk < n_chunk) *reinterpret_cast<uint4*>(dq + row * p.headdim + chunk * 8) = make_uint4(0, 0, 0, 0);
    }
  }
  lo = hi = 0;
  for (long long base = (long long)blockIdx.x * 16; base < k_rows; base += step) {
    const long long row = base + (threadIdx.x >> 4);
    const long long tok = row / p.nhead_k, h = row % p.nhead_k;
    const bool outside = tok < k_lo || tok >= k_hi;
    if (row < k_rows && chunk < n_chunk && outside) {
      *reinterpret_cast<uint4*>(dk + row * p.headdim + chunk * 8) = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(dv + row * p.headdim + chunk * 8) = make_uint4(0, 0, 0, 0);
    }
    if (!BF16) {
      float sq = 0.f;
      if (row < k_rows && chunk < n_chunk) {
        const uint4 a = *reinterpret_cast<const uint4*>(v + tok * v0 + h * v1 + chunk * 8);
        const uint32_t wa[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float x0, x1;
          unpack16<BF16>(wa[i], x0, x1);
          sq = fmaf(x0, x0, fmaf(x1, x1, sq));
        }
      }
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, s);
      if (row < k_rows && chunk == 0) {
        if (!outside) run.take(P.sp.max_v + (long long)first_token(p.cu_k, p.batch, (int)tok, lo, hi) * p.nhead_k + h, sqrtf(sq));
      }
    }
  }
  if (!BF16) run.flush();
}

// q-heads packed into a tile of at most `rows` rows: the largest power of two that divides the group
int pack_heads(int group, int rows) {
  int gp = 1;
  while (gp < rows && group % (gp * 2) == 0) gp *= 2;
  return gp;
}
int log2_of(int x) {
  int s = 0;
  while ((1 << s) < x) ++s;
  return s;
}
// rows of a streamed tile: `rows` split evenly into the fewest tiles of at most 64, rounded up to 16
int even_tile(int rows) {
  const int n = (rows + kBwdTile - 1) / kBwdTile;
  return ((rows + n - 1) / n + 15) / 16 * 16;
}

template <int D> constexpr size_t bwd_smem() { return 4u * 128u * D * 2u + 2u * kBwdStages * kBwdTile * D * 2u + sizeof(BwdControl); }
static_assert(bwd_smem<128>() <= 227u * 1024u, "shared memory of one CTA");

template <int D, bool BF16, bool KV>
cudaError_t launch_one(const BwdMaps& m, const BwdParams& P, cudaStream_t stream) {
  static SmemOptIn opt_in;
  cudaError_t e = opt_in.once(reinterpret_cast<const void*>(bwd_sm100_kernel<D, BF16, KV>), (int)bwd_smem<D>());
  if (e != cudaSuccess) return e;
  const long long resident = sm100_sm_count();
  const unsigned grid = (unsigned)(P.total_items < resident ? P.total_items : resident);
  bwd_sm100_kernel<D, BF16, KV><<<grid, kBwdThreads, bwd_smem<D>(), stream>>>(m, P);
  return cudaGetLastError();
}
template <int D>
cudaError_t launch_redo(const BwdMaps (&m)[2], const BwdParams (&P)[2], cudaStream_t stream) {
  static SmemOptIn opt_in;
  cudaError_t e = opt_in.once(reinterpret_cast<const void*>(bwd_redo_kernel<D>), (int)bwd_smem<D>());
  if (e != cudaSuccess) return e;
  bwd_redo_kernel<D><<<2 * sm100_sm_count(), kBwdThreads, bwd_smem<D>(), stream>>>(m[0], m[1], P[0], P[1]);
  return cudaGetLastError();
}

}  // namespace

size_t backward_sm100_workspace_bytes(long long total_q, long long total_k, int nhead_q, int nhead_k) {
  BwdSpace s;
  size_t zeroed;
  return carve_space(nullptr, total_q, total_k, nhead_q, nhead_k, &s, &zeroed);
}

const char* backward_sm100_ineligible_reason(const hbsa_backward_args& b, float scale) {
  const char* why = sm100_ineligible_reason(b.fwd, scale);
  if (why) return why;
  if (b.fwd.headdim > 128) return "headdim is above 128";
  if (b.do_stride[2] != 1) return "headdim stride of d_o is not 1";
  for (int i = 0; i < 2; ++i)
    if (b.do_stride[i] <= 0 || (b.do_stride[i] * 2) % 16 != 0) return "a token/head stride of d_o is not a positive multiple of 16 bytes";
  if ((uintptr_t)b.d_o % 16 != 0 || (uintptr_t)b.dq % 16 != 0 || (uintptr_t)b.dk % 16 != 0 || (uintptr_t)b.dv % 16 != 0)
    return "a gradient's base address is not 16-byte aligned";
  return nullptr;
}

int backward_sm100_kv_tile_rows(int kbs) { return even_tile(kbs); }

int launch_backward_sm100(const Problem& p, const Workspace& ws, const hbsa_backward_args& b, cudaStream_t stream, const char** err_text) {
  const hbsa_forward_args& a = b.fwd;
  EncodeTiledFn fn = sm100_encode_fn();
  if (!fn) { *err_text = "cuTensorMapEncodeTiled is not available from the CUDA driver"; return HBSA_ERR_DRIVER; }
  const bool bf16 = a.dtype == HBSA_DTYPE_BF16;
  BwdParams both[2] = {};                          // dQ, dK/dV
  BwdMaps maps[2];
  BwdParams& P = both[0];
  P.p = p;
  P.ws = ws;
  size_t zeroed;
  carve_space(static_cast<char*>(b.grad_workspace), a.total_q, a.total_k, a.nhead_q, a.nhead_k, &P.sp, &zeroed);
  P.total_q = a.total_q;
  P.total_k = a.total_k;
  P.scale_log2 = p.scale * kLog2e;
  P.wait_budget = sm100_wait_budget();
  P.debug_stall = sm100_debug_stall();
  cudaError_t e = cudaMemsetAsync(P.sp.head, 0, bf16 ? sizeof(BwdHeader) : zeroed, stream);
  if (e != cudaSuccess) { *err_text = cudaGetErrorString(e); return (int)e; }
  {
    const long long rows = (long long)a.total_q * a.nhead_q;
    const long long blocks = (rows + 15) / 16, most = 16ll * sm100_sm_count();
    const unsigned grid = (unsigned)(blocks < most ? blocks : most);
    const uint16_t *o = static_cast<const uint16_t*>(a.o), *d_o = static_cast<const uint16_t*>(b.d_o), *v = static_cast<const uint16_t*>(a.v);
    uint16_t *dq = static_cast<uint16_t*>(b.dq), *dk = static_cast<uint16_t*>(b.dk), *dv = static_cast<uint16_t*>(b.dv);
    if (bf16) bwd_prep_kernel<true><<<grid, 256, 0, stream>>>(P, o, a.o_stride[0], a.o_stride[1], d_o, b.do_stride[0], b.do_stride[1], v, a.v_stride[0], a.v_stride[1], a.lse, dq, dk, dv);
    else bwd_prep_kernel<false><<<grid, 256, 0, stream>>>(P, o, a.o_stride[0], a.o_stride[1], d_o, b.do_stride[0], b.do_stride[1], v, a.v_stride[0], a.v_stride[1], a.lse, dq, dk, dv);
    if ((e = cudaGetLastError()) != cudaSuccess) { *err_text = cudaGetErrorString(e); return (int)e; }
  }
  both[1] = both[0];
  for (int kv = 0; kv < 2; ++kv) {
    BwdParams& P = both[kv];
    if (kv) {
      P.gp = pack_heads(p.group, kBwdTile);
      P.tt = even_tile(p.qbs * P.gp) / P.gp;        // tokens x heads of a q-block, split evenly
      P.nt = P.tt * P.gp;
      P.n_msub = (p.kbs + 127) / 128;
      P.m_rows = ((p.kbs + P.n_msub - 1) / P.n_msub + 15) / 16 * 16;
      P.total_items = (long long)p.nhead_k * p.num_k_block * P.n_msub;
      P.out0 = b.dv;
      P.out1 = b.dk;
    } else {
      P.gp = pack_heads(p.group, 128);
      P.tt = 128 / P.gp;
      P.nt = p.kv_tile;
      P.tiles_per_qblock = (p.qbs + P.tt - 1) / P.tt;
      P.items_per_row = p.group / P.gp * P.tiles_per_qblock;
      P.total_items = (long long)p.nhead_k * p.num_q_block * P.items_per_row;
      P.out0 = b.dq;
      P.out1 = nullptr;
    }
    P.gp_shift = log2_of(P.gp);
    P.n_head_sub = p.group / P.gp;
    P.piece = kv && P.gp > 16 ? P.gp : 16;
    CUtensorMap q, g, k, v, xp, yp;
    const int qh = P.gp, qt = P.tt, kt = kv ? 128 : P.nt;
    const int pieces_ok = kv ? sm100_encode_map(fn, &xp, bf16, a.q, p.headdim, p.nhead_q, a.total_q, a.q_stride[0], a.q_stride[1], qh, P.piece / qh) &&
                               sm100_encode_map(fn, &yp, bf16, b.d_o, p.headdim, p.nhead_q, a.total_q, b.do_stride[0], b.do_stride[1], qh, P.piece / qh)
                             : sm100_encode_map(fn, &xp, bf16, a.k, p.headdim, p.nhead_k, a.total_k, a.k_stride[0], a.k_stride[1], 1, P.piece) &&
                               sm100_encode_map(fn, &yp, bf16, a.v, p.headdim, p.nhead_k, a.total_k, a.v_stride[0], a.v_stride[1], 1, P.piece);
    if (!pieces_ok || !sm100_encode_map(fn, &q, bf16, a.q, p.headdim, p.nhead_q, a.total_q, a.q_stride[0], a.q_stride[1], qh, qt) ||
        !sm100_encode_map(fn, &g, bf16, b.d_o, p.headdim, p.nhead_q, a.total_q, b.do_stride[0], b.do_stride[1], qh, qt) ||
        !sm100_encode_map(fn, &k, bf16, a.k, p.headdim, p.nhead_k, a.total_k, a.k_stride[0], a.k_stride[1], 1, kt) ||
        !sm100_encode_map(fn, &v, bf16, a.v, p.headdim, p.nhead_k, a.total_k, a.v_stride[0], a.v_stride[1], 1, kt)) {
      *err_text = "cuTensorMapEncodeTiled rejected a q/k/v/d_o layout";
      return HBSA_ERR_UNSUPPORTED;
    }
    maps[kv] = kv ? BwdMaps{k, v, q, g, xp, yp} : BwdMaps{q, g, k, v, xp, yp};
#define HBSA_LAUNCH_BWD(D_, BF_) (kv ? launch_one<D_, BF_, true>(maps[1], P, stream) : launch_one<D_, BF_, false>(maps[0], P, stream))
    if (p.headdim <= 64) e = bf16 ? HBSA_LAUNCH_BWD(64, true) : HBSA_LAUNCH_BWD(64, false);
    else e = bf16 ? HBSA_LAUNCH_BWD(128, true) : HBSA_LAUNCH_BWD(128, false);
#undef HBSA_LAUNCH_BWD
    if (e != cudaSuccess) { *err_text = cudaGetErrorString(e); return (int)e; }
  }
  if (!bf16) {
    e = p.headdim <= 64 ? launch_redo<64>(maps, both, stream) : launch_redo<128>(maps, both, stream);
    if (e != cudaSuccess) { *err_text = cudaGetErrorString(e); return (int)e; }
  }
  return 0;
}

}  // namespace hbsa
