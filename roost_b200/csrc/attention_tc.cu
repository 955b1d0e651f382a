// Causal grouped-query attention over the paged cache for prompt portions (rows with more than 16 packed rows), on the
// fifth-generation tensor cores: both products are tcgen05.mma with the accumulators in tensor memory, and the softmax
// weights go from registers to tensor memory, where the second product reads them as its first operand.
//
// Definition and numerics as in attention_mma.cu (src/Starlings.Roost.Ops/CpuOps.cs:181-298; 32-bit scores, maxima,
// exponentials, sums and output accumulation; the softmax weights rounded to bfloat16 as the operand of the second
// product, kernels/README.md:234-236). A CTA owns one or two groups of 128 packed rows (token r / G, head r % G) of one
// request and one key/value head and walks the keys in tiles of 128 at fixed absolute positions, so a row's bits do not
// depend on how the prompt was cut or on what else is in the batch.
//   warp 0 (producer): one 5-D tensor copy per row group brings its Q tile [128 rows x D] into 128-byte-swizzled shared
//     memory; per key tile it looks the pages up and its lanes issue the copies side by side: per page one copy per
//     64-column block of the keys, placed so that the tile's 128 key rows are consecutive in each block (one product then
//     takes them all), and one copy of the values. Keys and values have rings of their own: a tile's keys are free again
//     as soon as its scores are computed, its values only after the second product a tile later.
//   warp 1 (issuer, one lane): per key tile and row group, O += P V of the tile before (one product per 16 keys:
//     M 128, N = D, K 16, with P in tensor memory and V as the N-major operand exactly as the copy left it) and
//     S = Q K^T of this tile (M 128, N 128, K = D) into score columns of the group. With two row groups each has one set
//     of score columns and the products of one group run while the other group's softmax does; a CTA with one row group
//     has two sets and computes the scores of a tile while the softmax of the tile before runs.
//   warps 2.. (softmax, one thread a row, four warps a row group): read the row's 128 scores from tensor memory, scale,
//     mask by position, keep the running maximum and sum, write the weights as bfloat16 pairs over the scores they came
//     from, and at the end divide the accumulator by the sum and write the row out. The maximum a row's weights are taken
//     against moves only when the new maximum exceeds it by more than 2^8 (the weights then stay below 2^8, well inside
//     bfloat16's and float32's range, and the quotient at the end is the same): the row of the output accumulator is
//     rescaled in tensor memory only then.
// Wide weights (WIDE): a row's weights enter the second product as two bfloat16 operands, their rounding and what it left over, so that 16 bits
// of the 32-bit weights count: the second operands lie over the other half of the scores' columns, and every product with V is made twice. Rows of 1,500, 500 and 2,048 tokens, 16
// heads of 128 over 4, with a sink: 64 us, 243 with the mma.sync kernel that served wide weights before.
// Keys and values that are not paged (FLAT): entry r * stride + j is row r's token at position j of a dense tensor with the heads side by side, a
// key/value head a query head, keys wider than values by a part that all heads share (a tensor of its own, as the queries' last numbers are):
// what prompt portions of a latent attention carry out of their cache (rows of 2,048 and 1,000 tokens, 16 heads of 128 + 64 over a latent of 512:
// 69 us, with the gather and the two products before it 98; 1,204 in the latent space on mma.sync). The work items follow from q_indptr, the last tiles of a row first.
// Sigmoid weights (SIGMOID): a key's weight is the sigmoid of its score, less a slope a head times its distance, plus a bias a head; nothing divides
// by the weights' sum, so there is no running maximum and the accumulator is never rescaled; the output is multiplied by the sigmoid of a gate
// where there is one. Work items as for FLAT. A tile's chain bounds it (product, weights, product; an exponential and a reciprocal for each of 41 M
// weights would be 18 us of special-function time). Rows of 2,048 and 777 tokens, 16 heads of 64 over 4: 67 us, 125 + 48 on mma.sync with a second kernel that adds
// the sums of a long row's chunks.
// Value rows at positions the request does not hold yet (the rest of its last page) or before the CTA's first visible key
// are zeroed in shared memory before the second product, so that whatever the pool holds there cannot reach a result;
// their scores are masked by position. Every wait is bounded (see tma.cuh): a wait given up raises the CTA's abort flag
// and records a code that roost_attention_status() returns.
#include "tcgen05.cuh"

#include <initializer_list>

namespace roost {

constexpr float kLog2eTc = 1.4426950408889634f;
constexpr int kTcRows = 128;   // packed rows of a row group
constexpr int kTcKeys = 128;   // keys of a tile
constexpr float kTcLazyRescale = 8.0f;   // a row's reference maximum moves when the new one exceeds it by more than this (log2 units)
__device__ int g_attention_tc_error = 0;

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3, int c4) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];\n" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
               : "memory");
}

// 2^x in one special-function instruction (inputs here are at most 8 or -inf; results below 2^-126 flush to zero)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

template <int DK, int DV, int NG>
struct TcCfg {
  // what fits beside NG Q tiles in 227 KB: a key tile is 128 x DK x 2 bytes, a value tile 128 x DV x 2
  static constexpr int kKStages = DK == 192 ? 2 : DK == 128 ? (NG == 1 ? 3 : 2) : 3;
  static constexpr int kVStages = DV == 128 ? 2 : 3;
  static constexpr uint32_t kKTile = kTcKeys * DK * 2, kVTile = kTcKeys * DV * 2;
  static constexpr size_t kSmem = (size_t)NG * kTcRows * DK * 2 + (size_t)kKStages * kKTile + (size_t)kVStages * kVTile + 1024;
  static_assert(kSmem <= 227 * 1024, "shared memory of a CTA");
};

// What a FLAT launch has instead of pages: entries a row, batch rows, 64-column blocks of a head's own key part, k steps of a score.
struct TcFlat {
  int stride, rows, own_blocks, k_steps;
};

// What a SIGMOID launch has beside it: a slope and a bias a query head, the gate's rows (null: none), ld apart; the key tiles of a chunk, how many
// chunks a row of keys has at most (the last one takes what is left) and, with more than one, the chunks' sums [token][head][chunk][DV].
struct TcSigmoid {
  const float *slopes, *bias;
  const __nv_bfloat16* gate;
  int64_t ld_gate;
  int chunk_tiles, chunks;
  float* sums;
};

// The pairs of a launch that has no work list, found from the rows' lengths: rows in order, of a row chunk after chunk, of a chunk the items that
// see any of its keys, the last first, of an item the key/value heads. Pair `wi` as (batch row, first packed row, key/value head, chunk), row -1 beyond
// the last pair, and its row as (first token, tokens, position of the first). By a whole warp, a lane a row: with the walk over all rows in every
// thread the search grew with the square of a step's rows.
struct TcPair {
  int4 at;
  int q_start, n, pos0;
};
__device__ __forceinline__ TcPair tc_find_pair(int wi, const int32_t* q_indptr, const int32_t* kv_lens, int rows, int group, int kv_heads, int item_rows, int chunk_keys,
                                               int chunks) {
  const int lane = threadIdx.x & 31, item_tokens = item_rows / group;
  int item = wi / kv_heads;
  auto items_of = [&](int n, int pos0, int z) {       // a row's items whose last token sees keys of chunk z: the last ones
    const int tiles = (n + item_tokens - 1) / item_tokens, before = z * chunk_keys - pos0;
    return before <= 0 ? tiles : (before >= n ? 0 : tiles - before / item_tokens);
  };
  for (int r0 = 0; r0 < rows; r0 += 32) {
    const int r = r0 + lane;
    int n = 0, pos0 = 0, mine = 0, start = 0;
    if (r < rows) {
      start = q_indptr[r];
      n = q_indptr[r + 1] - start;
      pos0 = kv_lens[r] - n;
      if (pos0 >= 0)                                  // a padding row holds no keys
        for (int z = 0; z < chunks; ++z) mine += items_of(n, pos0, z);
    }
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int left = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += left;
    }
    const unsigned past = __ballot_sync(0xffffffffu, upto > item);
    if (past == 0) {
      item -= __shfl_sync(0xffffffffu, upto, 31);
      continue;
    }
    const int src = __ffs(past) - 1;
    item -= __shfl_sync(0xffffffffu, upto - mine, src);
    n = __shfl_sync(0xffffffffu, n, src);
    pos0 = __shfl_sync(0xffffffffu, pos0, src);
    start = __shfl_sync(0xffffffffu, start, src);
    int z = 0;
    for (int count = items_of(n, pos0, 0); item >= count; count = items_of(n, pos0, ++z)) item -= count;
    return {make_int4(r0 + src, ((n + item_tokens - 1) / item_tokens - 1 - item) * item_rows, wi % kv_heads, z), start, n, pos0};
  }
  return {make_int4(-1, 0, 0, 0), 0, 0, 0};
}
constexpr int kTcRounds = 32;      // pairs that a CTA of such a launch walks at most

// 1 / (1 + 2^x)
__device__ __forceinline__ float sigmoid_of_ex2(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(1.0f + ex2(x)));
  return y;
}

// work[i] = (batch row, first packed row of the item's NG x 128 rows); an item is run once for every key/value head.
// The grid is persistent: CTA c takes the (item, head) pairs c, c + gridDim.x, ... of the list, which the host has sorted
// longest first (FLAT and SIGMOID: the pairs of tc_find_pair, in its order). Tensor memory and the barriers are set up once; the rings of keys and values, the score columns and the
// barriers' phases run on from one pair to the next, so the copies of the next pair start while the last tiles of this
// one are still being computed.
template <int DK, int DV, int RPC, int NG, bool WIDE, bool FLAT, bool SIGMOID>
__global__ void __launch_bounds__(64 + NG * 128, 1)
    attention_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_q2,
                                const __grid_constant__ CUtensorMap map_k2, TcFlat flat, TcSigmoid sg, __nv_bfloat16* __restrict__ out, const int32_t* __restrict__ q_indptr,
                                const int32_t* __restrict__ kv_lens, const int32_t* __restrict__ kv_indptr,
                                const int32_t* __restrict__ kv_indices, const int2* __restrict__ work, int items, int q_heads, int kv_heads,
                                int page_size, float scale_log2, int window, const float* __restrict__ sinks) {
  const float sink = (window & ROOST_ATTENTION_SINK) ? 1.0f : 0.f;     // one more term, 2^(0 - m) or 2^(a head's stored number - m), in every row's denominator
  window &= ~(ROOST_ATTENTION_SINK | ROOST_ATTENTION_WIDE_WEIGHTS);
  using Cfg = TcCfg<DK, DV, NG>;
  constexpr int BM = kTcRows, TK = kTcKeys, KS = Cfg::kKStages, VS = Cfg::kVStages, NP = TK / RPC, CB = DK / 64;
  constexpr uint32_t kQBytes = BM * DK * 2;                 // one row group's Q tile
  constexpr uint32_t kKTile = Cfg::kKTile, kVTile = Cfg::kVTile;      // keys, and values, of TK positions
  constexpr uint32_t kVPage = (DV / 64) * RPC * 128;        // the values page copy by page copy: [column block][RPC rows][128 B]
  constexpr int kOps = NP * (CB + 1);                       // copies a tile takes: per page one per column block of keys, one of values
  static_assert(kOps <= 32, "one lane a copy");
  constexpr int SB = NG == 1 ? 2 : 1;                       // sets of score columns a row group has
  constexpr uint32_t kGroupCols = SB * TK + DV;             // tensor-memory columns of a row group: the scores (the weights over them) and the output
  constexpr uint32_t kTmemCols = NG * kGroupCols <= 256 ? 256 : 512;
  static_assert(NG * kGroupCols <= 512, "tensor memory has 512 columns");
  constexpr int kGroupBars = 2 * SB + 1;                    // s_full[SB], p_full[SB], o_done
  constexpr int kGroupThreads = 128;                        // one thread a row
  extern __shared__ unsigned char smem_raw[];
  const uint32_t smem_base = ((uint32_t)__cvta_generic_to_shared(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem_base;
  const uint32_t k_smem = q_smem + NG * kQBytes;
  const uint32_t v_smem = k_smem + KS * kKTile;
  __shared__ __align__(8) uint64_t bars[2 + 2 * KS + 2 * VS + NG * kGroupBars];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  constexpr bool FOUND = FLAT || SIGMOID;
  __shared__ TcPair found[FOUND ? kTcRounds : 1];
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars);
  const uint32_t q_full = bar0, q_empty = bar0 + 8u;
  auto k_full = [&](int s) { return bar0 + 8u * (2 + s); };
  auto k_empty = [&](int s) { return bar0 + 8u * (2 + KS + s); };
  auto v_full = [&](int s) { return bar0 + 8u * (2 + 2 * KS + s); };
  auto v_empty = [&](int s) { return bar0 + 8u * (2 + 2 * KS + VS + s); };
  auto s_full = [&](int g, int sb) { return bar0 + 8u * (2 + 2 * KS + 2 * VS + g * kGroupBars + sb); };
  auto p_full = [&](int g, int sb) { return bar0 + 8u * (2 + 2 * KS + 2 * VS + g * kGroupBars + SB + sb); };
  auto o_done = [&](int g) { return bar0 + 8u * (2 + 2 * KS + 2 * VS + g * kGroupBars + 2 * SB); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    abort_flag = 0;
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);        // the issuer hands the Q tiles back once the pair's last scores are computed
    for (int s = 0; s < KS; ++s) {
      mbar_init(k_full(s), 1);
      mbar_init(k_empty(s), 1);   // the issuer hands the keys back once every group's scores of the tile are computed
    }
    for (int s = 0; s < VS; ++s) {
      mbar_init(v_full(s), 1);
      mbar_init(v_empty(s), NG);  // every row group hands the values back (or the issuer does for a group that skips the tile)
    }
    for (int g = 0; g < NG; ++g) {
      for (int sb = 0; sb < SB; ++sb) {
        mbar_init(s_full(g, sb), 1);
        mbar_init(p_full(g, sb), 4);
      }
      mbar_init(o_done(g), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const int group = q_heads / kv_heads;
  const int total = items * kv_heads;
  // The pairs are sorted longest first (a work list's). CTA c takes, in round r, pair r G + c when r is even and r G + (G - 1 - c) when it
  // is odd: the CTA that got the longest pair of one round gets the shortest of the next, so every CTA walks about the
  // same number of tiles. (The last round may leave a CTA without a pair while a later one of the same round has one:
  // the walk then ends for it a round early, which costs it nothing.)
  auto pair_of = [&](int round) { return round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x); };
  if (FOUND) {      // the step's tables were there before its first kernel
    for (int round = warp; round < kTcRounds && pair_of(round) < total; round += 2 + 4 * NG) {
      const TcPair p = tc_find_pair(pair_of(round), q_indptr, kv_lens, flat.rows, group, kv_heads, NG * BM, sg.chunk_tiles * TK, sg.chunks);
      if (lane == 0) found[round] = p;
    }
  }
  pdl_launch_dependents();
  pdl_wait();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"((uint32_t)__cvta_generic_to_shared(&tmem_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_slot;
  auto tmem_s = [&](int g, int sb) { return tmem_base + (uint32_t)g * kGroupCols + (uint32_t)sb * TK; };   // the scores; the weights go over them
  auto tmem_o = [&](int g) { return tmem_base + (uint32_t)g * kGroupCols + SB * TK; };
  volatile int* abortp = &abort_flag;
  // What every thread derives of an (item, head) pair.
  struct Pair {
    int b, row0, kvh, z, q_start, kv_len, pos0, rows_total;
    int g_first[NG], g_last[NG];  // first and last key tile of each row group (last < first: none)
    int t0, ntiles, lo, hi;
  };
  auto load_pair = [&](int round, int wi, Pair& p) -> bool {
    int n;
    if (FOUND) {
      const TcPair f = found[round];
      p.b = f.at.x;
      p.row0 = f.at.y;
      p.kvh = f.at.z;
      p.z = f.at.w;
      p.q_start = f.q_start;
      n = f.n;
      p.kv_len = f.pos0 + n;
      if (p.b < 0) return false;
    } else {
      const int2 w = work[wi / kv_heads];
      p.b = w.x;
      p.row0 = w.y;
      p.kvh = wi % kv_heads;
      p.z = 0;
      if (p.b < 0) return false;  // padding of a fixed-size work list
      p.q_start = q_indptr[p.b];
      n = q_indptr[p.b + 1] - p.q_start;
      p.kv_len = kv_lens[p.b];
    }
    p.pos0 = p.kv_len - n;
    p.rows_total = n * group;
    // Key tiles of each row group: from its first row's window to its last row's position; a group past the request's
    // rows has none. The CTA walks the union (the groups' ranges overlap or touch: later rows see later keys).
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int r0 = p.row0 + g * BM;
      if (r0 < p.rows_total) {
        const int last_row = min(r0 + BM, p.rows_total) - 1;
        p.g_last[g] = (p.pos0 + last_row / group) / TK;
        p.g_first[g] = (window > 0 ? max(0, p.pos0 + r0 / group - window + 1) : 0) / TK;
      } else {
        p.g_first[g] = 1;
        p.g_last[g] = 0;
      }
      if (SIGMOID && sg.chunks > 1 && p.g_last[g] >= p.g_first[g]) {       // the chunk's tiles of them; of two groups the first may see none
        p.g_first[g] = p.z * sg.chunk_tiles;
        if (p.z < sg.chunks - 1) p.g_last[g] = min(p.g_last[g], p.g_first[g] + sg.chunk_tiles - 1);
        if (p.g_last[g] < p.g_first[g]) {
          p.g_first[g] = 1;
          p.g_last[g] = 0;
        }
      }
    }
    p.t0 = SIGMOID ? p.z * sg.chunk_tiles : p.g_first[0];
    int t1 = p.g_last[0];
#pragma unroll
    for (int g = 1; g < NG; ++g) {
      if (p.g_last[g] >= p.g_first[g]) t1 = max(t1, p.g_last[g]);
    }
    p.ntiles = t1 - p.t0 + 1;
    p.lo = window > 0 ? max(0, p.pos0 + p.row0 / group - window + 1) : 0;                              // first key any row of the pair sees
    p.hi = min(p.pos0 + (min(p.row0 + NG * BM, p.rows_total) - 1) / group, (t1 + 1) * TK - 1);          // last one
    return p.ntiles > 0;
  };

  if (warp == 0) {
    // ---- producer
    const int page_shift = FLAT ? 0 : 31 - __clz(page_size);  // a power of two here
    int kt = 0;        // tiles copied so far, over all pairs: the rings run on
    int pairs = 0;     // pairs begun so far
    bool ok = true;
    Pair p;
    for (int round = 0, wi = pair_of(0); wi < total && ok; wi = pair_of(++round)) {
      if (!load_pair(round, wi, p)) continue;
      const int32_t* pages = FLAT ? nullptr : kv_indices + kv_indptr[p.b];
      const int p_first = (p.t0 * TK) >> page_shift, p_last = FLAT ? -1 : p.hi >> page_shift;
      const int fallback = FLAT ? 0 : pages[p_last];
      auto row_of = [&](int pg, int entry) {  // first pool row of page pg of the request, given its block-table entry
        const bool visible = ((pg + 1) << page_shift) > p.lo && (pg << page_shift) <= p.hi;
        return ((visible && entry >= 0 ? entry : fallback) * kv_heads + p.kvh) << page_shift;
      };
      int batch0 = p_first;
      int cur = row_of(batch0 + lane, batch0 + lane <= p_last ? pages[batch0 + lane] : -1);
      int nxt_entry = batch0 + 32 + lane <= p_last ? pages[batch0 + 32 + lane] : -1;
      if (lane == 0) {
        if (pairs >= 1) ok = mbar_wait_limited(q_empty, (uint32_t)(pairs - 1) & 1u, abortp, 12, &g_attention_tc_error);
        if (ok) {
          mbar_expect_tx(q_full, NG * kQBytes);  // rows past the tensor's last token are filled with zeros and counted
          if constexpr (FLAT) {
#pragma unroll
            for (int c = 0; c < CB; ++c) {
              const bool own = c < flat.own_blocks;
              tma_load_3d(q_smem + c * (BM * 128), own ? &map_q : &map_q2, q_full, own ? c * 64 : 0, p.kvh, p.q_start + p.row0);
            }
          } else {
#pragma unroll
            for (int g = 0; g < NG; ++g) tma_load_5d(q_smem + g * kQBytes, &map_q, q_full, 0, 0, p.kvh, p.q_start + (p.row0 + g * BM) / group, 0);
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      ++pairs;
      for (int i = 0; i < p.ntiles && ok; ++i, ++kt) {
        const int ks = kt % KS, vs = kt % VS;
        const int j = (p.t0 + i) * TK;
        if (!FLAT && (j >> page_shift) >= batch0 + 32) {  // uniform in the warp
          batch0 += 32;
          cur = row_of(batch0 + lane, nxt_entry);
          nxt_entry = batch0 + 32 + lane <= p_last ? pages[batch0 + 32 + lane] : -1;
        }
        // lane L issues copy L of the tile: page copy L / (CB + 1); column block L % (CB + 1) of its keys, or its values.
        // A tile never straddles two batches of 32 pages: both start on tile boundaries.
        const int c = lane / (CB + 1), part = lane % (CB + 1);
        const int jc = j + (c < NP ? c : 0) * RPC;
        const int my_row = FLAT ? p.b * flat.stride + j : __shfl_sync(0xffffffffu, cur, ((jc >> page_shift) - batch0) & 31) + (jc & (page_size - 1));
        if (lane == 0) {
          if (kt >= KS) ok = mbar_wait_limited(k_empty(ks), (uint32_t)((kt / KS) - 1) & 1u, abortp, 1, &g_attention_tc_error);
          if (ok) mbar_expect_tx(k_full(ks), kKTile);
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;  // also orders the expected bytes before the copies
        if (ok && lane < kOps && part < CB) {
          const bool own = !FLAT || part < flat.own_blocks;
          tma_load_2d(k_smem + ks * kKTile + part * (TK * 128) + c * (RPC * 128), own ? &map_k : &map_k2, k_full(ks),
                      FLAT ? (own ? (p.kvh * flat.own_blocks + part) * 64 : 0) : part * 64, my_row);
        }
        if (lane == 0 && ok) {
          if (kt >= VS) ok = mbar_wait_limited(v_empty(vs), (uint32_t)((kt / VS) - 1) & 1u, abortp, 9, &g_attention_tc_error);
          if (ok) mbar_expect_tx(v_full(vs), kVTile);
        }
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (ok && lane < kOps && part == CB) {
          tma_load_3d(v_smem + vs * kVTile + c * kVPage, &map_v, v_full(vs), 0, my_row, FLAT ? p.kvh * (DV / 64) : 0);
        }
      }
    }
  } else if (warp == 1) {
    // ---- issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(BM, TK);
      constexpr uint32_t idesc_o = umma_idesc_bf16_b_mn(BM, DV);
      int kt0 = 0;            // tiles of the pairs before this one
      int pairs = 0;
      int jt0[NG];            // tiles of each group in the pairs before this one: which score columns, which phase
#pragma unroll
      for (int g = 0; g < NG; ++g) jt0[g] = 0;
      bool ok = true;
      Pair p;
      for (int round = 0, wi = pair_of(0); wi < total && ok; wi = pair_of(++round)) {
        if (!load_pair(round, wi, p)) continue;
        if (!(ok = mbar_wait_limited(q_full, (uint32_t)pairs & 1u, abortp, 2, &g_attention_tc_error))) break;
        ++pairs;
        tcgen05_fence_after();
        // O_g += P V of the pair's tile i (the group's tile j): the weights from tensor memory, the values from the ring
        auto issue_pv = [&](int g, int j, int i) {
          const int jt = jt0[g] + j, sb = jt % SB;
          if (!(ok = mbar_wait_limited(p_full(g, sb), (uint32_t)(jt / SB) & 1u, abortp, 3, &g_attention_tc_error))) return;
          tcgen05_fence_after();
          const uint32_t v0 = v_smem + ((kt0 + i) % VS) * kVTile;
#pragma unroll
          for (int kk = 0; kk < TK / 16; ++kk) {
            const uint32_t v_rows = v0 + (uint32_t)((kk * 16) / RPC) * kVPage + (uint32_t)((kk * 16) % RPC) * 128;
            const uint64_t b_desc = umma_desc_mn_major_sw128(v_rows, RPC * 128, 1024);
            tcgen05_mma_f16_ts(tmem_o(g), tmem_s(g, sb) + (uint32_t)(kk * 8), b_desc, idesc_o, (j > 0 || kk > 0) ? 1u : 0u);
            if (WIDE) tcgen05_mma_f16_ts(tmem_o(g), tmem_s(g, sb) + (uint32_t)(TK / 2 + kk * 8), b_desc, idesc_o, 1u);
          }
          tcgen05_commit(v_empty((kt0 + i) % VS));  // the values are free (for this group) once these products have read them
          if (p.g_first[g] + j == p.g_last[g]) tcgen05_commit(o_done(g));
        };
        // S_g = Q K^T of the pair's tile i
        auto issue_s = [&](int g, int j, int i) {
          const int jt = jt0[g] + j;
          const uint32_t k0 = k_smem + ((kt0 + i) % KS) * kKTile;
#pragma unroll
          for (int k = 0; k < DK / 16; ++k) {
            if (FLAT && k >= flat.k_steps) break;       // the rest of the shared part's block is padding
            const uint64_t a_desc = umma_desc_k_major_sw128(q_smem + g * kQBytes + (k / 4) * (BM * 128)) + (uint64_t)(2 * (k % 4));
            const uint64_t b_desc = umma_desc_k_major_sw128(k0 + (k / 4) * (TK * 128)) + (uint64_t)(2 * (k % 4));
            tcgen05_mma_f16(tmem_s(g, jt % SB), a_desc, b_desc, idesc_s, k > 0 ? 1u : 0u);
          }
          tcgen05_commit(s_full(g, jt % SB));
        };
        for (int i = 0; i <= p.ntiles && ok; ++i) {
          const int t = p.t0 + i;
          if (i < p.ntiles) {
            if (!(ok = mbar_wait_limited(k_full((kt0 + i) % KS), (uint32_t)((kt0 + i) / KS) & 1u, abortp, 4, &g_attention_tc_error))) break;
            tcgen05_fence_after();
          }
          if (SB == 2 && i < p.ntiles) {
            // two sets of score columns: this tile's scores are computed while the softmax of the tile before still runs.
            // (The set they go to held the weights of the group's tile two before, whose second product was issued an
            // iteration ago.)
#pragma unroll
            for (int g = 0; g < NG; ++g)
              if (t >= p.g_first[g] && t <= p.g_last[g]) issue_s(g, t - p.g_first[g], i);
          }
          if (i >= 1) {
            if (!(ok = mbar_wait_limited(v_full((kt0 + i - 1) % VS), (uint32_t)((kt0 + i - 1) / VS) & 1u, abortp, 5, &g_attention_tc_error))) break;
            tcgen05_fence_after();
          }
#pragma unroll
          for (int g = 0; g < NG; ++g) {
            if (i >= 1) {   // the second product of the tile before, which the group's softmax has finished meanwhile
              if (t - 1 >= p.g_first[g] && t - 1 <= p.g_last[g]) {
                issue_pv(g, t - 1 - p.g_first[g], i - 1);
                if (!ok) break;
              } else {
                mbar_arrive(v_empty((kt0 + i - 1) % VS));
              }
            }
            // one set of score columns: the scores overwrite the weights the product just issued reads (in issue order)
            if (SB == 1 && i < p.ntiles && t >= p.g_first[g] && t <= p.g_last[g]) issue_s(g, t - p.g_first[g], i);
          }
          if (ok && i < p.ntiles) tcgen05_commit(k_empty((kt0 + i) % KS));
          if (ok && i == p.ntiles - 1) tcgen05_commit(q_empty);   // the pair's last scores are on their way: Q may be replaced
        }
        kt0 += p.ntiles;
#pragma unroll
        for (int g = 0; g < NG; ++g) jt0[g] += max(0, p.g_last[g] - p.g_first[g] + 1);
      }
    }
  } else {
    // ---- softmax, correction, epilogue: one thread a row, four warps a row group
    const int g = (warp - 2) / 4;
    const int lane_group = warp & 3;               // the tensor-memory lanes this warp may touch
    const int row = lane_group * 32 + lane;        // row within the group
    const uint32_t lane_addr = (uint32_t)(lane_group * 32) << 16;
    const int tid_g = threadIdx.x - 64 - g * kGroupThreads;     // 0 .. 127 within the group
    int kt0 = 0;        // tiles of the pairs before this one (the rings' positions)
    int jt0 = 0;        // this group's tiles in the pairs before this one
    int outs = 0;       // pairs in which this group had rows: the phase of o_done
    bool ok = true;
    Pair p;
    for (int round = 0, wi = pair_of(0); wi < total && ok; wi = pair_of(++round)) {
      if (!load_pair(round, wi, p)) continue;
      const int pr = p.row0 + g * BM + row;
      const bool valid = pr < p.rows_total;
      const int qpos = valid ? p.pos0 + pr / group : -1;
      const int qlo = valid && window > 0 ? max(0, qpos - window + 1) : 0;
      const int my_tiles = p.g_last[g] - p.g_first[g] + 1;  // at most 0 for a group without rows
      const int head = p.kvh * group + (valid ? pr % group : 0);
      const float slope = SIGMOID ? sg.slopes[head] * kLog2eTc : 0.f, bias = SIGMOID ? sg.bias[head] * kLog2eTc : 0.f;
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < my_tiles && ok; ++j) {
        const int i = p.g_first[g] + j - p.t0;       // the pair's tile
        const int kt = kt0 + i;
        const int jt = jt0 + j, sb = jt % SB;
        const int j0 = (p.g_first[g] + j) * TK;
        if (!(ok = mbar_wait_limited(s_full(g, sb), (uint32_t)(jt / SB) & 1u, abortp, 6, &g_attention_tc_error))) break;
        tcgen05_fence_after();
        float s[TK];
        {
          uint32_t v[TK / 32][32];
#pragma unroll
          for (int c = 0; c < TK / 32; ++c) tcgen05_ld_32x32b_x32_nowait(tmem_s(g, sb) + lane_addr + c * 32, v[c]);
          tcgen05_wait_ld();
#pragma unroll
          for (int c = 0; c < TK / 32; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e) s[c * 32 + e] = __uint_as_float(v[c][e]);
        }
        if (!(j0 + TK - 1 <= qpos && j0 >= qlo)) {
#pragma unroll
          for (int e = 0; e < TK; ++e) {
            const int key = j0 + e;
            s[e] = (key <= qpos && key >= qlo) ? s[e] : -INFINITY;
          }
        }
        float corr = 1.0f, msafe = 0.f;
        if (!SIGMOID) {
          // the maximum of the raw scores (the scale is positive); four chains, so that it is not one long dependency
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int e = 0; e < TK; e += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(mx4[u], s[e + u]);
          }
          const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
          // the reference maximum moves only when it must: the weights of this tile are then at most 2^kTcLazyRescale
          if (mx > m + kTcLazyRescale || (m == -INFINITY && mx > -INFINITY)) {
            corr = ex2(m - mx);   // 0 when m is -inf
            m = mx;
          }
          msafe = m == -INFINITY ? 0.f : m;  // a row that has seen no key yet: every weight below is 0
        }
        const float at0 = SIGMOID ? fmaf(slope, (float)(j0 - qpos), bias) : 0.f;      // bias - slope (position - first key), in log2 units
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t packed[TK / 2], rest[WIDE ? TK / 2 : 1];
#pragma unroll
        for (int e = 0; e < TK; e += 2) {
          float p0, p1;
          if (SIGMOID) {
            p0 = sigmoid_of_ex2(-fmaf(s[e], scale_log2, fmaf(slope, (float)e, at0)));
            p1 = sigmoid_of_ex2(-fmaf(s[e + 1], scale_log2, fmaf(slope, (float)(e + 1), at0)));
          } else {
            p0 = ex2(fmaf(s[e], scale_log2, -msafe));
            p1 = ex2(fmaf(s[e + 1], scale_log2, -msafe));
            sum4[(e / 2) & 3] += p0 + p1;
          }
          __nv_bfloat162 pb = __floats2bfloat162_rn(p0, p1);
          packed[e / 2] = *reinterpret_cast<uint32_t*>(&pb);
          if (WIDE) {
            __nv_bfloat162 rb = __floats2bfloat162_rn(p0 - __uint_as_float(packed[e / 2] << 16), p1 - __uint_as_float(packed[e / 2] & 0xffff0000u));
            rest[e / 2] = *reinterpret_cast<uint32_t*>(&rb);
          }
        }
        if (!SIGMOID) l = l * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
        // The accumulator holds the pair's tiles 0 .. j - 1 once the second product of tile j - 1 is done. With one set
        // of score columns the scores of tile j were computed after it (the issuer's order). With two sets they were
        // issued before it: the group then waits for that product where it hands the values back.
        if (!SIGMOID && j >= 1 && __any_sync(0xffffffffu, corr != 1.0f)) {
          if (SB == 2) {
            if (!(ok = mbar_wait_limited(v_empty((kt - 1) % VS), (uint32_t)((kt - 1) / VS) & 1u, abortp, 10, &g_attention_tc_error))) break;
            tcgen05_fence_after();
          }
#pragma unroll 1
          for (int c = 0; c < DV / 32; ++c) {
            uint32_t v[32];
            tcgen05_ld_32x32b_x32(tmem_o(g) + lane_addr + c * 32, v);
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * corr);
            tcgen05_st_32x32b_x32(tmem_o(g) + lane_addr + c * 32, v);
          }
        }
        // value rows at positions the request does not hold yet, and rows before the first visible key (their page may
        // have been given back and replaced by another): zero, once the tile's values have landed. Every row group does
        // it before its own second product.
        if (j0 + TK > p.kv_len || j0 < p.lo) {
          if (!(ok = mbar_wait_limited(v_full(kt % VS), (uint32_t)(kt / VS) & 1u, abortp, 7, &g_attention_tc_error))) break;
          const uint32_t v0 = v_smem + (kt % VS) * kVTile;
          for (int idx = tid_g; idx < TK * (DV / 8); idx += kGroupThreads) {
            const int r = idx / (DV / 8), ch = idx % (DV / 8);
            if (j0 + r >= p.kv_len || j0 + r < p.lo) {
              const uint32_t addr = v0 + (uint32_t)(r / RPC) * kVPage + (uint32_t)(ch >> 3) * (RPC * 128) + (uint32_t)(r % RPC) * 128 +
                                    (uint32_t)(((ch & 7) ^ (r & 7)) << 4);
              asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(addr), "r"(0u) : "memory");
            }
          }
          asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the stores are visible to the tensor cores' reads
        }
        // the row's weights, two bfloat16 a column, over the first half of the scores' columns
#pragma unroll
        for (int c = 0; c < TK / 64; ++c) tcgen05_st_32x32b_x32_nowait(tmem_s(g, sb) + lane_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&packed[c * 32]));
        if (WIDE) {
#pragma unroll
          for (int c = 0; c < TK / 64; ++c)
            tcgen05_st_32x32b_x32_nowait(tmem_s(g, sb) + lane_addr + TK / 2 + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&rest[WIDE ? c * 32 : 0]));
        }
        tcgen05_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(g, sb));
      }
      // epilogue: O / l
      if (ok && my_tiles > 0) ok = mbar_wait_limited(o_done(g), (uint32_t)outs & 1u, abortp, 8, &g_attention_tc_error);
      if (ok && my_tiles > 0) {
        tcgen05_fence_after();
        if (!SIGMOID && sink != 0.f) l += ex2((sinks != nullptr && valid ? sinks[p.kvh * group + pr % group] * kLog2eTc : 0.f) - (m == -INFINITY ? 0.f : m));
        const float inv = SIGMOID ? 1.0f : (l > 0.f ? 1.0f / l : 0.f);
        const __nv_bfloat16* gate = SIGMOID && valid && sg.gate != nullptr ? sg.gate + (size_t)(p.q_start + pr / group) * sg.ld_gate + (size_t)head * DV : nullptr;
        __nv_bfloat16* dst = valid ? out + ((size_t)(p.q_start + pr / group) * q_heads + p.kvh * group + pr % group) * DV : nullptr;
        // a row that sees keys of several chunks leaves this one's sums for the kernel that adds them; one that sees none of the chunk, nothing
        float* sums = nullptr;
        bool writes = valid;
        if (SIGMOID && sg.chunks > 1 && valid) {
          writes = qpos >= p.z * sg.chunk_tiles * TK;
          if (qpos >= sg.chunk_tiles * TK) sums = sg.sums + (((size_t)(p.q_start + pr / group) * q_heads + head) * sg.chunks + p.z) * DV;
        }
#pragma unroll 1
        for (int c = 0; c < DV / 32; ++c) {
          uint32_t v[32];
          tcgen05_ld_32x32b_x32(tmem_o(g) + lane_addr + c * 32, v);
          if (SIGMOID && sums != nullptr && writes) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) *reinterpret_cast<uint4*>(sums + c * 32 + e) = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
          } else if (writes) {
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
              uint32_t o[4];
              if (SIGMOID && gate != nullptr) {
                float gv[8];
                Vec<__nv_bfloat16>::load(gate + c * 32 + e, gv);
#pragma unroll
                for (int u = 0; u < 8; ++u) v[e + u] = __float_as_uint(__uint_as_float(v[e + u]) * sigmoid_f(gv[u]));
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                __nv_bfloat162 ob = __floats2bfloat162_rn(__uint_as_float(v[e + 2 * u]) * inv, __uint_as_float(v[e + 2 * u + 1]) * inv);
                o[u] = *reinterpret_cast<uint32_t*>(&ob);
              }
              *reinterpret_cast<uint4*>(dst + c * 32 + e) = make_uint4(o[0], o[1], o[2], o[3]);
            }
          }
        }
        // the accumulator's columns are read: only now may this warp's arrival for the next pair's first weights come
        tcgen05_fence_before();
      }
      if (my_tiles > 0) {
        ++outs;
        jt0 += my_tiles;
      }
      kt0 += p.ntiles;
    }
  }

  __syncwarp();
  if (*abortp) {  // copies in flight land before shared memory is released
    const long long c0 = clock64();
    while (clock64() - c0 < 2000000LL) __nanosleep(256);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// The sums of a token's chunks, added in their order, then the output gate and the one rounding: a block a token, a thread four numbers. A token that
// sees one chunk has its output already.
__global__ void __launch_bounds__(256) sigmoid_tc_merge_kernel(const float* sums, __nv_bfloat16* out, const __nv_bfloat16* gate, int64_t ld_gate,
                                                              const int32_t* __restrict__ positions, int width, int dim, int chunk_keys, int chunks) {
  pdl_launch_dependents();
  const int t = blockIdx.x, own = min(positions[t] / chunk_keys + 1, chunks);
  pdl_wait();
  if (own <= 1) return;
  for (int i = threadIdx.x * 4; i < width; i += 1024) {
    const float* from = sums + ((size_t)t * (width / dim) + i / dim) * chunks * dim + i % dim;
    float4 a = *reinterpret_cast<const float4*>(from);
    for (int z = 1; z < own; ++z) {
      const float4 b = *reinterpret_cast<const float4*>(from + (size_t)z * dim);
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    if (gate != nullptr) {
      const uint2 g = *reinterpret_cast<const uint2*>(gate + (size_t)t * ld_gate + i);
      a.x *= sigmoid_f(__uint_as_float(g.x << 16)); a.y *= sigmoid_f(__uint_as_float(g.x & 0xffff0000u));
      a.z *= sigmoid_f(__uint_as_float(g.y << 16)); a.w *= sigmoid_f(__uint_as_float(g.y & 0xffff0000u));
    }
    __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
    *reinterpret_cast<uint2*>(out + (size_t)t * width + i) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
  }
}

// ------------------------------------------------------------------------------------------------ host side
static bool g_prefill_tc = true;

bool prefill_tc_serves(int head_dim, int q_heads, int kv_heads, int page_size, long long pool_pages, const void* k_pool, const void* v_pool,
                       const void* q) {
  if (!g_prefill_tc || pool_pages <= 0 || (head_dim != 64 && head_dim != 128) || kv_heads <= 0 || q_heads % kv_heads != 0) return false;
  const int group = q_heads / kv_heads;
  if (group > 128 || (group & (group - 1)) != 0) return false;  // a CTA's 128 packed rows are whole tokens
  if (page_size < 16 || (page_size & (page_size - 1)) != 0) return false;
  if (pool_pages * kv_heads * page_size >= (1LL << 31)) return false;
  const long long pool_bytes = pool_pages * kv_heads * page_size * head_dim * 2;
  const long long gap = (const char*)v_pool - (const char*)k_pool;
  if (gap < pool_bytes || gap % 16 != 0 || gap >= (1LL << 40)) return false;
  return (uintptr_t)k_pool % 128 == 0 && (q == nullptr || (uintptr_t)q % 16 == 0) && encode_tiled() != nullptr;
}

template <int DK, int DV, int RPC, int NG, bool WIDE, bool FLAT, bool SIGMOID = false>
static int launch_tc(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mq2, const CUtensorMap& mk2, TcFlat flat, TcSigmoid sg, void* out,
                     const int32_t* q_indptr, const int32_t* kv_lens, const int32_t* kv_indptr, const int32_t* kv_indices, const int32_t* work, int items,
                     int q_heads, int kv_heads, int page_size, float scale, int window, const float* sinks, cudaStream_t s) {
  constexpr size_t smem = TcCfg<DK, DV, NG>::kSmem;
  auto kernel = attention_prefill_tc_kernel<DK, DV, RPC, NG, WIDE, FLAT, SIGMOID>;
  static int sms[64] = {};   // per device: its SM count, and that the kernel's shared-memory size has been set there
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return fail(ROOST_ERR_UNSUPPORTED, "attention_prefill: device ordinal beyond 63");
  if (sms[dev] == 0) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
  }
  // One CTA fills an SM (shared memory, tensor memory). With a few pairs an SM the grid is persistent, one CTA an SM,
  // each walking its share of the sorted list (measured at 1 x 2048 tokens of 32/8 heads: 50 against 72 us); with many
  // pairs an SM every pair is a CTA of its own and the hardware hands them out as SMs fall free, which balances a long
  // list better than the fixed walk (8 x 8192 tokens: 1017 against 885 TFLOP/s).
  // Where keys are dealt in chunks most of the pairs that are counted here do not exist and those that do are of a length, so the walk goes on to
  // kTcRounds pairs.
  const long long pairs = (long long)items * kv_heads;
  const int rounds = SIGMOID && sg.chunks > 1 ? kTcRounds : 8;
  const int grid = (int)(pairs <= (long long)rounds * sms[dev] ? (pairs < sms[dev] ? pairs : sms[dev]) : pairs);
  launch_kernel(kernel, dim3(grid), dim3(64 + NG * 128), smem, s, mq, mk, mv, mq2, mk2, flat, sg, (__nv_bfloat16*)out, q_indptr, kv_lens, kv_indptr, kv_indices,
                (const int2*)work, items, q_heads, kv_heads, page_size, scale * kLog2eTc, window, sinks);
  return check_launch("attention_prefill_tc");
}

static int paged_box_rows(int page_size) { return page_size < 32 ? page_size : 32; }

static int paged_maps(const void* q, long long tokens, const void* k_pool, const void* v_pool, int q_heads, int kv_heads, int head_dim, int page_size,
                      long long pool_pages, CUtensorMap& mq, CUtensorMap& mk, CUtensorMap& mv) {
  const int group = q_heads / kv_heads, box_rows = paged_box_rows(page_size);
  {
    // q [tokens][kv_heads][group][D] as 64 columns x group x kv heads x tokens x column blocks; a box is 128 packed rows
    // of one key/value head: [column block][token][head of the group][64]
    const cuuint64_t dims[5] = {64u, (cuuint64_t)group, (cuuint64_t)kv_heads, (cuuint64_t)tokens, (cuuint64_t)head_dim / 64};
    const cuuint64_t strides[4] = {(cuuint64_t)head_dim * 2, (cuuint64_t)group * head_dim * 2, (cuuint64_t)q_heads * head_dim * 2, 128u};
    const cuuint32_t box[5] = {64u, (cuuint32_t)group, 1u, (cuuint32_t)(kTcRows / group), (cuuint32_t)head_dim / 64};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode_tiled()(&mq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(q), dims, strides, box, elem,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ROOST_ERR_CUDA, "attention_prefill: cuTensorMapEncodeTiled (q) failed with code " + std::to_string((int)r));
  }
  const cuuint64_t pool_rows = (cuuint64_t)(pool_pages * kv_heads * page_size);
  {
    const cuuint64_t dims[2] = {(cuuint64_t)head_dim, pool_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)head_dim * 2};
    const cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = encode_tiled()(&mk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(k_pool), dims, strides, box, elem,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ROOST_ERR_CUDA, "attention_prefill: cuTensorMapEncodeTiled (keys) failed with code " + std::to_string((int)r));
  }
  {
    const cuuint64_t dims[3] = {64u, pool_rows, (cuuint64_t)head_dim / 64};
    const cuuint64_t strides[2] = {(cuuint64_t)head_dim * 2, 128u};
    const cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, (cuuint32_t)head_dim / 64};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult r = encode_tiled()(&mv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(v_pool), dims, strides, box, elem,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ROOST_ERR_CUDA, "attention_prefill: cuTensorMapEncodeTiled (values) failed with code " + std::to_string((int)r));
  }
  return ROOST_OK;
}

int launch_prefill_tc(const void* q, long long tokens, void* out, const void* k_pool, const void* v_pool, const int32_t* q_indptr,
                      const int32_t* kv_lens, const int32_t* kv_indptr, const int32_t* kv_indices, const int32_t* work, int items, int tile_rows,
                      int q_heads, int kv_heads, int head_dim, int page_size, long long pool_pages, float scale, int window, const float* sinks, cudaStream_t s) {
  if (tile_rows != 128 && tile_rows != 256) return fail(ROOST_ERR_INVALID, "attention_prefill: the tcgen05 kernel takes work items of 128 or 256 packed rows");
  const int groups = tile_rows / kTcRows;
  const int box_rows = paged_box_rows(page_size);
  CUtensorMap mq, mk, mv;
  const int rc = paged_maps(q, tokens, k_pool, v_pool, q_heads, kv_heads, head_dim, page_size, pool_pages, mq, mk, mv);
  if (rc != ROOST_OK) return rc;
  const bool wide = (window & ROOST_ATTENTION_WIDE_WEIGHTS) != 0;
#define ROOST_TC_CASE(DD, RR, GG)                                                                                                              \
  if (head_dim == DD && box_rows == RR && groups == GG) {                                                                                      \
    if (wide)                                                                                                                                  \
      return launch_tc<DD, DD, RR, GG, true, false>(mq, mk, mv, mq, mk, TcFlat{}, TcSigmoid{}, out, q_indptr, kv_lens, kv_indptr, kv_indices, work, items,  \
                                                    q_heads, kv_heads, page_size, scale, window, sinks, s);                                    \
    return launch_tc<DD, DD, RR, GG, false, false>(mq, mk, mv, mq, mk, TcFlat{}, TcSigmoid{}, out, q_indptr, kv_lens, kv_indptr, kv_indices, work, items,   \
                                                   q_heads, kv_heads, page_size, scale, window, sinks, s);                                     \
  }
  ROOST_TC_CASE(128, 16, 1)
  ROOST_TC_CASE(128, 32, 1)
  ROOST_TC_CASE(64, 16, 1)
  ROOST_TC_CASE(64, 32, 1)
  ROOST_TC_CASE(128, 16, 2)
  ROOST_TC_CASE(128, 32, 2)
  ROOST_TC_CASE(64, 16, 2)
  ROOST_TC_CASE(64, 32, 2)
#undef ROOST_TC_CASE
  return fail(ROOST_ERR_UNSUPPORTED, "attention_prefill: no tcgen05 kernel for these sizes");
}

static bool flat_serves(int nope, int rope, int vdim) {
  return (nope == 64 || nope == 128) && (vdim == 64 || vdim == 128) && rope >= 0 && rope <= 64 && rope % 16 == 0 && encode_tiled() != nullptr;
}

// A tensor map of bfloat16 numbers with 128-byte swizzle; `strides` in bytes, of dimensions 1 ...
static int flat_map(CUtensorMap* m, const void* base, int rank, std::initializer_list<cuuint64_t> dims, std::initializer_list<cuuint64_t> strides,
                    std::initializer_list<cuuint32_t> box) {
  const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
  const CUresult r = encode_tiled()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims.begin(), strides.begin(), box.begin(), elem,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? ROOST_OK : fail(ROOST_ERR_CUDA, "carried_attention: cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
}

void set_prefill_tc(bool on) { g_prefill_tc = on; }

int* attention_tc_error_address() {
  int* p = nullptr;
  return cudaGetSymbolAddress((void**)&p, g_attention_tc_error) == cudaSuccess ? p : nullptr;
}

int prefill_tc_status() {
  int code = 0;
  if (cudaMemcpyFromSymbol(&code, g_attention_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (code != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_attention_tc_error, &zero, sizeof(int));
  }
  return code;
}

}  // namespace roost

using namespace roost;

extern "C" int roost_carried_attention_tc_supported(int nope, int rope, int vdim) { return flat_serves(nope, rope, vdim) ? 1 : 0; }

// q [tokens, heads x (nope + rope)], rows ld_q apart; keys [rows * stride, heads * nope], values [rows * stride, heads * vdim] and, with rope, the
// part of a key that all heads share, rope_keys [rows * stride, rope] with rows ld_rope apart: entry r * stride + j is row r's token at position j.
// A row's queries are its last q_indptr[r + 1] - q_indptr[r] positions before kv_lens[r]; window as in roost_attention_prefill; sinks: null, or
// exp(sinks[h]) joins head h's denominator. out [tokens, heads * vdim].
extern "C" int roost_carried_attention_tc(const void* q, int64_t ld_q, void* out, const void* keys, const void* values, const void* rope_keys, int64_t ld_rope,
                                          const int32_t* q_indptr, const int32_t* kv_lens, int tokens, int rows, int heads, int nope, int rope, int vdim,
                                          int stride, float scale, int window, const float* sinks, roost_stream_t stream) {
  ROOST_REQUIRE(tokens >= 0 && rows >= 0 && heads > 0 && stride > 0 && stride % kTcKeys == 0 && scale > 0.f && window >= 0,
                "carried_attention: sizes and the scale must be positive, a row's entries a multiple of 128");
  ROOST_REQUIRE(q && out && keys && values && q_indptr && kv_lens && (rope == 0 || rope_keys), "carried_attention: a pointer is null");
  if (!flat_serves(nope, rope, vdim)) return fail(ROOST_ERR_UNSUPPORTED, "carried_attention: sizes the tcgen05 form does not serve");
  ROOST_REQUIRE(ld_q >= (int64_t)heads * (nope + rope) && ld_q % 8 == 0 && (rope == 0 || (ld_rope >= rope && ld_rope % 8 == 0)),
                "carried_attention: rows are too narrow or not whole 16-byte pieces");
  ROOST_REQUIRE(((uintptr_t)q | (uintptr_t)out | (uintptr_t)keys | (uintptr_t)values | (uintptr_t)rope_keys) % 16 == 0, "carried_attention: a pointer is not aligned");
  const long long entries = (long long)rows * stride, items = (long long)tokens / kTcRows + rows;
  if (entries >= (1LL << 31) || items * heads >= (1LL << 30)) return fail(ROOST_ERR_UNSUPPORTED, "carried_attention: too many entries or heads");
  if (tokens == 0 || rows == 0) return ROOST_OK;
  const cuuint64_t E = (cuuint64_t)entries, H = (cuuint64_t)heads, head = (cuuint64_t)(nope + rope) * 2;
  CUtensorMap mq, mk, mv, mq2, mk2;
  int rc = flat_map(&mq, q, 3, {(cuuint64_t)nope, H, (cuuint64_t)tokens}, {head, (cuuint64_t)ld_q * 2}, {64u, 1u, (cuuint32_t)kTcRows});
  if (rc == ROOST_OK) rc = flat_map(&mk, keys, 2, {H * nope, E}, {H * nope * 2}, {64u, (cuuint32_t)kTcKeys});
  if (rc == ROOST_OK) rc = flat_map(&mv, values, 3, {64u, E, H * vdim / 64}, {H * vdim * 2, 128u}, {64u, (cuuint32_t)kTcKeys, (cuuint32_t)vdim / 64});
  mq2 = mq;
  mk2 = mk;
  if (rc == ROOST_OK && rope) {
    rc = flat_map(&mq2, (const char*)q + nope * 2, 3, {(cuuint64_t)rope, H, (cuuint64_t)tokens}, {head, (cuuint64_t)ld_q * 2}, {64u, 1u, (cuuint32_t)kTcRows});
    if (rc == ROOST_OK) rc = flat_map(&mk2, rope_keys, 2, {(cuuint64_t)rope, E}, {(cuuint64_t)ld_rope * 2}, {64u, (cuuint32_t)kTcKeys});
  }
  if (rc != ROOST_OK) return rc;
  const TcFlat flat = {stride, rows, nope / 64, (nope + rope) / 16};
  TcSigmoid whole = {};       // a row's keys in one chunk
  whole.chunk_tiles = whole.chunks = 1;
  const int w = window | (sinks != nullptr ? ROOST_ATTENTION_SINK : 0);
  const int dk = nope + (rope ? 64 : 0);
#define ROOST_TC_FLAT(KK, VV)                                                                                                                \
  if (dk == KK && vdim == VV)                                                                                                                \
    return launch_tc<KK, VV, 128, 1, true, true>(mq, mk, mv, mq2, mk2, flat, whole, out, q_indptr, kv_lens, nullptr, nullptr, nullptr, (int)items,  \
                                                 heads, heads, 1, scale, w, sinks, (cudaStream_t)stream);
  ROOST_TC_FLAT(64, 64)
  ROOST_TC_FLAT(64, 128)
  ROOST_TC_FLAT(128, 64)
  ROOST_TC_FLAT(128, 128)
  ROOST_TC_FLAT(192, 64)
  ROOST_TC_FLAT(192, 128)
#undef ROOST_TC_FLAT
  return fail(ROOST_ERR_UNSUPPORTED, "carried_attention: no tcgen05 kernel for these sizes");
}

// Sigmoid weights over the paged cache (two planes of one size), prompt portions and single tokens mixed: as roost_sigmoid_attention_mma. 0 where
// these sizes, pools or addresses are not served.
extern "C" int roost_sigmoid_attention_tc_supported(int dim, int vdim, int heads, int kv_heads, int page_size, long long pool_pages, const void* k_pool,
                                                    const void* v_pool, const void* q, const void* out, const void* gate, int64_t ld_gate) {
  return dim == vdim && prefill_tc_serves(dim, heads, kv_heads, page_size, pool_pages, k_pool, v_pool, q) && (uintptr_t)out % 16 == 0 &&
         (gate == nullptr || ((uintptr_t)gate % 16 == 0 && ld_gate % 8 == 0));
}

// `chunk_tiles`: the key tiles of 128 that a block takes of a row's keys; `chunks`: how many such chunks a row has at most, the last one takes what is
// left. With more than one: positions, and sums float[tokens * heads * chunks * dim], which a second kernel adds.
extern "C" int roost_sigmoid_attention_tc_chunks(const void* q, void* out, const void* k_pool, const void* v_pool, long long pool_pages, const void* gate, int64_t ld_gate,
                                                  const float* slopes, const float* head_bias, const int32_t* q_indptr, const int32_t* kv_lens, const int32_t* kv_indptr,
                                                  const int32_t* kv_indices, int tokens, int rows, int heads, int kv_heads, int dim, int page_size, float scale,
                                                  const int32_t* positions, float* sums, int chunk_tiles, int chunks, roost_stream_t stream) {
  ROOST_REQUIRE(tokens >= 0 && rows >= 0 && heads > 0 && kv_heads > 0 && page_size > 0 && heads % kv_heads == 0 && scale > 0.f, "sigmoid_attention_tc: sizes and the scale must be positive");
  ROOST_REQUIRE(chunk_tiles >= 1 && chunks >= 1 && chunk_tiles <= (1 << 20) && (chunks == 1 || (sums != nullptr && positions != nullptr && (uintptr_t)sums % 16 == 0)),
                "sigmoid_attention_tc: chunks of keys need a workspace for their sums");
  ROOST_REQUIRE(q && out && k_pool && v_pool && slopes && head_bias && q_indptr && kv_lens && kv_indptr && kv_indices, "sigmoid_attention_tc: a pointer is null");
  ROOST_REQUIRE(gate == nullptr || ld_gate >= (int64_t)heads * dim, "sigmoid_attention_tc: a gate's row is too narrow");
  if (!roost_sigmoid_attention_tc_supported(dim, dim, heads, kv_heads, page_size, pool_pages, k_pool, v_pool, q, out, gate, ld_gate))
    return fail(ROOST_ERR_UNSUPPORTED, "sigmoid_attention_tc: sizes or addresses the tcgen05 form does not serve");
  if (tokens == 0 || rows == 0) return ROOST_OK;
  CUtensorMap mq, mk, mv;
  const int rc = paged_maps(q, tokens, k_pool, v_pool, heads, kv_heads, dim, page_size, pool_pages, mq, mk, mv);
  if (rc != ROOST_OK) return rc;
  const int group = heads / kv_heads;
  // two row groups a CTA where every processor gets a pair of them; with less work the smaller items spread over more processors
  const int groups = (long long)tokens * heads >= 2LL * 148 * kTcRows ? 2 : 1;
  const long long items = ((long long)tokens * group / (groups * kTcRows) + rows) * chunks;
  if (items * kv_heads >= (1LL << 30)) return fail(ROOST_ERR_UNSUPPORTED, "sigmoid_attention_tc: too many tokens, heads or chunks");
  const TcFlat flat = {0, rows, 0, 0};
  const TcSigmoid sg = {slopes, head_bias, (const __nv_bfloat16*)gate, ld_gate, chunk_tiles, chunks, sums};
  const int box_rows = paged_box_rows(page_size);
  int launched = ROOST_ERR_UNSUPPORTED;
#define ROOST_TC_SIGMOID(DD, RR, GG)                                                                                                            \
  if (dim == DD && box_rows == RR && groups == GG)                                                                                             \
    launched = launch_tc<DD, DD, RR, GG, true, false, true>(mq, mk, mv, mq, mk, flat, sg, out, q_indptr, kv_lens, kv_indptr, kv_indices,       \
                                                            nullptr, (int)items, heads, kv_heads, page_size, scale, 0, nullptr,                \
                                                            (cudaStream_t)stream);
  ROOST_TC_SIGMOID(64, 16, 1)
  ROOST_TC_SIGMOID(64, 32, 1)
  ROOST_TC_SIGMOID(64, 16, 2)
  ROOST_TC_SIGMOID(64, 32, 2)
  ROOST_TC_SIGMOID(128, 16, 1)
  ROOST_TC_SIGMOID(128, 32, 1)
  ROOST_TC_SIGMOID(128, 16, 2)
  ROOST_TC_SIGMOID(128, 32, 2)
#undef ROOST_TC_SIGMOID
  if (launched == ROOST_ERR_UNSUPPORTED) return fail(ROOST_ERR_UNSUPPORTED, "sigmoid_attention_tc: no kernel for these sizes");
  if (launched == ROOST_OK && chunks > 1) {
    launch_kernel(sigmoid_tc_merge_kernel, dim3(tokens), dim3(256), 0, (cudaStream_t)stream, (const float*)sums, (__nv_bfloat16*)out, (const __nv_bfloat16*)gate, ld_gate,
                  positions, heads * dim, dim, chunk_tiles * kTcKeys, chunks);
    return check_launch("sigmoid_attention_tc");
  }
  return launched;
}

extern "C" int roost_sigmoid_attention_tc(const void* q, void* out, const void* k_pool, const void* v_pool, long long pool_pages, const void* gate, int64_t ld_gate,
                                          const float* slopes, const float* head_bias, const int32_t* q_indptr, const int32_t* kv_lens, const int32_t* kv_indptr,
                                          const int32_t* kv_indices, int tokens, int rows, int heads, int kv_heads, int dim, int page_size, float scale,
                                          roost_stream_t stream) {
  return roost_sigmoid_attention_tc_chunks(q, out, k_pool, v_pool, pool_pages, gate, ld_gate, slopes, head_bias, q_indptr, kv_lens, kv_indptr, kv_indices, tokens,
                                           rows, heads, kv_heads, dim, page_size, scale, nullptr, nullptr, 1, 1, stream);
}

ROOST_TRACE_TU(attention_tc)
