// out[m,n] = sum_k x[m,k] * w[n,k] in bfloat16 with 32-bit accumulation for the few rows of a decode step (m <= 16) and weights that the processors hold
// (19 MB at 16 pieces a lane, 14 at 8 or 12): the products of a small model, whose time is latency. Definition: src/Starlings.Roost.Ops/CpuOps.cs:395-437 (TransposeB, alpha 1, no bias, 32-bit
// accumulation, one rounding); with SWIGLU silu(gate) * up of two products (src/Starlings.Roost.Models.Tiny/RoostTiny.cs:51-53).
//
// Every CTA keeps its rows of w in registers: 8 to 32 rows, k dealt to its eight warps, at most 16 pieces of 16 bytes a lane, all asked for before
// pdl_wait(), while the kernel that makes x is running. What is left after the wait is one trip to L2 for x, a few mma.sync m16n8k16 (a lane's pieces of eight k
// are their operands as they lie: which k a product calls its first is free as long as both operands agree), and one exchange between the warps in shared
// memory. 256 threads of at most 128 registers, so that a CTA of the next kernel fits beside it and has its weights on the way as well.
// The order of a sum is fixed by (n, k): a row's bits do not depend on m.
//
// What bounds it: the trips between kernels. In a chain of its like, us, against the kernel that served it before (k split over clusters, or cuBLAS):
//   rows of x        1            8            16
//   4,096 x 1,024    2.3 (5.5)    2.6 (5.3)    3.2 (4.8)
//   1,024 x 2,048    1.7 (4.8)    2.1 (5.0)    3.0 (6.9)
//   1,024 x 3,072    2.0 (5.7)    2.6 (5.9)    3.3 (8.8)
//   1,024 x 1,024    1.5 (4.9)    1.6 (4.2)    2.1 (4.2)
//   64 x 1,024       1.1 (3.3)    1.3 (3.3)    1.5 (3.3)
// and a feed-forward of 1,024 by 3,072, two products with the activation on the first: 5.3 (11.9), 5.8 (12.8), 9.2 (15.7).
#include "mma.cuh"

namespace roost {

constexpr int kRowsWarps = 8;
constexpr int kRowsThreads = kRowsWarps * 32;
constexpr int kRowsMaxPieces = 16;

__device__ __forceinline__ uint4 load_weights16(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 load_x16(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// R8: groups of eight rows of w a CTA takes; KB: blocks of 32 k a warp takes; TT: groups of eight rows of x. With
// SWIGLU w's rows come in blocks of 256 (128 gate rows, then the 128 up rows of the same outputs), the groups are gate and up in turn.
// x carries no __restrict__: with it the compiler may load before pdl_wait().
template <typename TOut, int R8, int KB, int TT, bool SWIGLU>
__global__ void __launch_bounds__(kRowsThreads, 2) gemm_rows_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ w, TOut* out, int M, int N, int64_t ldx, int64_t ldw, int64_t ldo) {
  static_assert(R8 * KB <= kRowsMaxPieces, "weights in registers");
  __shared__ float red[kRowsWarps][R8 * 8][TT * 8 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int k0 = warp * KB * 32 + c * 8;
  pdl_launch_dependents();
  uint4 wr[R8][KB];
#pragma unroll
  for (int r = 0; r < R8; ++r) {
    int row;
    if constexpr (SWIGLU) {
      const int j = (blockIdx.x * (R8 / 2) + r / 2) * 8 + g;                 // the output whose gate (r even) or up row this is
      row = j / 128 * 256 + j % 128 + (r & 1) * 128;
    } else {
      row = (blockIdx.x * R8 + r) * 8 + g;
    }
    const __nv_bfloat16* p = w + (int64_t)min(row, N - 1) * ldw + k0;
#pragma unroll
    for (int b = 0; b < KB; ++b) wr[r][b] = load_weights16(p + b * 32);
  }
  // What follows runs twice: first without a row of x, ahead of the wait, so that its instructions are in the processor's cache when the rows are there (a
  // kernel of a step finds them gone: 6 other kernels ran since the layer before).
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (pass) pdl_wait();
    const int rows = pass ? M : 0;
    float acc[R8][TT][2][4];
#pragma unroll
    for (int r = 0; r < R8; ++r)
#pragma unroll
      for (int t = 0; t < TT; ++t)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[r][t][i / 4][i % 4] = 0.f;
    // pieces of x on their way at a time: up to eight (the loads are volatile, so that those of the next turn do not take registers in this one)
    constexpr int kAtOnce = KB * TT <= 8 ? KB : (KB == 12 ? (TT == 1 ? 6 : 4) : (KB == 6 ? 3 : 8 / TT));
    static_assert(KB % kAtOnce == 0, "whole turns");
#pragma unroll
    for (int b0 = 0; b0 < KB; b0 += kAtOnce) {
      uint4 xv[TT][kAtOnce];
#pragma unroll
      for (int t = 0; t < TT; ++t)
#pragma unroll
        for (int b = 0; b < kAtOnce; ++b)
          xv[t][b] = t * 8 + g < rows ? load_x16(x + (int64_t)(t * 8 + g) * ldx + k0 + (b0 + b) * 32) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int b = 0; b < kAtOnce; ++b) {
#pragma unroll
        for (int r = 0; r < R8; ++r) {
          // A piece is a product's first operand as it lies in its four registers: its pairs of k 0 and 2 are then row g of a tile of 16, pairs 1 and 3 row
          // g + 8. Against x's pairs 0 and 2 the first half of the sums is the row's, against its pairs 1 and 3 the second; the other halves are not used.
          // (Two pieces a tile of 16 rows would take half as many products, and twice the registers: four of one piece and four of the other would
          // have to change places.)
          const uint32_t a[4] = {wr[r][b0 + b].x, wr[r][b0 + b].y, wr[r][b0 + b].z, wr[r][b0 + b].w};
#pragma unroll
          for (int t = 0; t < TT; ++t) {
            mma_bf16(acc[r][t][0], a, xv[t][b].x, xv[t][b].z);
            mma_bf16(acc[r][t][1], a, xv[t][b].y, xv[t][b].w);
          }
        }
      }
    }
    // a lane's sums: row g, rows of x 2 c and 2 c + 1
#pragma unroll
    for (int r = 0; r < R8; ++r)
#pragma unroll
      for (int t = 0; t < TT; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) red[warp][r * 8 + g][t * 8 + 2 * c + i] = acc[r][t][0][i] + acc[r][t][1][2 + i];
    __syncthreads();
    constexpr int kOut = SWIGLU ? R8 * 4 : R8 * 8;
    for (int idx = threadIdx.x; idx < kOut * max(rows, 1); idx += kRowsThreads) {
      const int m = idx / kOut, j = idx % kOut, n = blockIdx.x * kOut + j;
      float s[2];
#pragma unroll
      for (int u = 0; u < (SWIGLU ? 2 : 1); ++u) {
        const int row = SWIGLU ? (j / 8 * 2 + u) * 8 + j % 8 : j;
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < kRowsWarps; ++q) v += red[q][row][m];
        s[u] = v;
      }
      const float y = SWIGLU ? s[0] / (1.0f + expf(-s[0])) * s[SWIGLU ? 1 : 0] : s[0];
      if (pass && n < (SWIGLU ? N / 2 : N)) out[(int64_t)m * ldo + n] = from_float<TOut>(y);
    }
    if (!pass) __syncthreads();       // the sums' room is free again
  }
}

struct RowsShape {
  int r8, kb;       // groups of eight rows a CTA, blocks of 32 k a warp; r8 0: not served
};

// The fewest rows a CTA with which the processors hold all CTAs beside those of the kernels around this one (a CTA has 48 to 114 registers a thread). Larger
// CTAs would do: 128 of 48 rows by 1,024 k (6,144 rows of w) take 1.1 us once all are there, but the last eight found no room until the attention
// ahead had ended, and then had their instructions and their rows to bring: 8 us.
static RowsShape rows_shape(int m, int n, int k, bool swiglu) {
  if (n < 1 || k % (32 * kRowsWarps) != 0) return {0, 0};
  const int kb = k / (32 * kRowsWarps);
  if (kb != 1 && kb != 2 && kb != 3 && kb != 4 && kb != 6 && kb != 8 && kb != 12 && kb != 16) return {0, 0};
  const int groups = (n + 7) / 8, sms = processors();
  for (int r8 : {1, 2, 4}) {
    if (swiglu && r8 == 1) continue;
    if (r8 * kb > kRowsMaxPieces) break;
    if ((groups + r8 - 1) / r8 <= (r8 * kb <= 8 && m <= 8 ? 3 : 2) * sms) return {r8, kb};
  }
  return {0, 0};
}

}  // namespace roost

using namespace roost;

struct RowsArgs {
  const __nv_bfloat16 *x, *w;
  void* out;
  int m, n, ctas;
  int64_t ldx, ldw, ldo;
  cudaStream_t stream;
};

template <typename TOut, int R8, int KB, bool SWIGLU>
static int launch_rows(const RowsArgs& g) {
  auto kernel = g.m <= 8 ? gemm_rows_kernel<TOut, R8, KB, 1, SWIGLU> : gemm_rows_kernel<TOut, R8, KB, 2, SWIGLU>;
  launch_kernel(kernel, dim3(g.ctas), dim3(kRowsThreads), 0, g.stream, g.x, g.w, (TOut*)g.out, g.m, g.n, g.ldx, g.ldw, g.ldo);
  return check_launch("gemm_rows");
}

template <typename TOut, int KB, bool SWIGLU>
static int launch_rows_of(int r8, const RowsArgs& g) {
  if constexpr (!SWIGLU) {
    if (r8 == 1) return launch_rows<TOut, 1, KB, SWIGLU>(g);
  }
  if constexpr (2 * KB <= kRowsMaxPieces) {
    if (r8 == 2) return launch_rows<TOut, 2, KB, SWIGLU>(g);
  }
  if constexpr (4 * KB <= kRowsMaxPieces) {
    if (r8 == 4) return launch_rows<TOut, 4, KB, SWIGLU>(g);
  }
  return fail(ROOST_ERR_UNSUPPORTED, "gemm_rows: sizes that no form serves");
}

template <typename TOut, bool SWIGLU>
static int dispatch_rows(const RowsShape& s, const RowsArgs& g) {
  switch (s.kb) {
    case 1: return launch_rows_of<TOut, 1, SWIGLU>(s.r8, g);
    case 2: return launch_rows_of<TOut, 2, SWIGLU>(s.r8, g);
    case 3: return launch_rows_of<TOut, 3, SWIGLU>(s.r8, g);
    case 4: return launch_rows_of<TOut, 4, SWIGLU>(s.r8, g);
    case 6: return launch_rows_of<TOut, 6, SWIGLU>(s.r8, g);
    case 8: return launch_rows_of<TOut, 8, SWIGLU>(s.r8, g);
    case 12: return launch_rows_of<TOut, 12, SWIGLU>(s.r8, g);
    case 16: return launch_rows_of<TOut, 16, SWIGLU>(s.r8, g);
  }
  return fail(ROOST_ERR_UNSUPPORTED, "gemm_rows: sizes that no form serves");
}

extern "C" int roost_gemm_rows_supported(int m, int n, int k, int64_t ldx, int64_t ldw, int swiglu) {
  if (m < 1 || m > 16 || n < 1 || k < 1 || ldx % 8 != 0 || ldw % 8 != 0 || ldx < k || ldw < k || (swiglu && n % 256 != 0)) return 0;
  return rows_shape(m, n, k, swiglu != 0).r8 != 0;
}

extern "C" int roost_gemm_rows(const void* x, const void* w, void* out, int m, int n, int k, int64_t ldx, int64_t ldw, int64_t ldo, int out_dtype, int swiglu,
                               roost_stream_t stream) {
  ROOST_REQUIRE(roost_gemm_rows_supported(m, n, k, ldx, ldw, swiglu), "gemm_rows: sizes that it does not serve");
  ROOST_REQUIRE((uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0, "gemm_rows: operands start on 16 bytes");
  ROOST_REQUIRE(ldo >= (swiglu ? n / 2 : n), "gemm_rows: a leading dimension is smaller than its row");
  ROOST_REQUIRE(out_dtype == ROOST_BF16 || (out_dtype == ROOST_F32 && !swiglu), "gemm_rows: the output is bfloat16, or float32 without the activation");
  const RowsShape s = rows_shape(m, n, k, swiglu != 0);
  const int groups = (n + 7) / 8;
  const RowsArgs g = {(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, out, m, n, (groups + s.r8 - 1) / s.r8, ldx, ldw, ldo, (cudaStream_t)stream};
  if (swiglu) return dispatch_rows<__nv_bfloat16, true>(s, g);
  return out_dtype == ROOST_F32 ? dispatch_rows<float, false>(s, g) : dispatch_rows<__nv_bfloat16, false>(s, g);
}
