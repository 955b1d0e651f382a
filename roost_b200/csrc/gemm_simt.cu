// out[m,n] = sum_k a[m,k] * w[n,k] with plain 32-bit FFMA: the products of the float32 model that gemm_f32_tc.cu does not take
// (short reductions, vocabulary-sized heads, rows of w that do not start on 16 bytes), also usable with bfloat16 operands for checks. Every output element sums
// over k in increasing order in one thread, so its bits do not depend on m's or n's extent or on the tile a
// row falls in. Definition: src/Starlings.Roost.Ops/CpuOps.cs:395-437 (TransposeB, Alpha 1, no bias).
//
// Two forms, bit for bit alike; the operands of both arrive by cp.async several stages of 32 k ahead, [row][k] as they lie in
// memory (bfloat16 operands and rows that are no whole 16-byte pieces: through registers, a stage ahead), and are read four k (16 bytes) at a time:
//   tiles: a thread makes TM x TN outputs of a block's BM x BN. Bound by issue slots and shared-memory reads together (78 %
//     and 68 % busy, the FMA pipe 64 %, at 2,048 x 4,096 x 4,096): 45 TFLOP/s there, 22.5 with the form before (one buffer,
//     scalar loads and reads); 512 x 6,144 x 1,024 170 us (337 before). Two outputs an instruction (fma.rn.f32x2) were
//     measured at 61 against 71 TFLOP/s for scalar ones when nothing else runs, and no faster here.
//   few rows (float32, whole 16-byte pieces, up to 8 rows): bound by reading the weights once; a lane keeps TN columns of RW
//     rows. 3 x 151,936 x 1,024: 120 us, 5.2 TB/s (939 us with a 64-row tile for three rows).
// What an earlier kernel of the step writes comes through pointers without __restrict__: with it the compiler may load before
// pdl_wait().
#include "common.cuh"

namespace roost {

// gemm_f32_tc.cu
bool gemm_f32_tc_takes(const void* w, int n, int k, int64_t ldw);
int launch_gemm_f32_tc(const float* a, const float* w, float* out, int m, int n, int k, int64_t lda, int64_t ldw, int64_t ldo, cudaStream_t stream);

constexpr int kSimtK = 32;           // k of a stage
constexpr int kSimtLd = kSimtK + 4;  // eight rows' 16-byte pieces of one k fall in different banks

__device__ __forceinline__ void simt_copy16(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}

// `ROWS` rows of one stage, [row][k], zeros beyond the matrix, in whole 16-byte pieces of floats by cp.async.
template <int ROWS, int NT>
__device__ __forceinline__ void simt_stage(float* dst, const float* p, int64_t ld, int row0, int rows, int k0, int K) {
#pragma unroll
  for (int i = 0; i < (ROWS * (kSimtK / 4) + NT - 1) / NT; ++i) {
    const int idx = threadIdx.x + i * NT, r = idx / (kSimtK / 4), kk = idx % (kSimtK / 4) * 4;
    if (ROWS * (kSimtK / 4) % NT != 0 && r >= ROWS) break;
    float* d = dst + r * kSimtLd + kk;
    if (row0 + r < rows && k0 + kk < K) simt_copy16(d, p + (int64_t)(row0 + r) * ld + k0 + kk);
    else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// The same an element at a time, through registers, so that a stage is on its way while the one before is multiplied.
// (Elements beyond the matrix are read at its end and replaced by zeros: with a condition around a load of 16 bits every load waited for the one
// before: 300 x 1,024 x 1,024 in bfloat16 106 us, 77 with the form before, whose tiles were 64 x 64.)
template <typename T, int ROWS, int NT>
__device__ __forceinline__ void simt_fetch(T (&held)[ROWS * kSimtK / NT], const T* p, int64_t ld, int row0, int rows, int k0, int K) {
  static_assert(ROWS * kSimtK % NT == 0, "whole passes");
#pragma unroll
  for (int i = 0; i < ROWS * kSimtK / NT; ++i) {
    const int idx = threadIdx.x + i * NT, r = min(row0 + idx / kSimtK, rows - 1), k = min(k0 + idx % kSimtK, K - 1);
    held[i] = p[(int64_t)r * ld + k];
  }
}
template <typename T, int ROWS, int NT>
__device__ __forceinline__ void simt_put(float* dst, const T (&held)[ROWS * kSimtK / NT], int row0, int rows, int k0, int K) {
#pragma unroll
  for (int i = 0; i < ROWS * kSimtK / NT; ++i) {
    const int idx = threadIdx.x + i * NT, r = idx / kSimtK, k = idx % kSimtK;
    dst[r * kSimtLd + k] = row0 + r < rows && k0 + k < K ? to_float(held[i]) : 0.f;
  }
}

template <typename TIn, typename TOut, int BM, int BN, int TM, int TN, int STAGES, bool ASYNC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_simt_kernel(const TIn* a, const TIn* w, TOut* out, int M, int N, int K, int64_t lda, int64_t ldw,
                                                                         int64_t ldo, int64_t batch_a, int64_t batch_w, int64_t batch_o) {
  constexpr int NX = BN / TN, NY = BM / TM, NT = NX * NY;
  extern __shared__ __align__(16) float sm[];
  float* ast = sm;                                    // [stages][BM][kSimtLd]
  float* wst = sm + STAGES * BM * kSimtLd;            // [stages][BN][kSimtLd]
  pdl_launch_dependents();
  pdl_wait();
  a += blockIdx.z * batch_a;   // a batch of products: one grid layer each (strides in elements; 0 for a single product)
  w += blockIdx.z * batch_w;
  out += blockIdx.z * batch_o;
  const int tx = threadIdx.x % NX, ty = threadIdx.x / NX;
  const int row_tiles = (M + BM - 1) / BM;                  // row tiles side by side: they share their weights in the cache
  const int m0 = blockIdx.x % row_tiles * BM, n0 = blockIdx.x / row_tiles * BN;
  const int steps = (K + kSimtK - 1) / kSimtK;
  auto issue = [&](int step) {
    if (step < steps) {
      const int buf = step % STAGES;
      simt_stage<BM, NT>(ast + buf * BM * kSimtLd, (const float*)a, lda, m0, M, step * kSimtK, K);
      simt_stage<BN, NT>(wst + buf * BN * kSimtLd, (const float*)w, ldw, n0, N, step * kSimtK, K);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  TIn ra[ASYNC ? 1 : BM * kSimtK / NT], rw[ASYNC ? 1 : BN * kSimtK / NT];
  auto fetch = [&](int step) {
    if constexpr (!ASYNC) {
      simt_fetch<TIn, BM, NT>(ra, a, lda, m0, M, step * kSimtK, K);
      simt_fetch<TIn, BN, NT>(rw, w, ldw, n0, N, step * kSimtK, K);
    }
  };
  auto put = [&](int step) {
    if constexpr (!ASYNC) {
      simt_put<TIn, BM, NT>(ast + step % STAGES * BM * kSimtLd, ra, m0, M, step * kSimtK, K);
      simt_put<TIn, BN, NT>(wst + step % STAGES * BN * kSimtLd, rw, n0, N, step * kSimtK, K);
    }
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  if constexpr (ASYNC) {
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue(s);
  } else {
    fetch(0);
    put(0);
  }
  for (int step = 0; step < steps; ++step) {
    if constexpr (ASYNC) asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();       // the stage has arrived for everyone, and the one before it has been read by everyone
    if constexpr (ASYNC) issue(step + STAGES - 1);
    else if (step + 1 < steps) fetch(step + 1);
    const float* as = ast + (step % STAGES) * BM * kSimtLd + ty * kSimtLd;      // a thread's rows and columns: every NY-th and every NX-th
    const float* ws = wst + (step % STAGES) * BN * kSimtLd + tx * kSimtLd;
    // the operands of the next four k are read while these are multiplied
    float4 x[2][TM], y[2][TN];
    auto read = [&](int k, int b) {
#pragma unroll
      for (int j = 0; j < TN; ++j) y[b][j] = *reinterpret_cast<const float4*>(ws + j * NX * kSimtLd + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) x[b][i] = *reinterpret_cast<const float4*>(as + i * NY * kSimtLd + k);
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < kSimtK; k += 4) {
      const int b = k / 4 & 1;
      if (k + 4 < kSimtK) read(k + 4, b ^ 1);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(x[b][i].x, y[b][j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(x[b][i].y, y[b][j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(x[b][i].z, y[b][j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(x[b][i].w, y[b][j].w, acc[i][j]);
    }
    if (!ASYNC && step + 1 < steps) put(step + 1);       // its buffer was read two steps ago
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + i * NY + ty;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + j * NX + tx;
      if (n < N) out[(int64_t)m * ldo + n] = from_float<TOut>(acc[i][j]);
    }
  }
}

constexpr int kFewK = 32, kFewStages = 4;

// WM warps side by side take RW rows each, 4 / WM groups of them BN / (4 / WM) columns each; a lane TN columns, 32 apart.
template <int WM, int RW, int TN>
__global__ void __launch_bounds__(128) gemm_simt_few_kernel(const float* a, const float* w, float* out, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldo,
                                                           int64_t batch_a, int64_t batch_w, int64_t batch_o) {
  constexpr int WN = 4 / WM, BM = WM * RW, BN = WN * 32 * TN, LD = kFewK + 4;      // a lane's 16-byte reads of 8 rows fall in different banks
  extern __shared__ __align__(16) float sm[];
  float* wst = sm;                                    // [stages][BN][LD]
  float* ast = sm + kFewStages * BN * LD;             // [stages][BM][LD]
  pdl_launch_dependents();
  a += blockIdx.z * batch_a;
  w += blockIdx.z * batch_w;
  out += blockIdx.z * batch_o;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % WM, wn = warp / WM;
  const int n0 = blockIdx.x * BN, steps = (K + kFewK - 1) / kFewK;
  auto issue = [&](int step) {
    if (step < steps) {
      const int buf = step % kFewStages, k0 = step * kFewK;
      for (int idx = tid; idx < BN * (kFewK / 4); idx += 128) {
        const int r = idx / (kFewK / 4), k = k0 + idx % (kFewK / 4) * 4;
        float* dst = wst + ((size_t)buf * BN + r) * LD + (k - k0);
        if (n0 + r < N && k < K) simt_copy16(dst, w + (int64_t)(n0 + r) * ldw + k);
        else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      for (int idx = tid; idx < BM * (kFewK / 4); idx += 128) {
        const int r = idx / (kFewK / 4), k = k0 + idx % (kFewK / 4) * 4;
        float* dst = ast + ((size_t)buf * BM + r) * LD + (k - k0);
        if (r < M && k < K) simt_copy16(dst, a + (int64_t)r * lda + k);
        else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  pdl_wait();
  float acc[RW][TN];
#pragma unroll
  for (int i = 0; i < RW; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < kFewStages - 1; ++s) issue(s);
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kFewStages - 2) : "memory");
    __syncthreads();       // the stage has arrived for everyone, and the one before it has been read by everyone
    issue(step + kFewStages - 1);
    const float* ws = wst + (size_t)(step % kFewStages) * BN * LD + (size_t)(wn * 32 * TN + lane) * LD;
    const float* as = ast + (size_t)(step % kFewStages) * BM * LD + (size_t)wm * RW * LD;
#pragma unroll
    for (int k = 0; k < kFewK; k += 4) {
      float4 x[RW], y[TN];
#pragma unroll
      for (int i = 0; i < RW; ++i) x[i] = *reinterpret_cast<const float4*>(as + i * LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) y[j] = *reinterpret_cast<const float4*>(ws + (size_t)j * 32 * LD + k);
#pragma unroll
      for (int i = 0; i < RW; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
          acc[i][j] = fmaf(x[i].w, y[j].w, fmaf(x[i].z, y[j].z, fmaf(x[i].y, y[j].y, fmaf(x[i].x, y[j].x, acc[i][j]))));
    }
  }
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    const int m = wm * RW + i;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + (wn * TN + j) * 32 + lane;
      if (m < M && n < N) out[(int64_t)m * ldo + n] = acc[i][j];
    }
  }
}

}  // namespace roost

using namespace roost;

struct SimtArgs {
  const void *a, *w;
  void* out;
  int batch, m, n, k;
  int64_t lda, ldw, ldo, batch_a, batch_w, batch_o;
  cudaStream_t stream;
};

template <typename TIn, typename TOut, int BM, int BN, int TM, int TN, int STAGES>
static int launch_simt_tiles(const SimtArgs& g, bool whole) {
  const long long tiles = (long long)((g.m + BM - 1) / BM) * ((g.n + BN - 1) / BN);
  if (tiles > INT32_MAX) return fail(ROOST_ERR_UNSUPPORTED, "gemm: too many tiles in one product");
  constexpr size_t smem = (size_t)STAGES * (BM + BN) * kSimtLd * sizeof(float);
  auto kernel = gemm_simt_kernel<TIn, TOut, BM, BN, TM, TN, STAGES, false>;
  if constexpr (sizeof(TIn) == 4)
    if (whole) kernel = gemm_simt_kernel<TIn, TOut, BM, BN, TM, TN, STAGES, true>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_kernel(kernel, dim3((unsigned)tiles, 1, g.batch), dim3((BM / TM) * (BN / TN)), smem, g.stream, (const TIn*)g.a, (const TIn*)g.w, (TOut*)g.out, g.m,
                g.n, g.k, g.lda, g.ldw, g.ldo, g.batch_a, g.batch_w, g.batch_o);
  return check_launch("gemm_simt");
}

template <int WM, int RW, int TN>
static int launch_simt_few(const SimtArgs& g) {
  constexpr int BM = WM * RW, BN = 4 / WM * 32 * TN;
  constexpr size_t smem = (size_t)kFewStages * (BM + BN) * (kFewK + 4) * sizeof(float);
  auto kernel = gemm_simt_few_kernel<WM, RW, TN>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_kernel(kernel, dim3((g.n + BN - 1) / BN, 1, g.batch), dim3(128), smem, g.stream, (const float*)g.a, (const float*)g.w, (float*)g.out, g.m, g.n, g.k,
                g.lda, g.ldw, g.ldo, g.batch_a, g.batch_w, g.batch_o);
  return check_launch("gemm_simt");
}

template <typename TIn, typename TOut>
static int launch_simt(const SimtArgs& g) {
  // whole pieces of 16 bytes in every row of both operands
  const bool whole = sizeof(TIn) == 4 && g.k % 4 == 0 && g.lda % 4 == 0 && g.ldw % 4 == 0 && g.batch_a % 4 == 0 && g.batch_w % 4 == 0 &&
                     (uintptr_t)g.a % 16 == 0 && (uintptr_t)g.w % 16 == 0;
  if constexpr (sizeof(TIn) == 4 && sizeof(TOut) == 4) {
    if (whole && g.m <= 8) {
      // a block takes 128 columns where two of them a processor remain, else 32 or 64 (a tile's weights are then read by fewer
      // threads, but by more processors: 3 x 1,024 x 3,072 39 us, 230 with 64 x 64 tiles)
      const bool wide = (long long)((g.n + 127) / 128) * g.batch >= 2 * 148;
      if (g.m <= 2) return wide ? launch_simt_few<1, 2, 1>(g) : launch_simt_few<2, 1, 1>(g);
      if (g.m <= 4) return wide ? launch_simt_few<1, 4, 1>(g) : launch_simt_few<4, 1, 1>(g);
      return wide ? launch_simt_few<2, 4, 2>(g) : launch_simt_few<4, 2, 1>(g);
    }
  }
  // Large tiles where they fill the processors (2,048 x 4,096 x 4,096: 1.53 ms; 1.81 with tiles of 32 x 64), small ones elsewhere (64 rows x 4,096
  // x 1,024: 36 us, 65 to 76 with the large tile), the smallest for decode batches (16 x 6,144 x 1,024: 21 us against 30 with 32 rows a tile).
  if (g.m <= 16) return launch_simt_tiles<TIn, TOut, 16, 64, 2, 4, 4>(g, whole);
  const long long big = (long long)((g.m + 127) / 128) * ((g.n + 63) / 64) * g.batch;
  if (big >= 148) return launch_simt_tiles<TIn, TOut, 128, 64, 8, 4, 3>(g, whole);
  return launch_simt_tiles<TIn, TOut, 32, 64, 4, 4, 4>(g, whole);
}

static int launch_gemm_simt(const void* a, const void* w, void* out, int batch, int m, int n, int k, int64_t lda, int64_t ldw, int64_t ldo,
                            int64_t batch_a, int64_t batch_w, int64_t batch_o, int in_dtype, int out_dtype, roost_stream_t stream) {
  ROOST_REQUIRE(m >= 0 && n > 0 && k > 0 && batch >= 0, "gemm: m, n and k must be positive");
  ROOST_REQUIRE(lda >= k && ldw >= k && ldo >= n, "gemm: a leading dimension is smaller than its row");
  if (m == 0 || batch == 0) return ROOST_OK;
  // the bound that callers have always had (tiles lay along the grid's y once)
  if (m > 64 * 65535) return fail(ROOST_ERR_UNSUPPORTED, "gemm: more than 4194240 rows in one product");
  if (batch > 65535) return fail(ROOST_ERR_UNSUPPORTED, "gemm: more than 65535 products in one batch");
  const SimtArgs g = {a, w, out, batch, m, n, k, lda, ldw, ldo, batch_a, batch_w, batch_o, (cudaStream_t)stream};
  if (in_dtype == ROOST_F32 && out_dtype == ROOST_F32) return launch_simt<float, float>(g);
  if (in_dtype == ROOST_BF16 && out_dtype == ROOST_BF16) return launch_simt<__nv_bfloat16, __nv_bfloat16>(g);
  if (in_dtype == ROOST_BF16 && out_dtype == ROOST_F32) return launch_simt<__nv_bfloat16, float>(g);
  return fail(ROOST_ERR_INVALID, "gemm: dtype codes must be (0,0), (1,1) or (1,0) for (in, out)");
}

extern "C" int roost_gemm_simt(const void* a, const void* w, void* out, int m, int n, int k, int64_t lda, int64_t ldw,
                               int64_t ldo, int in_dtype, int out_dtype, roost_stream_t stream) {
  if (in_dtype == ROOST_F32 && out_dtype == ROOST_F32 && m > 0 && m <= 64 * 65535 && n > 0 && k > 0 && lda >= k && ldw >= k && ldo >= n &&
      gemm_f32_tc_takes(w, n, k, ldw))
    return launch_gemm_f32_tc((const float*)a, (const float*)w, (float*)out, m, n, k, lda, ldw, ldo, (cudaStream_t)stream);
  return launch_gemm_simt(a, w, out, 1, m, n, k, lda, ldw, ldo, 0, 0, 0, in_dtype, out_dtype, stream);
}

extern "C" int roost_gemm_simt_batched(const void* a, const void* w, void* out, int batch, int m, int n, int k, int64_t lda, int64_t ldw,
                                       int64_t ldo, int64_t batch_a, int64_t batch_w, int64_t batch_o, int in_dtype, int out_dtype,
                                       roost_stream_t stream) {
  return launch_gemm_simt(a, w, out, batch, m, n, k, lda, ldw, ldo, batch_a, batch_w, batch_o, in_dtype, out_dtype, stream);
}
