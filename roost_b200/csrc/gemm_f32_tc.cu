// out[m,n] = sum_k a[m,k] * w[n,k] over float32 operands on the fifth-generation tensor cores: the products of the float32 model whose
// reduction is long enough (gemm_simt.cu decides, by n, k and w alone). Definition: src/Starlings.Roost.Ops/CpuOps.cs:395-437
// (TransposeB, Alpha 1, no bias).
//
// Every operand x is written as three bfloat16 numbers, h nearest to x, m what x - h has in eight bits, l = x - h - m: all 24 bits of a
// float32. Both operands are taken times 2^24 first and the sums times 2^-48 last, which changes no bit of either but leaves the parts of the smallest numbers
// within bfloat16's range. Six of the nine products of the parts are formed (l h, h l, m m, m h, h m, h h; m l and l m, which are left out, are each below 2^-24 of
// their term and of one sign, l l is below 2^-32), the small ones first. The tensor cores cut the running sum of a chain of products off instead
// of rounding it, so a chain ends after 32 k: its sum leaves tensor memory and is added in float32, to nearest. k is cut into four
// parts, each a chain of such additions of its own, and the parts are added in order. What an output's bits depend on is therefore its
// row of a, its row of w and k; not m, n, the tile, or which of the forms below ran.
// A sum that is not finite (an operand that is not, or is above 2^104, or sums above 2^80) is formed once more as a chain of
// FFMAs over k when the CTA's tiles are done, so infinities and NaN come out where they do there.
//
// Roles of a CTA, which owns a tile of 128 rows of w by NT rows of a (the accumulator lies transposed: a lane of tensor memory is a
// row of w, so that a warp's stores are 128 consecutive bytes of out):
//   a producer lane: TMA copies of 32 k of both operands, as they are, four to six blocks ahead;
//   warps 0..7: converters, two groups that take the blocks in turn. w's planes go to tensor memory, where the products read their first operand, a's
//     to shared memory as 64-byte-swizzled K-major tiles; two or four stages of both. (Loads of the operands into registers a block ahead, without the copies:
//     a warp has six scoreboards, and waiting for an old load waited for the new ones on the same one.)
//   two issuer lanes, which take the blocks in turn: the 12 products of a block. (One lane is held by its products' queue for as long as they take and
//     would look at the next block's barriers only then: 700 cycles between blocks.)
//   4 or 8 epilogue warps: add their lanes' columns of a finished chain to their registers; the other chain's accumulator is filled
//     meanwhile. The sum of the earlier parts of k waits in tensor memory (in `out` it cost 7 us a part: all CTAs write at once).
// Forms: whole tiles by persistent CTAs, or (CL) a cluster of four CTAs a tile, CTA r taking the r-th part of k and the sums meeting in
// distributed shared memory, for products of few tiles.
// What bounds it: the products, of which none takes less than 64 cycles (72 with these tiles, about 90 beside the converters' traffic), so a block's twelve
// 1,080; their floor at NT 96 is 580. 2,048 x 4,096 x 4,096: 439 us, 157 TFLOP/s of 32-bit products (1,527 us by FFMAs). A row of `a` that does not
// start on 16 bytes is read by the converters an element at a time.
#include "tcgen05.cuh"

namespace roost {

int* gemm_tcgen05_error_address();

namespace f32tc {

constexpr int kBlock = 32;                                 // k of a stage and of a chain in the tensor cores
constexpr int kParts = 4;
constexpr int kWRows = 128;
constexpr int kConverters = 256;                           // two groups of four warps, which take the blocks in turn
constexpr float kScale = 16777216.0f;                      // 2^24, of both operands: the last bit of the smallest float32 becomes 2^-125, a bfloat16 number
constexpr float kUnscale = 1.0f / (kScale * kScale);
constexpr uint32_t kWRaw = kWRows * kBlock * 4;            // bytes of a block of w in float32
constexpr uint32_t kWColumns = 3 * kBlock / 2;             // tensor-memory columns of a block of w: three planes, two numbers a column

template <int NT>
struct Cfg {
  static constexpr int kEpilogueWarps = NT <= 32 ? 4 : 8;
  static constexpr int kColumns = NT <= 32 ? NT : NT / 2;  // accumulator columns of an epilogue warp
  static constexpr int kThreads = kConverters + kEpilogueWarps * 32 + 96;
  static constexpr int kCtasAnSm = NT <= 32 ? 2 : 1;
  static constexpr int kStages = NT == 32 || NT == 128 ? 2 : 4;                                  // of planes: what tensor memory has left
  static constexpr int kRawStages = NT == 64 ? 6 : 4;                                            // what shared memory has left; even, as the stages: a
                                                                                                 // stage is one group's and one issuer's for good
  static constexpr uint32_t kPlane = NT * kBlock * 2;                                            // bytes of a plane of a
  static constexpr uint32_t kStage = 3 * kPlane;
  static constexpr uint32_t kRawStage = kWRaw + NT * kBlock * 4;
  static constexpr uint32_t kSums = 2 * NT, kW = 3 * NT;   // tensor memory: two accumulators, the sum of the earlier parts of k, the stages of w's planes
  static constexpr uint32_t kTmem = NT <= 32 ? 256 : 512;
  static constexpr size_t kSmem = kStages * (size_t)kStage + kRawStages * (size_t)kRawStage + 1024;
  static_assert(kStages % 2 == 0 && kRawStages % 2 == 0, "whose a stage is");
  static_assert(kW + kStages * kWColumns <= kTmem, "tensor memory");
  static_assert(kSmem * kCtasAnSm <= 227 * 1024 - (kCtasAnSm - 1) * 2048, "shared memory");
};

// Shared-memory matrix descriptor of a K-major tile whose rows are 64 bytes (32 bfloat16), 64-byte swizzle: eight-row groups are 512 bytes apart.
__device__ __forceinline__ uint64_t desc_k_major_sw64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
__device__ __forceinline__ void store8(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t p;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(p) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ void bits_of(uint64_t p, uint32_t& lo, uint32_t& hi) { asm("mov.b64 {%0, %1}, %2;\n" : "=r"(lo), "=r"(hi) : "l"(p)); }
// Four numbers times kScale as their three parts, packed in pairs: p[part][0] the first two, p[part][1] the others. With integer additions and masks: conversion
// instructions keep the special-function pipe at two thirds of its rate, and splitting by three additions of floats was 3 % slower. The scaling and the
// differences take two numbers an instruction: 2,048 x 4,096 x 4,096 439 us, 451 with one, 437 without the scaling.
__device__ __forceinline__ void split4(float4 v, uint32_t (&p)[3][2]) {
  const uint64_t scale = pair_of(kScale, kScale), minus = pair_of(-1.0f, -1.0f);
  uint64_t x[2] = {pair_of(v.x, v.y), pair_of(v.z, v.w)};
  asm("mul.rn.f32x2 %0, %0, %1;\n" : "+l"(x[0]) : "l"(scale));
  asm("mul.rn.f32x2 %0, %0, %1;\n" : "+l"(x[1]) : "l"(scale));
#pragma unroll
  for (int part = 0; part < 3; ++part) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t b0, b1;
      bits_of(x[i], b0, b1);
      if (part == 0) { b0 += 0x8000u; b1 += 0x8000u; }      // h to nearest; m cut off; l is whole
      p[part][i] = __byte_perm(b0, b1, 0x7632);
      if (part < 2) {
        const uint64_t h = pair_of(__uint_as_float(b0 & 0xFFFF0000u), __uint_as_float(b1 & 0xFFFF0000u));
        asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(x[i]) : "l"(h), "l"(minus));
      }
    }
  }
}
__device__ __forceinline__ void tmem_store8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// Four numbers of row `row` from column k on, an element at a time; zeros beyond the matrix.
__device__ __forceinline__ float4 fetch4(const float* p, int64_t ld, int row, int rows, int k, int K) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row >= rows) return v;
  const float* s = p + (int64_t)row * ld + k;
  if (k < K) v.x = s[0];
  if (k + 1 < K) v.y = s[1];
  if (k + 2 < K) v.z = s[2];
  if (k + 3 < K) v.w = s[3];
  return v;
}
__device__ __forceinline__ float4 load16(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ bool finite(float v) { return (__float_as_uint(v) & 0x7F800000u) != 0x7F800000u; }

// The outputs of rows m0 .. m1 - 1 of a and n0 .. n1 - 1 of w that are not finite, formed once more as chains of FFMAs over k. By all threads of a CTA when its
// tiles are done: inside the pipeline the roles that wait for one another with a limit would wait for it. A lane a row of w, eight rows of a at a time, so
// that a piece of w is read once for eight chains.
template <int THREADS>
__device__ __forceinline__ void redo_not_finite(const float* a, const float* w, float* out, int m0, int m1, int n0, int n1, int K, int64_t lda, int64_t ldw, int64_t ldo) {
  const int width = (n1 - n0 + 31) / 32 * 32, tasks = (m1 - m0 + 7) / 8 * width;      // whole warps
  for (int idx = threadIdx.x; idx < tasks; idx += THREADS) {
    const int n = n0 + idx % width, m = m0 + idx / width * 8;
    unsigned need = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (n < n1 && m + i < m1 && !finite(out[(int64_t)(m + i) * ldo + n])) need |= 1u << i;
    const unsigned any = __reduce_or_sync(0xffffffffu, need);
    if (any == 0) continue;
    const float* wr = w + (int64_t)min(n, n1 - 1) * ldw;
    const float* ar = a + (int64_t)m * lda;
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0.f;
    for (int k = 0; k < K; k += 4) {
      const float4 v = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (any >> i & 1) {
          const float* p = ar + i * lda + k;
          s[i] = fmaf(p[3], v.w, fmaf(p[2], v.z, fmaf(p[1], v.y, fmaf(p[0], v.x, s[i]))));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (need >> i & 1) out[(int64_t)(m + i) * ldo + n] = s[i];
  }
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(remote));
  return v;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr), "f"(v[0]), "f"(v[1]),
      "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]),
      "f"(v[14]), "f"(v[15])
      : "memory");
}

// Pointers carry no __restrict__: `a` is what an earlier kernel of the step writes, and a load must not move before pdl_wait().
// `a_whole`: rows of `a` are whole 16-byte pieces (tma_a is made); w's are always.
template <int NT, bool CL>
__global__ void __launch_bounds__(Cfg<NT>::kThreads, Cfg<NT>::kCtasAnSm)
    gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_a, const float* a, const float* w, float* out, int M,
                       int N, int K, int64_t lda, int64_t ldw, int64_t ldo, bool a_whole, int* error) {
  using C = Cfg<NT>;
  constexpr int R = C::kRawStages;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t raws = base + C::kStages * C::kStage;                              // [R][128 + NT][32] float32, behind the planes
  float* red = reinterpret_cast<float*>(smem_raw + (base - raw));          // [NT][128], over the stages (CL)
  __shared__ __align__(8) uint64_t bars[2 * C::kStages + 4 + 2 * R];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, redo_flag;       // redo: an output of this CTA is not finite
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (C::kStages + s); };
  auto acc_full = [&](int s) { return bar0 + 8u * (2 * C::kStages + s); };
  auto acc_empty = [&](int s) { return bar0 + 8u * (2 * C::kStages + 2 + s); };
  auto raw_full = [&](int s) { return bar0 + 8u * (2 * C::kStages + 4 + s); };
  auto raw_empty = [&](int s) { return bar0 + 8u * (2 * C::kStages + 4 + R + s); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = C::kThreads / 32 - 3, kIssuer = kProducer + 1;      // two issuers
  if (threadIdx.x == 0) {
    abort_flag = 0;
    redo_flag = 0;
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(full(s), 4);
      mbar_init(empty(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), C::kEpilogueWarps);
    }
    for (int s = 0; s < R; ++s) {
      mbar_init(raw_full(s), 1);
      mbar_init(raw_empty(s), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kIssuer) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"((uint32_t)__cvta_generic_to_shared(&tmem_slot)), "r"(C::kTmem)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  pdl_launch_dependents();
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();
  const uint32_t tmem = tmem_slot;
  volatile int* abortp = &abort_flag;
  // the tiles of this CTA (m fastest, so that neighbouring CTAs read the same rows of w) and its blocks of k
  const int m_tiles = (M + NT - 1) / NT, tiles = m_tiles * ((N + kWRows - 1) / kWRows), blocks = (K + kBlock - 1) / kBlock;
  const int first = CL ? blockIdx.x / kParts : blockIdx.x, step = CL ? tiles : gridDim.x, rank = CL ? blockIdx.x % kParts : 0;
  auto part_end = [&](int p) { return (int)((long long)blocks * (p + 1) / kParts); };
  const int kb0 = CL ? (int)((long long)blocks * rank / kParts) : 0, kb1 = CL ? part_end(rank) : blocks;

  if (warp == kProducer) {
    if (lane == 0) {
      const uint32_t bytes = a_whole ? C::kRawStage : kWRaw;
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = first; t < tiles && ok; t += step) {
        const int m0 = t % m_tiles * NT, n0 = t / m_tiles * kWRows;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!(ok = mbar_wait_limited(raw_empty(s), phase ^ 1u, abortp, 1, error))) break;
          mbar_expect_tx(raw_full(s), bytes);
          tma_load_2d(raws + s * C::kRawStage, &tma_w, raw_full(s), kb * kBlock, n0);
          if (a_whole) tma_load_2d(raws + s * C::kRawStage + kWRaw, &tma_a, raw_full(s), kb * kBlock, m0);
          if (++s == R) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp < kConverters / 32) {
    // w: row 32 (warp % 4) + lane, which is its lane of tensor memory. Its 16-byte pieces lie swizzled by the copy.
    // a: piece i is row r0 + 16 i, numbers 4 c .. 4 c + 3 of the block; all rows of a thread are alike modulo 8.
    const int tid = threadIdx.x & 127, group = threadIdx.x >> 7, r0 = tid >> 3, c = tid & 7;
    const uint32_t spot = (uint32_t)r0 * 64u + ((uint32_t)((c >> 1) ^ ((r0 >> 1) & 3)) << 4) + (uint32_t)(c & 1) * 8u;
    const uint32_t wdst = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::kW;
    int it = 0;
    bool ok = true;
    for (int t = first; t < tiles && ok; t += step) {
      const int m0 = t % m_tiles * NT;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % C::kStages, rs = it % R;
        if ((it & 1) != group) continue;
        if (!(ok = mbar_wait_limited(raw_full(rs), (uint32_t)(it / R) & 1u, abortp, 3, error))) break;
        if (!(ok = mbar_wait_limited(empty(s), ((uint32_t)(it / C::kStages) & 1u) ^ 1u, abortp, 2, error))) break;
        tcgen05_fence_after();
        const uint32_t src = raws + rs * C::kRawStage, dst = base + s * C::kStage + spot;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t planes[3][8];
          float4 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = load16(src + tid * 128u + ((uint32_t)((h * 4 + i) ^ (tid & 7)) << 4));
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t p[3][2];
            split4(v[i], p);
#pragma unroll
            for (int part = 0; part < 3; ++part) {
              planes[part][2 * i] = p[part][0];
              planes[part][2 * i + 1] = p[part][1];
            }
          }
#pragma unroll
          for (int part = 0; part < 3; ++part) tmem_store8(wdst + s * kWColumns + part * (kBlock / 2) + h * 8, planes[part]);
        }
        constexpr int kAtOnce = NT % 64 == 0 ? 4 : (NT % 32 == 0 ? 2 : 1);      // loads ahead of the first split: they and the stores keep their order
#pragma unroll
        for (int i0 = 0; i0 < NT / 16; i0 += kAtOnce) {
          float4 v[kAtOnce];
#pragma unroll
          for (int i = 0; i < kAtOnce; ++i)
            v[i] = a_whole ? load16(src + kWRaw + tid * 16u + (i0 + i) * 2048u) : fetch4(a, lda, m0 + r0 + 16 * (i0 + i), M, kb * kBlock + 4 * c, K);
#pragma unroll
          for (int i = 0; i < kAtOnce; ++i) {
            uint32_t p[3][2];
            split4(v[i], p);
#pragma unroll
            for (int part = 0; part < 3; ++part) store8(dst + part * C::kPlane + (i0 + i) * 1024u, p[part][0], p[part][1]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        tcgen05_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(full(s));
          mbar_arrive(raw_empty(rs));
        }
      }
    }
  } else if (warp >= kIssuer) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(kWRows, NT);
      int it = 0;
      bool ok = true;
      for (int t = first; t < tiles && ok; t += step) {
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % C::kStages, d = it & 1;
          if (d != warp - kIssuer) continue;
          if (!(ok = mbar_wait_limited(acc_empty(d), ((uint32_t)(it >> 1) & 1u) ^ 1u, abortp, 4, error))) break;
          if (!(ok = mbar_wait_limited(full(s), (uint32_t)(it / C::kStages) & 1u, abortp, 5, error))) break;
          tcgen05_fence_after();
          const uint32_t wp = tmem + C::kW + s * kWColumns, ap = base + s * C::kStage, acc = tmem + (uint32_t)d * NT;
          // the parts of w and of a that meet, the smallest products first
          constexpr int kOfW[6] = {2, 0, 1, 1, 0, 0}, kOfA[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
          for (int p = 0; p < 6; ++p) {
            const uint64_t da = desc_k_major_sw64(ap + kOfA[p] * C::kPlane);
#pragma unroll
            for (int j = 0; j < kBlock / 16; ++j)
              tcgen05_mma_f16_ts(acc, wp + kOfW[p] * (kBlock / 2) + j * 8, da + (uint64_t)(2 * j), idesc, p > 0 || j > 0 ? 1u : 0u);
          }
          tcgen05_commit(empty(s));
          tcgen05_commit(acc_full(d));
        }
      }
    }
  } else {
    const int ew = warp - kConverters / 32, group = warp & 3, col0 = ew / 4 * C::kColumns, row = group * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(group * 32) << 16);
    const uint32_t sums = lanes + C::kSums + col0;
    float acc[C::kColumns];
    int it = 0;
    bool ok = true;
    for (int t = first; t < tiles && ok; t += step) {
      const int m0 = t % m_tiles * NT + col0, n = t / m_tiles * kWRows + row;
      int part = 0;
#pragma unroll
      for (int j = 0; j < C::kColumns; ++j) acc[j] = 0.f;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it & 1;
        if (!(ok = mbar_wait_limited(acc_full(s), (uint32_t)(it >> 1) & 1u, abortp, 6, error))) break;
        tcgen05_fence_after();
#pragma unroll
        for (int j = 0; j < C::kColumns; j += 16) {
          uint32_t v[16];
          tcgen05_ld_32x32b_x16(lanes + (uint32_t)s * NT + col0 + j, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[j + i] += __uint_as_float(v[i]);
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(s));
        if (!CL && kb + 1 == part_end(part)) {     // a part of k is complete: added to the ones before it
          if (part > 0) {
#pragma unroll
            for (int j = 0; j < C::kColumns; j += 16) {
              uint32_t v[16];
              tcgen05_ld_32x32b_x16(sums + j, v);
#pragma unroll
              for (int i = 0; i < 16; ++i) acc[j + i] = __uint_as_float(v[i]) + acc[j + i];
            }
          }
          if (part + 1 < kParts) {
#pragma unroll
            for (int j = 0; j < C::kColumns; j += 16) tmem_store16(sums + j, acc + j);
            tcgen05_wait_st();
#pragma unroll
            for (int j = 0; j < C::kColumns; ++j) acc[j] = 0.f;
          }
          ++part;
        }
      }
      if (!ok) break;
      if constexpr (CL) {
#pragma unroll
        for (int j = 0; j < C::kColumns; ++j) red[(col0 + j) * kWRows + row] = acc[j];
      } else {
        if (n < N) {
#pragma unroll
          for (int j = 0; j < C::kColumns; ++j) {
            if (m0 + j < M) {
              if (!finite(acc[j])) redo_flag = 1;
              out[(int64_t)(m0 + j) * ldo + n] = acc[j] * kUnscale;
            }
          }
        }
      }
    }
  }
  __syncwarp();
  if constexpr (CL) {
    // every thread of every CTA of the cluster comes here, whatever its waits returned
    cluster_sync_all();
    if (!*abortp && first < tiles) {
      // CTA r adds up and writes 32 of the tile's rows of w: a warp a row of a at a time
      const int m0 = first % m_tiles * NT, n = first / m_tiles * kWRows + rank * 32 + lane;
      for (int m = warp; m < NT && m0 + m < M; m += C::kThreads / 32) {
        const uint32_t at = base + (uint32_t)(m * kWRows + rank * 32 + lane) * 4u;
        float v[kParts];
#pragma unroll
        for (int p = 0; p < kParts; ++p) v[p] = ld_cluster_f32(at, (uint32_t)p);
        float sum = v[0];
#pragma unroll
        for (int p = 1; p < kParts; ++p) sum += v[p];
        if (n < N) {
          if (!finite(sum)) redo_flag = 1;
          out[(int64_t)(m0 + m) * ldo + n] = sum * kUnscale;
        }
      }
    }
    cluster_sync_all();      // nobody leaves while another CTA still reads its shared memory
  }
  if (*abortp) {             // copies and products in flight have ended when the shared memory is given back
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) __nanosleep(256);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == kIssuer) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(C::kTmem) : "memory");
  }
  if (redo_flag && !*abortp) {
    for (int t = first; t < tiles; t += step) {
      const int m0 = t % m_tiles * NT, n0 = t / m_tiles * kWRows + (CL ? rank * (kWRows / kParts) : 0);
      if (n0 < N) redo_not_finite<C::kThreads>(a, w, out, m0, min(m0 + NT, M), n0, min(n0 + (CL ? kWRows / kParts : kWRows), N), K, lda, ldw, ldo);
    }
  }
}

struct Args {
  const float *a, *w;
  float* out;
  int m, n, k;
  int64_t lda, ldw, ldo;
  cudaStream_t stream;
};

// A [rows, k] float32 matrix with row stride ld as a tensor map with boxes of box_rows x 32.
static int make_map(CUtensorMap* map, const float* p, int rows, int k, int64_t ld, int box_rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return fail(ROOST_ERR_CUDA, "gemm_f32_tc: the driver does not export cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  const cuuint32_t box[2] = {(cuuint32_t)kBlock, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(p), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ROOST_ERR_CUDA, "gemm_f32_tc: cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return ROOST_OK;
}

template <int NT, bool CL>
static int launch(const Args& g, int sms) {
  using C = Cfg<NT>;
  auto kernel = gemm_f32_tc_kernel<NT, CL>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
  if (e != cudaSuccess) return fail(ROOST_ERR_CUDA, std::string("gemm_f32_tc: ") + cudaGetErrorString(e));
  int* error = gemm_tcgen05_error_address();
  if (!error) return fail(ROOST_ERR_CUDA, "gemm_f32_tc: the error word has no device address");
  const bool whole = g.lda % 4 == 0 && (uintptr_t)g.a % 16 == 0;
  CUtensorMap mw, ma;
  int rc = make_map(&mw, g.w, g.n, g.k, g.ldw, kWRows, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != ROOST_OK) return rc;
  ma = mw;
  if (whole && (rc = make_map(&ma, g.a, g.m, g.k, g.lda, NT, CU_TENSOR_MAP_SWIZZLE_NONE)) != ROOST_OK) return rc;
  const long long tiles = (long long)((g.m + NT - 1) / NT) * ((g.n + kWRows - 1) / kWRows), resident = (long long)sms * C::kCtasAnSm;
  const unsigned grid = (unsigned)(CL ? tiles * kParts : (tiles < resident ? tiles : resident));
  launch_kernel_cluster(kernel, dim3(grid), dim3(C::kThreads), C::kSmem, g.stream, CL ? kParts : 1, mw, ma, g.a, g.w, g.out, g.m, g.n, g.k, g.lda, g.ldw, g.ldo,
                        whole, error);
  return check_launch("gemm_f32_tc");
}

// Rows of `a` a tile, the cycles of an SM that a block of k of such a tile took (on a matrix of many rounds, 151,936 x 1,024, by 16 to 96 rows; 12 products of 128 x 96 x 16
// or fewer cannot take less than 770, whatever NT is), and how many CTAs of clusters an SM may be given in turn: they are not persistent. Narrow tiles
// start and end quickly: a row by 20,000 x 4,096 104 us in whole tiles, 78 in clusters; by 40,000 x 4,096 154 and 133. Wider ones do not: 512 rows by 4,096 x 4,096 152 us
// in whole tiles, 190 in clusters. 128 rows leave tensor memory for two stages of planes, which wait for one another, and are more than twice as slow as 64; they serve
// where 64 would need a second round of clusters, and only in clusters (in whole tiles 64 rows are expected to be quicker for any k that is taken).
struct Form {
  int rows;
  double cycles;
  int clusters;
};
constexpr Form kForms[] = {{16, 760, 16}, {32, 930, 4}, {64, 1250, 4}, {96, 1540, 4}, {128, 2700, 4}};

// What a product is expected to take: rounds of tiles on an SM, blocks of k, and what starts and ends a tile.
static double expected(const Form& f, bool cl, int m, int n, int k, int sms) {
  const long long tiles = (long long)((m + f.rows - 1) / f.rows) * ((n + kWRows - 1) / kWRows) * (cl ? kParts : 1), blocks = (k + kBlock - 1) / kBlock;
  const double rounds = (double)((tiles + sms - 1) / sms);
  return rounds * ((double)(cl ? (blocks + kParts - 1) / kParts : blocks) * f.cycles + (cl ? 5000.0 : 3000.0));
}

}  // namespace f32tc

// The rule on w alone that decides between the two products: an output's bits may not depend on how many rows are asked for together.
// Below 512 k the chain of FFMAs is short: not measured against, and no model's projections. Vocabulary-sized heads, of which a step wants a few rows, stay
// with the FFMAs, which read the weights at 5.2 TB/s there (3 x 151,936 x 1,024: 118 us, 130 here, where a block's 12 products take 770 cycles however few
// their rows). In between, us here (by FFMAs), for 1, 16 and 512 rows: 1,024 x 3,072 16 (50), 16 (50), 35 (185); 4,096 x 4,096 25 (72), 25 (76), 152 (448); 12,288 x 1,024
// 23 (25), 23 (37), 103 (336); 24,576 x 4,096 94 (92), 95 (160), 703 (2,383); 40,000 x 1,024 47 (39), 47 (74), 317 (936); 50,304 x 4,096 154 (170), 156 (324), 1,525 (4,742).
// A single row by 16,000 to 50,000 of a short k is the one shape that the FFMAs take less time for; the rows of a step, whose bits may not differ, are worth more.
bool gemm_f32_tc_takes(const void* w, int n, int k, int64_t ldw) {
  return k >= 512 && n < 65536 && k % 4 == 0 && ldw % 4 == 0 && (uintptr_t)w % 16 == 0;
}

int launch_gemm_f32_tc(const float* a, const float* w, float* out, int m, int n, int k, int64_t lda, int64_t ldw, int64_t ldo, cudaStream_t stream) {
  using namespace f32tc;
  const int count = processors();
  const Args g = {a, w, out, m, n, k, lda, ldw, ldo, stream};
  int rows = 0;
  bool cl = false;
  double least = 0;
  for (const Form& f : kForms) {
    for (int c = 0; c < 2; ++c) {
      const long long tiles = (long long)((m + f.rows - 1) / f.rows) * ((n + kWRows - 1) / kWRows);
      if (c ? tiles * kParts > (long long)f.clusters * count : f.rows == 128) continue;
      const double t = expected(f, c != 0, m, n, k, count);
      if (rows == 0 || t < least) {
        least = t;
        rows = f.rows;
        cl = c != 0;
      }
    }
  }
  switch (rows) {
    case 16: return cl ? launch<16, true>(g, count) : launch<16, false>(g, count);
    case 32: return cl ? launch<32, true>(g, count) : launch<32, false>(g, count);
    case 64: return cl ? launch<64, true>(g, count) : launch<64, false>(g, count);
    case 96: return cl ? launch<96, true>(g, count) : launch<96, false>(g, count);
    default: return launch<128, true>(g, count);
  }
}

}  // namespace roost
