// Attention of a decode step's few rows over short contexts (one query token a row), for bfloat16 heads of 64 or 128 numbers over a paged cache: grouped-query
// softmax attention (src/Starlings.Roost.Ops/CpuOps.cs:181-298) or, SIGMOID, weights sigmoid((q . k) scale - slope[h] (p - j) + bias[h]) that nothing
// divides, with the output gate of sigmoid_attention.cu. Rows, key/value heads and keys are dealt so that a warp has one or two blocks of 16 keys: a
// cluster of CTAs a (row, key/value head), eight warps a CTA, block b of the row's keys to warp b % (8 CTAs).
//
// Nothing passes through shared memory on its way to the products (mma.sync m16n8k16, the up to 16 heads of the group as the rows): a lane reads 16-byte
// pieces of keys and values that are operands as they lie. For the scores a lane's eight numbers of a key are two products' k in the order in which the
// query's pieces lie too; for the second product a lane's eight numbers of four keys are eight products' columns, packed in pairs of keys. The weights enter
// it as the sum of two (softmax) or three (SIGMOID: all their 24 bits) bfloat16 numbers. Warps and CTAs combine their (sum, maximum, denominator) in
// order through shared and distributed shared memory: no merge kernel.
//
// What bounds it: latency, one trip to memory for the keys behind one for the table's page. The kernel's instructions run once without keys ahead of the wait
// for the kernel in front (see gemm_rows.cu).
// 1 row x 1,000 keys, 16 heads of 128 over 8: 5.2 us behind the rotation, 7.4 to 8 by the copy-engine kernel; SIGMOID, 8 rows x 1,000 keys, 16 heads of 64 over
// 4: 7.5 us, 22 with the two kernels of sigmoid_attention.cu.
#include "mma.cuh"

namespace roost {

constexpr int kArWarps = 8;
constexpr int kArMaxSplits = 8;

struct AttentionRows {
  const __nv_bfloat16 *q, *k_base, *v_base, *gate;
  __nv_bfloat16* out;
  const int32_t *lens, *token_row, *kv_indptr, *kv_indices;      // lens: keys of a row, or (SIGMOID) the positions of the tokens
  const float *slopes, *head_bias;
  int64_t ld_gate;
  int entry, q_heads, kv_heads, page_size, page_shift;
  float scale;                                                   // softmax: times log2(e)
};

__device__ __forceinline__ uint4 ar_load16(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ar_word(const uint4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }
__device__ __forceinline__ float ar_remote(const float* p, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(remote));
  return v;
}
__device__ __forceinline__ void ar_cluster_sync() { asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory"); }
// What scores are taken relative to: their maximum, or 0 where there was none (no key, or none but -inf or NaN). Every weight is then exp2f of a difference: 0 for
// -inf, NaN for a NaN score, which so reaches the sums, the denominator and the output whatever the maximum is.
__device__ __forceinline__ float ar_base(float top) { return top == -INFINITY ? 0.f : top; }
// Two bfloat16 numbers with infinities (and NaN) as the largest finite number: what the weights' small parts, which may be zero or negative, are multiplied with. The
// large part meets the value itself.
__device__ __forceinline__ uint32_t ar_finite(uint32_t v) {
  const uint32_t most = 0x7F7F7F7Fu, least = 0xFF7FFF7Fu;
  const __nv_bfloat162 x = __hmax2(__hmin2(*reinterpret_cast<const __nv_bfloat162*>(&v), *reinterpret_cast<const __nv_bfloat162*>(&most)),
                                   *reinterpret_cast<const __nv_bfloat162*>(&least));
  return *reinterpret_cast<const uint32_t*>(&x);
}

template <int D, bool SIGMOID>
__global__ void __launch_bounds__(kArWarps * 32, 1) attention_rows_kernel(const AttentionRows a) {
  constexpr int DB = D / 32, U = D / 64, NT = D / 8, LD = D + 4, PARTS = SIGMOID ? 3 : 2;
  extern __shared__ __align__(16) float sm[];
  const int group = a.q_heads / a.kv_heads;
  float* so = sm;                                          // [warps][group][LD]: a warp's sums
  float* sml = so + kArWarps * group * LD;                 // [warps][group][2]: its maxima and denominators
  float* bo = sml + kArWarps * group * 2;                  // [group][D]: the CTA's sums
  float* bml = bo + group * D;                             // [group][2]
  const int rank = blockIdx.x, splits = gridDim.x, kvh = blockIdx.y, t = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  pdl_launch_dependents();
  const int len = SIGMOID ? a.lens[t] + 1 : a.lens[t];
  if (len <= 0) {                                          // a padding row: nothing is written
    pdl_wait();
    return;
  }
  const int32_t* pages = a.kv_indices + a.kv_indptr[a.token_row ? a.token_row[t] : t];
  const int blocks = (len + 15) >> 4, stride = splits * kArWarps, first = rank * kArWarps + warp;
  float slope[2] = {0.f, 0.f}, bias[2] = {0.f, 0.f};
  if constexpr (SIGMOID) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (g + 8 * r < group) {
        slope[r] = a.slopes[kvh * group + g + 8 * r];
        bias[r] = a.head_bias[kvh * group + g + 8 * r];
      }
    }
  }
  int entry_of = first + lane * stride < blocks ? pages[(first + lane * stride) * 16 >> a.page_shift] : 0;       // lane i: the page of the warp's i-th block
  float acc[NT][4], m[2], l[2];
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (pass) pdl_wait();
    uint32_t qa[DB][2][4];
#pragma unroll
    for (int b = 0; b < DB; ++b) {
      uint4 x[2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
        x[r] = pass && g + 8 * r < group ? ar_load16(a.q + ((size_t)t * a.q_heads + kvh * group + g + 8 * r) * D + 32 * b + 8 * c) : make_uint4(0, 0, 0, 0);
      qa[b][0][0] = x[0].x; qa[b][0][1] = x[1].x; qa[b][0][2] = x[0].y; qa[b][0][3] = x[1].y;
      qa[b][1][0] = x[0].z; qa[b][1][1] = x[1].z; qa[b][1][2] = x[0].w; qa[b][1][3] = x[1].w;
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
    for (int i = 0, blk = first; pass ? blk < blocks : i == 0; ++i, blk += stride) {
      // (a warp has at most eight blocks of the keys that kv_cap bounds; only rows longer than it was told come here)
      if (i > 0 && (i & 31) == 0) entry_of = blk + lane * stride < blocks ? pages[(blk + lane * stride) * 16 >> a.page_shift] : 0;
      const int page = __shfl_sync(0xffffffffu, entry_of, i & 31), key0 = blk * 16, seen = pass ? len - key0 : 0;       // the block's keys that there are
      const size_t at = (((size_t)page * a.kv_heads + kvh) * a.page_size + (key0 & (a.page_size - 1))) * a.entry;
      uint4 kx[2][DB], vx[4][U];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int b = 0; b < DB; ++b)
          kx[h][b] = 8 * h + g < seen ? ar_load16(a.k_base + at + (size_t)(8 * h + g) * a.entry + 32 * b + 8 * c) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int key = 2 * c + (x & 1) + 8 * (x >> 1);
#pragma unroll
        for (int u = 0; u < U; ++u)
          vx[x][u] = key < seen ? ar_load16(a.v_base + at + (size_t)key * a.entry + 64 * u + 8 * g) : make_uint4(0, 0, 0, 0);
      }
      float s[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int e = 0; e < 4; ++e) s[h][e] = 0.f;
#pragma unroll
        for (int b = 0; b < DB; ++b) {
          mma_bf16(s[h], qa[b][0], kx[h][b].x, kx[h][b].y);
          mma_bf16(s[h], qa[b][1], kx[h][b].z, kx[h][b].w);
        }
      }
      // s[h][2 r + e]: head g + 8 r, key 8 h + 2 c + e of the block
      if constexpr (SIGMOID) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = 8 * h + 2 * c + (e & 1);
            s[h][e] = key < seen ? sigmoid_f(s[h][e] * a.scale - slope[e >> 1] * (float)(len - 1 - key0 - key) + bias[e >> 1]) : 0.f;
          }
      } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float top = -INFINITY;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              s[h][2 * r + e] = 8 * h + 2 * c + e < seen ? s[h][2 * r + e] * a.scale : -INFINITY;
              top = fmaxf(top, s[h][2 * r + e]);
            }
          top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
          top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
          const float now = fmaxf(m[r], top), base = ar_base(now), fade = exp2f(m[r] - base);
          float sum = 0.f;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              s[h][2 * r + e] = exp2f(s[h][2 * r + e] - base);
              sum += s[h][2 * r + e];
            }
          l[r] = l[r] * fade + sum;               // of this lane's keys; the row's lanes are added at the end
          m[r] = now;
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            acc[n][2 * r] *= fade;
            acc[n][2 * r + 1] *= fade;
          }
        }
      }
      // the weights as operands of 16 heads x 16 keys, the small parts first
      uint32_t p[PARTS][4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float lo = s[x >> 1][2 * (x & 1)], hi = s[x >> 1][2 * (x & 1) + 1];
#pragma unroll
        for (int part = 0; part < PARTS; ++part) {
          const __nv_bfloat162 w = __floats2bfloat162_rn(lo, hi);
          p[PARTS - 1 - part][x] = *reinterpret_cast<const uint32_t*>(&w);
          lo -= __low2float(w);
          hi -= __high2float(w);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t pick = j & 1 ? 0x7632 : 0x5410;
          const uint32_t b0 = __byte_perm(ar_word(vx[0][u], j >> 1), ar_word(vx[1][u], j >> 1), pick);
          const uint32_t b1 = __byte_perm(ar_word(vx[2][u], j >> 1), ar_word(vx[3][u], j >> 1), pick);
          const uint32_t f0 = ar_finite(b0), f1 = ar_finite(b1);
#pragma unroll
          for (int part = 0; part < PARTS - 1; ++part) mma_bf16(acc[u * 8 + j], p[part], f0, f1);
          mma_bf16(acc[u * 8 + j], p[PARTS - 1], b0, b1);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    // acc[8 u + j][2 r + e]: head g + 8 r, number 64 u + 8 (2 c + e) + j
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int h = g + 8 * r;
      if (h >= group) continue;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) so[(warp * group + h) * LD + (n >> 3) * 64 + 8 * (2 * c + e) + (n & 7)] = acc[n][2 * r + e];
      if (c == 0) {
        sml[(warp * group + h) * 2] = m[r];
        sml[(warp * group + h) * 2 + 1] = l[r];
      }
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < group * D; idx += kArWarps * 32) {
      const int h = idx / D, d = idx % D;
      float top = -INFINITY, den = 0.f, sum = 0.f;
      if constexpr (!SIGMOID) {
#pragma unroll
        for (int w = 0; w < kArWarps; ++w) top = fmaxf(top, sml[(w * group + h) * 2]);
      }
      const float base = ar_base(top);
#pragma unroll
      for (int w = 0; w < kArWarps; ++w) {
        const float f = SIGMOID ? 1.f : exp2f(sml[(w * group + h) * 2] - base);
        sum += so[(w * group + h) * LD + d] * f;
        den += sml[(w * group + h) * 2 + 1] * f;
      }
      bo[h * D + d] = sum;
      if (d == 0) {
        bml[h * 2] = top;
        bml[h * 2 + 1] = den;
      }
    }
    if (!pass) {
      __syncthreads();       // the sums' room is free again
      continue;
    }
    if (splits > 1) ar_cluster_sync();
    else __syncthreads();
    for (int idx = rank * kArWarps * 32 + threadIdx.x; idx < group * D; idx += splits * kArWarps * 32) {
      const int h = idx / D, d = idx % D;
      float sum = 0.f, den = 0.f, top = -INFINITY, part[kArMaxSplits], pm[kArMaxSplits], pl[kArMaxSplits];
#pragma unroll
      for (int z = 0; z < kArMaxSplits; ++z) {
        part[z] = z < splits ? ar_remote(bo + h * D + d, z) : 0.f;
        pm[z] = !SIGMOID && z < splits ? ar_remote(bml + h * 2, z) : -INFINITY;
        pl[z] = !SIGMOID && z < splits ? ar_remote(bml + h * 2 + 1, z) : 0.f;
        top = fmaxf(top, pm[z]);
      }
      const float base = ar_base(top);
#pragma unroll
      for (int z = 0; z < kArMaxSplits; ++z) {
        const float f = SIGMOID ? 1.f : exp2f(pm[z] - base);
        sum += part[z] * f;
        den += pl[z] * f;
      }
      const size_t head = (size_t)t * a.q_heads + kvh * group + h;
      float y = sum;
      if constexpr (SIGMOID) {
        if (a.gate) y *= sigmoid_f(to_float(a.gate[(size_t)t * a.ld_gate + (size_t)(kvh * group + h) * D + d]));
      } else {
        y = den > 0.f ? sum / den : sum * 0.f;        // no weight at all: 0; a denominator of NaN: NaN, as the sum
      }
      a.out[head * D + d] = from_float<__nv_bfloat16>(y);
    }
    if (splits > 1) ar_cluster_sync();       // nobody leaves while another CTA still reads its shared memory
  }
}

// CTAs a (row, key/value head): as many as run at once (one a processor), at most one a 128 keys (a warp a block of 16). Clusters of eight need eight free
// processors of one group, which the kernels around this one leave for few: sixteen of them were slower than sixteen of four (2 rows of Qwen3 0.6B: 220 us
// a step of six layers, 196 in clusters of four).
static int rows_splits(int tokens, int kv_heads, int kv_cap) {
  const int sms = processors();
  int splits = 1;
  while (splits < kArMaxSplits && (long long)tokens * kv_heads * splits * 2 <= (splits * 2 == 8 ? sms / 2 : sms) && splits * 128 < kv_cap) splits *= 2;
  return splits;
}

}  // namespace roost

using namespace roost;

// Served where a warp has few blocks of keys: `kv_cap` is the bound on the rows' keys (of the captured step).
extern "C" int roost_attention_rows_supported(int tokens, int q_heads, int kv_heads, int head_dim, int page_size, int kv_cap, int sigmoid) {
  if (tokens < 1 || kv_heads < 1 || q_heads % kv_heads != 0 || q_heads / kv_heads > 16 || (head_dim != 64 && head_dim != 128)) return 0;
  if (page_size < 16 || (page_size & (page_size - 1)) != 0 || kv_cap < 1 || kv_heads > 65535 || tokens > 65535) return 0;
  const int blocks = (kv_cap + 15) / 16, each = rows_splits(tokens, kv_heads, kv_cap) * kArWarps, turns = (blocks + each - 1) / each;
  return (long long)tokens * kv_heads <= processors() && turns <= (sigmoid ? 8 : 2);
}

extern "C" int roost_attention_rows(const void* q, void* out, const void* k_base, const void* v_base, int entry, const int32_t* lens, const int32_t* token_row,
                                    const int32_t* kv_indptr, const int32_t* kv_indices, int tokens, int q_heads, int kv_heads, int head_dim, int page_size,
                                    float scale, int kv_cap, int sigmoid, const float* slopes, const float* head_bias, const void* gate, int64_t ld_gate,
                                    roost_stream_t stream) {
  ROOST_REQUIRE(q && out && k_base && v_base && lens && kv_indptr && kv_indices, "attention_rows: a pointer is null");
  ROOST_REQUIRE(!sigmoid || (slopes && head_bias && token_row), "attention_rows: sigmoid weights need slopes, biases and the tokens' rows");
  ROOST_REQUIRE(roost_attention_rows_supported(tokens, q_heads, kv_heads, head_dim, page_size, kv_cap, sigmoid), "attention_rows: sizes that it does not serve");
  ROOST_REQUIRE(((uintptr_t)q | (uintptr_t)k_base | (uintptr_t)v_base) % 16 == 0 && entry >= head_dim && entry % 8 == 0,
                "attention_rows: queries and cache entries start on 16 bytes");
  int shift = 0;
  while ((1 << shift) < page_size) ++shift;
  const AttentionRows a = {(const __nv_bfloat16*)q, (const __nv_bfloat16*)k_base, (const __nv_bfloat16*)v_base, (const __nv_bfloat16*)gate, (__nv_bfloat16*)out, lens, token_row,
                           kv_indptr, kv_indices, slopes, head_bias, ld_gate, entry, q_heads, kv_heads, page_size, shift, sigmoid ? scale : scale * 1.4426950408889634f};
  const int splits = rows_splits(tokens, kv_heads, kv_cap), group = q_heads / kv_heads;
  const size_t smem = ((size_t)kArWarps * group * (head_dim + 4 + 2) + (size_t)group * (head_dim + 2)) * sizeof(float);
  auto kernel = head_dim == 64 ? (sigmoid ? attention_rows_kernel<64, true> : attention_rows_kernel<64, false>)
                               : (sigmoid ? attention_rows_kernel<128, true> : attention_rows_kernel<128, false>);
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  launch_kernel_cluster(kernel, dim3(splits, kv_heads, tokens), dim3(kArWarps * 32), smem, (cudaStream_t)stream, splits, a);
  return check_launch("attention_rows");
}
