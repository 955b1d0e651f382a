// Causal grouped-query attention over the paged cache in 32-bit arithmetic: the path of the float32 model and
// of head sizes no tensor-core kernel serves.
//
// Definition: src/Starlings.Roost.Ops/CpuOps.cs:181-298. A query at absolute position p sees keys
// max(0, p - window + 1) .. p (no window: from 0); query head h reads key/value head h / (q_heads / kv_heads);
// score = q.k * scale; softmax with a running maximum; output = sum p_j v_j / sum p_j.
//
// Keys are visited in tiles of 32 at absolute positions that are multiples of 32, and what one query does with a tile (its
// scores, the tile's maximum, the sum of its weights, the output's sums) has one order, so the order of every sum depends
// on the query's position alone: the same token gives the same bits whether it arrives in a whole prompt, a portion or a
// single decode step, and whatever else is in the batch. Two forms, bit for bit alike:
//   paged_attention_generic_kernel (any sizes): a block per (query token, key/value head, group of 4 query heads), a
//     warp a query head, a lane a key.
//   paged_attention_rows_kernel (heads of up to 128 numbers in whole pieces of four, groups of up to 32): a block takes
//     up to 32 (token, head) rows of consecutive tokens of one request, so a key tile is read once for all of them, and
//     makes scores and outputs in register tiles. The next tile arrives by cp.async meanwhile. It is bound by reads of
//     shared memory; a prompt of 510 tokens, 16 heads of 128 over 8: 374 us a layer with the form above, 140 here.
#include "common.cuh"

namespace roost {

constexpr int kTile = 32;
constexpr int kWarps = 4;
constexpr int kMaxHeadDim = 512;

template <typename T>
__global__ void paged_attention_generic_kernel(const T* __restrict__ q, T* __restrict__ out, const T* __restrict__ k_pool,
                                               const T* __restrict__ v_pool, const int32_t* __restrict__ positions,
                                               const int32_t* __restrict__ token_row, const int32_t* __restrict__ kv_indptr,
                                               const int32_t* __restrict__ kv_indices, int q_heads, int kv_heads, int head_dim,
                                               int page_size, float scale, int window) {
  extern __shared__ float smem[];
  const int d = head_dim;
  const int dk = d + 1;                       // padded key rows: a lane per key reads without bank conflicts
  float* ks = smem;                           // [kTile][d + 1]
  float* vs = ks + kTile * dk;                // [kTile][d]
  float* qs = vs + kTile * d;                 // [kWarps][d]
  float* ps = qs + kWarps * d;                // [kWarps][kTile]

  const int t = blockIdx.x;
  const int kvh = blockIdx.y;
  const int group = q_heads / kv_heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = blockIdx.z * kWarps + warp;   // head within the group
  const bool active = g < group;
  const int h = kvh * group + g;

  const int pos = positions[t];
  const int b = token_row[t];
  const int32_t* pages = kv_indices + kv_indptr[b];
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;

  if (active) {
    const T* qv = q + ((size_t)t * q_heads + h) * d;
    for (int i = lane; i < d; i += 32) qs[warp * d + i] = to_float(qv[i]);
  }

  float m = -INFINITY, l = 0.f;
  float o[kMaxHeadDim / 32];
#pragma unroll
  for (int i = 0; i < kMaxHeadDim / 32; ++i) o[i] = 0.f;

  for (int j0 = (lo / kTile) * kTile; j0 <= pos; j0 += kTile) {
    __syncthreads();  // the previous tile has been consumed (and qs is written, the first time)
    // load the tile: keys j0 .. j0+31 that are visible
    for (int r = warp; r < kTile; r += kWarps) {
      const int j = j0 + r;
      if (j >= lo && j <= pos) {
        const int page = pages[j / page_size];
        const size_t base = (((size_t)page * kv_heads + kvh) * page_size + (j % page_size)) * d;
        for (int i = lane; i < d; i += 32) {
          ks[r * dk + i] = to_float(k_pool[base + i]);
          vs[r * d + i] = to_float(v_pool[base + i]);
        }
      } else {
        for (int i = lane; i < d; i += 32) {
          ks[r * dk + i] = 0.f;
          vs[r * d + i] = 0.f;
        }
      }
    }
    __syncthreads();
    if (active) {
      const int j = j0 + lane;
      const bool vis = j >= lo && j <= pos;
      float s = 0.f;
      const float* kr = ks + lane * dk;
      const float* qr = qs + warp * d;
      for (int i = 0; i < d; ++i) s = fmaf(qr[i], kr[i], s);
      s = vis ? s * scale : -INFINITY;
      const float m_new = fmaxf(m, warp_max(s));  // the tile holds at least one visible key
      const float p = vis ? expf(s - m_new) : 0.f;
      const float corr = expf(m - m_new);          // 0 on the first tile (m = -inf)
      l = l * corr + warp_sum(p);
      m = m_new;
      ps[warp * kTile + lane] = p;
      __syncwarp();
      const float* pr = ps + warp * kTile;
#pragma unroll
      for (int c = 0; c < kMaxHeadDim / 32; ++c) {
        const int i = c * 32 + lane;
        if (i < d) {
          float acc = o[c] * corr;
          for (int r = 0; r < kTile; ++r) acc = fmaf(pr[r], vs[r * d + i], acc);
          o[c] = acc;
        }
      }
      __syncwarp();
    }
  }
  if (active) {
    T* ov = out + ((size_t)t * q_heads + h) * d;
    const float inv = l > 0.f ? 1.0f / l : 0.f;
#pragma unroll
    for (int c = 0; c < kMaxHeadDim / 32; ++c) {
      const int i = c * 32 + lane;
      if (i < d) ov[i] = from_float<T>(o[c] * inv);
    }
  }
}

constexpr int kRows = 32;                 // (token, head) rows of a block
constexpr int kRowsLd = 132;              // floats of a staged row: heads of up to 128 numbers, eight rows' pieces in different banks

__device__ __forceinline__ void rows_copy16(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ float4 rows_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 rows_load4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}

// Block (x, kv head, z): the z-th run of tokens of one request among the tokens x * span .. x * span + span - 1. What the step's earlier
// kernels write comes through pointers without __restrict__: with it the compiler may load before pdl_wait().
template <typename T>
__global__ void __launch_bounds__(128) paged_attention_rows_kernel(const T* q, T* out, const T* k_pool, const T* v_pool, const int32_t* __restrict__ positions,
                                                                   const int32_t* __restrict__ token_row, const int32_t* __restrict__ kv_indptr,
                                                                   const int32_t* __restrict__ kv_indices, int tokens, int span, int q_heads,
                                                                   int kv_heads, int d, int page_size, float scale, int window) {
  extern __shared__ __align__(16) float smem[];
  float* kst = smem;                              // [2][kTile][kRowsLd]
  float* vst = kst + 2 * kTile * kRowsLd;         // [2][kTile][kRowsLd]
  float* qs = vst + 2 * kTile * kRowsLd;          // [kRows][kRowsLd]
  float* ps = qs + kRows * kRowsLd;               // [kRows][kTile + 4]
  float* fade = ps + kRows * (kTile + 4);         // [kRows]
  constexpr int PLD = kTile + 4;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = q_heads / kv_heads, kvh = blockIdx.y;
  pdl_launch_dependents();
  pdl_wait();
  // the run: boundaries are where the token's request is not the one before's
  const int base = blockIdx.x * span;
  const bool in = lane < span && base + lane < tokens;
  const int mine = in ? token_row[base + lane] : -1;
  const int before = __shfl_up_sync(0xffffffffu, mine, 1);
  unsigned starts = __ballot_sync(0xffffffffu, in && (lane == 0 || mine != before));
  for (int i = 0; i < (int)blockIdx.z && starts; ++i) starts &= starts - 1;
  if (starts == 0) return;
  const int s0 = __ffs(starts) - 1;
  starts &= starts - 1;
  const int s1 = starts ? __ffs(starts) - 1 : min(span, tokens - base);
  const int t0 = base + s0, count = s1 - s0, rows = count * group;
  const int32_t* pages = kv_indices + kv_indptr[token_row[t0]];
  // positions: a lane a token
  const int my_pos = lane < count ? positions[t0 + lane] : -1;
  const int last = __reduce_max_sync(0xffffffffu, my_pos);
  const int first_lo = __reduce_min_sync(0xffffffffu, lane < count ? (window > 0 ? max(0, my_pos - window + 1) : 0) : INT32_MAX);

  for (int idx = tid; idx < rows * (d / 4); idx += 128) {
    const int r = idx / (d / 4), i = idx % (d / 4) * 4;
    *reinterpret_cast<float4*>(qs + r * kRowsLd + i) = rows_load4(q + ((size_t)(t0 + r / group) * q_heads + kvh * group + r % group) * d + i);
  }
  // a warp's eight rows: scores of rows 8 w + 2 (lane / 8) + {0, 1} x keys (lane % 8) + 8 {0..3}; outputs of rows 8 w + 4 (lane / 16) + {0..3}
  // x columns 4 (lane % 16) + 64 {0, 1}
  const int row0 = warp * 8;
  float m[8], l[8];
  int pos[8], lo[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int row = row0 + r, at = __shfl_sync(0xffffffffu, my_pos, row < rows ? row / group : 0);
    pos[r] = row < rows ? at : -1;
    lo[r] = window > 0 ? max(0, pos[r] - window + 1) : 0;
    m[r] = -INFINITY;
    l[r] = 0.f;
  }
  float o[4][8];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) o[a][b] = 0.f;
  const bool live = row0 < rows;
  const int tile0 = first_lo / kTile * kTile;

  // the tile's keys and values that some row of the run may see, zeros elsewhere
  auto bring = [&](int j0, int buf) {
    const int key = j0 + lane;       // a lane looks one key's page up
    const bool wanted = key >= first_lo && key <= last;
    const int64_t slot = wanted ? ((int64_t)pages[key / page_size] * kv_heads + kvh) * page_size + key % page_size : -1;
#pragma unroll
    for (int i = 0; i < kTile / 4; ++i) {       // a warp a row of keys and of values
      const int r = warp + 4 * i;
      const int64_t from = __shfl_sync(0xffffffffu, slot, r);
      float* kd = kst + (buf * kTile + r) * kRowsLd + lane * 4;
      float* vd = vst + (buf * kTile + r) * kRowsLd + lane * 4;
      if (lane * 4 >= d) continue;
      if (from >= 0) {
        const size_t at = (size_t)from * d + lane * 4;
        if constexpr (sizeof(T) == 4) {
          rows_copy16(kd, (const float*)k_pool + at);
          rows_copy16(vd, (const float*)v_pool + at);
        } else {
          *reinterpret_cast<float4*>(kd) = rows_load4(k_pool + at);
          *reinterpret_cast<float4*>(vd) = rows_load4(v_pool + at);
        }
      } else {
        *reinterpret_cast<float4*>(kd) = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(vd) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  if (last >= 0) bring(tile0, 0);
  int buf = 0;
  for (int j0 = tile0; j0 <= last; j0 += kTile, buf ^= 1) {
    if (j0 + kTile <= last) {
      bring(j0 + kTile, buf ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();       // the tile (and, the first time, q) is there
    const float* kt = kst + buf * kTile * kRowsLd;
    const float* vt = vst + buf * kTile * kRowsLd;
    // A key that a row does not see has weight 0, and 0 times a value that is not finite must not reach the row's sums: the tile's values are
    // looked at, and where one is not finite the rows leave out what they do not see.
    bool odd = false;
#pragma unroll
    for (int i = 0; i < kTile / 4; ++i) {
      if (lane * 4 >= d) continue;
      const float4 v = *reinterpret_cast<const float4*>(vt + (warp + 4 * i) * kRowsLd + lane * 4);
      odd |= !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
    }
    if (live) {
      {
        const int ra = row0 + lane / 8 * 2, kx = lane % 8;
        float s[2][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) s[a][b] = 0.f;
        const float* qa = qs + ra * kRowsLd;
        const float* kb = kt + kx * kRowsLd;
#pragma unroll 4
        for (int i = 0; i < d; i += 4) {
          float4 x[2], y[4];
#pragma unroll
          for (int a = 0; a < 2; ++a) x[a] = *reinterpret_cast<const float4*>(qa + a * kRowsLd + i);
#pragma unroll
          for (int b = 0; b < 4; ++b) y[b] = *reinterpret_cast<const float4*>(kb + b * 8 * kRowsLd + i);
#pragma unroll
          for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) s[a][b] = fmaf(x[a].w, y[b].w, fmaf(x[a].z, y[b].z, fmaf(x[a].y, y[b].y, fmaf(x[a].x, y[b].x, s[a][b]))));
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) ps[(ra + a) * PLD + kx + 8 * b] = s[a][b];
      }
      __syncwarp();
      // a lane a key; a row that sees nothing of the tile keeps what it has
      const int j = j0 + lane;
      float z[8], corr[8], sum[8];
      bool takes[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        takes[r] = j0 <= pos[r] && j0 + kTile > lo[r];
        const float raw = ps[(row0 + r) * PLD + lane];
        z[r] = j >= lo[r] && j <= pos[r] ? raw * scale : -INFINITY;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float top = fmaxf(m[r], warp_max(z[r]));
        const float m_new = takes[r] ? top : m[r];
        z[r] = j >= lo[r] && j <= pos[r] ? expf(z[r] - m_new) : 0.f;
        corr[r] = takes[r] ? expf(m[r] - m_new) : 1.f;
        m[r] = m_new;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) sum[r] = warp_sum(z[r]);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        l[r] = takes[r] ? l[r] * corr[r] + sum[r] : l[r];
        ps[(row0 + r) * PLD + lane] = z[r];
        if (lane == 0) fade[row0 + r] = corr[r];
      }
    }
    odd = __syncthreads_or(odd);
    if (live) {
      const int ra = row0 + lane / 16 * 4, cx = lane % 16 * 4;
      if (cx < d) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float f = fade[ra + a];
#pragma unroll
          for (int b = 0; b < 8; ++b) o[a][b] *= f;
        }
        const bool right = cx + 64 < d;
        if (!odd) {
#pragma unroll 2
          for (int r = 0; r < kTile; r += 4) {
            float4 x[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) x[a] = *reinterpret_cast<const float4*>(ps + (ra + a) * PLD + r);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float4 u = *reinterpret_cast<const float4*>(vt + (r + e) * kRowsLd + cx);
              const float4 w = right ? *reinterpret_cast<const float4*>(vt + (r + e) * kRowsLd + cx + 64) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int a = 0; a < 4; ++a) {
                const float p = e == 0 ? x[a].x : (e == 1 ? x[a].y : (e == 2 ? x[a].z : x[a].w));
                o[a][0] = fmaf(p, u.x, o[a][0]);
                o[a][1] = fmaf(p, u.y, o[a][1]);
                o[a][2] = fmaf(p, u.z, o[a][2]);
                o[a][3] = fmaf(p, u.w, o[a][3]);
                o[a][4] = fmaf(p, w.x, o[a][4]);
                o[a][5] = fmaf(p, w.y, o[a][5]);
                o[a][6] = fmaf(p, w.z, o[a][6]);
                o[a][7] = fmaf(p, w.w, o[a][7]);
              }
            }
          }
        } else {
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const int row = ra + a, at = row < rows ? positions[t0 + row / group] : -1, from = window > 0 ? max(0, at - window + 1) : 0;
            for (int r = max(0, from - j0); r < kTile && j0 + r <= at; ++r) {
              const float p = ps[row * PLD + r];
              const float* v = vt + r * kRowsLd + cx;
#pragma unroll
              for (int b = 0; b < 8; ++b)
                if (b < 4 || right) o[a][b] = fmaf(p, v[b < 4 ? b : 60 + b], o[a][b]);
            }
          }
        }
      }
    }
    __syncthreads();       // the tile's buffer may be filled again
  }
  // the denominators by row, for the lanes that hold the row's outputs
#pragma unroll
  for (int r = 0; r < 8; ++r)
    if (lane == 0) fade[row0 + r] = l[r] > 0.f ? 1.0f / l[r] : 0.f;
  __syncwarp();
  const int ra = row0 + lane / 16 * 4, cx = lane % 16 * 4;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int row = ra + a;
    if (row >= rows) continue;
    const float inv = fade[row];
    T* ov = out + ((size_t)(t0 + row / group) * q_heads + kvh * group + row % group) * d;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int i = cx + (b < 4 ? b : 60 + b);
      if (i < d) ov[i] = from_float<T>(o[a][b] * inv);
    }
  }
}

}  // namespace roost

using namespace roost;

// `rows`: the requests that the step's tokens belong to (0: not known), which only chooses between the two forms.
extern "C" int roost_paged_attention_generic_rows(const void* q, void* out, const void* k_pool, const void* v_pool,
                                             const int32_t* positions, const int32_t* token_row,
                                             const int32_t* kv_indptr, const int32_t* kv_indices, int tokens,
                                             int q_heads, int kv_heads, int head_dim, int page_size, float scale,
                                             int window, int dtype, int rows, roost_stream_t stream) {
  ROOST_REQUIRE(tokens >= 0 && q_heads > 0 && kv_heads > 0 && head_dim > 0 && page_size > 0,
                "paged_attention: sizes must be positive");
  ROOST_REQUIRE(q_heads % kv_heads == 0, "paged_attention: q_heads must be a multiple of kv_heads");
  if (head_dim > kMaxHeadDim) return fail(ROOST_ERR_UNSUPPORTED, "paged_attention: head_dim beyond 512");
  if (kv_heads > 65535) return fail(ROOST_ERR_UNSUPPORTED, "paged_attention: more than 65535 key/value heads");
  if (tokens == 0) return ROOST_OK;
  const int group = q_heads / kv_heads;
  const uintptr_t piece = dtype == ROOST_F32 ? 16 : 8;      // four numbers
  // Where a block of many rows is the slower one: a prompt of a few tokens, whose one or two tiles are over before the larger block has begun (17 and 33
  // tokens, 16 heads of 128 over 8: 11.0 and 13.4 us, 7.4 and 12.5 in the other form; 15.8 and 15.4 at 64, 24 and 28 at 100), and steps that decode more tokens
  // than two blocks a processor, which is what its shared memory leaves (64 and 96 rows of 300 keys: 109 and 173 us, 100 and 111; 32 rows of 1,000: 167, 284).
  // A single token over fewer than thirty keys stays here although it is up to 2.5 us slower: the lengths are not known on the host.
  const bool single = rows > 0 && rows >= tokens;
  const bool many_rows = single ? (long long)tokens * kv_heads <= 2 * 148 : tokens > 64;
  if (many_rows && head_dim % 4 == 0 && head_dim <= 128 && group <= kRows && ((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) % piece == 0) {
    const int span = kRows / group;
    dim3 tiles((tokens + span - 1) / span, kv_heads, min(span, tokens));
    const size_t bytes = ((size_t)4 * kTile * kRowsLd + (size_t)kRows * kRowsLd + (size_t)kRows * (kTile + 4) + kRows) * sizeof(float);
    ROOST_DISPATCH_DTYPE(dtype, T, {
      auto kernel = paged_attention_rows_kernel<T>;
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      launch_kernel(kernel, tiles, dim3(128), bytes, (cudaStream_t)stream, (const T*)q, (T*)out, (const T*)k_pool, (const T*)v_pool, positions, token_row,
                    kv_indptr, kv_indices, tokens, span, q_heads, kv_heads, head_dim, page_size, scale, window);
    });
    return check_launch("paged_attention_generic");
  }
  dim3 grid(tokens, kv_heads, (group + kWarps - 1) / kWarps);
  const size_t smem = ((size_t)kTile * (head_dim + 1) + (size_t)kTile * head_dim + (size_t)kWarps * head_dim + kWarps * kTile) * sizeof(float);
  ROOST_DISPATCH_DTYPE(dtype, T, {
    auto kernel = paged_attention_generic_kernel<T>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<grid, kWarps * 32, smem, (cudaStream_t)stream>>>((const T*)q, (T*)out, (const T*)k_pool, (const T*)v_pool,
                                                              positions, token_row, kv_indptr, kv_indices, q_heads, kv_heads,
                                                              head_dim, page_size, scale, window);
  });
  return check_launch("paged_attention_generic");
}

extern "C" int roost_paged_attention_generic(const void* q, void* out, const void* k_pool, const void* v_pool, const int32_t* positions, const int32_t* token_row,
                                             const int32_t* kv_indptr, const int32_t* kv_indices, int tokens, int q_heads, int kv_heads, int head_dim, int page_size,
                                             float scale, int window, int dtype, roost_stream_t stream) {
  return roost_paged_attention_generic_rows(q, out, k_pool, v_pool, positions, token_row, kv_indptr, kv_indices, tokens, q_heads, kv_heads, head_dim, page_size, scale,
                                            window, dtype, 0, stream);
}
