// What the attentions of sink_attention.cu and sigmoid_attention.cu do to a token's heads before they attend, for heads of 64 and 128 numbers in
// whole 16-byte pieces: rotation (interleaved pairs or split halves), division by the head's root mean square, a weight a number, a temperature of
// the queries, the cache write. A lane holds one piece of a head, so a warp takes several heads at a time; the cosines and sines of its numbers
// are made once a token. A warp takes a token, or four warps do where a step has few. Bound by memory where a step has many tokens: 4,048 tokens
// of 16 + 4 + 4 heads of 128 18.7 us (39 a number at a time, a block a token), 2,825 of 16 + 4 + 4 heads of 64 6.4 (24).
#pragma once

#include "common.cuh"

namespace roost {

struct HeadPrepare {
  int64_t ld;
  int entry, tokens, heads, kv_heads, vdim, page_size;
  const double* inv_freq;
  int rot_dims, halves;
  float amplitude, eps;             // eps 0: no norm
  const float *q_w, *k_w;           // null: none
  float temp_coef;
  int temp_every;
  const int32_t *positions, *slot_mapping;
};

// WPT: warps that share a token.
template <typename T, int DIM, int WPT>
__global__ void __launch_bounds__(128) head_prepare_kernel(T* qkv, T* q_out, T* k_base, T* v_base, const HeadPrepare a) {
  constexpr int N = Vec<T>::N, LPH = DIM / N, HPW = 32 / LPH;      // numbers a lane, lanes a head, heads a warp
  constexpr int BATCH = 4;                                         // passes whose pieces are on their way at once
  __shared__ float angles[4][2 * (DIM / 2)];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane % LPH;
  const int t = blockIdx.x * (4 / WPT) + warp / WPT, share = warp % WPT;
  if (t >= a.tokens) { pdl_wait(); return; }                                       // no barrier of the block below
  const int pos = a.positions[t], slot = a.slot_mapping[t];
  const int half = a.rot_dims / 2;
  float* cs = angles[warp];
  float* sn = cs + DIM / 2;
  for (int i = lane; i < half; i += 32) {
    double ang = (double)pos * a.inv_freq[i];
    ang -= 6.283185307179586476925286766559 * rint(ang * 0.15915494309189533576888376337251);
    float s, c;
    sincosf((float)ang, &s, &c);
    sn[i] = s * a.amplitude;
    cs[i] = c * a.amplitude;
  }
  __syncwarp();
  float c[N], s[N];       // of the lane's numbers: x' = c x + s partner, the sign of the number's place in its pair in s
#pragma unroll
  for (int e = 0; e < N; ++e) {
    const int i = sub * N + e;
    const bool turned = i < a.rot_dims;
    const int pair = a.halves ? (i < half ? i : i - half) : i / 2;
    const bool first = a.halves ? i < half : (i & 1) == 0;
    c[e] = turned ? cs[pair] : 1.f;
    s[e] = turned ? (first ? -sn[pair] : sn[pair]) : 0.f;
  }
  const float temp = a.temp_coef != 0.f && pos >= 0 ? 1.0f + a.temp_coef * logf((float)((pos + 1) / a.temp_every + 1)) : 1.0f;
  const int total = a.heads + a.kv_heads, reach = half / N;        // lanes between the numbers of a pair of split halves
  const size_t page = slot >= 0 ? slot / a.page_size : 0, off = slot >= 0 ? slot % a.page_size : 0;
  T* row = qkv + (size_t)t * a.ld;
  pdl_wait();
  for (int h0 = share * HPW; h0 < total; h0 += HPW * WPT * BATCH) {
    float x[BATCH][N];
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int h = h0 + b * HPW * WPT + lane / LPH;
#pragma unroll
      for (int e = 0; e < N; ++e) x[b][e] = 0.f;
      if (h < total) Vec<T>::load(row + (size_t)h * DIM + sub * N, x[b]);
    }
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      if (h0 + b * HPW * WPT >= total) break;                      // the same for the whole warp
      const int h = h0 + b * HPW * WPT + lane / LPH;
      if (a.rot_dims) {
        float y[N];
        if (a.halves) {
#pragma unroll
          for (int e = 0; e < N; ++e) y[e] = __shfl_xor_sync(0xffffffffu, x[b][e], reach);
        } else {
#pragma unroll
          for (int e = 0; e < N; ++e) y[e] = x[b][e ^ 1];
        }
#pragma unroll
        for (int e = 0; e < N; ++e)
          if (sub * N + e < a.rot_dims) x[b][e] = x[b][e] * c[e] + y[e] * s[e];       // a number beside the rotated part has no partner
      }
      float inv = 1.0f;
      if (a.eps > 0.f) {
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < N; ++e) ss = fmaf(x[b][e], x[b][e], ss);
#pragma unroll
        for (int o = LPH / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        inv = 1.0f / sqrtf(ss / (float)DIM + a.eps);
      }
      if (h >= total) continue;
      const bool is_q = h < a.heads;
      const float* w = is_q ? a.q_w : a.k_w;
#pragma unroll
      for (int e = 0; e < N; ++e) {
        x[b][e] *= inv;
        if (w != nullptr) x[b][e] *= w[sub * N + e];
        if (is_q) x[b][e] *= temp;
      }
      if (!is_q && slot < 0) continue;                             // a padding token: no key is written
      T* dst = !is_q ? k_base + ((page * a.kv_heads + (h - a.heads)) * a.page_size + off) * a.entry
                     : (q_out != nullptr ? q_out + ((size_t)t * a.heads + h) * DIM : row + (size_t)h * DIM);
      Vec<T>::store(dst + sub * N, x[b]);
    }
  }
  if (slot < 0) return;
  const T* from = row + (size_t)total * DIM;
  for (int i = (share * 32 + lane) * N; i < a.kv_heads * a.vdim; i += 32 * WPT * N)
    *reinterpret_cast<uint4*>(v_base + ((page * a.kv_heads + i / a.vdim) * a.page_size + off) * a.entry + i % a.vdim) = *reinterpret_cast<const uint4*>(from + i);
}

// Whether the form above serves: whole pieces everywhere, and pairs of split halves whose numbers lie a power of two of lanes apart.
inline bool head_prepare_serves(const void* qkv, const void* q_out, const void* k_base, const void* v_base, int dim, const HeadPrepare& a, int dtype) {
  if (dtype != ROOST_F32 && dtype != ROOST_BF16) return false;
  const int n = dtype == ROOST_F32 ? 4 : 8, reach = a.rot_dims / 2 / n;
  if ((dim != 64 && dim != 128) || a.vdim % n || a.entry % n || a.ld % n) return false;
  if (a.halves && a.rot_dims && (a.rot_dims / 2 % n || (reach & (reach - 1)))) return false;
  return ((uintptr_t)qkv | (uintptr_t)q_out | (uintptr_t)k_base | (uintptr_t)v_base) % 16 == 0;
}

template <typename T>
inline void launch_head_prepare(void* qkv, void* q_out, void* k_base, void* v_base, int dim, const HeadPrepare& a, cudaStream_t stream) {
  const bool few = a.tokens < 4 * 148;       // a warp a token would leave most of the processors idle
  auto kernel = dim == 64 ? (few ? head_prepare_kernel<T, 64, 4> : head_prepare_kernel<T, 64, 1>) : (few ? head_prepare_kernel<T, 128, 4> : head_prepare_kernel<T, 128, 1>);
  launch_kernel(kernel, dim3(few ? a.tokens : (a.tokens + 3) / 4), dim3(128), 0, stream, (T*)qkv, (T*)q_out, (T*)k_base, (T*)v_base, a);
}

}  // namespace roost
