// The Mamba-2 recurrence of mamba2.cu for prompt portions in bfloat16, 64 tokens at a time on the tensor cores. With the decays' logarithms
// l_t = -exp(A_log) dt_t summed within a chunk, e_t = l_1 + .. + l_t, and S the state before it:
//   y_t  = exp(e_t) S C_t + sum_{s <= t} [exp(e_t - e_s) dt_s (C_t . B_s)] x_s + D x_t,
//   S'   = exp(e_n) S + sum_s [exp(e_n - e_s) dt_s x_s] B_s^T.
// B, C and x are bfloat16 and enter the products as they are. What the walk keeps in 32 bits stays so: the state and the bracketed weights
// enter as three bfloat16 operands each, whose sum is the 24 bits of the float; sums are float32, a few products from zero each, added to nearest (mma.cuh
// says why: outputs 1.1e-7 from 64 bits, the walk's 1.6e-7, 2.1e-7 with all products in one chain); e_t is summed in double and kept as two floats.
//
// A block takes a head of a row and walks its chunks in order, the state in registers, so nothing of it goes through memory between chunks.
// Eight warps: warp (pw, nh) keeps S for 16 of the head's 64 values and half of the state's N indices, as sums of a product, which have the
// layout of a first operand: S C^T needs no shared memory for S. The two warps of a pw exchange their halves of it and then own half of the
// chunk's tokens each. The weights of (t, s) are made once a block, from C B^T by all warps, and pass through shared memory.
//
// One long row would leave most processors idle, so steps of more tokens than a segment cut their rows into segments of whole chunks, as long as the
// step's tokens make them (a row's bits may then depend on what else is in its step; three launches): MODE 1 walks every segment but a row's last from an empty state, making no outputs, and leaves its state and the product of its
// decays; a carry gives every segment the state it starts from; MODE 2 walks all segments from there. MODE 0 walks whole rows.
//
// A product multiplies what a token must not see by zero, so where a chunk's outputs are not finite the chunk is taken again a token at a time.
//
// What bounds it is the chain of a chunk's phases (about 5 us a chunk with two blocks a processor; mma.sync's 4 M multiply-adds a head and
// chunk would take 2). Measured, bfloat16, 64 heads of 64 x 128, rows of 2,048, 1,037 and 1,011 tokens: the layer 490 us (471 with the chains), 1,180 with the two
// walks in 32-bit arithmetic (398 + 592 us of it); whole rows without segments 593. 32 heads, one row of 1,619: 120 us a layer, 351 before.
#include "mma.cuh"

#include <type_traits>

namespace roost {

constexpr int kM2Tokens = 64;      // tokens of a chunk
constexpr int kM2P = 64;           // values of a head

template <int NS>
struct Mamba2Tiles {
  static constexpr int kRow = NS * 2;                         // bytes of a token's B
  static constexpr int kB = 0, kC = kM2Tokens * kRow, kX = 2 * kM2Tokens * kRow, kStage = kX + kM2Tokens * kM2P * 2;
  static constexpr int kW = 2 * kStage;                       // three planes [t][s] of the weights; before them the exchanged halves of S C^T
  static constexpr int kScalars = kW + 3 * kM2Tokens * kM2Tokens * 2;
  static constexpr int kBytes = kScalars + 2 * (5 * kM2Tokens + 1) * 4 + 8;
};

template <int NS, int MODE>
__global__ void __launch_bounds__(256, 2) mamba2_chunks_kernel(const __nv_bfloat16* xbc, const __nv_bfloat16* u, int64_t ld_u, int dt_col, float* y,
                                                               const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                                                               const float* __restrict__ d_skip, float* state, int64_t state_stride,
                                                               const int32_t* __restrict__ q_indptr, const int32_t* __restrict__ slots, int rows, int heads,
                                                               int groups, int segment, float* ws_state, float* ws_decay) {
  using M = Mamba2Tiles<NS>;
  constexpr int KB = M::kRow;
  constexpr int JN = NS / 16;            // 8-column tiles of a warp's half of the state
  constexpr int KN = NS / 32;            // k steps of that half
  extern __shared__ __align__(128) char smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  float* exchange = reinterpret_cast<float*>(smem + M::kW);
  pdl_launch_dependents();
  const int h = blockIdx.x, grp = h / (heads / groups);
  int r = blockIdx.y, start, end;
  bool last = true;        // the row ends with this block's tokens
  if (MODE == 0) {
    start = q_indptr[r];
    end = q_indptr[r + 1];
  } else {                 // rows in order, each with ceil(tokens / segment) segments
    int k = blockIdx.y, count = 0;
    for (r = 0; r < rows; ++r) {
      count = (q_indptr[r + 1] - q_indptr[r] + segment - 1) / segment;
      if (k < count) break;
      k -= count;
    }
    if (r == rows) { pdl_wait(); return; }
    last = k == count - 1;
    if (MODE == 1 && last) { pdl_wait(); return; }       // nobody starts from the state a row's last segment ends with
    start = q_indptr[r] + k * segment;
    end = min(start + segment, q_indptr[r + 1]);
  }
  const int inner = heads * kM2P, channels = inner + 2 * groups * NS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int pw = warp >> 1, nh = warp & 1;
  const float bias = dt_bias[h], rate = -expf(a_log[h]), skip = d_skip[h];
  const size_t at_state = ((size_t)pw * 16 + g) * NS + nh * (NS / 2) + 2 * c;       // of a head
  float* Sg = state + (size_t)slots[r] * state_stride + (size_t)h * kM2P * NS + at_state;
  float* Sw = MODE == 0 ? nullptr : ws_state + ((size_t)blockIdx.y * heads + h) * kM2P * NS + at_state;
  pdl_wait();
  if (end <= start) return;
  const __nv_bfloat16* b_from = xbc + inner + (size_t)grp * NS;
  const __nv_bfloat16* x_from = xbc + (size_t)h * kM2P;

  auto bring = [&](int t0, int n, int buf) {
    const uint32_t at = sbase + buf * M::kStage;
    for (int idx = tid; idx < kM2Tokens * (NS / 8); idx += 256) {
      const int t = idx / (NS / 8), piece = idx % (NS / 8);
      const uint32_t to = at + swizzled<KB>(t, piece);
      if (t < n) {
        const __nv_bfloat16* from = b_from + (size_t)(t0 + t) * channels + piece * 8;
        copy16_async(to + M::kB, from);
        copy16_async(to + M::kC, from + (size_t)groups * NS);
      } else {
        zero16(to + M::kB);
        zero16(to + M::kC);
      }
    }
    for (int idx = tid; idx < kM2Tokens * (kM2P / 8); idx += 256) {
      const int t = idx / (kM2P / 8), piece = idx % (kM2P / 8);
      const uint32_t to = at + M::kX + swizzled<kM2P * 2>(t, piece);
      if (t < n) copy16_async(to, x_from + (size_t)(t0 + t) * channels + piece * 8);
      else zero16(to);
    }
    copy_commit();
  };
  // by warp 0: a chunk's [e_t in two parts | exp(e_t) | exp(e_n - e_t) dt_t | dt_t | exp(e_n)]
  auto scalars_of = [&](int buf) { return reinterpret_cast<float*>(smem + M::kScalars) + buf * (5 * kM2Tokens + 1); };
  float raw[2] = {0.f, 0.f};       // of warp 0: the next chunk's step projections
  auto fetch = [&](int t0, int n) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (2 * lane + i < n) raw[i] = to_float(u[(size_t)(t0 + 2 * lane + i) * ld_u + dt_col + h]);
  };
  auto steps = [&](int n, int buf) {
    float* sc = scalars_of(buf);
    float dt[2];
    double e[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      dt[i] = 0.f;
      float l = 0.f;
      if (t < n) {
        const float z = raw[i] + bias;
        dt[i] = z > 20.f ? z : log1pf(expf(z));
        l = rate * dt[i];
        if (l < -1e4f) l = -1e4f;        // exp is zero from -104 on; sums stay finite
      }
      e[i] = l;
    }
    const double both = e[0] + e[1];
    double sum = both;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double left = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += left;
    }
    const double before = __shfl_up_sync(0xffffffffu, sum, 1), total = __shfl_sync(0xffffffffu, sum, 31);
    e[0] += lane ? before : 0.0;
    e[1] = sum;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      const float top = (float)e[i], rest = (float)(e[i] - (double)top);
      sc[t] = top;
      sc[kM2Tokens + t] = rest;
      sc[2 * kM2Tokens + t] = expf(top) * (1.f + rest);
      sc[3 * kM2Tokens + t] = expf((float)(total - e[i])) * dt[i];
      sc[4 * kM2Tokens + t] = dt[i];
    }
    if (lane == 0) sc[5 * kM2Tokens] = expf((float)total);
  };

  bring(start, min(kM2Tokens, end - start), 0);
  if (warp == 0) {
    fetch(start, min(kM2Tokens, end - start));
    steps(min(kM2Tokens, end - start), 0);
  }
  float S[JN][4], decays = 1.f;
#pragma unroll
  for (int j = 0; j < JN; ++j) {
    const float* from = (MODE == 0 ? Sg : Sw) + 8 * j;
    float2 a = make_float2(0.f, 0.f), b = a;
    if (MODE != 1) {
      a = *reinterpret_cast<const float2*>(from);
      b = *reinterpret_cast<const float2*>(from + (size_t)8 * NS);
    }
    S[j][0] = a.x; S[j][1] = a.y; S[j][2] = b.x; S[j][3] = b.y;
  }
  int t0 = start, buf = 0, careful_until = start;
  while (t0 < end) {
    const bool careful = t0 < careful_until;
    const int n = careful ? 1 : min(kM2Tokens, end - t0), next = min(kM2Tokens, end - t0 - n);
    copy_wait<0>();
    __syncthreads();
    if (!careful && next > 0) {
      bring(t0 + n, next, buf ^ 1);
      if (warp == 0) fetch(t0 + n, next);
    }
    const uint32_t tb = sbase + buf * M::kStage + M::kB, tc = sbase + buf * M::kStage + M::kC, tx = sbase + buf * M::kStage + M::kX;
    const float* sc = scalars_of(buf);

    if (MODE != 1) {
    // this warp's half of (S C^T)[p][t] for all tokens, by tiles of eight
    float Y[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) Y[j][0] = Y[j][1] = Y[j][2] = Y[j][3] = 0.f;
#pragma unroll
    for (int k = 0; k < KN; ++k) {
      uint32_t a[3][4];
      split3(S[2 * k][0], S[2 * k][1], a[0][0], a[1][0], a[2][0]);
      split3(S[2 * k][2], S[2 * k][3], a[0][1], a[1][1], a[2][1]);
      split3(S[2 * k + 1][0], S[2 * k + 1][1], a[0][2], a[1][2], a[2][2]);
      split3(S[2 * k + 1][2], S[2 * k + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
      for (int half = 0; half < 2; ++half) {       // four independent sums between two products of one
        if (32 * half >= n) break;
        uint32_t b[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
          ldsm_x4(b[j], tc + swizzled<KB>(32 * half + 16 * j + (lane & 7) + ((lane >> 4) << 3), nh * (NS / 16) + 2 * k + ((lane >> 3) & 1)));
        float part[4][4];       // from zero, then added in float32 (see mma_bf16_zero)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          mma_bf16_zero(part[2 * j], a[2], b[j][0], b[j][1]);
          mma_bf16_zero(part[2 * j + 1], a[2], b[j][2], b[j][3]);
        }
#pragma unroll
        for (int q = 1; q >= 0; --q)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            mma_bf16(part[2 * j], a[q], b[j][0], b[j][1]);
            mma_bf16(part[2 * j + 1], a[q], b[j][2], b[j][3]);
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) Y[4 * half + j][e] += part[j][e];
      }
    }
    // the other half's owner gets its tokens' share
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) exchange[((warp * 4 + i) * 4 + e) * 32 + lane] = nh ? Y[i][e] : Y[4 + i][e];
    // (C B^T)[t][s] for 16 tokens t = 16 pw .. and half of the tiles of s up to them
    float G[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) G[i][0] = G[i][1] = G[i][2] = G[i][3] = 0.f;
    if (16 * pw < n) {
#pragma unroll
      for (int k = 0; k < NS / 16; k += 2) {
        uint32_t a0[4], a1[4];
        ldsm_x4(a0, tc + swizzled<KB>(16 * pw + (lane & 15), 2 * k + (lane >> 4)));
        ldsm_x4(a1, tc + swizzled<KB>(16 * pw + (lane & 15), 2 * k + 2 + (lane >> 4)));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i > pw) break;
          uint32_t b[4];
          ldsm_x4(b, tb + swizzled<KB>(8 * (nh * (pw + 1) + i) + (lane & 7), 2 * k + (lane >> 3)));
          float part[4];
          mma_bf16_zero(part, a0, b[0], b[1]);
          mma_bf16(part, a1, b[2], b[3]);
#pragma unroll
          for (int e = 0; e < 4; ++e) G[i][e] += part[e];
        }
      }
    }
    if (!careful && next > 0 && warp == 0) steps(next, buf ^ 1);       // pw 0 has the fewest tiles above
    __syncthreads();
    float Z[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float e0 = sc[2 * kM2Tokens + 32 * nh + 8 * i + 2 * c], e1 = sc[2 * kM2Tokens + 32 * nh + 8 * i + 2 * c + 1];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float mine = nh ? Y[4 + i][e] : Y[i][e], other = exchange[(((warp ^ 1) * 4 + i) * 4 + e) * 32 + lane];
        Z[i][e] = (mine + other) * (e & 1 ? e1 : e0);
      }
    }
    __syncthreads();       // the exchanged halves have been read; the weights take their place
    if (16 * pw < n) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i > pw) break;
        const int s = 8 * (nh * (pw + 1) + i) + 2 * c;
        const float es0 = sc[s], es1 = sc[s + 1], er0 = sc[kM2Tokens + s], er1 = sc[kM2Tokens + s + 1];
        const float dt0 = sc[4 * kM2Tokens + s], dt1 = sc[4 * kM2Tokens + s + 1];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int t = 16 * pw + g + 8 * half;
          const float et = sc[t], er = sc[kM2Tokens + t];
          float w0 = s <= t ? G[i][2 * half] * (expf((et - es0) + (er - er0)) * dt0) : 0.f;
          float w1 = s + 1 <= t ? G[i][2 * half + 1] * (expf((et - es1) + (er - er1)) * dt1) : 0.f;
          if (s == t) w0 += skip;
          if (s + 1 == t) w1 += skip;
          uint32_t w[3];
          split3(w0, w1, w[0], w[1], w[2]);
#pragma unroll
          for (int q = 0; q < 3; ++q)
            *reinterpret_cast<uint32_t*>(smem + M::kW + q * kM2Tokens * kM2Tokens * 2 + swizzled<kM2Tokens * 2>(t, s >> 3) + (s & 7) * 2) = w[q];
        }
      }
    }
    __syncthreads();
    // the chunk's own share of its outputs, for this warp's half of the tokens
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k > 2 * nh + 1 || 32 * nh >= n) break;
      uint32_t a[4];
      ldsm_x4_trans(a, tx + swizzled<kM2P * 2>(16 * k + (lane & 7) + ((lane >> 4) << 3), 2 * pw + ((lane >> 3) & 1)));
      float part[4][4];
#pragma unroll
      for (int pl = 2; pl >= 0; --pl)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int tt = 2 * nh + q;       // tokens 16 tt ..
          if (k > tt || 16 * tt >= n) continue;
          uint32_t b[4];
          ldsm_x4(b, sbase + M::kW + pl * kM2Tokens * kM2Tokens * 2 + swizzled<kM2Tokens * 2>(16 * tt + (lane & 7) + ((lane >> 4) << 3), 2 * k + ((lane >> 3) & 1)));
          if (pl == 2) {
            mma_bf16_zero(part[2 * q], a, b[0], b[1]);
            mma_bf16_zero(part[2 * q + 1], a, b[2], b[3]);
          } else {
            mma_bf16(part[2 * q], a, b[0], b[1]);
            mma_bf16(part[2 * q + 1], a, b[2], b[3]);
          }
        }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (k > 2 * nh + q || 16 * (2 * nh + q) >= n) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          Z[2 * q][e] += part[2 * q][e];
          Z[2 * q + 1][e] += part[2 * q + 1][e];
        }
      }
    }
    if (n > 1) {
      bool odd = false;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) odd |= 32 * nh + 8 * i + 2 * c + (e & 1) < n && !isfinite(Z[i][e]);
      if (__syncthreads_or(odd)) {       // again, a token at a time
        careful_until = t0 + n;
        copy_wait<0>();
        __syncthreads();
        bring(t0, 1, buf);
        if (warp == 0) {
          fetch(t0, 1);
          steps(1, buf);
        }
        continue;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 32 * nh + 8 * i + 2 * c + (e & 1);
        if (t < n) y[(size_t)(t0 + t) * inner + h * kM2P + pw * 16 + g + (e >> 1) * 8] = Z[i][e];
      }
    } else if (!careful && next > 0 && warp == 0) {
      steps(next, buf ^ 1);
    }
    // the state after the chunk
    const float fade = sc[5 * kM2Tokens];
    decays *= fade;
#pragma unroll
    for (int j = 0; j < JN; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] *= fade;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (16 * k >= n) break;
      uint32_t x[4], a[3][4];
      ldsm_x4_trans(x, tx + swizzled<kM2P * 2>(16 * k + (lane & 7) + ((lane >> 4) << 3), 2 * pw + ((lane >> 3) & 1)));
      const float* w = sc + 3 * kM2Tokens + 16 * k + 2 * c;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float w0 = w[(i >> 1) * 8], w1 = w[(i >> 1) * 8 + 1];
        split3(__uint_as_float(x[i] << 16) * w0, __uint_as_float(x[i] & 0xffff0000u) * w1, a[0][i], a[1][i], a[2][i]);
      }
#pragma unroll
      for (int j = 0; j < JN; j += 4) {
        uint32_t b[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) ldsm_x4_trans(b[i], tb + swizzled<KB>(16 * k + (lane & 15), nh * (NS / 16) + j + 2 * i + (lane >> 4)));
        float part[4][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_bf16_zero(part[2 * i], a[2], b[i][0], b[i][1]);
          mma_bf16_zero(part[2 * i + 1], a[2], b[i][2], b[i][3]);
        }
#pragma unroll
        for (int q = 1; q >= 0; --q)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            mma_bf16(part[2 * i], a[q], b[i][0], b[i][1]);
            mma_bf16(part[2 * i + 1], a[q], b[i][2], b[i][3]);
          }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j + i][e] += part[i][e];
      }
    }
    t0 += n;
    if (careful) {
      if (t0 < end) {
        __syncthreads();
        const int m = t0 < careful_until ? 1 : min(kM2Tokens, end - t0);
        bring(t0, m, buf);
        if (warp == 0) {
          fetch(t0, m);
          steps(m, buf);
        }
      }
    } else {
      buf ^= 1;
    }
  }
  if (MODE == 1 && tid == 0) ws_decay[(size_t)blockIdx.y * heads + h] = decays;
  if (!last && MODE == 2) return;
  float* to = MODE == 1 ? Sw : Sg;
#pragma unroll
  for (int j = 0; j < JN; ++j) {
    *reinterpret_cast<float2*>(to + 8 * j) = make_float2(S[j][0], S[j][1]);
    *reinterpret_cast<float2*>(to + (size_t)8 * NS + 8 * j) = make_float2(S[j][2], S[j][3]);
  }
}

// Per row and four entries of a head's state, in segment order: the state a segment starts from replaces the segment's own.
__global__ void __launch_bounds__(256) mamba2_segment_carry_kernel(float* ws_state, const float* ws_decay, const float* state, int64_t state_stride,
                                                                  const int32_t* __restrict__ q_indptr, const int32_t* __restrict__ slots, int heads, int per,
                                                                  int segment) {
  pdl_launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, e = (blockIdx.z * 256 + threadIdx.x) * 4;
  if (e >= per) { pdl_wait(); return; }
  int first = 0;
  for (int i = 0; i < r; ++i) first += (q_indptr[i + 1] - q_indptr[i] + segment - 1) / segment;
  const int count = (q_indptr[r + 1] - q_indptr[r] + segment - 1) / segment;
  const float2* slot = reinterpret_cast<const float2*>(state + (size_t)slots[r] * state_stride + (size_t)h * per + e);
  pdl_wait();
  if (count == 0) return;
  const float2 lo = slot[0], hi = slot[1];
  float4 run = make_float4(lo.x, lo.y, hi.x, hi.y);
  for (int k0 = 0; k0 < count; k0 += 4) {       // the segments' own states do not depend on one another
    float4 own[4];
    float decay[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k0 + j < count - 1) {
        own[j] = *reinterpret_cast<const float4*>(ws_state + ((size_t)(first + k0 + j) * heads + h) * per + e);
        decay[j] = ws_decay[(size_t)(first + k0 + j) * heads + h];
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k0 + j < count) {
        *reinterpret_cast<float4*>(ws_state + ((size_t)(first + k0 + j) * heads + h) * per + e) = run;
        if (k0 + j < count - 1)
          run = make_float4(fmaf(decay[j], run.x, own[j].x), fmaf(decay[j], run.y, own[j].y), fmaf(decay[j], run.z, own[j].z), fmaf(decay[j], run.w, own[j].w));
      }
  }
}

// A row of one token takes a block as long as a chunk does, so steps of few tokens a row stay with the walk. On this side of the line, 64 heads, a prompt of
// 480 tokens beside 31 and 63 rows that decode: 250 and 543 us a layer, 509 and 1,186 with the walk; fewer than eight tokens a row were not measured.
bool mamba2_chunks_serve(int rows, int tokens, int heads, int head_dim, int state_rows, int groups, int dtype) {
  return dtype == ROOST_BF16 && head_dim == kM2P && (state_rows == 64 || state_rows == 128) && rows <= 65535 && heads <= 65535 && tokens >= 8LL * rows;
}

// Tokens of a segment: whole chunks, at least four (the first walk of a segment costs two fifths of the second), about two segments for
// each of the two blocks that a processor holds. 0: whole rows.
int mamba2_segment_tokens(int rows, int tokens, int heads) {
  const long long chunks = (tokens + kM2Tokens - 1) / kM2Tokens;
  const long long each = chunks * heads / (4 * 148);
  const int segment = (int)(each < 4 ? 4 : each) * kM2Tokens;
  return tokens / segment + rows <= 65535 && tokens > segment ? segment : 0;
}

int mamba2_chunks(const void* xbc, const void* u, int64_t ld_u, int dt_col, float* y, const float* dt_bias, const float* a_log, const float* d_skip, float* state,
                  int64_t state_stride, const int32_t* q_indptr, const int32_t* slots, int rows, int tokens, int heads, int state_rows, int groups, float* ws_state,
                  float* ws_decay, cudaStream_t stream) {
  const int segment = ws_state != nullptr ? mamba2_segment_tokens(rows, tokens, heads) : 0;
  auto go = [&](auto kernel, int bytes, int parts) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    launch_kernel(kernel, dim3(heads, parts), dim3(256), (size_t)bytes, stream, (const __nv_bfloat16*)xbc, (const __nv_bfloat16*)u, ld_u, dt_col, y, dt_bias, a_log,
                  d_skip, state, state_stride, q_indptr, slots, rows, heads, groups, segment, ws_state, ws_decay);
  };
  auto all = [&](auto ns) {
    constexpr int NS = decltype(ns)::value;
    if (segment == 0) {
      go(mamba2_chunks_kernel<NS, 0>, Mamba2Tiles<NS>::kBytes, rows);
      return;
    }
    const int parts = tokens / segment + rows;
    go(mamba2_chunks_kernel<NS, 1>, Mamba2Tiles<NS>::kBytes, parts);
    launch_kernel(mamba2_segment_carry_kernel, dim3(rows, heads, (kM2P * NS + 1023) / 1024), dim3(256), 0, stream, ws_state, (const float*)ws_decay,
                  (const float*)state, state_stride, q_indptr, slots, heads, kM2P * NS, segment);
    go(mamba2_chunks_kernel<NS, 2>, Mamba2Tiles<NS>::kBytes, parts);
  };
  if (state_rows == 64) all(std::integral_constant<int, 64>());
  else all(std::integral_constant<int, 128>());
  return check_launch("mamba2_scan");
}

}  // namespace roost

using namespace roost;

extern "C" int roost_mamba2_scan_parts(int rows, int tokens, int heads, int head_dim, int state_rows, int groups, int dtype) {
  if (!mamba2_chunks_serve(rows, tokens, heads, head_dim, state_rows, groups, dtype)) return -1;
  const int segment = mamba2_segment_tokens(rows, tokens, heads);
  return segment ? tokens / segment + rows : 0;
}
