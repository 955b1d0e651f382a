// Gated linear attention (gated_linear_attention.cu says what it is) for prompt portions in bfloat16, heads of 64 keys and 128 values, 16 tokens at a
// time on the tensor cores. With alpha the decays of a key channel, P_t = alpha_1 .. alpha_t and Q_t = alpha_(t+1) .. alpha_n within a chunk of n
// tokens, and S the state before it:
//   o_t = S^T (P_t q_t) + sum_{s <= t} A[t][s] v_s,   A[t][s] = sum_d q_t[d] k_s[d] alpha_(s+1)[d] .. alpha_t[d],
//   S'  = diag(P_n) S + sum_s (Q_s k_s) v_s^T.
// Products of decays only ever shrink, so nothing overflows whatever the decays are. Values are bfloat16 and enter the products as they are; what is
// kept in 32 bits stays so: the state, the decayed queries and keys and A enter as three bfloat16 operands each, whose sum is the 24 bits of the
// float (six products where both sides are split, as many as count), sums are float32: a few products from zero each, added to nearest (mma.cuh says why).
// Outputs are no further from 64 bits than the walk's (1.1e-7 and 1.2e-7 of their norm; 6e-7 with all products of an output in one chain).
//
// A block takes a head of a row, eight warps 16 of its 128 values each with all 64 keys: a warp's part of S^T stays in registers as sums of a
// product, which have the layout of a first operand. Per chunk all threads make the decayed queries and keys and A (a thread a key token and four
// channels walks the queries after it) and leave them in shared memory; the next chunk's inputs arrive meanwhile. Rows are cut into segments as in
// mamba2_chunks.cu (by the step's tokens): MODE 1 leaves a segment's own state and the products of its decays, the carry kernel every segment's true starting state, MODE
// 2 makes the outputs; MODE 0 walks whole rows. A chunk whose outputs are not finite is taken again a token at a time (a product multiplies what a
// token must not see by zero). What bounds it is the chain of a chunk's phases. Rows of 3,000 and 1,096 tokens, 16 heads: the layer 263 us (256 to 259 with the chains), 447 with the
// two walks on the FMA pipe (97 + 194 us of it) and a number a thread in the norm after it; 382 tokens 73 us, 293 before.
#include "mma.cuh"

namespace roost {

constexpr int kGcTokens = 16, kGcD = 64, kGcV = 128;
constexpr int kGcLdA = 68;                                           // floats of a staged row of decays
constexpr int kGcAlpha = 0, kGcQ = kGcTokens * kGcLdA * 4, kGcK = kGcQ + kGcTokens * kGcD * 2, kGcVal = kGcK + kGcTokens * kGcD * 2,
              kGcStage = kGcVal + kGcTokens * kGcV * 2;
constexpr int kGcPq = 2 * kGcStage, kGcPk = kGcPq + 3 * kGcTokens * kGcD * 2, kGcPa = kGcPk + 3 * kGcTokens * kGcD * 2,
              kGcFade = kGcPa + 3 * kGcTokens * kGcTokens * 2, kGcBytes = kGcFade + kGcD * 4;
static_assert(kGcStage % 128 == 0 && kGcQ % 128 == 0, "swizzled tiles");

template <int MODE>
__global__ void __launch_bounds__(256, 2) gla_chunks_kernel(const __nv_bfloat16* u, int64_t ld, float q_scale, const float* alpha, float* out, float* state,
                                                            int64_t state_stride, const int32_t* __restrict__ q_indptr, const int32_t* __restrict__ slots, int rows,
                                                            int heads, int segment, float* ws, float* ws_keep) {
  extern __shared__ __align__(128) char smem[];
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  pdl_launch_dependents();
  const int h = blockIdx.x, QK = heads * kGcD;
  int r = blockIdx.y, start, end;
  bool last = true;
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
    if (MODE == 1 && last) { pdl_wait(); return; }
    start = q_indptr[r] + k * segment;
    end = min(start + segment, q_indptr[r + 1]);
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  // the slot holds S [64][128]: the thread's entries are columns 16 warp + g and + 8 of the rows 8 j + 2 c and + 1
  const size_t at_state = (size_t)(2 * c) * kGcV + warp * 16 + g;
  float* Sg = state + (size_t)slots[r] * state_stride + (size_t)h * kGcD * kGcV + at_state;
  float* Sw = MODE == 0 ? nullptr : ws + ((size_t)blockIdx.y * heads + h) * kGcD * kGcV + at_state;
  pdl_wait();
  if (end <= start) return;

  auto bring = [&](int t0, int n, int buf) {
    const uint32_t to = sbase + buf * kGcStage;
    {                                              // decays: 16 pieces a token; beyond the chunk ones are as good as any (k is zero there)
      const int t = tid >> 4, i = tid & 15;
      const uint32_t dst = to + kGcAlpha + t * kGcLdA * 4 + i * 16;
      if (t < n) copy16_async(dst, alpha + (size_t)(t0 + t) * QK + h * kGcD + i * 4);
      else asm volatile("st.shared.v4.f32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst), "f"(1.0f) : "memory");
    }
    {                                              // queries and keys: 8 pieces a token each
      const int which = tid >> 7, t = (tid >> 3) & 15, i = tid & 7;
      const uint32_t dst = to + (which ? kGcK : kGcQ) + t * kGcD * 2 + i * 16;
      if (t < n) copy16_async(dst, u + (size_t)(t0 + t) * ld + which * QK + h * kGcD + i * 8);
      else zero16(dst);
    }
    {                                              // values: 16 pieces a token
      const int t = tid >> 4, i = tid & 15;
      const uint32_t dst = to + kGcVal + swizzled<kGcV * 2>(t, i);
      if (t < n) copy16_async(dst, u + (size_t)(t0 + t) * ld + 2 * QK + h * kGcV + i * 8);
      else zero16(dst);
    }
    copy_commit();
  };

  float S[8][4];           // S^T: rows are values, columns keys
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[j][e] = MODE == 1 ? 0.f : (MODE == 0 ? Sg : Sw)[(size_t)(8 * j + (e & 1)) * kGcV + (e >> 1) * 8];
  float keep = 1.f;        // MODE 1, thread d < 64: the product of the segment's decays of channel d
  bring(start, min(kGcTokens, end - start), 0);
  int t0 = start, buf = 0, careful_until = start;
  while (t0 < end) {
    const bool careful = t0 < careful_until;
    const int n = careful ? 1 : min(kGcTokens, end - t0), next = min(kGcTokens, end - t0 - n);
    copy_wait<0>();
    __syncthreads();
    if (!careful && next > 0) bring(t0 + n, next, buf ^ 1);
    const float* al = reinterpret_cast<const float*>(smem + buf * kGcStage + kGcAlpha);
    const __nv_bfloat16* qs = reinterpret_cast<const __nv_bfloat16*>(smem + buf * kGcStage + kGcQ);
    const __nv_bfloat16* ks = reinterpret_cast<const __nv_bfloat16*>(smem + buf * kGcStage + kGcK);
    const uint32_t tv = sbase + buf * kGcStage + kGcVal;
    float* fade = reinterpret_cast<float*>(smem + kGcFade);

    // decayed queries and keys: a thread takes two channels of two tokens; the eight threads of a pair of channels lie side by side
    {
      const int part = tid & 7, d = (tid >> 3) * 2, t = part * 2;
      const float2 a0 = *reinterpret_cast<const float2*>(al + t * kGcLdA + d), a1 = *reinterpret_cast<const float2*>(al + (t + 1) * kGcLdA + d);
      float2 own = make_float2(a0.x * a1.x, a0.y * a1.y), pre = own, post = own;       // products up to and from this part on
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const float px = __shfl_up_sync(0xffffffffu, pre.x, o, 8), py = __shfl_up_sync(0xffffffffu, pre.y, o, 8);
        const float sx = __shfl_down_sync(0xffffffffu, post.x, o, 8), sy = __shfl_down_sync(0xffffffffu, post.y, o, 8);
        if (part >= o) { pre.x *= px; pre.y *= py; }
        if (part + o < 8) { post.x *= sx; post.y *= sy; }
      }
      if (part == 7) *reinterpret_cast<float2*>(fade + d) = pre;                        // the whole chunk's
      float2 before = make_float2(__shfl_up_sync(0xffffffffu, pre.x, 1, 8), __shfl_up_sync(0xffffffffu, pre.y, 1, 8));
      float2 after = make_float2(__shfl_down_sync(0xffffffffu, post.x, 1, 8), __shfl_down_sync(0xffffffffu, post.y, 1, 8));
      if (part == 0) before = make_float2(1.f, 1.f);
      if (part == 7) after = make_float2(1.f, 1.f);
      uint32_t p[3];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t off = swizzled<kGcD * 2>(t + i, d >> 3) + (d & 7) * 2;
        if (MODE != 1) {
          const uint32_t qv = *reinterpret_cast<const uint32_t*>(qs + (t + i) * kGcD + d);
          const float fx = i ? pre.x : before.x * a0.x, fy = i ? pre.y : before.y * a0.y;
          split3_nearest(__uint_as_float(qv << 16) * q_scale * fx, __uint_as_float(qv & 0xffff0000u) * q_scale * fy, p[0], p[1], p[2]);
#pragma unroll
          for (int pl = 0; pl < 3; ++pl) *reinterpret_cast<uint32_t*>(smem + kGcPq + pl * kGcTokens * kGcD * 2 + off) = p[pl];
        }
        const uint32_t kv = *reinterpret_cast<const uint32_t*>(ks + (t + i) * kGcD + d);
        const float fx = i ? after.x : after.x * a1.x, fy = i ? after.y : after.y * a1.y;
        split3(__uint_as_float(kv << 16) * fx, __uint_as_float(kv & 0xffff0000u) * fy, p[0], p[1], p[2]);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl) *reinterpret_cast<uint32_t*>(smem + kGcPk + pl * kGcTokens * kGcD * 2 + off) = p[pl];
      }
    }
    if (MODE != 1) {
      // A: a thread takes key token s and four channels, and the queries after it; sixteen threads' sums of every query end in one of them
      const int s = warp * 2 + (lane >> 4), dq = (lane & 15) * 4;
      float a[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) a[t] = 0.f;
      if (warp * 2 < n) {
        const uint2 kr = *reinterpret_cast<const uint2*>(ks + s * kGcD + dq);
        float w[4] = {__uint_as_float(kr.x << 16), __uint_as_float(kr.x & 0xffff0000u), __uint_as_float(kr.y << 16), __uint_as_float(kr.y & 0xffff0000u)};
#pragma unroll
        for (int t = 0; t < 16; ++t) {
          if (t < warp * 2) continue;              // the same for the whole warp
          const float4 f = *reinterpret_cast<const float4*>(al + t * kGcLdA + dq);
          if (t > s) { w[0] *= f.x; w[1] *= f.y; w[2] *= f.z; w[3] *= f.w; }
          const uint2 qr = *reinterpret_cast<const uint2*>(qs + t * kGcD + dq);
          float sum = __uint_as_float(qr.x << 16) * w[0];
          sum = fmaf(__uint_as_float(qr.x & 0xffff0000u), w[1], sum);
          sum = fmaf(__uint_as_float(qr.y << 16), w[2], sum);
          sum = fmaf(__uint_as_float(qr.y & 0xffff0000u), w[3], sum);
          a[t] = t >= s ? sum : 0.f;
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {            // lane i keeps the queries whose bits agree with its own
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const bool up = lane & o;
          const float give = up ? a[i] : a[i + o], mine = up ? a[i + o] : a[i];
          a[i] = mine + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      const int t = lane & 15;
      uint32_t p[3];
      split3(a[0] * q_scale, 0.f, p[0], p[1], p[2]);
#pragma unroll
      for (int pl = 0; pl < 3; ++pl) *reinterpret_cast<uint16_t*>(smem + kGcPa + pl * kGcTokens * kGcTokens * 2 + t * kGcTokens * 2 + s * 2) = (uint16_t)p[pl];
    }
    __syncthreads();
    uint32_t v[4];         // V^T: rows 16 values of the warp, k the chunk's tokens
    ldsm_x4_trans(v, tv + swizzled<kGcV * 2>((lane & 7) + ((lane >> 4) << 3), 2 * warp + ((lane >> 3) & 1)));
    if (MODE != 1) {
      // the products of leading parts are summed from zero and added in float32, rounded to nearest; the others, 2^-8 of them, in chains
      float Y[2][4], low[2][4];
#pragma unroll
      for (int pl = 2; pl >= 0; --pl) {
        uint32_t b[4];     // tokens t = 0 .. 7 at s 0 .. 7, 8 .. 15, then t = 8 .. 15
        ldsm_x4(b, sbase + kGcPa + pl * kGcTokens * kGcTokens * 2 + ((lane & 7) + ((lane >> 4) << 3)) * kGcTokens * 2 + ((lane >> 3) & 1) * 16);
        if (pl == 1) {
          mma_bf16(low[0], v, b[0], b[1]);
          mma_bf16(low[1], v, b[2], b[3]);
        } else {
          mma_bf16_zero(pl == 2 ? low[0] : Y[0], v, b[0], b[1]);
          mma_bf16_zero(pl == 2 ? low[1] : Y[1], v, b[2], b[3]);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t a[3][4], b[3][4];
        split3_nearest(S[2 * k][0], S[2 * k][1], a[0][0], a[1][0], a[2][0]);
        split3_nearest(S[2 * k][2], S[2 * k][3], a[0][1], a[1][1], a[2][1]);
        split3_nearest(S[2 * k + 1][0], S[2 * k + 1][1], a[0][2], a[1][2], a[2][2]);
        split3_nearest(S[2 * k + 1][2], S[2 * k + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
        for (int pl = 0; pl < 3; ++pl)
          ldsm_x4(b[pl], sbase + kGcPq + pl * kGcTokens * kGcD * 2 + swizzled<kGcD * 2>((lane & 7) + ((lane >> 4) << 3), 2 * k + ((lane >> 3) & 1)));
        // the parts' products down to 2^-16 of the largest, the least first; what is left out lies below the sums' last place
#pragma unroll
        for (int o = 2; o >= 1; --o)
#pragma unroll
          for (int x = 0; x <= o; ++x) {
            mma_bf16(low[0], a[x], b[o - x][0], b[o - x][1]);
            mma_bf16(low[1], a[x], b[o - x][2], b[o - x][3]);
          }
        float top[2][4];
        mma_bf16_zero(top[0], a[0], b[0][0], b[0][1]);
        mma_bf16_zero(top[1], a[0], b[0][2], b[0][3]);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) Y[j][e] += top[j][e];
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) Y[j][e] += low[j][e];
      if (n > 1) {
        bool odd = false;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) odd |= 8 * j + 2 * c + (e & 1) < n && !isfinite(Y[j][e]);
        if (__syncthreads_or(odd)) {       // again, a token at a time
          careful_until = t0 + n;
          copy_wait<0>();
          __syncthreads();
          bring(t0, 1, buf);
          continue;
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = 8 * j + 2 * c + (e & 1);
          if (t < n) out[(size_t)(t0 + t) * heads * kGcV + (size_t)h * kGcV + warp * 16 + g + (e >> 1) * 8] = Y[j][e];
        }
    }
    // the state after the chunk
    if (MODE == 1 && tid < kGcD) keep *= fade[tid];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float low[2][4], top[2][4];
#pragma unroll
      for (int pl = 2; pl >= 0; --pl) {
        uint32_t b[4];
        ldsm_x4_trans(b, sbase + kGcPk + pl * kGcTokens * kGcD * 2 + swizzled<kGcD * 2>(lane & 15, j + (lane >> 4)));
        if (pl == 1) {
          mma_bf16(low[0], v, b[0], b[1]);
          mma_bf16(low[1], v, b[2], b[3]);
        } else {
          mma_bf16_zero(pl == 2 ? low[0] : top[0], v, b[0], b[1]);
          mma_bf16_zero(pl == 2 ? low[1] : top[1], v, b[2], b[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 f = *reinterpret_cast<const float2*>(fade + 8 * (j + i) + 2 * c);
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j + i][e] = fmaf(S[j + i][e], e & 1 ? f.y : f.x, top[i][e] + low[i][e]);
      }
    }
    t0 += n;
    if (careful) {
      if (t0 < end) {
        __syncthreads();
        bring(t0, t0 < careful_until ? 1 : min(kGcTokens, end - t0), buf);
      }
    } else {
      buf ^= 1;
    }
  }
  if (MODE == 1 && tid < kGcD) ws_keep[((size_t)blockIdx.y * heads + h) * kGcD + tid] = keep;
  if (MODE == 2 && !last) return;
  float* to = MODE == 1 ? Sw : Sg;
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) to[(size_t)(8 * j + (e & 1)) * kGcV + (e >> 1) * 8] = S[j][e];
}

// Per row, in segment order, four values of a key: the state a segment starts from replaces the segment's own.
__global__ void __launch_bounds__(256) gla_segment_carry_kernel(float* ws, const float* ws_keep, const float* state, int64_t state_stride,
                                                               const int32_t* __restrict__ q_indptr, const int32_t* __restrict__ slots, int heads, int segment) {
  pdl_launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, e = (blockIdx.z * 256 + threadIdx.x) * 4, per = kGcD * kGcV;
  int first = 0;
  for (int i = 0; i < r; ++i) first += (q_indptr[i + 1] - q_indptr[i] + segment - 1) / segment;
  const int count = (q_indptr[r + 1] - q_indptr[r] + segment - 1) / segment;
  const float* slot = state + (size_t)slots[r] * state_stride + (size_t)h * per + e;
  pdl_wait();
  if (count == 0) return;
  float4 run = make_float4(slot[0], slot[1], slot[2], slot[3]);
  for (int k0 = 0; k0 < count; k0 += 4) {       // the segments' own states do not depend on one another
    float4 own[4];
    float keep[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k0 + j < count - 1) {
        own[j] = *reinterpret_cast<const float4*>(ws + ((size_t)(first + k0 + j) * heads + h) * per + e);
        keep[j] = ws_keep[((size_t)(first + k0 + j) * heads + h) * kGcD + e / kGcV];
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k0 + j < count) {
        *reinterpret_cast<float4*>(ws + ((size_t)(first + k0 + j) * heads + h) * per + e) = run;
        if (k0 + j < count - 1)
          run = make_float4(fmaf(keep[j], run.x, own[j].x), fmaf(keep[j], run.y, own[j].y), fmaf(keep[j], run.z, own[j].z), fmaf(keep[j], run.w, own[j].w));
      }
  }
}

// Tokens of a segment: whole chunks, at least 64 tokens, about three segments for each of the two blocks that a processor holds. 0: whole rows.
static int gla_segment_tokens(int rows, int tokens, int heads) {
  const long long chunks = (tokens + kGcTokens - 1) / kGcTokens;
  const long long each = chunks * heads / (6 * 148);
  const int segment = (int)(each < 4 ? 4 : each) * kGcTokens;
  return tokens / segment + rows <= 65535 && tokens > segment ? segment : 0;
}

}  // namespace roost

using namespace roost;

// Steps of few tokens a row stay with the walk, as in mamba2_chunks.cu: 16 heads, a prompt of 480 tokens beside 31 and 63 rows that decode 79 and 154 us a
// layer here, 319 and 347 with the walk; fewer than eight tokens a row were not measured.
extern "C" int roost_gla_chunks_parts(int rows, int tokens, int heads, int dim, int vdim, int dtype) {
  if (dtype != ROOST_BF16 || dim != kGcD || vdim != kGcV || rows <= 0 || rows > 65535 || heads > 65535 || tokens < 8LL * rows) return -1;
  const int segment = gla_segment_tokens(rows, tokens, heads);
  return segment ? tokens / segment + rows : 0;
}

extern "C" int roost_gla_chunks(const void* u, int64_t ld, float q_scale, const float* alpha, float* out, float* state, int64_t state_stride,
                                const int32_t* q_indptr, const int32_t* slots, int rows, int tokens, int heads, float* ws, float* ws_keep, roost_stream_t stream) {
  ROOST_REQUIRE(rows >= 0 && tokens >= 0 && heads > 0, "gla_chunks: sizes must be positive");
  ROOST_REQUIRE(u && alpha && out && state && q_indptr && slots, "gla_chunks: a pointer is null");
  ROOST_REQUIRE(ld >= (int64_t)heads * (2 * kGcD + kGcV) && ld % 8 == 0 && state_stride >= (int64_t)heads * kGcD * kGcV, "gla_chunks: a row or a slot is too narrow, or not whole pieces");
  ROOST_REQUIRE(((uintptr_t)u | (uintptr_t)alpha | (uintptr_t)ws) % 16 == 0, "gla_chunks: a pointer is not aligned");
  if (rows == 0 || tokens == 0) return ROOST_OK;
  if (rows > 65535 || heads > 65535) return fail(ROOST_ERR_UNSUPPORTED, "gla_chunks: too many rows or heads");
  cudaStream_t s = (cudaStream_t)stream;
  const int segment = ws != nullptr && ws_keep != nullptr ? gla_segment_tokens(rows, tokens, heads) : 0;
  auto go = [&](auto kernel, int parts) {
    launch_kernel(kernel, dim3(heads, parts), dim3(256), (size_t)kGcBytes, s, (const __nv_bfloat16*)u, ld, q_scale, alpha, out, state, state_stride, q_indptr, slots,
                  rows, heads, segment, ws, ws_keep);
  };
  if (segment == 0) {
    go(gla_chunks_kernel<0>, rows);
  } else {
    const int parts = tokens / segment + rows;
    go(gla_chunks_kernel<1>, parts);
    launch_kernel(gla_segment_carry_kernel, dim3(rows, heads, kGcD * kGcV / 1024), dim3(256), 0, s, ws, (const float*)ws_keep, (const float*)state, state_stride,
                  q_indptr, slots, heads, segment);
    go(gla_chunks_kernel<2>, parts);
  }
  return check_launch("gla_chunks");
}
