// Fused row-wise kernels of one decode step (everything between the GEMMs):
//   uv_embed_norm     token embedding gather + the two RMS norms that open the step
//   uv_qkv_post       value-embedding gate, per-head QK RMS norm, partial RoPE, int8 quantise + cache append
//   uv_resid_norm     lambda-weighted residual add + RMS norm (output feeds the next GEMM)
//   uv_swiglu         silu(gate) * up
// All of them keep the reference's rounding points: every elementwise result is rounded to the activation dtype
// where the reference's half-precision torch ops round (ultraviolet/kernels/fast_decode.py:272-334,
// ultraviolet/model.py:302-320, :567-571, :388-391), norms accumulate in fp32 with eps = 2^-23.
#include <stdlib.h>

#include <type_traits>

#include "common.cuh"
#include "qkv_post.cuh"

namespace uv {

template <typename T> struct Vec2;
template <> struct Vec2<__half> { using type = __half2; };
template <> struct Vec2<__nv_bfloat16> { using type = __nv_bfloat162; };

template <typename T> __device__ __forceinline__ float2 ld2(const T* p) {
  typename Vec2<T>::type v = *reinterpret_cast<const typename Vec2<T>::type*>(p);
  return make_float2(to_f32<T>(v.x), to_f32<T>(v.y));
}
template <typename T> __device__ __forceinline__ void st2(T* p, float a, float b) {
  typename Vec2<T>::type v;
  v.x = from_f32<T>(a);
  v.y = from_f32<T>(b);
  *reinterpret_cast<typename Vec2<T>::type*>(p) = v;
}

// two values at a time through the packed converters (the scalar ones go to a quarter-rate unit)
template <typename T> __device__ __forceinline__ typename Vec2<T>::type pair(float a, float b);
template <> __device__ __forceinline__ __half2 pair<__half>(float a, float b) { return __floats2half2_rn(a, b); }
template <> __device__ __forceinline__ __nv_bfloat162 pair<__nv_bfloat16>(float a, float b) {
  return __floats2bfloat162_rn(a, b);
}
template <typename T> __device__ __forceinline__ float2 rnd2(float a, float b) {
  const typename Vec2<T>::type v = pair<T>(a, b);
  return make_float2(to_f32<T>(v.x), to_f32<T>(v.y));
}

// ------------------------------------------------------------------------------------------------ embed + norms
// A warp owns a row; rows of up to ROW_MAX elements live in registers as 16-byte vectors (lane owns elements
// 8*lane + 256*j .. +7): one global read and one write per element, three or four memory instructions per lane.
constexpr int ROW_MAX = 1024;
constexpr int ROW_J = ROW_MAX / 256;

template <typename T> __device__ __forceinline__ void ld8(const T* p, float (&v)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const typename Vec2<T>::type* h = reinterpret_cast<const typename Vec2<T>::type*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[2 * i] = to_f32<T>(h[i].x), v[2 * i + 1] = to_f32<T>(h[i].y);
}
template <typename T> __device__ __forceinline__ void st8(T* p, const float (&v)[8]) {
  uint4 u;
  typename Vec2<T>::type* h = reinterpret_cast<typename Vec2<T>::type*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i].x = from_f32<T>(v[2 * i]), h[i].y = from_f32<T>(v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

// x = rms_norm(embed[tok]); xn = rms_norm(x)   (fast_decode.py:284 and the first layer's pre-norm, :303)
template <typename T>
__global__ void __launch_bounds__(128) embed_norm_kernel(const int64_t* __restrict__ tok, const T* __restrict__ embed,
                                                         int64_t vocab, int d, T* __restrict__ x, T* __restrict__ xn,
                                                         int B, const int64_t* __restrict__ pos,
                                                         const float* __restrict__ inv_freq, int n_pairs,
                                                         float* __restrict__ rope_cs, float* __restrict__ ss_out,
                                                         int ss_parts, int ss_ld) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  pdl_wait();
  pdl_trigger();
  if (row >= B) return;
  if (rope_cs != nullptr) {
    // the step's RoPE table: cos / sin of pos * inv_freq rounded to T, as apply_rope's operands are
    // (fast_decode.py:286-290); every layer's q / k rotation reads it instead of evaluating cosf / sinf
    const float pf = (float)pos[row];
    for (int j = lane; j < n_pairs; j += 32) {
      const float th = pf * inv_freq[j];
      rope_cs[(int64_t)row * 2 * n_pairs + j] = rnd<T>(cosf(th));
      rope_cs[(int64_t)row * 2 * n_pairs + n_pairs + j] = rnd<T>(sinf(th));
    }
  }
  int64_t t = tok[row];
  if (t < 0 || t >= vocab) t = 0;  // out-of-range ids read row 0 instead of faulting
  const T* e = embed + t * d;
  float v[ROW_J][8];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < ROW_J; ++j) {
    const int i = 8 * lane + 256 * j;
    if (i < d) {
      ld8<T>(e + i, v[j]);
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += v[j][k] * v[j][k];
    }
  }
  float inv = rsqrtf(warp_sum(ss) / (float)d + RMS_EPS);
  ss = 0.f;
#pragma unroll
  for (int j = 0; j < ROW_J; ++j) {
    if (8 * lane + 256 * j < d) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        v[j][k] = rnd<T>(v[j][k] * inv);
        ss += v[j][k] * v[j][k];
      }
    }
  }
  ss = warp_sum(ss);
  if (ss_out != nullptr && lane < ss_parts) {
    // the row's sum of squares in the per-tile form the tensor-core GEMMs read (deferred RMS norm): all of it in
    // part 0, zeros in the others
    ss_out[(int64_t)lane * ss_ld + row] = lane == 0 ? ss : 0.f;
  }
  inv = rsqrtf(ss / (float)d + RMS_EPS);
#pragma unroll
  for (int j = 0; j < ROW_J; ++j) {
    const int i = 8 * lane + 256 * j;
    if (i < d) {
      st8<T>(x + (int64_t)row * d + i, v[j]);
      if (xn != nullptr) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j][k] *= inv;
        st8<T>(xn + (int64_t)row * d + i, v[j]);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ residual + norm
// h = l0 * x + l1 * a (each product and the sum rounded to T, Block.finish, model.py:567-571); hn = rms_norm(h)
template <typename T>
__global__ void __launch_bounds__(128) resid_norm_kernel(const T* __restrict__ x, const T* __restrict__ a,
                                                         const float* __restrict__ lambdas, int d,
                                                         T* __restrict__ h, T* __restrict__ hn, int B) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  pdl_wait();
  pdl_trigger();
  if (row >= B) return;
  const float l0 = lambdas[0], l1 = lambdas[1];
  const int64_t ro = (int64_t)row * d;
  float v[ROW_J][8];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < ROW_J; ++j) {
    const int i = 8 * lane + 256 * j;
    if (i < d) {
      float xv[8], av[8];
      ld8<T>(x + ro + i, xv);
      ld8<T>(a + ro + i, av);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        v[j][k] = rnd<T>(rnd<T>(l0 * xv[k]) + rnd<T>(l1 * av[k]));
        ss += v[j][k] * v[j][k];
      }
    }
  }
  const float inv = rsqrtf(warp_sum(ss) / (float)d + RMS_EPS);
#pragma unroll
  for (int j = 0; j < ROW_J; ++j) {
    const int i = 8 * lane + 256 * j;
    if (i < d) {
      st8<T>(h + ro + i, v[j]);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[j][k] *= inv;
      st8<T>(hn + ro + i, v[j]);
    }
  }
}

// ------------------------------------------------------------------------------------------------ SwiGLU
// act = silu(g) * u with gu = [g | u] (B, 2f) (MLP.forward fused branch, model.py:388-391)
template <typename T>
__global__ void __launch_bounds__(256) swiglu_kernel(const T* __restrict__ gu, int f, T* __restrict__ act,
                                                     int64_t n_pairs) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // pair index over (B, f/2)
  pdl_wait();
  pdl_trigger();
  if (i >= n_pairs) return;
  const int half_f = f / 2;
  const int64_t row = i / half_f;
  const int col = (int)(i % half_f) * 2;
  const float2 g = ld2<T>(gu + row * 2 * f + col);
  const float2 u = ld2<T>(gu + row * 2 * f + f + col);
  const float s0 = rnd<T>(g.x / (1.0f + __expf(-g.x))), s1 = rnd<T>(g.y / (1.0f + __expf(-g.y)));
  st2<T>(act + row * f + col, s0 * u.x, s1 * u.y);
}

// act = silu(g) * u of the gate|up projection of UN-normalised rows h: [g | u] = (h . W^T) * rs with
// rs = rsqrt(mean(h^2) + eps) formed here.  A row is cut over SWR_SPLIT CTAs of SWR_THREADS threads (each re-forms rs
// from the 1-2 KB row: cheaper than one long CTA per row).  Every thread first requests everything it will need -- its
// 16-byte pieces of h and of g and u -- so the sum of squares and the projection arrive in one round trip.
constexpr int SWR_THREADS = 64;
constexpr int SWR_SPLIT = 4;
constexpr int SWR_HV = 2;     // 16-byte pieces of h per thread: d <= 8 * 64 * 2 = 1024 without the tail loop
constexpr int SWR_VMAX = 2;   // 8-feature vectors per thread: f <= 8 * 64 * 2 * SWR_SPLIT = 4096 on this path

template <typename T>
__global__ void __launch_bounds__(SWR_THREADS) swiglu_rs_kernel(const T* __restrict__ gu, const T* __restrict__ hrow,
                                                                int d, int f, T* __restrict__ act) {
  __shared__ float red[SWR_THREADS / 32];
  const int row = blockIdx.x / SWR_SPLIT, part = blockIdx.x % SWR_SPLIT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();
  const T* hr = hrow + (int64_t)row * d;
  const T* g = gu + (int64_t)row * 2 * f;
  const int nvec = f / 8;
  const int per = (nvec + SWR_SPLIT - 1) / SWR_SPLIT, v0 = part * per;
  const int v1 = v0 + per < nvec ? v0 + per : nvec;
  float hv[SWR_HV][8], gv[SWR_VMAX][8], uv[SWR_VMAX][8];
  // all loads first
#pragma unroll
  for (int j = 0; j < SWR_HV; ++j) {
    const int i = 8 * (tid + j * SWR_THREADS);
    if (i < d) {
      ld8<T>(hr + i, hv[j]);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) hv[j][k] = 0.f;
    }
  }
#pragma unroll
  for (int j = 0; j < SWR_VMAX; ++j) {
    const int v = v0 + tid + j * SWR_THREADS;
    if (v < v1) {
      ld8<T>(g + 8 * v, gv[j]);
      ld8<T>(g + f + 8 * v, uv[j]);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < SWR_HV; ++j)
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += hv[j][k] * hv[j][k];
  for (int i = 8 * (tid + SWR_HV * SWR_THREADS); i < d; i += 8 * SWR_THREADS) {  // rows wider than 1024 elements
    float more[8];
    ld8<T>(hr + i, more);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += more[k] * more[k];
  }
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < SWR_THREADS / 32; ++w) tot += red[w];
  const float rs = rsqrtf(tot / (float)d + RMS_EPS);
#pragma unroll
  for (int j = 0; j < SWR_VMAX; ++j) {
    const int v = v0 + tid + j * SWR_THREADS;
    if (v < v1) {
      float o[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float g0 = rnd<T>(gv[j][k] * rs), u0 = rnd<T>(uv[j][k] * rs);
        o[k] = rnd<T>(g0 / (1.0f + __expf(-g0))) * u0;
      }
      st8<T>(act + (int64_t)row * f + 8 * v, o);
    }
  }
}

// The same for launches of many rows: a warp owns a row, requests all of it (16-byte pieces of h, g and u) before it
// uses any, and forms rs once.  At prefill sizes the kernel above is bound by its own traffic -- four CTAs a row read
// h four times and leave 48 bytes a thread in flight; this one streams.  20,500 rows of f = 1664: 99 us -> 49 us (bf16; 45 in
// fp16; 231 MB: 35 us at the measured copy rate).  The results are those of the kernel above bit for bit -- a row's bits must
// not depend on how many rows came with it -- so the squares are summed in its order and the quotient is the rounded one.
constexpr int SWM_WARPS = 8;
constexpr int SWM_ROWS = 768;
constexpr int SWM_V = 7;      // 8-feature vectors a lane holds at a time

// the row's norm factor as swiglu_rs_kernel forms it: its two warps take the 256-element groups of the row in turn
template <typename T> __device__ __forceinline__ float swiglu_row_factor(const T* row, int d, int lane) {
  uint4 u[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = 8 * lane + 256 * j;
    u[j] = i < d ? *reinterpret_cast<const uint4*>(row + i) : make_uint4(0u, 0u, 0u, 0u);
  }
  float ss[2] = {0.f, 0.f};
  auto add = [](float& s, const uint4& w) {
    const T* v = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float f = to_f32<T>(v[k]);
      s += f * f;
    }
  };
#pragma unroll
  for (int j = 0; j < 4; ++j) add(ss[j & 1], u[j]);
  for (int i = 8 * lane + 1024; i < d; i += 512) {  // rows wider than 1024 elements
    add(ss[0], *reinterpret_cast<const uint4*>(row + i));
    if (i + 256 < d) add(ss[1], *reinterpret_cast<const uint4*>(row + i + 256));
  }
  return rsqrtf((warp_sum(ss[0]) + warp_sum(ss[1])) / (float)d + RMS_EPS);
}

// q[k] = g[k] / (1 + exp(-g[k])), the rounded quotient, without the division's code: the quotient by the approximate reciprocal
// plus its remainder (exact in an FMA) times that reciprocal, one step of Newton's method.  That is off from the rounded
// quotient only where the true one lies within 2^-45 of itself from the middle between two floats, which no g of 16 bits
// does (all of them are compared in the tests).  Without a remainder (zeros keep their sign, infinities, NaN) the first quotient
// stands; divisors too large for the reciprocal give results that are zero in fp16, and in bf16 are divided properly.
// 20,500 rows, bf16 / fp16: 49.2 / 45.4 us, 47.9 / 43.5 with __fdividef (which is off by up to 2 units), 63 with the division;
// 4096 rows: 16.0 / 14.4 us, 16.7 / 16.1 with __fdividef.
template <typename T> __device__ __forceinline__ void silu8(const float (&g)[8], float (&q)[8]) {
  float least = INFINITY;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float b = 1.0f + __expf(-g[k]);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    const float q0 = g[k] * r, rem = fmaf(-q0, b, g[k]);
    q[k] = fabsf(rem) > 0.f ? fmaf(rem, r, q0) : q0;   // (no remainder, or NaN)
    least = fminf(least, fabsf(q0));
  }
  if (!std::is_same<T, __half>::value && least < 0x1p-100f) {
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = g[k] / (1.0f + __expf(-g[k]));
  }
}

template <typename T>
__global__ void __launch_bounds__(SWM_WARPS * 32) swiglu_rows_kernel(const T* __restrict__ gu, const T* __restrict__ hrow,
                                                                     int d, int f, T* __restrict__ act, int B) {
  const int lane = threadIdx.x & 31, row = blockIdx.x * SWM_WARPS + (threadIdx.x >> 5);
  pdl_wait();
  pdl_trigger();
  if (row >= B) return;
  const T* g = gu + (int64_t)row * 2 * f;
  const int nvec = f / 8;
  uint4 gv[SWM_V], uv[SWM_V];
  auto request = [&](int v0) {
#pragma unroll
    for (int j = 0; j < SWM_V; ++j) {
      const int v = v0 + 32 * j + lane;
      if (v < nvec) {
        gv[j] = __ldcs(reinterpret_cast<const uint4*>(g) + v);
        uv[j] = __ldcs(reinterpret_cast<const uint4*>(g + f) + v);
      }
    }
  };
  request(0);
  const float rs = swiglu_row_factor<T>(hrow + (int64_t)row * d, d, lane);
  for (int v0 = 0; v0 < nvec; v0 += 32 * SWM_V) {
    if (v0) request(v0);
#pragma unroll
    for (int j = 0; j < SWM_V; ++j) {
      const int v = v0 + 32 * j + lane;
      if (v >= nvec) break;
      const typename Vec2<T>::type *a = reinterpret_cast<const typename Vec2<T>::type*>(&gv[j]),
                                   *b = reinterpret_cast<const typename Vec2<T>::type*>(&uv[j]);
      float g8[8], s8[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 g2 = rnd2<T>(to_f32<T>(a[k].x) * rs, to_f32<T>(a[k].y) * rs);
        g8[2 * k] = g2.x, g8[2 * k + 1] = g2.y;
      }
      silu8<T>(g8, s8);
      uint4 out;
      typename Vec2<T>::type* o = reinterpret_cast<typename Vec2<T>::type*>(&out);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 u2 = rnd2<T>(to_f32<T>(b[k].x) * rs, to_f32<T>(b[k].y) * rs);
        const float2 s = rnd2<T>(s8[2 * k], s8[2 * k + 1]);
        o[k] = pair<T>(s.x * u2.x, s.y * u2.y);
      }
      *(reinterpret_cast<uint4*>(act + (int64_t)row * f) + v) = out;
    }
  }
}

// ------------------------------------------------------------------------------------------------ QKV post
// One warp per (row b, head slot), in place on the packed GEMM output; the arithmetic lives in qkv_post.cuh.
// W warps per CTA, one (row, item) per warp.  COOP (xn_raw launches whose items per row are a multiple of W): the W
// items of a CTA belong to ONE row, whose sum of squares the CTA forms once -- every thread one 16-byte piece -- instead
// of each warp reading the whole row for itself (18 readers per 1.3 KB row otherwise: at a few thousand rows that
// redundant L2 traffic is what the launch costs).
template <typename T, int HD, bool TABLE, int W, bool COOP>
__global__ void __launch_bounds__(W * 32) qkv_post_kernel(const __grid_constant__ QkvPostParams P) {
  constexpr int E = HD >= 32 ? HD / 32 : 1;
  const int lane = threadIdx.x & 31;
  const int slots = P.H + 2 * P.K;
  const int per_row = slots + (P.gate_out ? P.H : 0);  // head slots, then one gate item per query head
  const int item = blockIdx.x * W + (threadIdx.x >> 5);
  pdl_wait();
  pdl_trigger();
  if (item >= P.B * per_row) return;  // (COOP: the item count is a multiple of W, so this is CTA-uniform)
  const int b = item / per_row, hs = item % per_row;
  const bool raw = P.xn_raw != 0;
  // the slot's own values are requested before the row reduction below needs its loads: one round trip, not two
  const bool act0 = lane * E < HD;
  float x0[E];
  if (hs < slots) {
    const T* vec0 = static_cast<const T*>(P.qkv) + ((int64_t)b * slots + hs) * HD;
#pragma unroll
    for (int i = 0; i < E; ++i) x0[i] = act0 ? to_f32<T>(vec0[lane * E + i]) : 0.f;
  }
  // so is where a key / value slot will land (position, cache row): three more loads off the tail of the chain
  QkvSlot dest{};
  const bool appends = hs >= P.H && hs < slots && P.k_cache != nullptr;
  if (appends) dest = qkv_post_slot(P, b);
  float rs = 1.0f;
  if constexpr (COOP) {
    __shared__ float part[W];
    const uint4* row = reinterpret_cast<const uint4*>(static_cast<const T*>(P.xn) + (int64_t)b * P.d);
    float ss = 0.f;
    for (int p = threadIdx.x; p * 8 < P.d; p += W * 32) {
      const uint4 u = row[p];
      const T* v = reinterpret_cast<const T*>(&u);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float f = to_f32<T>(v[k]);
        ss += f * f;
      }
    }
    ss = warp_sum(ss);
    if (lane == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) tot += part[w];
    rs = rsqrtf(tot / (float)P.d + RMS_EPS);
  } else {
    if (raw) rs = row_rms_factor<T>(static_cast<const T*>(P.xn) + (int64_t)b * P.d, P.d, lane);
  }
  if (hs >= slots) {
    const int head = hs - slots;
    const float g = head_gate<T>(static_cast<const T*>(P.xn) + (int64_t)b * P.d,
                                 static_cast<const T*>(P.gate_w) + (int64_t)head * P.gate_ch, P.gate_ch, lane, rs,
                                 raw);
    if (lane == 0) P.gate_out[(int64_t)b * P.H + head] = g;
    return;
  }
  const bool act = lane * E < HD;
  T* vec = static_cast<T*>(P.qkv) + ((int64_t)b * slots + hs) * HD;
  float x[E];
#pragma unroll
  for (int i = 0; i < E; ++i) x[i] = x0[i];
  if (raw) {  // the projection of the un-normalised row, scaled: what the GEMM on the normalised row would hold
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = rnd<T>(x[i] * rs);
  }
  qkv_post_compute<T, HD, TABLE>(P, b, hs, lane, x, rs, raw);
#pragma unroll
  for (int i = 0; i < E; ++i)
    if (act) vec[lane * E + i] = from_f32<T>(x[i]);
  if (appends) qkv_post_append<T, HD>(P, b, hs, lane, x, &dest);
}

// The same for launches of many rows (xn_raw, RoPE from the table): a warp owns a row -- the norm factor is formed once
// from registers that then feed the gates -- and a head slot is a group of HD / 8 lanes with 16 bytes each, so a row of
// ten 64-wide slots is three passes.  The kernel above spends a warp on every slot and gate, eighteen a row, each with
// its own chain of loads: right when rows are few, three times the instructions and 2-byte-a-lane traffic when they are
// not.  20,500 rows: 136 us -> 41 us (78 MB: 12 us at the measured copy rate).
// The results are those of the kernel above bit for bit (a row's bits must not depend on how many rows came with it): every
// sum adds the same partial sums in the same order, which takes a butterfly for each of them; lanes that would hold copies
// of several such sums keep one each instead.  COOP: as the cooperative form of that kernel sums a row's squares, one sum
// for 256 elements, else one for the row.
constexpr int QPR_WARPS = 8;
constexpr int QPR_ROWS = 768;
constexpr int QPR_GCH = 128;   // channels a gate may read

// N sums over the lanes of a group of LG, each as the butterfly of xor LG/2, ..., 1 adds it, left where the index's high bits
// are the lane's: v[i] of lane l is sum number (l / (LG / min(LG, N))) * (N / min(LG, N)) + i.
template <int LG, int N> __device__ __forceinline__ void group_sums(float (&v)[N], int lane) {
  int n = N;
#pragma unroll
  for (int o = LG / 2; o > 0; o >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < N / 2; ++i)
        if (i < n) {
          const float send = up ? v[i] : v[i + n];
          v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, send, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
}

template <typename T, int HD, bool COOP>
__global__ void __launch_bounds__(QPR_WARPS * 32) qkv_post_rows_kernel(const __grid_constant__ QkvPostParams P) {
  constexpr int LG = HD / 8, NG = 32 / LG;              // lanes a slot, slots a pass
  constexpr int E = HD >= 32 ? HD / 32 : 1, NP = 8 / E; // elements of a slot that the kernel above has in a lane
  extern __shared__ __align__(16) unsigned char qpr_smem[];
  // (H, 32, 4) then (K, 32, 4): channels lane, lane + 32, lane + 64, lane + 96 of a gate side by side, zeros past its last
  T* const gw = reinterpret_cast<T*>(qpr_smem);
  T* const vw = gw + (P.gate_out ? P.H * QPR_GCH : 0);
  const int lane = threadIdx.x & 31, grp = lane / LG, gl = lane % LG;
  const int slots = P.H + 2 * P.K;
  auto stage = [&](T* to, const void* from, int n, int channels) {
    for (int i = threadIdx.x; i < n * QPR_GCH; i += QPR_WARPS * 32) {
      const int c = ((i >> 2) & 31) + 32 * (i & 3);
      to[i] = c < channels ? static_cast<const T*>(from)[(i / QPR_GCH) * channels + c] : from_f32<T>(0.f);
    }
  };
  if (P.gate_out) stage(gw, P.gate_w, P.H, P.gate_ch);
  if (P.ve_gate) stage(vw, P.ve_gate, P.K, P.ve_ch);
  const int channels = max(P.gate_out ? P.gate_ch : 0, P.ve_gate ? P.ve_ch : 0);
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  auto unpack = [](const uint4& u, float (&v)[8]) {
    const typename Vec2<T>::type* h = reinterpret_cast<const typename Vec2<T>::type*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[2 * k] = to_f32<T>(h[k].x), v[2 * k + 1] = to_f32<T>(h[k].y);
  };
  auto pack = [](const float (&v)[8]) {
    uint4 u;
    typename Vec2<T>::type* h = reinterpret_cast<typename Vec2<T>::type*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = pair<T>(v[2 * k], v[2 * k + 1]);
    return u;
  };
  auto scale = [](float (&v)[8], float s) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const float2 r = rnd2<T>(v[k] * s, v[k + 1] * s);
      v[k] = r.x, v[k + 1] = r.y;
    }
  };
  // this lane's share of one gate's product with the normalised channels, in the order of head_gate
  auto gate_dot = [](const float (&xs)[4], const T* w) {
    const uint2 u = *reinterpret_cast<const uint2*>(w);
    const typename Vec2<T>::type* h = reinterpret_cast<const typename Vec2<T>::type*>(&u);
    float acc = 0.f;
    acc += xs[0] * to_f32<T>(h[0].x), acc += xs[1] * to_f32<T>(h[0].y);
    acc += xs[2] * to_f32<T>(h[1].x), acc += xs[3] * to_f32<T>(h[1].y);
    return acc;
  };
  auto gate_of = [](float dot) {
    return rnd<T>(2.0f * rnd<T>(1.0f / (1.0f + __expf(-rnd<T>(dot)))));
  };
  auto group_max = [](float v) {
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  };
  for (int b = blockIdx.x * QPR_WARPS + (threadIdx.x >> 5); b < P.B; b += gridDim.x * QPR_WARPS) {
    const T* xr = static_cast<const T*>(P.xn) + (int64_t)b * P.d;
    T* const qr = static_cast<T*>(P.qkv) + (int64_t)b * slots * HD;
    uint4 xu[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = 8 * lane + 256 * j;
      xu[j] = i < P.d ? *reinterpret_cast<const uint4*>(xr + i) : make_uint4(0u, 0u, 0u, 0u);
    }
    float xs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) xs[j] = lane + 32 * j < channels ? to_f32<T>(xr[lane + 32 * j]) : 0.f;
    uint4 raw = grp < slots ? *reinterpret_cast<const uint4*>(qr + grp * HD + 8 * gl) : make_uint4(0u, 0u, 0u, 0u);
    const QkvSlot dest = qkv_post_slot(P, b);
    const float* cs = P.inv_freq ? P.rope_cs + (int64_t)b * 2 * P.n_pairs : nullptr;
    float x[8], part[4] = {0.f, 0.f, 0.f, 0.f}, ss;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      unpack(xu[j], x);
#pragma unroll
      for (int k = 0; k < 8; ++k) part[COOP ? j : 0] += x[k] * x[k];
    }
    if constexpr (COOP) {
      group_sums<32, 4>(part, lane);
      ss = __shfl_sync(0xffffffffu, part[0], 0);
#pragma unroll
      for (int j = 1; j < 4; ++j) ss += __shfl_sync(0xffffffffu, part[0], 8 * j);
    } else {
      ss = warp_sum(part[0]);
    }
    const float rs = rsqrtf(ss / (float)P.d + RMS_EPS);
    // ---- head gates, eight at a time
#pragma unroll
    for (int j = 0; j < 4; ++j) xs[j] = rnd<T>(xs[j] * rs);
    if (P.gate_out) {
      for (int h0 = 0; h0 < P.H; h0 += 8) {
        float dot[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) dot[i] = h0 + i < P.H ? gate_dot(xs, gw + ((h0 + i) * 32 + lane) * 4) : 0.f;
        group_sums<32, 8>(dot, lane);
        const int h = h0 + (lane >> 2);
        const float g = gate_of(dot[0]);
        if (h < P.H && (lane & 3) == 0) P.gate_out[(int64_t)b * P.H + h] = g;
      }
    }
    // ---- head slots, NG at a time
    for (int s0 = 0; s0 < slots; s0 += NG) {
      const int hs = s0 + grp;
      const bool live = hs < slots, isv = hs >= P.H + P.K;
      const uint4 cur = raw;
      if (s0 + NG < slots)
        raw = hs + NG < slots ? *reinterpret_cast<const uint4*>(qr + (hs + NG) * HD + 8 * gl) : make_uint4(0u, 0u, 0u, 0u);
      unpack(cur, x);
      scale(x, rs);
      float sq[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        sq[i] = 0.f;
#pragma unroll
        for (int k = 0; k < E; ++k) sq[i] += x[i * E + k] * x[i * E + k];
      }
      group_sums<LG, NP>(sq, lane);
      constexpr int LEFT = NP > LG ? NP / LG : 1;       // sums that stayed in a lane, then added in the butterfly's order
#pragma unroll
      for (int o = LG / 2, m = NP; o > 0 && m > 1; o >>= 1, m >>= 1)
#pragma unroll
        for (int i = 0; i < LEFT; ++i) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
#pragma unroll
      for (int m = LEFT / 2; m > 0; m >>= 1)
#pragma unroll
        for (int i = 0; i < m; ++i) sq[i] += sq[i + m];
      const float inv = rsqrtf(sq[0] / (float)HD + RMS_EPS);
      if (!isv) scale(x, inv);
      if (cs != nullptr) {                              // dim j < n_pairs turns with dim j + n_pairs
        const int np8 = P.n_pairs / 8;
        const bool turns = !isv && gl < 2 * np8;
        const float* c = cs + 8 * (gl & (np8 - 1));
        const float sgn = gl < np8 ? -1.f : 1.f;        // x1 c - x2 s, x1 s + x2 c: every product and sum rounded
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const float o0 = __shfl_xor_sync(0xffffffffu, x[k], np8), o1 = __shfl_xor_sync(0xffffffffu, x[k + 1], np8);
          if (turns) {
            const float2 cc = *reinterpret_cast<const float2*>(c + k), sn = *reinterpret_cast<const float2*>(c + P.n_pairs + k);
            const float2 a = rnd2<T>(x[k] * cc.x, x[k + 1] * cc.y), d = rnd2<T>(o0 * sn.x, o1 * sn.y);
            const float2 y = rnd2<T>(a.x + sgn * d.x, a.y + sgn * d.y);
            x[k] = y.x, x[k + 1] = y.y;
          }
        }
      }
      if (P.ve_gate != nullptr && s0 + NG > P.H + P.K) {  // some slot of this pass is a value head (warp-uniform)
        const int kh = isv && live ? hs - P.H - P.K : 0;
        float acc = 0.f;
        for (int k0 = 0; k0 < P.K; ++k0) {
          const float p = warp_sum(gate_dot(xs, vw + (k0 * 32 + lane) * 4));
          if (k0 == kh) acc = p;
        }
        if (isv && live) {
          const float g = gate_of(acc);
          int64_t t = P.tok[b];
          if (t < 0 || t >= P.vocab) t = 0;
          float ve[8];
          unpack(*reinterpret_cast<const uint4*>(static_cast<const T*>(P.value_embed) + (t * P.K + kh) * HD + 8 * gl), ve);
#pragma unroll
          for (int k = 0; k < 8; k += 2) {
            const float2 a = rnd2<T>(g * ve[k], g * ve[k + 1]), y = rnd2<T>(x[k] + a.x, x[k + 1] + a.y);
            x[k] = y.x, x[k + 1] = y.y;
          }
        }
      }
      if (live) *reinterpret_cast<uint4*>(qr + hs * HD + 8 * gl) = pack(x);
      if (P.k_cache != nullptr && s0 + NG > P.H) {      // quantise + append (quantize_lane, common.cuh, 8 values a lane)
        float amax = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(x[k]));
        amax = group_max(amax);
        if (live && hs >= P.H) {
          int64_t p = dest.pos;
          bool keep = true;
          if (P.ring) {
            keep = !(dest.last >= 0 && p + P.S <= dest.last);   // else a newer token of this launch owns the slot
            p = ((p % P.S) + P.S) % P.S;
          }
          if (keep && (p < 0 || p >= P.S)) {
            keep = false;
            if (gl == 0 && P.oob) atomicAdd(P.oob, 1);
          }
          if (keep) {
            const __half s16 = __float2half_rn(__fdiv_rn(amax, 127.0f));
            const float sf = fmaxf(__half2float(s16), 1e-30f);
            uint32_t w8[2] = {0u, 0u};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float r = fminf(fmaxf(rintf(__fdiv_rn(x[k], sf)), -127.0f), 127.0f);
              w8[k / 4] |= ((uint32_t)__float2int_rn(r) & 0xffu) << (8 * (k & 3));
            }
            const int kh = isv ? hs - P.H - P.K : hs - P.H;
            const int64_t dst = (dest.row * P.K + kh) * P.S_alloc + p;
            *reinterpret_cast<uint2*>((isv ? P.v_cache : P.k_cache) + dst * HD + 8 * gl) = make_uint2(w8[0], w8[1]);
            if (gl == 0) (isv ? P.v_scale : P.k_scale)[dst] = __half_as_ushort(s16);
          }
        }
      }
    }
  }
}

template <typename T>
static int launch_qkv_post(const QkvPostParams& P, int hd, cudaStream_t st) {
  const int per_row = P.H + 2 * P.K + (P.gate_out ? P.H : 0);
  const int64_t items = (int64_t)P.B * per_row;
  // cooperative row reduction when the launch defers the norm and a row's items fill whole CTAs of 6 or 4 warps
  static const bool coop_on = [] {
    const char* v = getenv("UVDECODE_QKV_POST_COOP");
    return !(v && v[0] == '0');
  }();
  const int coop = (P.xn_raw && coop_on) ? (per_row % 6 == 0 ? 6 : (per_row % 4 == 0 ? 4 : 0)) : 0;
  // many rows: a warp a row.  Below QPR_ROWS rows a row's own chain is what counts, and a warp for every slot shortens it
  // (256 rows: 4.2 us against 7.0; 768: 7.7 against 7.3; 4096: 12.9 with this one).
  const bool rows_ok = P.B >= QPR_ROWS && P.xn_raw && P.d <= 1024 && (!P.gate_out || P.gate_ch <= QPR_GCH) &&
                       (!P.ve_gate || P.ve_ch <= QPR_GCH) && aligned16(P.qkv) &&
                       (!P.ve_gate || aligned16(P.value_embed)) &&
                       (!P.k_cache || (((uintptr_t)P.k_cache | (uintptr_t)P.v_cache) & 7) == 0) &&
                       (!P.inv_freq || (P.rope_cs && ((uintptr_t)P.rope_cs & 7) == 0 &&
                                        (P.n_pairs == 8 || P.n_pairs == 16 || P.n_pairs == 32 || P.n_pairs == 64)));
  const size_t smem = (size_t)((P.gate_out ? P.H : 0) + (P.ve_gate ? P.K : 0)) * QPR_GCH * sizeof(T);   // the gates' weights
  if (rows_ok && smem <= 48 * 1024) {
    const int64_t ctas = ((int64_t)P.B + QPR_WARPS - 1) / QPR_WARPS;
    const unsigned grid = (unsigned)(ctas < 148 * 6 ? ctas : 148 * 6);
#define UV_QKV_POST_ROWS(HD_)                                                                                             \
  case HD_:                                                                                                               \
    if (coop) launch_pdl(qkv_post_rows_kernel<T, HD_, true>, dim3(grid), dim3(QPR_WARPS * 32), smem, st, P);              \
    else launch_pdl(qkv_post_rows_kernel<T, HD_, false>, dim3(grid), dim3(QPR_WARPS * 32), smem, st, P);                  \
    break;
    switch (hd) {
      UV_QKV_POST_ROWS(16)
      UV_QKV_POST_ROWS(32)
      UV_QKV_POST_ROWS(64)
      UV_QKV_POST_ROWS(128)
      default: return UV_ERR_SHAPE;
    }
#undef UV_QKV_POST_ROWS
    return check_launch();
  }
  const int wpc = coop ? coop : 4;
  const unsigned grid = (unsigned)((items + wpc - 1) / wpc);
  // with the step's RoPE table the kernel carries no cosf / sinf code at all
#define UV_QKV_POST_W(HD_, TABLE_)                                                                              \
  do {                                                                                                          \
    if (coop == 6) launch_pdl(qkv_post_kernel<T, HD_, TABLE_, 6, true>, dim3(grid), dim3(192), 0, st, P);       \
    else if (coop == 4) launch_pdl(qkv_post_kernel<T, HD_, TABLE_, 4, true>, dim3(grid), dim3(128), 0, st, P);  \
    else launch_pdl(qkv_post_kernel<T, HD_, TABLE_, 4, false>, dim3(grid), dim3(128), 0, st, P);                \
  } while (0)
#define UV_QKV_POST(HD_)                       \
  case HD_:                                    \
    if (P.rope_cs) UV_QKV_POST_W(HD_, true);   \
    else UV_QKV_POST_W(HD_, false);            \
    break;
  switch (hd) {
    UV_QKV_POST(16)
    UV_QKV_POST(32)
    UV_QKV_POST(64)
    UV_QKV_POST(128)
    default: return UV_ERR_SHAPE;
  }
#undef UV_QKV_POST
#undef UV_QKV_POST_W
  return check_launch();
}

}  // namespace uv

using namespace uv;

extern "C" int uv_embed_norm_rope(const int64_t* tok, const void* embed, int dtype, int64_t vocab, int d, void* x,
                                  void* xn, int B, const int64_t* pos, const float* inv_freq, int n_pairs,
                                  float* rope_cs, void* stream) {
  if (!xn) return B == 0 ? UV_OK : UV_ERR_ARG;
  return uv_embed_norm_ss(tok, embed, dtype, vocab, d, x, xn, B, pos, inv_freq, n_pairs, rope_cs, nullptr, 0, 0,
                          stream);
}

extern "C" int uv_embed_norm_ss(const int64_t* tok, const void* embed, int dtype, int64_t vocab, int d, void* x,
                                void* xn, int B, const int64_t* pos, const float* inv_freq, int n_pairs,
                                float* rope_cs, float* ss_out, int ss_parts, int ss_ld, void* stream) {
  if (B == 0) return UV_OK;
  if (!tok || !embed || !x || B < 0 || vocab < 1) return UV_ERR_ARG;
  if (!xn && !ss_out) return UV_ERR_ARG;
  if (ss_out && (ss_parts < 1 || ss_parts > 32 || ss_ld < B)) return UV_ERR_ARG;
  if (rope_cs && (!pos || !inv_freq || n_pairs < 1)) return UV_ERR_ARG;
  if (d < 8 || (d & 7) || d > ROW_MAX) return UV_ERR_SHAPE;  // rows are moved as 16-byte vectors
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)((B + 3) / 4);
  if (dtype == UV_F16)
    launch_pdl(embed_norm_kernel<__half>, dim3(grid), dim3(128), 0, st, tok, static_cast<const __half*>(embed), vocab,
               d, static_cast<__half*>(x), static_cast<__half*>(xn), B, pos, inv_freq, n_pairs, rope_cs, ss_out, ss_parts,
               ss_ld);
  else if (dtype == UV_BF16)
    launch_pdl(embed_norm_kernel<__nv_bfloat16>, dim3(grid), dim3(128), 0, st, tok,
               static_cast<const __nv_bfloat16*>(embed), vocab, d, static_cast<__nv_bfloat16*>(x),
               static_cast<__nv_bfloat16*>(xn), B, pos, inv_freq, n_pairs, rope_cs, ss_out, ss_parts, ss_ld);
  else return UV_ERR_DTYPE;
  return check_launch();
}

extern "C" int uv_embed_norm(const int64_t* tok, const void* embed, int dtype, int64_t vocab, int d, void* x,
                             void* xn, int B, void* stream) {
  return uv_embed_norm_rope(tok, embed, dtype, vocab, d, x, xn, B, nullptr, nullptr, 0, nullptr, stream);
}

extern "C" int uv_qkv_post_args(const uv_qkv_args* a, void* stream) {
  if (!a) return UV_ERR_ARG;
  if (a->B == 0) return UV_OK;
  QkvPostParams P{};
  const int rc = qkv_post_params(&P, a->qkv, a->xn, a->tok, a->value_embed, a->ve_gate, a->inv_freq, a->pos, a->k_cache,
                                 a->v_cache, a->k_scale, a->v_scale, a->row_map, a->oob_count, a->vocab, a->B, a->H,
                                 a->K, a->hd, a->d, a->S, a->S_alloc, a->ring, a->ve_ch, a->n_pairs);
  if (rc != UV_OK) return rc;
  P.rope_cs = a->inv_freq ? a->rope_cs : nullptr;
  if (a->gate_out) {
    if (!a->gate_w || !a->xn || a->gate_ch < 1 || a->gate_ch > a->d) return UV_ERR_ARG;
    P.gate_w = a->gate_w, P.gate_out = a->gate_out, P.gate_ch = a->gate_ch;
  }
  P.last_pos = a->last_pos;
  if (a->xn_raw) {
    if (!a->xn || a->d < 8 || (a->d & 7) || !aligned16(a->xn)) return UV_ERR_ARG;
    P.xn_raw = 1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a->dtype == UV_F16) return launch_qkv_post<__half>(P, a->hd, st);
  if (a->dtype == UV_BF16) return launch_qkv_post<__nv_bfloat16>(P, a->hd, st);
  return UV_ERR_DTYPE;
}

extern "C" int uv_resid_norm(const void* x, const void* a, const float* lambdas, int dtype, int d, void* h, void* hn,
                             int B, void* stream) {
  if (B == 0) return UV_OK;
  if (!x || !a || !lambdas || !h || !hn || B < 0) return UV_ERR_ARG;
  if (d < 8 || (d & 7) || d > ROW_MAX) return UV_ERR_SHAPE;  // rows are moved as 16-byte vectors
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)((B + 3) / 4);
  if (dtype == UV_F16)
    launch_pdl(resid_norm_kernel<__half>, dim3(grid), dim3(128), 0, st, static_cast<const __half*>(x),
               static_cast<const __half*>(a), lambdas, d, static_cast<__half*>(h), static_cast<__half*>(hn), B);
  else if (dtype == UV_BF16)
    launch_pdl(resid_norm_kernel<__nv_bfloat16>, dim3(grid), dim3(128), 0, st, static_cast<const __nv_bfloat16*>(x),
               static_cast<const __nv_bfloat16*>(a), lambdas, d, static_cast<__nv_bfloat16*>(h),
               static_cast<__nv_bfloat16*>(hn), B);
  else return UV_ERR_DTYPE;
  return check_launch();
}

extern "C" int uv_swiglu(const void* gu, int dtype, int f, void* act, int B, void* stream) {
  if (B == 0) return UV_OK;
  if (!gu || !act || B < 0) return UV_ERR_ARG;
  if (f < 2 || (f & 1)) return UV_ERR_SHAPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t n = (int64_t)B * (f / 2);
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (dtype == UV_F16)
    launch_pdl(swiglu_kernel<__half>, dim3(grid), dim3(256), 0, st, static_cast<const __half*>(gu), f,
               static_cast<__half*>(act), n);
  else if (dtype == UV_BF16)
    launch_pdl(swiglu_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(gu), f,
               static_cast<__nv_bfloat16*>(act), n);
  else return UV_ERR_DTYPE;
  return check_launch();
}

extern "C" int uv_swiglu_rs(const void* gu, const void* h, int dtype, int d, int f, void* act, int B, void* stream) {
  if (B == 0) return UV_OK;
  if (!gu || !h || !act || B < 0) return UV_ERR_ARG;
  if (f < 8 || (f & 7) || f > 8 * SWR_THREADS * SWR_VMAX * SWR_SPLIT || d < 8 || (d & 7)) return UV_ERR_SHAPE;
  if (!aligned16(h) || !aligned16(gu) || !aligned16(act)) return UV_ERR_ALIGN;  // rows move as 16-byte vectors
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // From SWM_ROWS rows on the launch is bound by what it moves; below, by one row's chain of loads, which four CTAs a row
  // shorten (256 rows: 3.2 us against 4.9; 768: 5.2 against 5.0; 2048: 6.3 with this one).
  if (B >= SWM_ROWS) {
    const dim3 grid((unsigned)((B + SWM_WARPS - 1) / SWM_WARPS)), block(SWM_WARPS * 32);
    if (dtype == UV_F16)
      launch_pdl(swiglu_rows_kernel<__half>, grid, block, 0, st, static_cast<const __half*>(gu),
                 static_cast<const __half*>(h), d, f, static_cast<__half*>(act), B);
    else if (dtype == UV_BF16)
      launch_pdl(swiglu_rows_kernel<__nv_bfloat16>, grid, block, 0, st, static_cast<const __nv_bfloat16*>(gu),
                 static_cast<const __nv_bfloat16*>(h), d, f, static_cast<__nv_bfloat16*>(act), B);
    else return UV_ERR_DTYPE;
    return check_launch();
  }
  if (dtype == UV_F16)
    launch_pdl(swiglu_rs_kernel<__half>, dim3((unsigned)B * SWR_SPLIT), dim3(SWR_THREADS), 0, st, static_cast<const __half*>(gu),
               static_cast<const __half*>(h), d, f, static_cast<__half*>(act));
  else if (dtype == UV_BF16)
    launch_pdl(swiglu_rs_kernel<__nv_bfloat16>, dim3((unsigned)B * SWR_SPLIT), dim3(SWR_THREADS), 0, st,
               static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(h), d, f,
               static_cast<__nv_bfloat16*>(act));
  else return UV_ERR_DTYPE;
  return check_launch();
}

extern "C" int uv_qkv_post(void* qkv, const void* xn, const int64_t* tok, const void* value_embed,
                           const void* ve_gate, const float* inv_freq, const int64_t* pos, int8_t* k_cache,
                           int8_t* v_cache, uint16_t* k_scale, uint16_t* v_scale, const int64_t* row_map,
                           int* oob_count, int dtype, int64_t vocab, int B, int H, int K, int hd, int d, int S,
                           int S_alloc, int ring, int ve_ch, int n_pairs, void* stream) {
  if (B == 0) return UV_OK;
  QkvPostParams P{};
  const int rc = qkv_post_params(&P, qkv, xn, tok, value_embed, ve_gate, inv_freq, pos, k_cache, v_cache, k_scale,
                                 v_scale, row_map, oob_count, vocab, B, H, K, hd, d, S, S_alloc, ring, ve_ch, n_pairs);
  if (rc != UV_OK) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == UV_F16) return launch_qkv_post<__half>(P, hd, st);
  if (dtype == UV_BF16) return launch_qkv_post<__nv_bfloat16>(P, hd, st);
  return UV_ERR_DTYPE;
}
