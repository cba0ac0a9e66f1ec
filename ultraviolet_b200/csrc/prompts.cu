// Packing of a left-padded prompt batch, the final norm of its last tokens, and the softcap of full logits: the small
// launches around a packed prefill pass and around MathLM.logits.  Each replaces a string of tensor operations whose
// launches and host round trips cost more than the bytes they moved (a boolean selection per packed array; five passes
// over the (B, V) matrix for the softcap, 16 MB each at 256 rows).
#include "common.cuh"
#include "qkv_post.cuh"

namespace uv {

// prefix sums of the prompts' lengths and of their 16-token tiles, one CTA
__global__ void __launch_bounds__(1024) prompt_offsets_kernel(const int64_t* starts, int T, int n, int32_t* cu,
                                                              int32_t* tile_cu) {
  __shared__ int wl[32], wt[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int base_l = 0, base_t = 0;
  if (tid == 0) cu[0] = 0, tile_cu[0] = 0;
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + tid;
    int64_t len = i < n ? (int64_t)T - starts[i] : 0;
    len = len < 0 ? 0 : len > T ? T : len;
    int a = (int)len, t = ((int)len + 15) / 16;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) a += x, t += y;
    }
    if (lane == 31) wl[warp] = a, wt[warp] = t;
    __syncthreads();
    int add_l = base_l, add_t = base_t;
    for (int w = 0; w < warp; ++w) add_l += wl[w], add_t += wt[w];
    if (i < n) cu[i + 1] = a + add_l, tile_cu[i + 1] = t + add_t;
    for (int w = 0; w < 32; ++w) base_l += wl[w], base_t += wt[w];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(128) pack_prompts_kernel(const int64_t* idx, int64_t ld, int T, const int64_t* starts,
                                                           const int64_t* rows, const int32_t* cu, int64_t M, int64_t* tok,
                                                           int64_t* pos, int64_t* row, int64_t* last) {
  const int i = blockIdx.x, len = cu[i + 1] - cu[i];
  const int64_t s = T - len, r = rows[i], o = cu[i];
  for (int j = threadIdx.x; j < len && o + j < M; j += 128) {
    tok[o + j] = idx[i * ld + s + j];
    pos[o + j] = s + j, row[o + j] = r, last[o + j] = T - 1;
  }
}

template <typename T>
__global__ void __launch_bounds__(128) gather_norm_kernel(const T* x, int d, const int32_t* cu, int n, T* out) {
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;
  const bool empty = cu[i + 1] == cu[i];
  const T* r = x + (int64_t)(empty ? 0 : cu[i + 1] - 1) * d;
  const float rs = empty ? 0.f : row_rms_factor<T>(r, d, lane);
  for (int c = lane; c < d; c += 32) out[(int64_t)i * d + c] = from_f32<T>(empty ? 0.f : to_f32<T>(r[c]) * rs);
}

template <typename T>
__global__ void __launch_bounds__(256) softcap_kernel(const T* x, int64_t n, float a, float b, float c, float* out) {
  constexpr int W = 16 / sizeof(T);
  const int64_t nv = n / W, step = (int64_t)gridDim.x * 256;
  auto cap = [=](float v) { return a / (1.0f + expf(-((v + b) / c))); };
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < nv; i += step) {
    const uint4 u = __ldcs(reinterpret_cast<const uint4*>(x) + i);
    const T* v = reinterpret_cast<const T*>(&u);
#pragma unroll
    for (int k = 0; k < W; k += 4)
      *reinterpret_cast<float4*>(out + i * W + k) = make_float4(cap(to_f32<T>(v[k])), cap(to_f32<T>(v[k + 1])),
                                                                cap(to_f32<T>(v[k + 2])), cap(to_f32<T>(v[k + 3])));
  }
  for (int64_t i = nv * W + (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += step) out[i] = cap(to_f32<T>(x[i]));
}

}  // namespace uv

using namespace uv;

extern "C" int uv_pack_prompts(const int64_t* idx, int64_t ld, int T, const int64_t* starts, const int64_t* rows, int n,
                               int64_t M, int32_t* cu, int32_t* tile_cu, int64_t* tok, int64_t* pos, int64_t* row,
                               int64_t* last, void* stream) {
  if (n == 0) return UV_OK;
  if (!idx || !starts || !rows || !cu || !tile_cu || !tok || !pos || !row || !last || n < 0 || T < 1 || M < 0) return UV_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  prompt_offsets_kernel<<<1, 1024, 0, st>>>(starts, T, n, cu, tile_cu);
  pack_prompts_kernel<<<(unsigned)n, 128, 0, st>>>(idx, ld, T, starts, rows, cu, M, tok, pos, row, last);
  return check_launch();
}

extern "C" int uv_gather_norm(const void* x, int dtype, int d, const int32_t* cu, int n, void* out, void* stream) {
  if (n == 0) return UV_OK;
  if (!x || !cu || !out || n < 0) return UV_ERR_ARG;
  if (d < 8 || (d & 7)) return UV_ERR_SHAPE;
  if (!aligned16(x)) return UV_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)((n + 3) / 4);
  if (dtype == UV_F16)
    gather_norm_kernel<__half><<<grid, 128, 0, st>>>(static_cast<const __half*>(x), d, cu, n, static_cast<__half*>(out));
  else if (dtype == UV_BF16)
    gather_norm_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>(static_cast<const __nv_bfloat16*>(x), d, cu, n,
                                                            static_cast<__nv_bfloat16*>(out));
  else return UV_ERR_DTYPE;
  return check_launch();
}

extern "C" int uv_softcap(const void* x, int dtype, int64_t n, float a, float b, float c, float* out, void* stream) {
  if (n == 0) return UV_OK;
  if (!x || !out || n < 0) return UV_ERR_ARG;
  if (!aligned16(x) || !aligned16(out)) return UV_ERR_ALIGN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t want = (n / 8 + 255) / 256 + 1;
  const unsigned grid = (unsigned)(want < 148 * 8 ? want : 148 * 8);
  if (dtype == UV_F16) softcap_kernel<__half><<<grid, 256, 0, st>>>(static_cast<const __half*>(x), n, a, b, c, out);
  else if (dtype == UV_BF16)
    softcap_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x), n, a, b, c, out);
  else return UV_ERR_DTYPE;
  return check_launch();
}
