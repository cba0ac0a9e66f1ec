// Weight publication: every fused inference weight of the decode engine from the trainer's parameters, in one launch.
//
// What bounds it: HBM.  UV-50M reads 204 MB of fp32 parameters and writes 100 MB (47 us at the measured copy rate); as
// some 25 tensor operations a layer, with the residual lambdas fetched to the host one by one, it took 2.79 ms; as this
// launch 0.13 ms with the host side of the call and its synchronisation.
// Layout: a block copies 4096 elements of one matrix, four 16-byte loads (fp32) a thread in flight; which matrix follows
// from comparing the block number with the matrices' block counts, the same in every layer (grid.y).  Blocks of wo and
// w_down form their layer's folded coefficient themselves, from the at most 2 * layer + 2 lambdas before it.
#include "common.cuh"

namespace uv {

constexpr int FW_THREADS = 256;
constexpr int FW_BLOCK = FW_THREADS * 16;
constexpr int FW_MAXL = 32;
constexpr int FW_NSEG = 7;   // wq wk wv wo w_gate w_up w_down

struct FuseP {
  uv_fuse_layer layer[FW_MAXL];
  const void *embed, *value_embed;
  void *d_embed, *d_value_embed;
  int64_t n_embed, n_value_embed;
  int64_t n[FW_NSEG];
  int first[FW_NSEG + 1];    // block number at which each matrix of a layer starts
  int L, H, n_ve, n_gate, fold;
  float limit;
  int* status;
};

// dst[i] = D(P(src[i] * mul)) -- or D((float(src[i]) * a) * b), products in fp32 -- for this block's elements
template <typename P, typename D, typename F>
__device__ __forceinline__ void fw_copy(const P* src, D* dst, int64_t n, int64_t i0, F f) {
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 && i0 + FW_BLOCK <= n) {
    constexpr int W = 16 / sizeof(P);                   // elements of a 16-byte load
    constexpr int J = 16 / W;
    uint4 u[J];
#pragma unroll
    for (int j = 0; j < J; ++j) u[j] = __ldcs(reinterpret_cast<const uint4*>(src + i0) + j * FW_THREADS + threadIdx.x);
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const P* v = reinterpret_cast<const P*>(&u[j]);
      D o[W];
#pragma unroll
      for (int k = 0; k < W; ++k) o[k] = f(v[k]);
      D* to = dst + i0 + (int64_t)(j * FW_THREADS + threadIdx.x) * W;
      if constexpr (W == 4) *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(o);
      else *reinterpret_cast<uint4*>(to) = *reinterpret_cast<const uint4*>(o);
    }
    return;
  }
  for (int64_t i = i0 + threadIdx.x; i < n && i < i0 + FW_BLOCK; i += FW_THREADS) dst[i] = f(src[i]);
}

template <typename P, typename D>
__global__ void __launch_bounds__(FW_THREADS) fuse_weights_kernel(const __grid_constant__ FuseP A) {
  const int tid = threadIdx.x, l = blockIdx.y;
  auto plain = [](P x) { return from_f32<D>(to_f32<P>(x)); };
  if (l == A.L) {                                       // the embeddings
    const int64_t nb = (A.n_embed + FW_BLOCK - 1) / FW_BLOCK;
    for (int64_t b = blockIdx.x; b < nb; b += gridDim.x)
      fw_copy<P, D>(static_cast<const P*>(A.embed), static_cast<D*>(A.d_embed), A.n_embed, b * FW_BLOCK, plain);
    const int64_t nv = A.value_embed ? (A.n_value_embed + FW_BLOCK - 1) / FW_BLOCK : 0;
    for (int64_t b = blockIdx.x; b < nv; b += gridDim.x)
      fw_copy<P, D>(static_cast<const P*>(A.value_embed), static_cast<D*>(A.d_value_embed), A.n_value_embed, b * FW_BLOCK,
                    plain);
    return;
  }
  const uv_fuse_layer& Y = A.layer[l];
  auto lam = [&](const void* p) { return rnd<D>(to_f32<P>(*static_cast<const P*>(p))); };   // as the step uses them
  if ((int)blockIdx.x == A.first[FW_NSEG]) {            // the small ones of the layer
    for (int i = tid; i < A.n_ve && Y.ve_gate; i += FW_THREADS)
      static_cast<D*>(Y.d_ve_gate)[i] = plain(static_cast<const P*>(Y.ve_gate)[i]);
    for (int i = tid; i < A.n_gate && Y.attn_gate; i += FW_THREADS)
      static_cast<D*>(Y.d_attn_gate)[i] = plain(static_cast<const P*>(Y.attn_gate)[i]);
    for (int i = tid; i < A.H && Y.xsa_alpha; i += FW_THREADS)
      Y.d_xsa[i] = tanhf(to_f32<P>(static_cast<const P*>(Y.xsa_alpha)[i]));
    if (tid < 4)
      Y.d_lambdas[tid] = lam(tid == 0 ? Y.resid_attn : tid == 1 ? Y.post_attn : tid == 2 ? Y.resid_mlp : Y.post_mlp);
    return;
  }
  int seg = 0;
  while (seg + 1 < FW_NSEG && (int)blockIdx.x >= A.first[seg + 1]) ++seg;
  const int64_t i0 = (int64_t)((int)blockIdx.x - A.first[seg]) * FW_BLOCK;
  const P* src = static_cast<const P*>(seg == 0 ? Y.wq : seg == 1 ? Y.wk : seg == 2 ? Y.wv : seg == 3 ? Y.wo
                                       : seg == 4 ? Y.w_gate : seg == 5 ? Y.w_up : Y.w_down);
  const int64_t n = A.n[seg];
  if (seg < 3) {
    D* dst = static_cast<D*>(Y.d_wqkv) + (seg > 0 ? A.n[0] : 0) + (seg > 1 ? A.n[1] : 0);
    const float s = to_f32<P>(*static_cast<const P*>(Y.qkv_scale));
    fw_copy<P, D>(src, dst, n, i0, [s](P x) { return from_f32<D>(to_f32<P>(from_f32<P>(to_f32<P>(x) * s))); });
  } else if (seg == 4 || seg == 5) {
    fw_copy<P, D>(src, static_cast<D*>(Y.d_gu) + (seg == 5 ? A.n[4] : 0), n, i0, plain);
  } else if (!A.fold) {
    if (seg == 6) {
      fw_copy<P, D>(src, static_cast<D*>(Y.d_down), n, i0, plain);
    } else {
      const float s = to_f32<P>(*static_cast<const P*>(Y.o_scale));
      fw_copy<P, D>(src, static_cast<D*>(Y.d_wo), n, i0,
                    [s](P x) { return from_f32<D>(to_f32<P>(from_f32<P>(to_f32<P>(x) * s))); });
    }
  } else {
    // the stream the kernels carry is x / s: s the product of the residual lambdas so far
    __shared__ float r[2 * FW_MAXL];
    for (int i = tid; i < 2 * (l + 1); i += FW_THREADS)
      r[i] = lam(i & 1 ? A.layer[i >> 1].resid_mlp : A.layer[i >> 1].resid_attn);
    const float post = lam(seg == 3 ? Y.post_attn : Y.post_mlp);
    const float o = seg == 3 ? to_f32<P>(*static_cast<const P*>(Y.o_scale)) : 1.0f;
    __syncthreads();
    double s = 1.0;
    for (int i = 0; i < 2 * l + (seg == 3 ? 1 : 2); ++i) s *= (double)r[i];
    const float c = (float)((double)post / s);
    if (seg == 6 && i0 == 0 && tid == 0) {
      const float least = fminf(fabsf(r[2 * l]), fabsf(r[2 * l + 1]));
      const double a = fabs(s);
      if (!(least >= 0.015625f) || !(a > 1.0 / (double)A.limit && a < (double)A.limit)) atomicOr(A.status, 1);
    }
    D* dst = static_cast<D*>(seg == 3 ? Y.d_wo : Y.d_down);
    if (seg == 3) fw_copy<P, D>(src, dst, n, i0, [o, c](P x) { return from_f32<D>(to_f32<P>(x) * o * c); });
    else fw_copy<P, D>(src, dst, n, i0, [c](P x) { return from_f32<D>(to_f32<P>(x) * c); });
  }
}

template <typename P, typename D> static int launch_fuse(const FuseP& A, cudaStream_t st) {
  const dim3 grid((unsigned)(A.first[FW_NSEG] + 1), (unsigned)(A.L + 1));
  fuse_weights_kernel<P, D><<<grid, FW_THREADS, 0, st>>>(A);
  return check_launch();
}

}  // namespace uv

extern "C" int uv_fuse_weights(const uv_fuse_args* a, void* stream) {
  using namespace uv;
  if (!a || !a->h_layers || !a->embed || !a->d_embed || !a->status) return UV_ERR_ARG;
  if (a->n_layers < 1 || a->d < 1 || a->H < 1 || a->K < 1 || a->hd < 1 || a->f < 1 || a->vocab < 1) return UV_ERR_ARG;
  if (a->n_layers > FW_MAXL) return UV_ERR_SHAPE;
  if ((a->value_embed == nullptr) != (a->d_value_embed == nullptr)) return UV_ERR_ARG;
  if (a->dst_dtype != UV_F16 && a->dst_dtype != UV_BF16) return UV_ERR_DTYPE;
  FuseP A{};
  for (int l = 0; l < a->n_layers; ++l) {
    const uv_fuse_layer& y = a->h_layers[l];
    for (const void* p : {y.wq, y.wk, y.wv, y.wo, y.w_gate, y.w_up, y.w_down, y.qkv_scale, y.o_scale, y.resid_attn,
                          y.post_attn, y.resid_mlp, y.post_mlp, (const void*)y.d_wqkv, (const void*)y.d_wo,
                          (const void*)y.d_gu, (const void*)y.d_down, (const void*)y.d_lambdas})
      if (!p) return UV_ERR_ARG;
    if ((y.ve_gate && !y.d_ve_gate) || (y.attn_gate && !y.d_attn_gate) || (y.xsa_alpha && !y.d_xsa)) return UV_ERR_ARG;
    A.layer[l] = y;
  }
  const int64_t d = a->d, q = (int64_t)a->H * a->hd, kv = (int64_t)a->K * a->hd, f = a->f;
  const int64_t n[FW_NSEG] = {q * d, kv * d, kv * d, d * q, f * d, f * d, d * f};
  int64_t at = 0;
  for (int s = 0; s < FW_NSEG; ++s) {
    A.n[s] = n[s], A.first[s] = (int)at;
    at += (n[s] + FW_BLOCK - 1) / FW_BLOCK;
  }
  if (at > 0x7ffffff0) return UV_ERR_SHAPE;
  A.first[FW_NSEG] = (int)at;
  A.embed = a->embed, A.d_embed = a->d_embed, A.n_embed = a->vocab * d;
  A.value_embed = a->value_embed, A.d_value_embed = a->d_value_embed, A.n_value_embed = a->vocab * kv;
  A.L = a->n_layers, A.H = a->H, A.n_ve = a->K * a->ve_ch, A.n_gate = a->H * a->gate_ch, A.fold = a->fold;
  A.limit = a->dst_dtype == UV_BF16 ? 16777216.0f : 64.0f;   // fp16 has 5 exponent bits: keep the stream near x
  A.status = a->status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool half = a->dst_dtype == UV_F16;
  switch (a->src_dtype) {
    case UV_F32: return half ? launch_fuse<float, __half>(A, st) : launch_fuse<float, __nv_bfloat16>(A, st);
    case UV_F16: return half ? launch_fuse<__half, __half>(A, st) : launch_fuse<__half, __nv_bfloat16>(A, st);
    case UV_BF16:
      return half ? launch_fuse<__nv_bfloat16, __half>(A, st) : launch_fuse<__nv_bfloat16, __nv_bfloat16>(A, st);
    default: return UV_ERR_DTYPE;
  }
}
