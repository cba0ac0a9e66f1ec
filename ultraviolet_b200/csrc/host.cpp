// Host paths that are called often enough for their Python to cost more than their kernels, as one extension module
// (ultraviolet_b200._uvhost): reading tensor metadata, filling argument blocks and launching through libuvdecode's C ABI.
// Each function returns None for arguments it does not take as they are (other devices or layouts, tensor subclasses,
// dispatch modes); the caller's Python then handles or rejects them.
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <cublas_v2.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/uvdecode.h"

namespace {

using at::Tensor;

// ---- libuvdecode, loaded by the ctypes binding before
struct Lib {
  decltype(&uv_error_string) error_string;
  decltype(&uv_last_cuda_error) last_cuda_error;
  decltype(&uv_default_splits) default_splits;
  decltype(&uv_decode_attn) decode_attn;
  decltype(&uv_decode_attn_workspace_bytes) workspace_bytes;
  decltype(&uv_sample) sample;
  decltype(&uv_embed_norm_rope) embed_norm_rope;
  decltype(&uv_embed_norm) embed_norm;
  decltype(&uv_qkv_post_args) qkv_post;
  decltype(&uv_prefill_attn) prefill_attn;
  decltype(&uv_swiglu_rs) swiglu_rs;
  decltype(&uv_pack_prompts) pack_prompts;
  decltype(&uv_gather_norm) gather_norm;
};
Lib L;
PyObject* error_type = nullptr;

void init(const std::string& path, py::object uv_error) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
  auto get = [&](const char* name) {
    void* p = dlsym(h, name);
    if (!p) throw std::runtime_error(path + " has no symbol " + name);
    return p;
  };
#define UV_GET(field, name) L.field = reinterpret_cast<decltype(L.field)>(get(name))
  UV_GET(error_string, "uv_error_string");
  UV_GET(last_cuda_error, "uv_last_cuda_error");
  UV_GET(default_splits, "uv_default_splits");
  UV_GET(decode_attn, "uv_decode_attn");
  UV_GET(workspace_bytes, "uv_decode_attn_workspace_bytes");
  UV_GET(sample, "uv_sample");
  UV_GET(embed_norm_rope, "uv_embed_norm_rope");
  UV_GET(embed_norm, "uv_embed_norm");
  UV_GET(qkv_post, "uv_qkv_post_args");
  UV_GET(prefill_attn, "uv_prefill_attn");
  UV_GET(swiglu_rs, "uv_swiglu_rs");
  UV_GET(pack_prompts, "uv_pack_prompts");
  UV_GET(gather_norm, "uv_gather_norm");
#undef UV_GET
  error_type = uv_error.release().ptr();
}

void check(int code, const char* what) {
  if (code == UV_OK) return;
  std::string msg = std::string(what) + ": " + L.error_string(code);
  if (code == UV_ERR_CUDA) msg += " [cudaError " + std::to_string(L.last_cuda_error()) + "]";
  msg += " (code " + std::to_string(code) + ")";
  PyErr_SetString(error_type, msg.c_str());
  throw py::error_already_set();
}

int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return UV_F32;
    case at::kHalf: return UV_F16;
    case at::kBFloat16: return UV_BF16;
    case at::kChar: return UV_I8;
    default: return -1;
  }
}

// a tensor whose metadata and memory can be taken at face value on CUDA device `dev` (no wrapper, nor a view that stands for
// other values than those in memory)
bool plain(const Tensor& t, c10::Device dev) {
  constexpr c10::DispatchKeySet others({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                        c10::DispatchKey::Conjugate, c10::DispatchKey::ZeroTensor,
                                        c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
  return t.defined() && t.device() == dev && t.layout() == at::kStrided && !t.key_set().has_any(others) &&
         !(t.requires_grad() && at::GradMode::is_enabled()) && !t._fw_grad(0).defined();
}
// nothing watches or rewrites the calls of this thread: no dispatch or function mode, transform or tracer
bool modes_off() {
  constexpr c10::DispatchKeySet watchers({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::Tracer,
                                          c10::DispatchKey::Functionalize, c10::DispatchKey::PreDispatch,
                                          c10::DispatchKey::Python, c10::DispatchKey::PythonDispatcher});
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
         !c10::impl::tls_local_dispatch_key_set().included_.has_any(watchers);
}
// the tensor of a Python object that is a torch.Tensor or a parameter, not one of a subclass; else null
const Tensor* exact(py::handle h) {
  return THPVariable_CheckExact(h.ptr()) ? &THPVariable_Unpack(h.ptr()) : nullptr;
}
// a call on these tensors may go to kernels directly: memory on one CUDA device, no gradient wanted, nothing watching
bool plain_call(const std::vector<py::object>& objects) {
  if (!modes_off()) return false;
  for (const py::object& o : objects) {
    const Tensor* t = exact(o);
    if (!t || !t->is_cuda() || !plain(*t, exact(objects[0])->device())) return false;
  }
  return true;
}
const void* ro(const Tensor& t) { return t.const_data_ptr(); }

// ---- kernels.decode_attention on an int8 cache
// slots really allocated per row of [:, :, :S] views of a longer allocation (kernels/decode_attn.py:_row_alloc)
int64_t row_alloc(const Tensor& k, const Tensor& v, const Tensor& ks, const Tensor& vs, int64_t S) {
  const int64_t hd = k.size(3);
  if (k.stride(2) != hd || k.stride(1) % hd) return S;
  const int64_t alloc = k.stride(1) / hd;
  if (alloc <= S || v.stride(1) != alloc * hd || ks.stride(1) != alloc || vs.stride(1) != alloc) return S;
  const Tensor* t[4] = {&k, &v, &ks, &vs};
  for (int i = 0; i < 4; ++i) {
    const int64_t row = i < 2 ? alloc * hd : alloc;
    const int64_t last = t[i]->storage_offset() + (t[i]->size(0) - 1) * t[i]->stride(0) +
                         (t[i]->size(1) - 1) * t[i]->stride(1) + row;
    if (last * (int64_t)t[i]->element_size() > (int64_t)t[i]->storage().nbytes()) return S;
  }
  return alloc;
}

constexpr int64_t kAutoSplits = INT32_MIN;

std::optional<Tensor> decode_attention(py::handle hq, py::handle hk, py::handle hv, py::handle hpos, py::handle hstarts,
                                       double scale, int64_t window, int64_t ring, py::handle hks, py::handle hvs,
                                       int64_t ctx, int64_t splits) {
  const Tensor* in[7];
  const py::handle from[7] = {hq, hk, hv, hpos, hstarts, hks, hvs};
  for (int i = 0; i < 7; ++i)
    if (!(in[i] = exact(from[i]))) return std::nullopt;
  const Tensor &q_ = *in[0], &k = *in[1], &v = *in[2], &pos = *in[3], &starts = *in[4], &ks = *in[5], &vs = *in[6];
  if (!q_.is_cuda() || !modes_off()) return std::nullopt;
  const c10::Device dev = q_.device();
  for (const Tensor* t : {&q_, &k, &v, &pos, &starts, &ks, &vs})
    if (!plain(*t, dev)) return std::nullopt;
  if (q_.dim() != 3 || k.dim() != 4 || v.dim() != 4 || ks.dim() != 3 || vs.dim() != 3 || k.scalar_type() != at::kChar ||
      v.scalar_type() != at::kChar || ks.scalar_type() != at::kHalf || vs.scalar_type() != at::kHalf ||
      pos.scalar_type() != at::kLong || starts.scalar_type() != at::kLong || !pos.is_contiguous() ||
      !starts.is_contiguous() || q_.stride(2) != 1 || (q_.scalar_type() != at::kHalf && q_.scalar_type() != at::kBFloat16))
    return std::nullopt;
  const int64_t B = q_.size(0), H = q_.size(1), hd = q_.size(2), KH = k.size(1), S = k.size(2);
  if (B == 0 || KH == 0 || pos.numel() != B || starts.numel() != B) return std::nullopt;
  c10::cuda::CUDAGuard guard(dev);
  if (splits == kAutoSplits) {
    int64_t c = ctx > 0 ? ctx : S;
    if (window > 0 && window < c) c = window;
    splits = L.default_splits((int)(B * KH), (int)c, at::cuda::getCurrentDeviceProperties()->multiProcessorCount);
  }
  Tensor out = at::empty({B, H, hd}, q_.options()), ws;
  uv_attn_args a{};
  a.q = ro(q_), a.q_dtype = code_of(q_.scalar_type()), a.sqb = q_.stride(0), a.sqh = q_.stride(1);
  a.k_cache = ro(k), a.v_cache = ro(v), a.kv_dtype = UV_I8;
  a.skb = k.stride(0), a.skh = k.stride(1), a.sks = k.stride(2);
  a.svb = v.stride(0), a.svh = v.stride(1), a.svs = v.stride(2);
  a.k_scale = static_cast<const uint16_t*>(ro(ks)), a.v_scale = static_cast<const uint16_t*>(ro(vs));
  a.ssb = ks.stride(0), a.ssh = ks.stride(1), a.stb = vs.stride(0), a.sth = vs.stride(1);
  a.pos = pos.const_data_ptr<int64_t>(), a.starts = starts.const_data_ptr<int64_t>();
  a.out = out.mutable_data_ptr(), a.sob = out.stride(0), a.soh = out.stride(1);
  a.B = (int)B, a.H = (int)H, a.KH = (int)KH, a.hd = (int)hd, a.S = (int)S, a.S_alloc = (int)row_alloc(k, v, ks, vs, S);
  a.window = (int)window, a.ring = ring < 0 ? window > 0 : ring != 0, a.scale = (float)scale, a.num_splits = (int)splits;
  if (splits > 1) {
    const size_t n = L.workspace_bytes((int)B, (int)KH, (int)(H / KH), (int)hd, (int)splits);
    if (n) {
      ws = at::empty({(int64_t)(n / 4)}, q_.options().dtype(at::kFloat));
      a.workspace = ws.mutable_data_ptr(), a.workspace_bytes = n;
    }
  }
  check(L.decode_attn(&a, at::cuda::getCurrentCUDAStream().stream()), "uv_decode_attn");
  return out;
}

// ---- kernels.fused_sample
std::optional<std::pair<Tensor, Tensor>> fused_sample(py::handle hx, py::handle hu, double a, double b, double c,
                                                      double temperature, double top_p) {
  const Tensor *px = exact(hx), *pu = exact(hu);
  if (!px || !pu) return std::nullopt;
  const Tensor &x = *px, &u = *pu;
  if (!x.is_cuda() || !modes_off() || !plain(x, x.device()) || !plain(u, x.device())) return std::nullopt;
  if (x.dim() != 2 || x.stride(1) != 1 || u.scalar_type() != at::kFloat || !u.is_contiguous() || u.numel() < x.size(0))
    return std::nullopt;
  const int code = code_of(x.scalar_type());
  if (code < 0 || code == UV_I8) return std::nullopt;
  c10::cuda::CUDAGuard guard(x.device());
  Tensor tok = at::empty({x.size(0)}, x.options().dtype(at::kLong)), lp = at::empty({x.size(0)}, x.options().dtype(at::kFloat));
  check(L.sample(ro(x), code, x.stride(0), (int)x.size(0), (int)x.size(1), 0, (float)a, (float)b, (float)c,
                 (float)temperature, (float)top_p, u.const_data_ptr<float>(), 0, nullptr, nullptr,
                 tok.mutable_data_ptr<int64_t>(), lp.mutable_data_ptr<float>(), nullptr, nullptr,
                 at::cuda::getCurrentCUDAStream().stream()),
        "uv_sample");
  return std::make_pair(tok, lp);
}

// c = x . w^T (accumulate: c += x . w^T) for contiguous row-major x (M, K), w (N, K), c (M, N): the cuBLAS call that torch.mm
// makes (torch's handle, workspace and stream; fp32 accumulation) while its switches are at their defaults
// (engine.py: default_matmul), without the operator dispatch in front of it, which costs more than the launch
void gemm(int M, const void* x, const Tensor& w, void* c, bool accumulate = false) {
  const int K = (int)w.size(1), N = (int)w.size(0);
  const cudaDataType_t type = w.scalar_type() == at::kHalf ? CUDA_R_16F : CUDA_R_16BF;
  const float one = 1.0f, beta = accumulate ? 1.0f : 0.0f;
  const cublasStatus_t s = cublasGemmEx(at::cuda::getCurrentCUDABlasHandle(), CUBLAS_OP_T, CUBLAS_OP_N, N, M, K, &one,
                                        ro(w), type, K, x, type, K, &beta, c, type, N, CUBLAS_COMPUTE_32F,
                                        CUBLAS_GEMM_DEFAULT_TENSOR_OP);
  TORCH_CHECK(s == CUBLAS_STATUS_SUCCESS, "cublasGemmEx failed with status ", (int)s);
}

// ---- what a prepared launch over a list of tensors was prepared for: their memory, types, sizes and strides
class TensorFacts {
 public:
  explicit TensorFacts(const std::vector<Tensor>& ts) {
    for (const Tensor& t : ts)
      facts_.push_back({t.const_data_ptr(), t.scalar_type(), t.device(), t.sizes().vec(), t.strides().vec(), plain(t), t.is_contiguous()});
  }
  bool match(const std::vector<Tensor>& ts) const {
    if (ts.size() != facts_.size()) return false;
    for (size_t i = 0; i < ts.size(); ++i) {
      const Fact& f = facts_[i];
      const Tensor& t = ts[i];
      if (!f.plain || !plain(t) || t.const_data_ptr() != f.data || t.scalar_type() != f.type || t.device() != f.device ||
          t.sizes() != f.sizes || t.strides() != f.strides)
        return false;
    }
    return true;
  }
  // all of them contiguous, of one type, on t's device
  bool uniform_with(const Tensor& t) const {
    for (const Fact& f : facts_)
      if (!f.plain || !f.contiguous || f.type != facts_[0].type || f.device != t.device()) return false;
    return !facts_.empty();
  }

 private:
  struct Fact {
    const void* data;
    at::ScalarType type;
    c10::Device device;
    std::vector<int64_t> sizes, strides;
    bool plain, contiguous;
  };
  static bool plain(const Tensor& t) {
    return t.layout() == at::kStrided && !t.unsafeGetTensorImpl()->key_set().has(c10::DispatchKey::Python);
  }
  std::vector<Fact> facts_;
};

// ---- one packed prompt pass through every layer (DecodeEngine.trunk with packed=..., folded stream)
struct LayerFacts {
  Tensor wqkv, wo, gu, down;
  const void *ve_gate, *attn_gate;
  const float* xsa_alpha;
  bool ring, rope;
  int window;
};

class PrefillTrunk {
 public:
  PrefillTrunk(std::vector<Tensor> wqkv, std::vector<Tensor> wo, std::vector<Tensor> gu, std::vector<Tensor> down,
               std::vector<int64_t> ve_gate, std::vector<int64_t> attn_gate, std::vector<int64_t> xsa,
               std::vector<bool> ring, std::vector<bool> rope, std::vector<int64_t> window, Tensor embed,
               std::optional<Tensor> value_embed, Tensor inv_freq, int64_t H, int64_t K, int64_t hd, int64_t f,
               int64_t n_pairs, int64_t gate_ch, int64_t ve_ch, double scale, double xsa_eps)
      : embed_(embed), value_embed_(value_embed), inv_freq_(inv_freq), H_((int)H), K_((int)K), hd_((int)hd), f_((int)f),
        n_pairs_((int)n_pairs), gate_ch_((int)gate_ch), ve_ch_((int)ve_ch), scale_((float)scale), eps_((float)xsa_eps) {
    for (size_t l = 0; l < wqkv.size(); ++l)
      layers_.push_back({wqkv[l], wo[l], gu[l], down[l], reinterpret_cast<const void*>(ve_gate[l]),
                         reinterpret_cast<const void*>(attn_gate[l]), reinterpret_cast<const float*>(xsa[l]), ring[l],
                         rope[l], (int)window[l]});
    code_ = code_of(embed.scalar_type());
  }

  // oob: device word that counts skipped cache writes; k .. vs: the state's layers.  Returns the normed rows of the prompts'
  // last tokens (zeros for an empty prompt).  M >= 1.
  Tensor run(const Tensor& idx, const Tensor& starts, const Tensor& rows, int64_t M, int64_t max_tiles, Tensor oob,
             const std::vector<Tensor>& k, const std::vector<Tensor>& v, const std::vector<Tensor>& ks,
             const std::vector<Tensor>& vs) {
    for (const auto* layers : {&k, &v, &ks, &vs})
      TORCH_CHECK_INDEX(layers->size() >= layers_.size(), "the decode state has ", layers->size(), " layers, the model ",
                        layers_.size());
    at::AutoDispatchBelowADInplaceOrView below;         // no autograd bookkeeping on the library calls below
    c10::cuda::CUDAGuard guard(embed_.device());
    void* st = at::cuda::getCurrentCUDAStream().stream();
    const int n = (int)idx.size(0), T = (int)idx.size(1), d = (int)embed_.size(1), m = (int)M;
    const int64_t vocab = embed_.size(0);
    // The activations of the pass, one block of the allocator's pool that goes back to it at the end: passes come in every
    // size, so buffers kept per size would add up without bound, and passes on several streams or threads have their own.
    const int slots = H_ + 2 * K_;
    const int64_t widths[8] = {2 * d, 2 * d, 2 * slots * hd_, 2 * H_ * hd_, 4 * f_, 2 * f_, 4 * H_, 8 * n_pairs_};
    int64_t at[9] = {0};
    for (int b = 0; b < 8; ++b) at[b + 1] = at[b] + (widths[b] * M + 255) / 256 * 256;
    const Tensor block = at::empty({at[8]}, embed_.options().dtype(at::kByte));
    char* const base = static_cast<char*>(block.mutable_data_ptr());
    void *const x = base, *const xn = base + at[1], *const qkv = base + at[2], *const z = base + at[3];
    void *const gu = base + at[4], *const act = base + at[5];
    float *const gate = reinterpret_cast<float*>(base + at[6]), *const rope_cs = reinterpret_cast<float*>(base + at[7]);
    // tok, pos, row, last of every packed row and the two prefix sums, in one allocation each
    Tensor packed = at::empty({4, M}, idx.options()), cu = at::empty({2, n + 1}, idx.options().dtype(at::kInt));
    int64_t *tok = packed.mutable_data_ptr<int64_t>(), *pos = tok + M, *row = pos + M, *last = row + M;
    int32_t *cu_p = cu.mutable_data_ptr<int32_t>(), *tile_p = cu_p + n + 1;
    check(L.pack_prompts(idx.const_data_ptr<int64_t>(), idx.stride(0), T, starts.const_data_ptr<int64_t>(),
                         rows.const_data_ptr<int64_t>(), n, M, cu_p, tile_p, tok, pos, row, last, st),
          "uv_pack_prompts");
    if (n_pairs_ > 0)
      check(L.embed_norm_rope(tok, ro(embed_), code_, vocab, d, x, xn, m, pos, inv_freq_.const_data_ptr<float>(), n_pairs_, rope_cs,
                              st),
            "uv_embed_norm_rope");
    else
      check(L.embed_norm(tok, ro(embed_), code_, vocab, d, x, xn, m, st), "uv_embed_norm");
    for (size_t l = 0; l < layers_.size(); ++l) {
      const LayerFacts& y = layers_[l];
      gemm(m, x, y.wqkv, qkv);
      uv_qkv_args q{};
      q.qkv = qkv, q.xn = x, q.tok = tok, q.pos = pos, q.row_map = row, q.last_pos = last;
      q.value_embed = value_embed_ ? ro(*value_embed_) : nullptr, q.ve_gate = y.ve_gate;
      if (y.rope && n_pairs_ > 0) q.inv_freq = inv_freq_.const_data_ptr<float>(), q.rope_cs = rope_cs;
      q.k_cache = k[l].mutable_data_ptr<int8_t>(), q.v_cache = v[l].mutable_data_ptr<int8_t>();
      q.k_scale = static_cast<uint16_t*>(ks[l].mutable_data_ptr()), q.v_scale = static_cast<uint16_t*>(vs[l].mutable_data_ptr());
      q.oob_count = oob.mutable_data_ptr<int>(), q.dtype = code_, q.vocab = vocab, q.B = m, q.H = H_, q.K = K_, q.hd = hd_;
      q.d = d, q.S = (int)k[l].size(2), q.S_alloc = (int)(k[l].stride(1) / hd_), q.ring = y.ring, q.ve_ch = ve_ch_;
      q.n_pairs = n_pairs_, q.xn_raw = 1;
      if (gate_ch_ > 0) q.gate_w = y.attn_gate, q.gate_out = gate, q.gate_ch = gate_ch_;
      check(L.qkv_post(&q, st), "uv_qkv_post");
      uv_prefill_attn_args p{};
      p.qkv = qkv, p.dtype = code_, p.ld = slots * hd_, p.cu_seqlens = cu_p, p.tile_cu = tile_p, p.n_seq = n;
      p.max_tiles = (int)max_tiles, p.out = z, p.ldo = H_ * hd_, p.H = H_, p.K = K_, p.hd = hd_;
      p.window = y.window, p.scale = scale_, p.xsa_alpha = y.xsa_alpha, p.xsa_eps = eps_;
      if (gate_ch_ > 0) p.gate_vals = gate;
      check(L.prefill_attn(&p, st), "uv_prefill_attn");
      gemm(m, z, y.wo, x, true);
      gemm(m, x, y.gu, gu);
      check(L.swiglu_rs(gu, x, code_, d, f_, act, m, st), "uv_swiglu_rs");
      gemm(m, act, y.down, x, true);
    }
    Tensor out = at::empty({n, d}, embed_.options());
    check(L.gather_norm(x, code_, d, cu_p, n, out.mutable_data_ptr(), st), "uv_gather_norm");
    return out;
  }

 private:
  std::vector<LayerFacts> layers_;
  Tensor embed_;
  std::optional<Tensor> value_embed_;
  Tensor inv_freq_;
  int H_, K_, hd_, f_, n_pairs_, gate_ch_, ve_ch_, code_ = -1;
  float scale_, eps_;
};

}  // namespace

PYBIND11_MODULE(_uvhost, m) {
  m.def("init", &init);
  m.def("plain_call", &plain_call);
  m.def("decode_attention", &decode_attention);
  m.def("fused_sample", &fused_sample);
  py::class_<TensorFacts>(m, "TensorFacts")
      .def(py::init<const std::vector<Tensor>&>())
      .def("match", &TensorFacts::match)
      .def("uniform_with", &TensorFacts::uniform_with);
  py::class_<PrefillTrunk>(m, "PrefillTrunk")
      .def(py::init<std::vector<Tensor>, std::vector<Tensor>, std::vector<Tensor>, std::vector<Tensor>, std::vector<int64_t>,
                    std::vector<int64_t>, std::vector<int64_t>, std::vector<bool>, std::vector<bool>, std::vector<int64_t>,
                    Tensor, std::optional<Tensor>, Tensor, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                    double, double>())
      .def("run", &PrefillTrunk::run);
}
