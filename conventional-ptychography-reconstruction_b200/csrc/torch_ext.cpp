// torch_ext.cpp -- the fused loss, the complex MLP and the Fourier upsampling as C++
// torch autograd functions over the C ABI.
//
// fused_loss (Recovery.py:288-307, backward at :316) needs an autograd node
// whose backward scales the gradients the forward already computed.  Written
// in Python, every step pays the Python Function machinery twice (forward and,
// from the autograd engine's thread, backward).  Here the node is C++: the
// forward calls ptycho_fwd_adj, the backward ptycho_scale_pair, both through
// addresses handed over by `bind` (taken from the ctypes handle of
// libptycho_b200.so, so there is one copy of the library in the process).
// The MLP's Python Function converted eleven parameters to views, and as many
// gradients back, on every call: 327 us of host work for a forward and backward, the
// time of 600,000 coordinates on the GPU; 204 us here (an upsampling 107, now 62).
// No computation happens here; a non-zero library status raises RuntimeError,
// bad arguments raise ValueError / TypeError as the Python path does.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cstdint>
#include <mutex>
#include <optional>
#include <unordered_map>

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;

typedef int (*fwd_adj_fn)(const float*, int, int, const float*, int, int, const int32_t*, const float*, int,
                          const int32_t*, int, int, double*, double*, float*, float*, unsigned, void*, size_t,
                          int32_t*, void*);
typedef int (*scale_pair_fn)(const float*, float*, long long, const float*, float*, long long, const double*,
                             void*);
typedef size_t (*ws_size_fn)(int, int, int, int, int);
typedef const char* (*status_string_fn)(int);
typedef int (*cmlp_pack_fn)(const float*, const float*, const float*, const float*, const float*, const float*,
                            const float*, const float*, const float*, const float*, const float*, void*, void*);
typedef int (*cmlp_fwd_fn)(const void*, const float*, int, float*, int32_t*, void*);
typedef int (*cmlp_bwd_fn)(const void*, const float*, const float*, int, float*, float*, float*, void*, size_t,
                           int32_t*, void*);
typedef int (*upsample_fn)(const float*, int, int, int, float*, void*, size_t, void*);

fwd_adj_fn g_fwd_adj = nullptr;
scale_pair_fn g_scale_pair = nullptr;
ws_size_fn g_ws_size = nullptr;
status_string_fn g_status_string = nullptr;

cmlp_pack_fn g_cmlp_pack = nullptr;
cmlp_fwd_fn g_cmlp_fwd[2] = {nullptr, nullptr};  // [N][32] features, feature-major
cmlp_bwd_fn g_cmlp_bwd[2] = {nullptr, nullptr};
size_t (*g_cmlp_bwd_ws)(int) = nullptr;
int64_t g_cmlp_packed_bytes = 0, g_cmlp_grad_floats = 0;
upsample_fn g_upsample[2] = {nullptr, nullptr};  // forward, adjoint
size_t (*g_upsample_ws)(int, int, int) = nullptr;

constexpr int64_t kMaxProbeDim = 4096;

void check(int rc, const char* where) {
  TORCH_CHECK(rc == 0, where, ": ", g_status_string ? g_status_string(rc) : "error", " (status ", rc, ")");
}

// as a kernel reads it: contiguous, no pending conjugation or negation (contiguous()
// alone keeps those)
Tensor plain(Tensor t) {
  if (t.is_conj()) t = t.resolve_conj();
  if (t.is_neg()) t = t.resolve_neg();
  return t.contiguous();
}

template <typename T>
T* fptr(const Tensor& t) {
  return t.defined() ? reinterpret_cast<T*>(t.data_ptr()) : nullptr;
}

// One growing workspace per (device, stream): calls on one stream are ordered,
// calls on different streams must not share scratch.  The Python entry points
// use the same cache, so a process holds one workspace per stream.
std::mutex g_ws_mu;
std::unordered_map<uint64_t, Tensor> g_ws;

// At most kMaxWorkspaces entries: a caller that keeps creating streams would
// otherwise keep every old stream's workspace alive.  Dropping an entry is
// safe: each workspace was allocated on its own stream, and the caching
// allocator reuses freed memory in that stream's order.
constexpr size_t kMaxWorkspaces = 16;

Tensor workspace_on(const Tensor& like, cudaStream_t s, size_t bytes) {
  const uint64_t key = (uint64_t(like.device().index()) << 56) ^ reinterpret_cast<uintptr_t>(s);
  std::lock_guard<std::mutex> lock(g_ws_mu);
  if (g_ws.size() >= kMaxWorkspaces && g_ws.find(key) == g_ws.end()) g_ws.clear();
  Tensor& w = g_ws[key];
  if (!w.defined() || size_t(w.numel()) < bytes)
    w = torch::empty({int64_t(bytes < 256 ? 256 : bytes)}, like.options().dtype(torch::kUInt8));
  return w;
}

cudaStream_t current_stream(const Tensor& t) {
  return at::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

// Nothing throws inside the node's forward: the wrapper below checks and
// converts every argument before apply(), and a library error is handed out
// through `rc` and raised after apply() has returned.
class FusedLoss : public torch::autograd::Function<FusedLoss> {
 public:
  // O [H, W] c64, P [M, N] c64 on one CUDA device; tl [F, 2] int32, Imeas
  // [F, M, N] float32, batch [B] int32 frame ids (none: all F frames) and the
  // status word [1] int32, all contiguous on that device.  The batch is an
  // optional (not an undefined tensor): autograd records a device for every
  // tensor argument.
  static Tensor forward(AutogradContext* ctx, Tensor O, Tensor P, const Tensor& tl, const Tensor& Imeas,
                        int64_t loss_code, const std::optional<Tensor>& batch, const Tensor& status, bool need_grad,
                        int* rc) {
    O = plain(O);
    P = plain(P);
    const int64_t H = O.size(0), W = O.size(1), M = P.size(0), N = P.size(1);
    const int64_t F = tl.size(0);
    const bool has_batch = batch.has_value() && batch->defined();
    const int64_t B = has_batch ? batch->numel() : F;
    cudaStream_t s = current_stream(O);
    Tensor loss = torch::empty({}, O.options().dtype(torch::kFloat64));
    Tensor dO, dP;
    if (need_grad) {
      dO = torch::empty({H, W}, O.options());
      dP = torch::empty({M, N}, P.options());
    }
    Tensor ws = workspace_on(O, s, g_ws_size(int(H), int(W), int(M), int(N), int(B)));
    *rc = g_fwd_adj(fptr<const float>(O), int(H), int(W), fptr<const float>(P), int(M), int(N),
                    fptr<const int32_t>(tl), fptr<const float>(Imeas), int(F),
                    has_batch ? fptr<const int32_t>(*batch) : nullptr, int(B), int(loss_code), nullptr,
                    fptr<double>(loss), fptr<float>(dO), fptr<float>(dP), 0u, ws.data_ptr(), size_t(ws.numel()),
                    fptr<int32_t>(status), s);
    ctx->save_for_backward({dO, dP});
    return loss;
  }

  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    auto saved = ctx->get_saved_variables();
    const Tensor& dO = saved[0];
    const Tensor& dP = saved[1];
    const bool nO = ctx->needs_input_grad(0) && dO.defined() && grads[0].defined();
    const bool nP = ctx->needs_input_grad(1) && dP.defined() && grads[0].defined();
    Tensor gO, gP;
    if (nO || nP) {
      Tensor g = plain(grads[0].to(torch::kFloat64));
      gO = nO ? torch::empty_like(dO) : Tensor();
      gP = nP ? torch::empty_like(dP) : Tensor();
      // one launch scales both (out of place: the saved gradients stay valid for a second backward)
      check(g_scale_pair(nO ? fptr<const float>(dO) : nullptr, fptr<float>(gO), nO ? 2 * dO.numel() : 0,
                         nP ? fptr<const float>(dP) : nullptr, fptr<float>(gP), nP ? 2 * dP.numel() : 0,
                         fptr<const double>(g), current_stream(g)),
            "ptycho_scale_pair");
    }
    return {gO, gP, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

void bind(int64_t fwd_adj, int64_t scale_pair, int64_t ws_size, int64_t status_string) {
  g_fwd_adj = reinterpret_cast<fwd_adj_fn>(fwd_adj);
  g_scale_pair = reinterpret_cast<scale_pair_fn>(scale_pair);
  g_ws_size = reinterpret_cast<ws_size_fn>(ws_size);
  g_status_string = reinterpret_cast<status_string_fn>(status_string);
}

// fused_loss(O, P, tl, Imeas, loss_code, batch|None, status): the caller has
// checked the loss name and the complex64 dtypes
Tensor fused_loss(const Tensor& O, const Tensor& P, const Tensor& tl_in, const Tensor& Imeas_in,
                  int64_t loss_code, const std::optional<Tensor>& batch_in, const Tensor& status) {
  TORCH_CHECK(g_fwd_adj && g_scale_pair && g_ws_size, "bind() was not called");
  TORCH_CHECK_VALUE(O.is_cuda() && P.is_cuda(), "object and probe must be CUDA tensors (there is no CPU path)");
  TORCH_CHECK_VALUE(P.device() == O.device(), "object and probe must be on one device");
  TORCH_CHECK_TYPE(O.scalar_type() == torch::kComplexFloat && P.scalar_type() == torch::kComplexFloat,
                   "object and probe must be complex64");
  TORCH_CHECK_VALUE(O.dim() == 2, "object must be [H, W]");
  TORCH_CHECK_VALUE(P.dim() == 2 && P.size(0) >= 1 && P.size(0) <= kMaxProbeDim && P.size(1) >= 1 &&
                        P.size(1) <= kMaxProbeDim,
                    "probe must be [M, N] with 1 <= M, N <= ", kMaxProbeDim, ", got ", P.sizes());
  TORCH_CHECK_VALUE(status.is_cuda() && status.device() == O.device() && status.scalar_type() == torch::kInt32,
                    "status must be the device's int32 status word");
  const auto dev = O.device();
  c10::cuda::CUDAGuard guard(dev);
  // windows, measurements and frame ids carry no gradient (the node returns none for them)
  const Tensor tl = tl_in.detach().to(dev, torch::kInt32).contiguous();
  const Tensor Imeas = plain(Imeas_in.detach().to(dev, torch::kFloat32));
  std::optional<Tensor> batch;
  if (batch_in.has_value() && batch_in->defined()) batch = batch_in->detach().to(dev, torch::kInt32).contiguous();
  const int64_t F = tl.dim() == 2 ? tl.size(0) : -1;
  TORCH_CHECK_VALUE(tl.dim() == 2 && tl.size(1) == 2, "windows must be [F, 2] (tlY, tlX)");
  TORCH_CHECK_VALUE(Imeas.dim() == 3 && Imeas.size(0) == F && Imeas.size(1) == P.size(0) &&
                        Imeas.size(2) == P.size(1),
                    "measurements must be [F, M, N] = (", F, ", ", P.size(0), ", ", P.size(1), "), got ",
                    Imeas.sizes());
  const bool need = torch::GradMode::is_enabled() && (O.requires_grad() || P.requires_grad());
  int rc = 0;
  Tensor loss = FusedLoss::apply(O, P, tl, Imeas, loss_code, batch, status, need, &rc);
  check(rc, "ptycho_fwd_adj");
  return loss;
}

// ---------------------------------------------------------------------------
// Complex MLP (cmlp.py): parameters in the order omega_0, weight, bias of three
// layers, output weight and bias.
// ---------------------------------------------------------------------------
constexpr int kCmlpParams = 11;

// a parameter's values as contiguous float32 (complex64 as pairs); no copy when
// that is what it is
Tensor floats_of(const Tensor& p) {
  Tensor t = p.detach();
  if (t.is_complex()) t = torch::view_as_real(plain(t));
  return plain(t).to(torch::kFloat32);
}

// [N, 32] float32 view of a feature-major [32, N] buffer (the encoder's output)
bool is_planar(const Tensor& x) {
  return x.dim() == 2 && x.size(1) == 32 && x.size(0) > 1 && x.stride(0) == 1 && x.stride(1) == x.size(0);
}

class Cmlp : public torch::autograd::Function<Cmlp> {
 public:
  // x [N, 32] float32, feature-major or contiguous (checked by the caller)
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& om1, const Tensor& W1, const Tensor& b1,
                        const Tensor& om2, const Tensor& W2, const Tensor& b2, const Tensor& om3, const Tensor& W3,
                        const Tensor& b3, const Tensor& Wo, const Tensor& bo, const Tensor& status, int* rc) {
    const Tensor ps[kCmlpParams] = {W1, b1, om1, W2, b2, om2, W3, b3, om3, Wo, bo};  // ptycho_cmlp_pack's order
    Tensor f[kCmlpParams];
    for (int i = 0; i < kCmlpParams; ++i) f[i] = floats_of(ps[i]);
    void* s = current_stream(x);
    const int64_t N = x.size(0);
    Tensor packed = torch::empty({g_cmlp_packed_bytes}, x.options().dtype(torch::kUInt8));
    Tensor y = torch::empty({N, 1}, x.options().dtype(torch::kComplexFloat));
    const int planar = is_planar(x);
    *rc = g_cmlp_pack(fptr<const float>(f[0]), fptr<const float>(f[1]), fptr<const float>(f[2]), fptr<const float>(f[3]),
                      fptr<const float>(f[4]), fptr<const float>(f[5]), fptr<const float>(f[6]), fptr<const float>(f[7]),
                      fptr<const float>(f[8]), fptr<const float>(f[9]), fptr<const float>(f[10]), packed.data_ptr(), s);
    if (*rc == 0)
      *rc = g_cmlp_fwd[planar](packed.data_ptr(), fptr<const float>(x), int(N), fptr<float>(y), fptr<int32_t>(status), s);
    ctx->save_for_backward({x, packed});
    ctx->saved_data["status"] = status;  // not a saved variable: reading it out clears it in place
    const Tensor in[kCmlpParams] = {om1, W1, b1, om2, W2, b2, om3, W3, b3, Wo, bo};
    std::vector<int64_t> types;
    std::vector<c10::IValue> sizes;
    for (const Tensor& p : in) {
      types.push_back(int64_t(p.scalar_type()));
      sizes.emplace_back(p.sizes().vec());
    }
    ctx->saved_data["types"] = types;
    ctx->saved_data["sizes"] = c10::ivalue::Tuple::create(sizes);
    return y;
  }

  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &packed = saved[1];
    const Tensor status = ctx->saved_data["status"].toTensor();
    c10::cuda::CUDAGuard guard(x.device());
    void* s = current_stream(x);
    const int64_t N = x.size(0);
    const Tensor gy = plain(grads[0].reshape({N}).to(torch::kComplexFloat));
    const int planar = is_planar(x);
    Tensor grad = torch::empty({g_cmlp_grad_floats}, x.options());
    Tensor ws = torch::empty({int64_t(g_cmlp_bwd_ws(int(N)))}, x.options().dtype(torch::kUInt8));
    // the features' gradient goes back in their own layout
    Tensor gx;
    if (ctx->needs_input_grad(0)) gx = planar ? torch::empty({32, N}, x.options()) : torch::empty({N, 32}, x.options());
    check(g_cmlp_bwd[planar](packed.data_ptr(), fptr<const float>(x), fptr<const float>(gy), int(N), fptr<float>(gx),
                             fptr<float>(grad), nullptr, ws.data_ptr(), size_t(ws.numel()), fptr<int32_t>(status), s),
          planar ? "ptycho_cmlp_backward_planar" : "ptycho_cmlp_backward");
    tensor_list out(1 + kCmlpParams + 2);
    if (gx.defined()) out[0] = planar ? gx.t() : gx;
    // offset and length of each parameter's gradient in the blob (floats), complex or not
    struct Part {
      int64_t off, n;
      bool cplx;
    };
    static constexpr Part parts[kCmlpParams] = {{1056, 1, false},   {0, 1024, false},   {1024, 32, false}, {3170, 1, false},
                                                {1058, 2048, true}, {3106, 64, true},   {5284, 1, false},  {3172, 2048, true},
                                                {5220, 64, true},   {5286, 64, true},   {5350, 2, true}};
    const auto types = ctx->saved_data["types"].toIntVector();
    const auto sizes = ctx->saved_data["sizes"].toTuple();
    for (int i = 0; i < kCmlpParams; ++i) {
      if (!ctx->needs_input_grad(1 + i)) continue;
      Tensor g = grad.narrow(0, parts[i].off, parts[i].n);
      if (parts[i].cplx) g = torch::view_as_complex(g.view({-1, 2}));
      out[1 + i] = g.reshape(sizes->elements()[i].toIntVector()).to(torch::ScalarType(types[i]));
    }
    return out;
  }
};

// (y [N, 1] complex64, library status of the forward)
std::pair<Tensor, int> cmlp(const Tensor& x_in, const std::vector<Tensor>& p, const Tensor& status) {
  TORCH_CHECK(g_cmlp_pack && g_cmlp_bwd_ws, "bind_inr() was not called");
  TORCH_CHECK_VALUE(x_in.is_cuda(), "features must be a CUDA tensor (there is no CPU path)");
  TORCH_CHECK_VALUE(x_in.dim() == 2 && x_in.size(1) == 32, "features must be [N, 32], got ", x_in.sizes());
  TORCH_CHECK_VALUE(p.size() == size_t(kCmlpParams), "the MLP has eleven parameters");
  // the library reads these sizes at the parameters' addresses
  struct Want {
    int64_t numel;
    bool cplx;
  };
  static constexpr Want want[kCmlpParams] = {{1, false}, {1024, false}, {32, false}, {1, false}, {1024, true}, {32, true},
                                             {1, false}, {1024, true},  {32, true},  {32, true}, {1, true}};
  for (int i = 0; i < kCmlpParams; ++i) {
    TORCH_CHECK_VALUE(p[i].device() == x_in.device(), "parameter ", i, " of the MLP is on ", p[i].device(),
                      ", the features are on ", x_in.device());
    TORCH_CHECK_VALUE(p[i].numel() == want[i].numel && p[i].is_complex() == want[i].cplx, "parameter ", i,
                      " of the MLP has shape ", p[i].sizes(), " and type ", p[i].scalar_type());
  }
  TORCH_CHECK_VALUE(status.device() == x_in.device() && status.scalar_type() == torch::kInt32,
                    "status must be the device's int32 status word");
  c10::cuda::CUDAGuard guard(x_in.device());
  Tensor x = x_in.to(torch::kFloat32).resolve_neg();
  if (!is_planar(x)) x = x.contiguous();
  int rc = 0;
  Tensor y = Cmlp::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8], p[9], p[10], status, &rc);
  return {y, rc};
}

// ---------------------------------------------------------------------------
// Fourier upsampling (resample.py)
// ---------------------------------------------------------------------------
class Upsample : public torch::autograd::Function<Upsample> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& x, int64_t s, int* rc) {
    const Tensor xc = plain(x.to(torch::kComplexFloat));
    const int64_t h = x.size(0), w = x.size(1);
    Tensor y = torch::empty({h * s, w * s}, xc.options());
    Tensor ws = torch::empty({int64_t(g_upsample_ws(int(h), int(w), int(s)))}, xc.options().dtype(torch::kUInt8));
    *rc = g_upsample[0](fptr<const float>(xc), int(h), int(w), int(s), fptr<float>(y), ws.data_ptr(), size_t(ws.numel()),
                        current_stream(xc));
    ctx->saved_data["h"] = h;
    ctx->saved_data["w"] = w;
    ctx->saved_data["s"] = s;
    return y;
  }

  static tensor_list backward(AutogradContext* ctx, tensor_list grads) {
    const int64_t h = ctx->saved_data["h"].toInt(), w = ctx->saved_data["w"].toInt(), s = ctx->saved_data["s"].toInt();
    const Tensor g = plain(grads[0].to(torch::kComplexFloat));
    c10::cuda::CUDAGuard guard(g.device());
    Tensor gx = torch::empty({h, w}, g.options());
    Tensor ws = torch::empty({int64_t(g_upsample_ws(int(h), int(w), int(s)))}, g.options().dtype(torch::kUInt8));
    check(g_upsample[1](fptr<const float>(g), int(h), int(w), int(s), fptr<float>(gx), ws.data_ptr(), size_t(ws.numel()),
                        current_stream(g)),
          "ptycho_fourier_upsample_adjoint");
    return {gx, Tensor(), Tensor()};
  }
};

// (y [h s, w s] complex64, library status); the caller has checked shape and scale
std::pair<Tensor, int> upsample(const Tensor& x, int64_t s) {
  TORCH_CHECK(g_upsample[0] && g_upsample_ws, "bind_inr() was not called");
  TORCH_CHECK_VALUE(x.is_cuda(), "x must be a CUDA tensor (there is no CPU path)");
  c10::cuda::CUDAGuard guard(x.device());
  int rc = 0;
  Tensor y = Upsample::apply(x, s, &rc);
  return {y, rc};
}

void bind_inr(const std::vector<int64_t>& a, int64_t packed_bytes, int64_t grad_floats) {
  TORCH_CHECK(a.size() == 9, "bind_inr: nine addresses");
  g_cmlp_pack = reinterpret_cast<cmlp_pack_fn>(a[0]);
  g_cmlp_fwd[0] = reinterpret_cast<cmlp_fwd_fn>(a[1]);
  g_cmlp_fwd[1] = reinterpret_cast<cmlp_fwd_fn>(a[2]);
  g_cmlp_bwd[0] = reinterpret_cast<cmlp_bwd_fn>(a[3]);
  g_cmlp_bwd[1] = reinterpret_cast<cmlp_bwd_fn>(a[4]);
  g_cmlp_bwd_ws = reinterpret_cast<size_t (*)(int)>(a[5]);
  g_upsample[0] = reinterpret_cast<upsample_fn>(a[6]);
  g_upsample[1] = reinterpret_cast<upsample_fn>(a[7]);
  g_upsample_ws = reinterpret_cast<size_t (*)(int, int, int)>(a[8]);
  g_cmlp_packed_bytes = packed_bytes;
  g_cmlp_grad_floats = grad_floats;
}

// the cached workspace of the current stream of `like`'s device, at least `bytes` long
Tensor workspace(const Tensor& like, int64_t bytes) {
  TORCH_CHECK_VALUE(like.is_cuda() && bytes >= 0, "workspace needs a CUDA tensor and a size");
  return workspace_on(like, current_stream(like), size_t(bytes));
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind", &bind, "bind(fwd_adj, scale_pair, workspace_size, status_string) function addresses");
  m.def("fused_loss", &fused_loss, "fused forward + loss + adjoint as one autograd node");
  m.def("workspace", &workspace, "the per-stream ptycho_fwd_adj workspace");
  m.def("bind_inr", &bind_inr, "addresses of the MLP and upsampling entry points");
  m.def("cmlp", &cmlp, "complex MLP as one autograd node: (y, status)");
  m.def("upsample", &upsample, "Fourier upsampling as one autograd node: (y, status)");
}
