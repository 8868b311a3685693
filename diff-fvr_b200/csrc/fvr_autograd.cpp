// Native autograd binding of the differentiable calls.
//
// A Python autograd node costs about 45 us of host time per call forward and
// needs the interpreter lock on the autograd engine's thread backward; the
// calls below are one library launch sequence per direction (kernels of 70 to
// 135 us at ordinary sizes), so the host was the bound: one pose of the
// pinhole renderer 155 us from the Python node, 97 from here; the explicit rays
// 201 and 130; the image step 190 and 112; the registration loss 181 and 149.
//
// Each node calls the C ABI through addresses the Python side hands over once
// (bind); this file holds no kernels.  What a model, lattice or engine keeps
// between calls travels as a plan: a reference-counted record of tensors and
// sizes, from which pointers are taken at each call.
//
// The spectral-NCC loss:
//
// The reference's loss (src/fvr/torch_engine.py:292-307, forward_spectral_ncc)
// is differentiated by PyTorch's autograd.  Here the forward pass already
// computes the pose gradient (the moments kernel and its dependent epilogue,
// fvr_tc_sncc_value_and_grad in libfvr_b200.so), so the autograd node only has
// to keep dL/dposes and scale it by the upstream gradient.  Written as a C++
// torch::autograd::Function, one forward call costs one pybind call, two
// allocations and the foreign launch, and the backward runs on the autograd
// engine's device thread without taking the Python interpreter lock.
//
// The launch itself is reached through the C ABI only: the Python side hands
// over the address of fvr_tc_sncc_value_and_grad and every argument that is
// fixed for a prepared call (stencil storage, shape, views, target spectra,
// high-pass table, launch variant, workspace); this file holds no kernels.
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <array>
#include <cstdint>
#include <map>
#include <string>
#include <vector>

#include "fvr_b200.h"

namespace {

// ---------------------------------------------------------------- C ABI

struct Api {
  decltype(&fvr_status_string) status = nullptr;
  decltype(&fvr_pou_pinhole_forward) pinhole_forward = nullptr;
  decltype(&fvr_pou_pinhole_backward_chunked) pinhole_backward = nullptr;
  decltype(&fvr_pou_pinhole_backward_chunked_workspace) pinhole_backward_workspace = nullptr;
  decltype(&fvr_pou_rays_forward) rays_forward = nullptr;
  decltype(&fvr_pou_rays_backward) rays_backward = nullptr;
  decltype(&fvr_pou_rays_backward_workspace) rays_backward_workspace = nullptr;
  decltype(&fvr_tc_image) image = nullptr;
  decltype(&fvr_tc_image_backward) image_backward = nullptr;
  decltype(&fvr_cncc_image) cncc_image = nullptr;
  decltype(&fvr_cncc_image_workspace) cncc_image_workspace = nullptr;
  decltype(&fvr_reg_loss_forward) reg_loss_forward = nullptr;
  decltype(&fvr_reg_loss_backward) reg_loss_backward = nullptr;
  decltype(&fvr_reg_loss_workspace) reg_loss_workspace = nullptr;
  int64_t geo_stride = 0, reg_stats = 0;
};
Api api;

// The package's FvrError, in a forward as in a backward (the autograd engine
// hands its Python type on).  Everything else, an allocation that fails among
// it, keeps the type it has in torch.
PyObject* error_type = nullptr;
struct LibraryError : torch::PyTorchError {
  using PyTorchError::PyTorchError;
  PyObject* python_type() override { return error_type ? error_type : PyExc_RuntimeError; }
};

void check(int rc, const char* name, const char* (*status)(int) = nullptr) {
  if (rc == 0) return;
  if (!status) status = api.status;
  throw LibraryError(std::string(name) + " failed with status " + std::to_string(rc) + ": " +
                     (status ? status(rc) : ""));
}

void* current_stream(c10::DeviceIndex device) { return c10::cuda::getCurrentCUDAStream(device).stream(); }

at::TensorOptions on(at::Device d, at::ScalarType t) { return at::TensorOptions().dtype(t).device(d); }

// A contiguous tensor of the given type on the device (the same one where it already is).
at::Tensor as(const at::Tensor& t, at::Device d, at::ScalarType type) {
  at::Tensor x = t.detach();
  if (x.device() != d || x.scalar_type() != type) x = x.to(d, type);
  return x.contiguous();
}

at::Tensor to_type(at::Tensor t, int64_t type) {
  const auto want = static_cast<at::ScalarType>(type);
  return t.scalar_type() == want ? t : t.to(want);
}

const float* fptr(const at::Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

template <typename T>
c10::IValue keep(const c10::intrusive_ptr<T>& p) {
  return c10::IValue::make_capsule(p);
}
template <typename T>
c10::intrusive_ptr<T> kept(const c10::IValue& v) {
  return c10::static_intrusive_pointer_cast<T>(v.toCapsule());
}

// ---------------------------------------------------------------- cone beam

// Block spectra and geometry constants of a PerspectiveSlabFVR.
struct PouModel : torch::CustomClassHolder {
  int dtype = 0;
  int64_t B = 0, P = 0;
  double ds = 0.0;
  at::Tensor stencil, scales, centers, freqs;
  at::Device device() const { return stencil.device(); }
  double vscale() const { return static_cast<double>(P) * ds; }
  double c() const { return static_cast<double>(P / 2); }
};

// Separable ray tables and detector basis of a pinhole lattice.
struct PouLattice : torch::CustomClassHolder {
  int64_t H = 0, W = 0;
  std::array<double, 12> base{};
  at::Tensor rxc, ryr, ic;
};

using ModelPtr = c10::intrusive_ptr<PouModel>;
using LatticePtr = c10::intrusive_ptr<PouLattice>;

class Pinhole : public torch::autograd::Function<Pinhole> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& mats, ModelPtr m, LatticePtr l,
                            int64_t chunk) {
    const at::Device d = m->device();
    c10::cuda::CUDAGuard guard(d);
    const at::Tensor x = as(mats, d, at::kFloat);
    TORCH_CHECK(x.dim() == 3 && x.size(1) == 4 && x.size(2) == 4, "pose matrices must have shape (N, 4, 4)");
    const int64_t N = x.size(0);
    at::Tensor geo = at::empty({N, api.geo_stride}, on(d, at::kDouble)), offs = at::empty({m->B, N, 3}, on(d, at::kDouble));
    at::Tensor imgs = at::empty({m->B, N, m->P, m->P}, on(d, at::kFloat));
    at::Tensor out = at::empty({N, 1, l->H, l->W}, on(d, at::kFloat));
    check(api.pinhole_forward(m->dtype, m->stencil.data_ptr(), fptr(m->scales), m->B, m->P, fptr(x), N,
                              l->base.data(), m->vscale(), fptr(m->centers), fptr(m->freqs), fptr(l->rxc),
                              fptr(l->ryr), fptr(l->ic), l->H, l->W, 1.0 / m->ds, m->c(), geo.data_ptr<double>(),
                              offs.data_ptr<double>(), imgs.data_ptr<float>(), out.data_ptr<float>(),
                              current_stream(d.index())),
          "fvr_pou_pinhole_forward");
    // the obliquity table may be the caller's own tensor: kept as one, so that a write to it before the backward is seen
    // (an inference tensor has no version and cannot be kept by a node)
    ctx->save_for_backward({geo, offs, imgs, l->ic.is_inference() ? at::Tensor() : l->ic});
    ctx->saved_data["model"] = keep(m);
    ctx->saved_data["lattice"] = keep(l);
    ctx->saved_data["chunk"] = chunk;  // poses whose image gradients are held at a time
    ctx->saved_data["type"] = static_cast<int64_t>(mats.scalar_type());
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list go) {
    if (!go[0].defined()) return {at::Tensor(), at::Tensor(), at::Tensor(), at::Tensor()};
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &geo = saved[0], &offs = saved[1], &imgs = saved[2];
    const ModelPtr m = kept<PouModel>(ctx->saved_data["model"]);
    const LatticePtr l = kept<PouLattice>(ctx->saved_data["lattice"]);
    const at::Tensor& ic = saved[3].defined() ? saved[3] : l->ic;
    const at::Device d = m->device();
    c10::cuda::CUDAGuard guard(d);
    const int64_t N = geo.size(0), chunk = std::min(N, ctx->saved_data["chunk"].toInt());
    const int64_t ws_bytes = api.pinhole_backward_workspace(m->B, N, l->H, l->W, chunk);
    const at::Tensor g = as(go[0], d, at::kFloat);
    at::Tensor ws = at::empty({ws_bytes}, on(d, at::kByte));
    at::Tensor gimgs = at::empty({m->B, chunk, m->P, m->P}, on(d, at::kFloat));
    at::Tensor grad = at::empty({N, 4, 4}, on(d, at::kFloat));
    check(api.pinhole_backward(m->dtype, m->stencil.data_ptr(), fptr(m->scales), m->B, m->P, geo.data_ptr<double>(),
                               offs.data_ptr<double>(), N, l->base.data(), m->vscale(), fptr(m->centers),
                               fptr(m->freqs), fptr(imgs), fptr(l->rxc), fptr(l->ryr), fptr(ic), l->H, l->W,
                               1.0 / m->ds, m->c(), fptr(g), chunk, gimgs.data_ptr<float>(), ws.data_ptr(), ws_bytes,
                               grad.data_ptr<float>(), current_stream(d.index())),
          "fvr_pou_pinhole_backward_chunked");
    return {to_type(grad, ctx->saved_data["type"].toInt()), at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

class LatticeRays : public torch::autograd::Function<LatticeRays> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& srcs, const at::Tensor& trg,
                            ModelPtr m) {
    const at::Device d = m->device();
    c10::cuda::CUDAGuard guard(d);
    const at::Tensor s = as(srcs, d, at::kFloat), t = as(trg, d, at::kFloat);
    TORCH_CHECK(t.dim() == 4 && t.size(3) == 3 && s.dim() == 2 && s.size(0) == t.size(0) && s.size(1) == 3,
                "expected sources (N, 3) and detector points (N, H, W, 3)");
    const int64_t N = t.size(0), H = t.size(1), W = t.size(2);
    at::Tensor geo = at::empty({N, api.geo_stride}, on(d, at::kDouble)), offs = at::empty({m->B, N, 3}, on(d, at::kDouble));
    at::Tensor rays = at::empty({3, N, H * W}, on(d, at::kFloat));
    at::Tensor imgs = at::empty({m->B, N, m->P, m->P}, on(d, at::kFloat));
    at::Tensor out = at::empty({N, H, W}, on(d, at::kFloat));
    check(api.rays_forward(m->dtype, m->stencil.data_ptr(), fptr(m->scales), m->B, m->P, fptr(s), fptr(t), N, H, W,
                           m->vscale(), fptr(m->centers), fptr(m->freqs), 1.0 / m->ds, m->c(), geo.data_ptr<double>(),
                           offs.data_ptr<double>(), rays.data_ptr<float>(), imgs.data_ptr<float>(),
                           out.data_ptr<float>(), current_stream(d.index())),
          "fvr_pou_rays_forward");
    ctx->save_for_backward({t, geo, offs, rays, imgs});
    ctx->saved_data["model"] = keep(m);
    ctx->saved_data["stype"] = static_cast<int64_t>(srcs.scalar_type());
    ctx->saved_data["ttype"] = static_cast<int64_t>(trg.scalar_type());
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list go) {
    if (!go[0].defined()) return {at::Tensor(), at::Tensor(), at::Tensor()};
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &t = saved[0], &geo = saved[1], &offs = saved[2], &rays = saved[3], &imgs = saved[4];
    const ModelPtr m = kept<PouModel>(ctx->saved_data["model"]);
    const at::Device d = m->device();
    c10::cuda::CUDAGuard guard(d);
    const int64_t N = t.size(0), H = t.size(1), W = t.size(2);
    const int64_t ws_bytes = api.rays_backward_workspace(m->B, N, H, W);
    const at::Tensor g = as(go[0], d, at::kFloat);
    at::Tensor ws = at::empty({ws_bytes}, on(d, at::kByte)), gimgs = at::empty_like(imgs);
    at::Tensor gs = at::empty({N, 3}, on(d, at::kFloat)), gt = at::empty_like(t);
    check(api.rays_backward(m->dtype, m->stencil.data_ptr(), fptr(m->scales), m->B, m->P, fptr(t), N, H, W,
                            m->vscale(), fptr(m->centers), fptr(m->freqs), 1.0 / m->ds, m->c(),
                            geo.data_ptr<double>(), offs.data_ptr<double>(), fptr(rays), fptr(imgs), fptr(g),
                            gimgs.data_ptr<float>(), ws.data_ptr(), ws_bytes, gs.data_ptr<float>(),
                            gt.data_ptr<float>(), current_stream(d.index())),
          "fvr_pou_rays_backward");
    return {to_type(gs, ctx->saved_data["stype"].toInt()), to_type(gt, ctx->saved_data["ttype"].toInt()),
            at::Tensor()};
  }
};

// ---------------------------------------------------------------- parallel beam images

// Spectrum storage of an engine with the tables of one output size.
struct ImagePlan : torch::CustomClassHolder {
  int dtype = 0;
  int64_t D = 0, H = 0, W = 0, R = 0;
  double kappa = 0.0;
  at::Tensor stencil, scales, lin, tw;
};
using ImagePtr = c10::intrusive_ptr<ImagePlan>;

class Image : public torch::autograd::Function<Image> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& poses, ImagePtr k, int64_t view) {
    const at::Device d = k->stencil.device();
    c10::cuda::CUDAGuard guard(d);
    const at::Tensor p = as(poses, d, at::kFloat);
    const int64_t C = p.size(0);
    at::Tensor img = at::empty({C, 1, k->R, k->R}, on(d, at::kFloat));
    check(api.image(k->dtype, k->stencil.data_ptr(), fptr(k->scales), k->D, k->H, k->W, fptr(p), C,
                    static_cast<int>(view), fptr(k->lin), k->R, k->kappa, k->tw.data_ptr(), img.data_ptr<float>(),
                    current_stream(d.index())),
          "fvr_tc_image");
    ctx->save_for_backward({p, img});
    ctx->saved_data["plan"] = keep(k);
    ctx->saved_data["view"] = view;
    ctx->saved_data["type"] = static_cast<int64_t>(poses.scalar_type());
    return img;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list go) {
    if (!go[0].defined()) return {at::Tensor(), at::Tensor(), at::Tensor()};
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &p = saved[0], &img = saved[1];
    const ImagePtr k = kept<ImagePlan>(ctx->saved_data["plan"]);
    const at::Device d = p.device();
    c10::cuda::CUDAGuard guard(d);
    const at::Tensor g = as(go[0], d, at::kFloat);
    at::Tensor grad = at::empty({p.size(0), 6}, on(d, at::kFloat));
    check(api.image_backward(k->dtype, k->stencil.data_ptr(), fptr(k->scales), k->D, k->H, k->W, fptr(p), p.size(0),
                             static_cast<int>(ctx->saved_data["view"].toInt()), fptr(k->lin), k->R, k->kappa,
                             k->tw.data_ptr(), fptr(img), fptr(g), grad.data_ptr<float>(), current_stream(d.index())),
          "fvr_tc_image_backward");
    return {to_type(grad, ctx->saved_data["type"].toInt()), at::Tensor(), at::Tensor()};
  }
};

// Image spectral NCC: the forward keeps dloss/dpred, the backward scales it.
// That gradient's own dependence on pred is not recorded, so neither is its
// product with the upstream gradient: a second derivative is refused instead of
// losing that term.
class ImageNcc : public torch::autograd::Function<ImageNcc> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& pred, const at::Tensor& target,
                            const c10::optional<at::Tensor>& hp, const at::Tensor& tw0, const at::Tensor& tw1,
                            bool need) {
    const at::Device d = pred.device();
    c10::cuda::CUDAGuard guard(d);
    const at::Tensor x = as(pred, d, at::kFloat), t = as(target, d, at::kFloat);
    const int64_t H = pred.size(-2), W = pred.size(-1), n = H * W;
    const int64_t B = x.numel() / n, Bt = t.numel() / n, ws_bytes = api.cncc_image_workspace(B);
    at::Tensor loss = at::empty({}, on(d, at::kFloat)), ws = at::empty({std::max<int64_t>(ws_bytes, 8)}, on(d, at::kByte));
    at::Tensor grad;
    if (need) grad = at::empty(pred.sizes(), on(d, at::kFloat));
    check(api.cncc_image(fptr(x), fptr(t), B, Bt, H, W, hp ? fptr(*hp) : nullptr, tw0.data_ptr(), tw1.data_ptr(), ws.data_ptr(),
                         ws_bytes, loss.data_ptr<float>(), need ? grad.data_ptr<float>() : nullptr,
                         current_stream(d.index())),
          "fvr_cncc_image");
    if (need) ctx->save_for_backward({grad});
    ctx->saved_data["type"] = static_cast<int64_t>(pred.scalar_type());
    return loss;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list go) {
    torch::autograd::variable_list out(6);
    if (!go[0].defined()) return out;
    const at::Tensor grad = ctx->get_saved_variables()[0];
    out[0] = to_type(grad * go[0].detach().to(grad.device(), grad.scalar_type()), ctx->saved_data["type"].toInt());
    return out;
  }
};

// ---------------------------------------------------------------- registration loss

class RegLoss : public torch::autograd::Function<RegLoss> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& a, const at::Tensor& b,
                            const at::Tensor& ra, const at::Tensor& rb, int64_t crop, double ms_weight,
                            double edge_weight) {
    const at::Device d = a.device();
    c10::cuda::CUDAGuard guard(d);
    const std::array<at::Tensor, 4> t{as(a, d, at::kFloat), as(b, d, at::kFloat), as(ra, d, at::kFloat),
                                      as(rb, d, at::kFloat)};
    const int64_t B = a.size(0), H = a.size(2), W = a.size(3), ws_bytes = api.reg_loss_workspace(2, B, H, W);
    at::Tensor ws = at::empty({ws_bytes}, on(d, at::kByte)), stats = at::empty({2 * B, api.reg_stats}, on(d, at::kDouble));
    at::Tensor out = at::empty({B}, on(d, at::kFloat));
    const float* imgs[2] = {fptr(t[0]), fptr(t[1])};
    const float* refs[2] = {fptr(t[2]), fptr(t[3])};
    const int64_t rbatch[2] = {ra.size(0), rb.size(0)};
    check(api.reg_loss_forward(imgs, refs, rbatch, 2, B, H, W, crop, static_cast<float>(ms_weight),
                               static_cast<float>(edge_weight), ws.data_ptr(), ws_bytes, stats.data_ptr<double>(),
                               out.data_ptr<float>(), current_stream(d.index())),
          "fvr_reg_loss_forward");
    ctx->save_for_backward({t[0], t[1], t[2], t[3], stats});
    ctx->saved_data["crop"] = crop;
    ctx->saved_data["ms"] = ms_weight;
    ctx->saved_data["edge"] = edge_weight;
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list go) {
    torch::autograd::variable_list out(7);
    if (!go[0].defined()) return out;
    const auto s = ctx->get_saved_variables();
    const at::Device d = s[0].device();
    c10::cuda::CUDAGuard guard(d);
    const at::Tensor g = as(go[0], d, at::kFloat);
    out[0] = at::empty_like(s[0]);
    out[1] = at::empty_like(s[1]);
    const float* imgs[2] = {fptr(s[0]), fptr(s[1])};
    const float* refs[2] = {fptr(s[2]), fptr(s[3])};
    const int64_t rbatch[2] = {s[2].size(0), s[3].size(0)};
    float* grads[2] = {out[0].data_ptr<float>(), out[1].data_ptr<float>()};
    check(api.reg_loss_backward(imgs, refs, rbatch, 2, s[0].size(0), s[0].size(2), s[0].size(3),
                                ctx->saved_data["crop"].toInt(), static_cast<float>(ctx->saved_data["ms"].toDouble()),
                                static_cast<float>(ctx->saved_data["edge"].toDouble()), s[4].data_ptr<double>(),
                                fptr(g), 1, grads, current_stream(d.index())),
          "fvr_reg_loss_backward");
    return out;
  }
};

// ---------------------------------------------------------------- spectral NCC

using SnccValueAndGrad = int (*)(int, const void*, const float*, int64_t, int64_t, int64_t, const float*, int64_t,
                                 int, const int*, const void* const*, const float*, const float*, int64_t, double,
                                 int, const float*, int64_t, void*, int64_t, float*, float*, float*, int, void*);
using StatusString = const char* (*)(int);

// One prepared launch: the arguments of fvr_tc_sncc_value_and_grad that do
// not change between calls, and the tensors that own the memory they name.
struct SnccCall {
  SnccValueAndGrad fn = nullptr;
  StatusString status = nullptr;
  int dtype = 0;
  const void* stencil = nullptr;
  const float* scales = nullptr;
  int64_t D = 0, H = 0, W = 0, C = 0, R = 0;
  std::vector<int> views;
  std::vector<const void*> ftargs;
  const float* hp = nullptr;
  const float* lin = nullptr;
  double kappa = 0.0;
  int variant = 0;
  void* ws = nullptr;
  int64_t ws_bytes = 0;
  int device = 0;
  std::vector<at::Tensor> keep;
};

template <typename T>
T as_ptr(int64_t v) {
  return reinterpret_cast<T>(static_cast<intptr_t>(v));
}

// dL/dposes as the forward kept it, tied to the poses it was formed at: its own
// derivative is not computed, so asking for it is an error (the derivative by
// the upstream gradient, which only scales it, is there).
class FirstOrder : public torch::autograd::Function<FirstOrder> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext*, const at::Tensor& grad, const at::Tensor&) {
    return grad.view(grad.sizes());
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext*, torch::autograd::variable_list) {
    TORCH_CHECK(false, "the spectral NCC loss has no second derivative in the poses");
  }
};

class SnccLoss : public torch::autograd::Function<SnccLoss> {
 public:
  // Returns sum_v loss_v as a 0-dim tensor; keeps dL/dposes for backward.
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& poses, int64_t handle) {
    const SnccCall& k = *as_ptr<const SnccCall*>(handle);
    at::Tensor p = poses.detach();
    if (!p.is_cuda() || p.get_device() != k.device || p.scalar_type() != at::kFloat)
      p = p.to(at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(k.device)), at::kFloat);
    p = p.contiguous();
    if (p.dim() != 2 || p.size(0) != k.C || p.size(1) != 6)
      throw LibraryError("poses must have shape (" + std::to_string(k.C) + ", 6)");
    const auto opts = at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, k.device);
    const int nv = static_cast<int>(k.views.size());
    at::Tensor grad = at::empty({k.C, 6}, opts);
    at::Tensor loss = at::empty({nv + 1}, opts);
    cudaStream_t s = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(k.device)).stream();
    check(k.fn(k.dtype, k.stencil, k.scales, k.D, k.H, k.W, p.data_ptr<float>(), k.C, nv, k.views.data(),
               k.ftargs.data(), k.hp, k.lin, k.R, k.kappa, k.variant, nullptr, 0, k.ws, k.ws_bytes,
               loss.data_ptr<float>(), nullptr, grad.data_ptr<float>(), 0, s),
          "fvr_tc_sncc_value_and_grad", k.status);
    ctx->save_for_backward({grad});
    ctx->saved_data["poses"] = poses;  // for the graph only: later writes to them are no matter
    ctx->saved_data["pdt"] = static_cast<int64_t>(poses.scalar_type());
    return loss.select(0, nv);
  }

  // dL/dposes scaled by the upstream gradient of the (scalar) loss.
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list go) {
    at::Tensor grad = ctx->get_saved_variables()[0];
    if (at::GradMode::is_enabled()) grad = FirstOrder::apply(grad, ctx->saved_data["poses"].toTensor());
    at::Tensor r = go[0].defined() ? grad * go[0].to(grad.scalar_type()) : at::zeros_like(grad);
    const auto pdt = static_cast<at::ScalarType>(ctx->saved_data["pdt"].toInt());
    if (r.scalar_type() != pdt) r = r.to(pdt);
    return {r, at::Tensor()};
  }
};

at::Tensor sncc_loss(const at::Tensor& poses, const SnccCall& call) {
  return SnccLoss::apply(poses, reinterpret_cast<int64_t>(&call));
}

}  // namespace

// What tells tensors apart that a preparation may be kept for: addresses, shapes,
// strides and types; and their versions, which a write in place advances
// (inference tensors have none).
std::pair<pybind11::bytes, pybind11::bytes> tensor_keys(const std::vector<at::Tensor>& tensors) {
  std::vector<int64_t> key, versions;
  key.reserve(8 * tensors.size());
  versions.reserve(tensors.size());
  for (const at::Tensor& t : tensors) {
    key.push_back(reinterpret_cast<intptr_t>(t.const_data_ptr()));
    key.push_back(static_cast<int64_t>(t.scalar_type()));
    key.push_back(t.dim());
    for (int64_t n : t.sizes()) key.push_back(n);
    for (int64_t n : t.strides()) key.push_back(n);
    versions.push_back(t.is_inference() ? 0 : static_cast<int64_t>(t._version()));
  }
  auto bytes = [](const std::vector<int64_t>& v) {
    return pybind11::bytes(reinterpret_cast<const char*>(v.data()), v.size() * sizeof(int64_t));
  };
  return {bytes(key), bytes(versions)};
}

void bind(const std::map<std::string, int64_t>& a, int64_t geo_stride, int64_t reg_stats) {
  auto set = [&](auto& f, const char* name) {
    const auto it = a.find(name);
    TORCH_CHECK(it != a.end() && it->second != 0, "no address for ", name);
    f = as_ptr<std::decay_t<decltype(f)>>(it->second);
  };
  set(api.status, "fvr_status_string");
  set(api.pinhole_forward, "fvr_pou_pinhole_forward");
  set(api.pinhole_backward, "fvr_pou_pinhole_backward_chunked");
  set(api.pinhole_backward_workspace, "fvr_pou_pinhole_backward_chunked_workspace");
  set(api.rays_forward, "fvr_pou_rays_forward");
  set(api.rays_backward, "fvr_pou_rays_backward");
  set(api.rays_backward_workspace, "fvr_pou_rays_backward_workspace");
  set(api.image, "fvr_tc_image");
  set(api.image_backward, "fvr_tc_image_backward");
  set(api.cncc_image, "fvr_cncc_image");
  set(api.cncc_image_workspace, "fvr_cncc_image_workspace");
  set(api.reg_loss_forward, "fvr_reg_loss_forward");
  set(api.reg_loss_backward, "fvr_reg_loss_backward");
  set(api.reg_loss_workspace, "fvr_reg_loss_workspace");
  api.geo_stride = geo_stride;
  api.reg_stats = reg_stats;
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  m.doc() = "Native autograd binding of libfvr_b200.so";
  m.def("bind", &bind, "addresses of the C entry points and two record sizes", py::arg("addresses"),
        py::arg("geo_stride"), py::arg("reg_stats"));
  py::class_<PouModel, ModelPtr>(m, "PouModel")
      .def(py::init([](int dtype, at::Tensor stencil, c10::optional<at::Tensor> scales, int64_t B, int64_t P, double ds,
                       at::Tensor centers, at::Tensor freqs) {
        auto k = c10::make_intrusive<PouModel>();
        k->dtype = dtype;
        k->stencil = std::move(stencil);
        if (scales) k->scales = *scales;
        k->B = B;
        k->P = P;
        k->ds = ds;
        k->centers = std::move(centers);
        k->freqs = std::move(freqs);
        return k;
      }));
  py::class_<PouLattice, LatticePtr>(m, "PouLattice")
      .def(py::init([](const std::vector<double>& base, at::Tensor rxc, at::Tensor ryr, at::Tensor ic) {
        TORCH_CHECK(base.size() == 12 && ic.dim() == 2, "a detector basis of 12 numbers and a 2-d obliquity table");
        auto k = c10::make_intrusive<PouLattice>();
        std::copy(base.begin(), base.end(), k->base.begin());
        k->H = ic.size(0);
        k->W = ic.size(1);
        k->rxc = std::move(rxc);
        k->ryr = std::move(ryr);
        k->ic = std::move(ic);
        return k;
      }));
  py::class_<ImagePlan, ImagePtr>(m, "ImagePlan")
      .def(py::init([](int dtype, at::Tensor stencil, c10::optional<at::Tensor> scales, int64_t D, int64_t H, int64_t W,
                       int64_t R, double kappa, at::Tensor lin, at::Tensor tw) {
        auto k = c10::make_intrusive<ImagePlan>();
        k->dtype = dtype;
        k->stencil = std::move(stencil);
        if (scales) k->scales = *scales;
        k->D = D;
        k->H = H;
        k->W = W;
        k->R = R;
        k->kappa = kappa;
        k->lin = std::move(lin);
        k->tw = std::move(tw);
        return k;
      }));
  m.def("tensor_keys", torch::wrap_pybind_function(tensor_keys), "(identity, versions) of the tensors, as bytes");
  m.def("set_error_type", [](py::object type) { error_type = type.release().ptr(); },
        "the exception raised for a library status");
  // wrapped: torch's own exceptions (out of memory among them) and ours arrive as their Python types
  m.def("pinhole", torch::wrap_pybind_function([](const at::Tensor& mats, ModelPtr k, LatticePtr l, int64_t chunk) {
          return Pinhole::apply(mats, k, l, chunk);
        }));
  m.def("lattice_rays", torch::wrap_pybind_function([](const at::Tensor& srcs, const at::Tensor& trg, ModelPtr k) {
          return LatticeRays::apply(srcs, trg, k);
        }));
  m.def("image", torch::wrap_pybind_function([](const at::Tensor& poses, ImagePtr k, int64_t view) {
          return Image::apply(poses, k, view);
        }));
  m.def("image_ncc",
        torch::wrap_pybind_function([](const at::Tensor& pred, const at::Tensor& target, c10::optional<at::Tensor> hp,
                                       const at::Tensor& tw0, const at::Tensor& tw1) {
          const bool need = at::GradMode::is_enabled() && pred.requires_grad();
          return ImageNcc::apply(pred, target.detach(), hp, tw0, tw1, need);
        }));
  m.def("reg_loss",
        torch::wrap_pybind_function([](const at::Tensor& a, const at::Tensor& b, const at::Tensor& ra,
                                       const at::Tensor& rb, int64_t crop, double ms, double edge) {
          return RegLoss::apply(a, b, ra.detach(), rb.detach(), crop, ms, edge);
        }));
  pybind11::class_<SnccCall>(m, "SnccCall")
      .def(pybind11::init([](int64_t fn, int64_t status, int dtype, int64_t stencil, int64_t scales, int64_t D,
                             int64_t H, int64_t W, int64_t C, std::vector<int> views, std::vector<int64_t> ftargs,
                             int64_t hp, int64_t lin, int64_t R, double kappa, int variant, int64_t ws,
                             int64_t ws_bytes, int device, std::vector<at::Tensor> keep) {
             TORCH_CHECK(fn != 0 && stencil != 0 && lin != 0 && ws != 0, "null pointer in a prepared launch");
             TORCH_CHECK(!views.empty() && views.size() == ftargs.size(), "one target spectrum per view");
             auto* k = new SnccCall();
             k->fn = as_ptr<SnccValueAndGrad>(fn);
             k->status = as_ptr<StatusString>(status);
             k->dtype = dtype;
             k->stencil = as_ptr<const void*>(stencil);
             k->scales = as_ptr<const float*>(scales);
             k->D = D;
             k->H = H;
             k->W = W;
             k->C = C;
             k->R = R;
             k->views = std::move(views);
             for (int64_t f : ftargs) k->ftargs.push_back(as_ptr<const void*>(f));
             k->hp = as_ptr<const float*>(hp);
             k->lin = as_ptr<const float*>(lin);
             k->kappa = kappa;
             k->variant = variant;
             k->ws = as_ptr<void*>(ws);
             k->ws_bytes = ws_bytes;
             k->device = device;
             k->keep = std::move(keep);
             return k;
           }),
           pybind11::arg("fn"), pybind11::arg("status"), pybind11::arg("dtype"), pybind11::arg("stencil"),
           pybind11::arg("scales"), pybind11::arg("D"), pybind11::arg("H"), pybind11::arg("W"), pybind11::arg("C"),
           pybind11::arg("views"), pybind11::arg("ftargs"), pybind11::arg("hp"), pybind11::arg("lin"),
           pybind11::arg("R"), pybind11::arg("kappa"), pybind11::arg("variant"), pybind11::arg("ws"),
           pybind11::arg("ws_bytes"), pybind11::arg("device"), pybind11::arg("keep"));
  m.def("sncc_loss", torch::wrap_pybind_function(sncc_loss), "sum_v spectral-NCC loss of the prepared call; differentiable in poses",
        pybind11::arg("poses"), pybind11::arg("call"));
}
