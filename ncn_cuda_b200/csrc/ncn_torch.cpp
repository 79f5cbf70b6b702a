// PyTorch autograd nodes of the NCN operators (extension module _ncn_torch).
//
// What the reference does in Python -- one autograd.Function per stage and a loop over the stages
// (ncn_cuda/ncn_pytorch_wrapper_v2.py:9-50, 107-144) -- is one C++ node per call here: a fused net
// (or a stack of residual ones) or a chain of stages, with the C ABI of include/ncn_b200.h below it.
//
// Why native: at small batches the host is the bound.  A training step of a 1024 x 1024 net runs 59 us
// of kernels; through Python autograd functions, ctypes and torch.stack / unbind it took 294 us.
// A chain of stages keeps its inner activations in one node, so that the engine hands over once per
// direction instead of once per stage, the weights of a fused net are gathered by its own kernel
// and their gradients returned as views of one buffer (as torch.stack and its backward would).
//
// Saved tensors go through SavedVariable, so in-place changes, saved-tensor hooks and a second backward
// without retain_graph behave as for any autograd operator.  Without gradients no state is stored.
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/engine.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/ncn_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::edge_list;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// A non-zero status as the NCNError of _lib.py; also from the engine's threads, which do not hold the GIL.
void check_status(const char* fn, int status) {
  if (status == NCN_OK) return;
  py::gil_scoped_acquire gil;
  try {
    py::module_::import("ncn_cuda_b200._lib").attr("check")(fn, status);
  } catch (py::error_already_set& e) {
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}

void check_activations(const Tensor& x, const Tensor& xa) {
  if (!x.is_cuda()) throw std::runtime_error("NCN kernels run on CUDA tensors only; there is no CPU path in this package");
  if (x.dim() != 3) throw py::value_error("expected [B, N, E] tensors");
  if (xa.sizes() != x.sizes() || xa.scalar_type() != x.scalar_type() || xa.device() != x.device())
    throw py::value_error("x, xa (and the cotangents) must agree in shape, dtype and device");
  if (x.scalar_type() != at::kFloat && x.scalar_type() != at::kBFloat16)
    throw py::type_error(std::string("NCN kernels take float32 or bfloat16 tensors, got ") + c10::toString(x.scalar_type()));
}

int dtype_code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? NCN_BF16 : NCN_F32; }

// The weights as the kernels take them: fp32, contiguous, on the activations' device.
Tensor plain_weights(const Tensor& W, int64_t numel, const at::Device& dev) {
  if (W.numel() != numel)
    throw py::value_error("weight has " + std::to_string(W.numel()) + " elements, expected " + std::to_string(numel));
  if (W.scalar_type() == at::kFloat && W.is_contiguous() && W.device() == dev) return W;
  return W.detach().to(dev, at::kFloat).contiguous();
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

Tensor cotangent(const Tensor& g, const Tensor& like) {
  return g.defined() ? g.contiguous() : at::zeros_like(like, at::MemoryFormat::Contiguous);
}

bool wants_grad(const Tensor& x, const Tensor& xa, const variable_list& ws) {
  if (!at::GradMode::is_enabled()) return false;
  if (x.requires_grad() || xa.requires_grad()) return true;
  for (const Tensor& w : ws)
    if (w.requires_grad()) return true;
  return false;
}

struct NcnNode : public Node {
  at::IntArrayRef shape() const { return shape_; }
  std::vector<int64_t> shape_;          // [B, N, E]
  at::TensorOptions options_;           // of the activations
  std::vector<std::vector<int64_t>> wshape_;
  std::vector<at::TensorOptions> wopt_;  // of the weights as the caller holds them

  void attach(const Tensor& x, const Tensor& xa, const variable_list& ws) {
    edge_list e;
    e.reserve(2 + ws.size());
    e.push_back(torch::autograd::impl::gradient_edge(x));
    e.push_back(torch::autograd::impl::gradient_edge(xa));
    for (const Tensor& w : ws) {
      e.push_back(torch::autograd::impl::gradient_edge(w));
      wshape_.push_back(w.sizes().vec());
      wopt_.push_back(w.options());
    }
    set_next_edges(std::move(e));
    shape_ = x.sizes().vec();
    options_ = x.options();
  }
  // the caller's cotangents, zeros where none arrived
  void incoming(const variable_list& g, Tensor& dy, Tensor& dya) const {
    const Tensor& any = g[0].defined() ? g[0] : g[1];
    if (any.defined()) {
      dy = cotangent(g[0], any);
      dya = cotangent(g[1], any);
    } else {
      dy = at::zeros(shape_, options_);
      dya = at::zeros(shape_, options_);
    }
  }
  // The gradient of weight k, `offset` floats into the buffer of all of them.  A tensor over the same storage, put
  // together by hand: narrow + view cost 4 us for each weight in the engine's thread.
  Tensor weight_grad(const Tensor& all, int64_t offset, size_t k) const {
    Tensor g = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(all.storage()), all.key_set(), all.dtype());
    g.unsafeGetTensorImpl()->set_storage_offset(offset);
    g.unsafeGetTensorImpl()->set_sizes_contiguous(wshape_[k]);
    return as_weight(std::move(g), k);
  }
  // an fp32 gradient in the type and on the device of weight k
  Tensor as_weight(Tensor g, size_t k) const {
    if (wopt_[k].dtype() == at::kFloat && wopt_[k].device() == g.device()) return g;
    return g.to(wopt_[k].device(), c10::typeMetaToScalarType(wopt_[k].dtype()));
  }
};


// ---------------------------------------------------------------- fused nets
// `layers` nets of L stages each (more than one only as residual layers), every net one kernel per direction.
struct FusedCfg {
  double alpha;
  int act, n, C, first, L, layers, every, dt;
  bool recompute, residual, tape;
  int flags() const { return (residual ? NCN_RESIDUAL : 0) | (recompute ? NCN_RECOMPUTE : 0) | (tape ? NCN_TAPE : 0); }
};

struct FusedNode : public NcnNode {
  FusedCfg c{};
  bool gathered = false;                       // W was put together from one tensor per stage
  SavedVariable W;                             // [layers, L, 2E]
  std::vector<SavedVariable> s0, s1, ckpt;     // per layer: what the backward starts from, stored states

  std::string name() const override { return "NCNNetBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    W.reset_data();
    for (auto* v : {&s0, &s1, &ckpt})
      for (SavedVariable& t : *v) t.reset_data();
  }
  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    at::NoGradGuard no_grad;
    Tensor dy, dya;
    incoming(g, dy, dya);
    const c10::cuda::OptionalCUDAGuard guard(dy.device());
    const int64_t B = shape_[0], N = shape_[1], E = shape_[2];
    const Tensor w = plain_weights(W.unpack(), (int64_t)c.layers * c.L * 2 * E, dy.device());
    const Tensor dW = at::empty({(int64_t)c.layers * c.L * 2 * E}, dy.options().dtype(at::kFloat));
    const size_t ws_bytes = ncn_bwd_workspace_bytes(B, N, E, c.n, c.C, c.L, c.dt);
    const Tensor ws = at::empty({(int64_t)ws_bytes}, dy.options().dtype(at::kByte));
    void* const st = stream_of(dy);
    const bool release = !torch::autograd::get_current_graph_task_keep_graph();  // (as ChainNode)
    for (int k = c.layers - 1; k >= 0; --k) {
      Tensor a, b, ck;
      if (!c.tape) {
        // the only layer whose saved tensors can be the node's own outputs is the last one
        const bool own = !c.recompute && k == c.layers - 1;
        a = own ? s0[k].unpack(shared_from_this()) : s0[k].unpack();
        b = own ? s1[k].unpack(shared_from_this()) : s1[k].unpack();
      }
      if (!ckpt.empty()) ck = ckpt[k].unpack();
      Tensor dx = at::empty(shape_, options_), dxa = at::empty(shape_, options_);
      check_status("ncn_net_bwd",
                   ncn_net_bwd(a.defined() ? a.data_ptr() : nullptr, b.defined() ? b.data_ptr() : nullptr, dy.data_ptr(),
                               dya.data_ptr(), w.const_data_ptr<float>() + (int64_t)k * c.L * 2 * E, dx.data_ptr(),
                               dxa.data_ptr(), nullptr, nullptr, dW.mutable_data_ptr<float>() + (int64_t)k * c.L * 2 * E,
                               ck.defined() ? ck.const_data_ptr<float>() : nullptr, c.every, ws.data_ptr(), ws_bytes, B, N, E,
                               c.n, c.C, c.first, c.L, c.alpha, c.act, c.dt, c.flags(), 0, st));
      dy = std::move(dx);
      dya = std::move(dxa);
      if (release) {
        for (auto* v : {&s0, &s1, &ckpt})
          if (!v->empty()) (*v)[k].reset_data();
      }
    }
    variable_list out;
    out.reserve(num_outputs());
    out.push_back(std::move(dy));
    out.push_back(std::move(dya));
    if (!gathered) {
      out.push_back(weight_grad(dW, 0, 0));
    } else {
      for (size_t l = 0; l < wshape_.size(); ++l) out.push_back(weight_grad(dW, (int64_t)l * 2 * E, l));
    }
    return out;
  }
};

std::tuple<Tensor, Tensor> fused_forward(const Tensor& x_in, const Tensor& xa_in, const variable_list& ws, bool gathered,
                                         FusedCfg c) {
  const bool grad = wants_grad(x_in, xa_in, ws);
  const c10::cuda::OptionalCUDAGuard guard(x_in.device());
  std::shared_ptr<FusedNode> node;
  if (grad) {
    node = std::shared_ptr<FusedNode>(new FusedNode(), torch::autograd::deleteNode);
    node->attach(x_in, xa_in, ws);
  }
  Tensor y, ya;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor x = x_in.contiguous(), xa = xa_in.contiguous();
    const int64_t B = x.size(0), N = x.size(1), E = x.size(2);
    c.dt = dtype_code(x);
    const Tensor W = gathered ? at::empty({(int64_t)ws.size() * 2 * E}, x.options().dtype(at::kFloat))
                              : plain_weights(ws[0], (int64_t)c.layers * c.L * 2 * E, x.device());
    std::vector<Tensor> each;  // gathered: the weights one by one, which the kernel gathers into W
    std::vector<const float*> list;
    if (gathered) {
      each.reserve(ws.size());
      list.reserve(ws.size());
      for (const Tensor& w : ws) {
        each.push_back(plain_weights(w, 2 * E, x.device()));
        list.push_back(each.back().const_data_ptr<float>());
      }
    }
    if (!grad) {  // nothing will be walked back: no states are stored
      c.every = 0;
      c.tape = c.recompute = false;
    }
    const int flags = (c.residual ? NCN_RESIDUAL : 0) | (c.tape ? NCN_TAPE : 0);
    const size_t ck_bytes = ncn_ckpt_bytes(B, N, E, c.L, c.every, flags);
    void* const st = stream_of(x);
    Tensor in = x, ina = xa;
    for (int k = 0; k < c.layers; ++k) {
      y = at::empty_like(x);
      ya = at::empty_like(xa);
      Tensor ck;
      if (ck_bytes) ck = at::empty({(int64_t)(ck_bytes / 4)}, x.options().dtype(at::kFloat));
      float* const ckp = ck.defined() ? ck.mutable_data_ptr<float>() : nullptr;
      if (gathered)
        check_status("ncn_net_fwd",
                     ncn_net_fwd_list(in.data_ptr(), ina.data_ptr(), list.data(), W.mutable_data_ptr<float>(), y.data_ptr(),
                                      ya.data_ptr(), ckp, c.every, B, N, E, c.n, c.C, c.first, c.L, c.alpha, c.act, c.dt, flags, st));
      else
        check_status("ncn_net_fwd",
                     ncn_net_fwd(in.data_ptr(), ina.data_ptr(), W.const_data_ptr<float>() + (int64_t)k * c.L * 2 * E, y.data_ptr(),
                                 ya.data_ptr(), ckp, c.every, B, N, E, c.n, c.C, c.first, c.L, c.alpha, c.act, c.dt, flags, st));
      if (grad) {
        if (c.recompute) {
          node->s0.emplace_back(k == 0 && x.is_same(x_in) ? x_in : in, false);
          node->s1.emplace_back(k == 0 && xa.is_same(xa_in) ? xa_in : ina, false);
        } else if (!c.tape && k + 1 < c.layers) {
          node->s0.emplace_back(y, false);
          node->s1.emplace_back(ya, false);
        }
        if (ck.defined()) node->ckpt.emplace_back(ck, false);
      }
      in = y;
      ina = ya;
    }
    if (grad) {
      node->c = c;
      node->gathered = gathered;
      node->W = SavedVariable(!gathered && W.is_same(ws[0]) ? ws[0] : W, false);
    }
  }
  if (grad) {
    torch::autograd::set_history(y, node);
    torch::autograd::set_history(ya, node);
    if (!c.tape && !c.recompute) {
      node->s0.emplace_back(y, true);
      node->s1.emplace_back(ya, true);
    }
  }
  return {y, ya};
}

// ---------------------------------------------------------------- chains of stages
enum Keep : int { KEEP_OUTPUT = 0, KEEP_INPUT = 1, KEEP_MID = 2 };  // set_stage_backward in ncn_pytorch_wrapper_v2.py

struct ChainCfg {
  double alpha;
  int act, n, C, first, L, keep, dt;
};

struct ChainNode : public NcnNode {
  ChainCfg c{};
  std::vector<SavedVariable> y, ya, mid, W;  // per stage
  SavedVariable x0, xa0, ctxlen;
  bool has_ctx = false;

  std::string name() const override { return has_ctx ? "NCNContextBackward" : "NCNStagesBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto* v : {&y, &ya, &mid, &W})
      for (SavedVariable& t : *v) t.reset_data();
    x0.reset_data();
    xa0.reset_data();
    ctxlen.reset_data();
  }
  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    at::NoGradGuard no_grad;
    Tensor dy, dya;
    incoming(g, dy, dya);
    const c10::cuda::OptionalCUDAGuard guard(dy.device());
    const int64_t B = shape_[0], N = shape_[1], E = shape_[2];
    // The stages leave their partial sums side by side in the workspace, and one launch adds up those of all (of as many as
    // fit: a stage uses a fraction of the ws_bytes that always suffice).
    const size_t ws_bytes = ncn_bwd_workspace_bytes(B, N, E, c.n, c.C, 1, c.dt);
    const Tensor ws = at::empty({(int64_t)ws_bytes}, dy.options().dtype(at::kByte));
    char* const ws_base = static_cast<char*>(ws.data_ptr());
    size_t used = 0;
    std::vector<const float*> partial;
    std::vector<int> partial_rows;
    std::vector<float*> partial_out;
    std::vector<Tensor> dW(c.L);  // a tensor of its own per stage: a weight's .grad holds no other's memory
    const size_t mid_bytes = c.keep == KEEP_MID ? ncn_stage_mid_bytes(B, N, E, c.n, c.dt) : 0;
    const Tensor cl = has_ctx ? ctxlen.unpack() : Tensor();
    void* const st = stream_of(dy);
    auto out_of = [&](std::vector<SavedVariable>& v, int l) {
      return l == c.L - 1 ? v[l].unpack(shared_from_this()) : v[l].unpack();
    };
    // What a stage kept is released behind it, unless the graph is kept: a node per stage would do the same.
    const bool release = !torch::autograd::get_current_graph_task_keep_graph();
    // The walk ends at the first stage whose gradient is asked for: at stage 0 where the input's is.
    const bool inputs = task_should_compute_output(0) || task_should_compute_output(1);
    int last = 0;
    if (!inputs)
      while (last < c.L - 1 && !task_should_compute_output(2 + last)) ++last;
    const bool several = last < c.L - 1;  // a single stage sums its own: no launch would be saved
    if (several) {
      partial.reserve(c.L - last);
      partial_rows.reserve(c.L - last);
      partial_out.reserve(c.L - last);
    }
    auto reduce = [&]() {
      if (partial.empty()) return;
      check_status("ncn_reduce_partials", ncn_reduce_partials(partial.data(), partial_rows.data(), partial_out.data(),
                                                              (int)partial.size(), 2 * E, st));
      partial.clear();
      partial_rows.clear();
      partial_out.clear();
      used = 0;
    };
    for (int l = c.L - 1; l >= last; --l) {
      const Tensor w = plain_weights(W[l].unpack(), 2 * E, dy.device());
      const Tensor yl = out_of(y, l), yal = out_of(ya, l);
      Tensor dx = at::empty(shape_, options_), dxa = at::empty(shape_, options_);
      dW[l] = at::empty(wshape_[l], dy.options().dtype(at::kFloat));
      Tensor xc, xac, m;
      int keep = NCN_KEEP_OUTPUT;
      const char* call = "ncn_stage_bwd";
      if (has_ctx) {
        keep = NCN_KEEP_CTX;
        call = "ncn_stage_bwd_ctx";
      } else if (c.keep == KEEP_INPUT) {
        keep = NCN_KEEP_INPUT;
        call = "ncn_stage_bwd_saved";
        xc = (l == 0 ? x0.unpack() : y[l - 1].unpack()).contiguous();
        xac = (l == 0 ? xa0.unpack() : ya[l - 1].unpack()).contiguous();
      } else if (mid_bytes) {
        keep = NCN_KEEP_MID;
        call = "ncn_stage_bwd_mid";
        m = mid[l].unpack();
      }
      auto ptr = [](const Tensor& t) -> const void* { return t.defined() ? t.const_data_ptr() : nullptr; };
      const void *yp = yl.const_data_ptr(), *yap = yal.const_data_ptr(), *dyp = dy.const_data_ptr(), *dyap = dya.const_data_ptr();
      const int* const clp = has_ctx ? cl.const_data_ptr<int>() : nullptr;
      const float* const wp = w.const_data_ptr<float>();
      float* const dwp = dW[l].mutable_data_ptr<float>();
      void *dxp = dx.data_ptr(), *dxap = dxa.data_ptr();
      const int module_l = c.first + l;
      int rc, rows = 0;
      if (!several) {
        switch (keep) {
          case NCN_KEEP_CTX:
            rc = ncn_stage_bwd_ctx(yp, yap, dyp, dyap, wp, clp, dxp, dxap, nullptr, nullptr, dwp, ws_base, ws_bytes, B, N, E, c.n, c.C,
                                   module_l, c.alpha, c.act, c.dt, st);
            break;
          case NCN_KEEP_INPUT:
            rc = ncn_stage_bwd_saved(ptr(xc), ptr(xac), yp, yap, dyp, dyap, wp, dxp, dxap, dwp, ws_base, ws_bytes, B, N, E, c.n, c.C,
                                     module_l, c.alpha, c.act, c.dt, st);
            break;
          case NCN_KEEP_MID:
            rc = ncn_stage_bwd_mid(yp, yap, ptr(m), mid_bytes, dyp, dyap, wp, dxp, dxap, dwp, ws_base, ws_bytes, B, N, E, c.n, c.C,
                                   module_l, c.alpha, c.act, c.dt, st);
            break;
          default:
            rc = ncn_stage_bwd(yp, yap, dyp, dyap, wp, dxp, dxap, nullptr, nullptr, dwp, ws_base, ws_bytes, B, N, E, c.n, c.C, module_l,
                               c.alpha, c.act, c.dt, st);
        }
      } else {
        auto walk = [&]() {
          return ncn_stage_bwd_partial(keep, ptr(xc), ptr(xac), yp, yap, ptr(m), mid_bytes, clp, dyp, dyap, wp, dxp, dxap, ws_base + used,
                                       ws_bytes - used, &rows, B, N, E, c.n, c.C, module_l, c.alpha, c.act, c.dt, st);
        };
        rc = used < ws_bytes ? walk() : NCN_ERR_WORKSPACE;
        if (rc == NCN_ERR_WORKSPACE && used > 0) {  // (nothing has been launched)
          reduce();
          rc = walk();
        }
      }
      check_status(call, rc);
      if (several) {
        partial.push_back(reinterpret_cast<const float*>(ws_base + used));
        partial_rows.push_back(rows);
        partial_out.push_back(dwp);
        used += ((size_t)rows * 2 * E * sizeof(float) + 255) / 256 * 256;
      }
      dy = std::move(dx);
      dya = std::move(dxa);
      if (release) {
        for (auto* v : {&y, &ya, &mid, &W})
          if (!v->empty()) (*v)[l].reset_data();
      }
    }
    reduce();
    variable_list out(2 + wshape_.size());
    if (inputs) {
      out[0] = std::move(dy);
      out[1] = std::move(dya);
    }
    for (int l = last; l < c.L; ++l) out[2 + l] = as_weight(std::move(dW[l]), l);
    return out;
  }
};

std::tuple<Tensor, Tensor> chain_forward(const Tensor& x_in, const Tensor& xa_in, const variable_list& ws, const Tensor& ctx_in,
                                         ChainCfg c) {
  const bool grad = wants_grad(x_in, xa_in, ws);
  if (grad && !x_in.requires_grad() && !xa_in.requires_grad() && !ws[0].requires_grad()) {
    // Stages that nothing is asked of come first: they run without a node, and store nothing.
    size_t first = 1;
    while (!ws[first].requires_grad()) ++first;
    ChainCfg frozen = c, rest = c;
    frozen.L = (int)first;
    rest.L = c.L - (int)first;
    rest.first = c.first + (int)first;
    const auto mid = chain_forward(x_in, xa_in, variable_list(ws.begin(), ws.begin() + first), ctx_in, frozen);
    return chain_forward(std::get<0>(mid), std::get<1>(mid), variable_list(ws.begin() + first, ws.end()), ctx_in, rest);
  }
  const c10::cuda::OptionalCUDAGuard guard(x_in.device());
  std::shared_ptr<ChainNode> node;
  if (grad) {
    node = std::shared_ptr<ChainNode>(new ChainNode(), torch::autograd::deleteNode);
    node->attach(x_in, xa_in, ws);
  }
  Tensor y, ya;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor x = x_in.contiguous(), xa = xa_in.contiguous();
    const int64_t B = x.size(0), N = x.size(1), E = x.size(2);
    c.dt = dtype_code(x);
    Tensor ctx;
    if (ctx_in.defined()) {
      if (ctx_in.numel() != B)
        throw py::value_error("ctxlen has " + std::to_string(ctx_in.numel()) + " entries for " + std::to_string(B) + " batch rows");
      ctx = ctx_in.to(x.device(), at::kInt).contiguous();
    }
    const size_t mid_bytes = grad && !ctx.defined() && c.keep == KEEP_MID ? ncn_stage_mid_bytes(B, N, E, c.n, c.dt) : 0;
    void* const st = stream_of(x);
    Tensor in = x, ina = xa;
    for (int l = 0; l < c.L; ++l) {
      const Tensor w = plain_weights(ws[l], 2 * E, x.device());
      const float* const wp = w.const_data_ptr<float>();
      const int module_l = c.first + l;
      y = at::empty_like(x);
      ya = at::empty_like(xa);
      if (ctx.defined()) {
        check_status("ncn_stage_fwd_ctx",
                     ncn_stage_fwd_ctx(in.data_ptr(), ina.data_ptr(), wp, ctx.const_data_ptr<int>(), y.data_ptr(), ya.data_ptr(), B,
                                       N, E, c.n, c.C, module_l, c.alpha, c.act, c.dt, st));
      } else if (mid_bytes) {
        Tensor m = at::empty({(int64_t)(mid_bytes / 4)}, x.options().dtype(at::kFloat));
        check_status("ncn_stage_fwd_mid",
                     ncn_stage_fwd_mid(in.data_ptr(), ina.data_ptr(), wp, y.data_ptr(), ya.data_ptr(), m.data_ptr(), mid_bytes, B, N,
                                       E, c.n, c.C, module_l, c.alpha, c.act, c.dt, st));
        node->mid.emplace_back(m, false);
      } else {
        check_status("ncn_stage_fwd", ncn_stage_fwd(in.data_ptr(), ina.data_ptr(), wp, y.data_ptr(), ya.data_ptr(), B, N, E, c.n,
                                                    c.C, module_l, c.alpha, c.act, c.dt, st));
      }
      if (grad) {
        node->W.emplace_back(w.is_same(ws[l]) ? ws[l] : w, false);
        if (l + 1 < c.L) {
          node->y.emplace_back(y, false);
          node->ya.emplace_back(ya, false);
        }
      }
      in = y;
      ina = ya;
    }
    if (grad) {
      node->c = c;
      if (c.keep == KEEP_INPUT) {
        node->x0 = SavedVariable(x_in, false);
        node->xa0 = SavedVariable(xa_in, false);
      }
      if (ctx.defined()) {
        node->ctxlen = SavedVariable(ctx, false);
        node->has_ctx = true;
      }
    }
  }
  if (grad) {
    torch::autograd::set_history(y, node);
    torch::autograd::set_history(ya, node);
    node->y.emplace_back(y, true);
    node->ya.emplace_back(ya, true);
  }
  return {y, ya};
}

// ---------------------------------------------------------------- Python entry points
// What an entry returns where the Python Function (ncn_pytorch_wrapper_v2.py) has to take the call: nothing.
using Result = std::optional<std::tuple<Tensor, Tensor>>;

// Tensors the nodes can take: the memory is the value.  Not those with a forward gradient (the nodes have no
// forward-mode rule and would drop it), nor wrappers of functorch or of Python subclasses with their own dispatch.
bool plain(const Tensor& t) {
  constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                         c10::DispatchKey::BatchedNestedTensor, c10::DispatchKey::Functionalize,
                                         c10::DispatchKey::Python});
  return !t.key_set().has_any(wrapped) && !t._fw_grad(/*level=*/0).defined();
}

// A call the native nodes must not answer: it goes through the Function, which records, transforms or refuses it as
// any custom Function is.  Under torch.jit.trace the kernels leave no trace of themselves, and the graph would hold
// the allocations of their results alone; with a functorch transform or a dispatch mode in effect the nodes would
// pass it by.
bool needs_function(const Tensor& x, const Tensor& xa, const variable_list& ws) {
  const c10::impl::LocalDispatchKeySet tls = c10::impl::tls_local_dispatch_key_set();
  constexpr c10::DispatchKeySet modes({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::Python});
  if (torch::jit::tracer::isTracing() || tls.included_.has_any(modes)) return true;
  if (!plain(x) || !plain(xa)) return true;
  for (const Tensor& w : ws)
    if (!plain(w)) return true;
  return false;
}

Result py_net(const Tensor& x, const Tensor& xa, const Tensor& W, double alpha, int act, int n, int C, int first,
                                  int L, int layers, bool recompute, int every, bool tape, bool residual) {
  if (needs_function(x, xa, {W})) return std::nullopt;
  check_activations(x, xa);
  py::gil_scoped_release nogil;
  return fused_forward(x, xa, {W}, false, FusedCfg{alpha, act, n, C, first, L, layers, every, 0, recompute, residual, tape});
}

Result py_stages(const Tensor& x, const Tensor& xa, const variable_list& ws, double alpha, int act, int n, int C,
                                     int first, int keep) {
  if (needs_function(x, xa, ws)) return std::nullopt;
  check_activations(x, xa);
  py::gil_scoped_release nogil;
  return chain_forward(x, xa, ws, Tensor(), ChainCfg{alpha, act, n, C, first, (int)ws.size(), keep, 0});
}

Result py_stage_ctx(const Tensor& x, const Tensor& xa, const Tensor& W, const Tensor& ctxlen, double alpha, int act,
                                        int n, int C, int module_l) {
  if (needs_function(x, xa, {W})) return std::nullopt;
  check_activations(x, xa);
  py::gil_scoped_release nogil;
  return chain_forward(x, xa, {W}, ctxlen, ChainCfg{alpha, act, n, C, module_l, 1, KEEP_OUTPUT, 0});
}

// A net given as one weight tensor per stage: fused where the library covers the shape, else stage by stage.
Result py_net_list(const Tensor& x, const Tensor& xa, const variable_list& ws, double alpha, int act, int n, int C,
                                       bool recompute, int every, bool tape, int keep) {
  if (needs_function(x, xa, ws)) return std::nullopt;
  check_activations(x, xa);
  py::gil_scoped_release nogil;
  const int L = (int)ws.size();
  bool fused = false;
  if (act != 3) {  // leaky-relu has per-stage kernels only
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const int flags = (recompute ? NCN_RECOMPUTE : 0) | (tape ? NCN_TAPE : 0);
    fused = ncn_net_supported_from(x.size(0), x.size(1), x.size(2), n, C, 0, L, dtype_code(x), flags, every) != 0;
  }
  if (fused) return fused_forward(x, xa, ws, true, FusedCfg{alpha, act, n, C, 0, L, 1, every, 0, recompute, false, tape});
  return chain_forward(x, xa, ws, Tensor(), ChainCfg{alpha, act, n, C, 0, L, keep, 0});
}

// ---------------------------------------------------------------- activations that live on the host
// Forward and backward of a fused net, chunk of rows by chunk (host.py): copies in, kernels and copies out on a stream each, two
// chunks of inputs and three of results on the device.  in: x, xa, dy, dya; out: y, ya, dx, dxa; dW [L, 2E] on the device gains the
// weight gradient chunk after chunk.  Returns when the results are on the host.
//
// Native because a chunk's 8 copies, 3 launches and 4 events cost 220 us in Python against 75 here, which sets the smallest chunk and
// with it how much of the first copy in and the last copy out nothing overlaps.
void py_host_step(const variable_list& in, const variable_list& out, const Tensor& weights, const Tensor& dW, double alpha, int act, int n, int C,
                  bool recompute, int every, bool tape, const std::vector<std::pair<int64_t, int64_t>>& chunks) {
  py::gil_scoped_release nogil;
  at::NoGradGuard no_grad;
  const c10::cuda::CUDAGuard guard(weights.device());
  const c10::DeviceIndex dev = weights.device().index();
  using Stream = c10::cuda::CUDAStream;
  const Stream s_in = c10::cuda::getStreamFromPool(false, dev), s_k = c10::cuda::getStreamFromPool(false, dev),
               s_out = c10::cuda::getStreamFromPool(false, dev);
  int64_t rows = 0;
  for (const auto& c : chunks) rows = std::max(rows, c.second - c.first);
  std::vector<int64_t> shape = in[0].sizes().vec();
  if (!shape.empty()) shape[0] = rows;
  const at::TensorOptions opt = in[0].options().device(weights.device()).pinned_memory(false);
  constexpr int SI = 2, SO = 3;
  // All memory comes from the caller's stream, which the others wait for: on streams of the pool, another three in every call, each
  // would gather a cache of its own.
  const int L = (int)weights.size(0);
  Tensor bin[SI][4], bout[SO][4], ck, ws;
  for (int k = 0; k < SO; ++k)
    for (int q = 0; q < 4; ++q) {
      if (k >= (int)chunks.size()) continue;
      if (k < SI) bin[k][q] = at::empty(shape, opt);
      bout[k][q] = at::empty(shape, opt);
    }
  if (chunks.empty()) return;
  check_activations(bin[0][0], bin[0][1]);
  const int64_t N = shape[1], E = shape[2];
  const int dt = dtype_code(bin[0][0]);
  const Tensor W = plain_weights(weights, (int64_t)L * 2 * E, weights.device());
  ws = at::empty({(int64_t)ncn_bwd_workspace_bytes(rows, N, E, n, C, L, dt)}, opt.dtype(at::kByte));
  if (const size_t bytes = ncn_ckpt_bytes(rows, N, E, L, every, tape ? NCN_TAPE : 0)) ck = at::empty({(int64_t)(bytes / 4)}, opt.dtype(at::kFloat));
  at::cuda::CUDAEvent start;
  start.record(c10::cuda::getCurrentCUDAStream(dev));
  for (const Stream& s : {s_in, s_k, s_out}) start.block(s);

  at::cuda::CUDAEvent ev_in[SI], ev_free[SI], ev_f[SO], ev_b[SO], ev_out[SO];
  try {
    int ci = 0;
    for (const auto& c : chunks) {
      const int ki = ci % SI, ko = ci % SO;
      const int64_t B = c.second - c.first;
      {
        const c10::cuda::CUDAStreamGuard on(s_in);
        if (ci >= SI) ev_free[ki].block(s_in);
        for (int q = 0; q < 4; ++q) bin[ki][q].slice(0, 0, B).copy_(in[q].slice(0, c.first, c.second), true);
        ev_in[ki].record(s_in);
      }
      {
        const c10::cuda::CUDAStreamGuard on(s_k);
        if (ci >= SO) ev_out[ko].block(s_k);
        ev_in[ki].block(s_k);
        void *const x = bin[ki][0].data_ptr(), *const xa = bin[ki][1].data_ptr(), *const y = bout[ko][0].data_ptr(), *const ya = bout[ko][1].data_ptr();
        float* const ckp = ck.defined() ? ck.mutable_data_ptr<float>() : nullptr;
        check_status("ncn_net_fwd", ncn_net_fwd(x, xa, W.const_data_ptr<float>(), y, ya, ckp, every, B, N, E, n, C, 0, L, alpha, act, dt,
                                                tape ? NCN_TAPE : 0, s_k.stream()));
        ev_f[ko].record(s_k);
        const void *const s0 = tape ? nullptr : recompute ? x : y, *const s1 = tape ? nullptr : recompute ? xa : ya;
        check_status("ncn_net_bwd",
                     ncn_net_bwd(s0, s1, bin[ki][2].data_ptr(), bin[ki][3].data_ptr(), W.const_data_ptr<float>(), bout[ko][2].data_ptr(),
                                 bout[ko][3].data_ptr(), nullptr, nullptr, dW.mutable_data_ptr<float>(), ckp, every, ws.data_ptr(),
                                 (size_t)ws.numel(), B, N, E, n, C, 0, L, alpha, act, dt, (recompute ? NCN_RECOMPUTE : 0) | (tape ? NCN_TAPE : 0),
                                 1, s_k.stream()));
        ev_b[ko].record(s_k);
        ev_free[ki].record(s_k);
      }
      {
        const c10::cuda::CUDAStreamGuard on(s_out);
        for (int q = 0; q < 4; ++q) {
          if (q == 0) ev_f[ko].block(s_out);  // the outputs leave while the backward still runs
          if (q == 2) ev_b[ko].block(s_out);
          out[q].slice(0, c.first, c.second).copy_(bout[ko][q].slice(0, 0, B), true);
        }
        ev_out[ko].record(s_out);
      }
      ++ci;
    }
    s_out.synchronize();
    s_k.synchronize();
  } catch (...) {  // nothing may be on its way to or from buffers that are given back
    for (const Stream& s : {s_in, s_k, s_out}) cudaStreamSynchronize(s.stream());
    throw;
  }
}

}  // namespace

PYBIND11_MODULE(_ncn_torch, m) {
  m.doc() = "autograd nodes of the NCN operators over the C ABI of libncn_b200.so";
  m.def("net", &py_net);
  m.def("net_list", &py_net_list);
  m.def("stages", &py_stages);
  m.def("stage_ctx", &py_stage_ctx);
  m.def("host_step", &py_host_step);
}
