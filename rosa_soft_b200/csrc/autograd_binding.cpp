// The differentiable operator as one native call: argument check, dropout seed, hard forward and the
// autograd node whose backward is the surrogate VJP.  Same order of work as soft.py's Python form
// (reference rosa_soft/soft.py:259-508), which stays for tracing and for everything that is not a
// plain call; going through the interpreter and a Python autograd function cost more host time than
// the kernels of a small step take.
#include <ATen/core/dispatch/Dispatcher.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <cmath>
#include <limits>
#include <optional>
#include <tuple>

#include "autograd_binding.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using Triple = std::tuple<Tensor, Tensor, Tensor>;

Triple call_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, int64_t W) {
  if (!cu.defined()) {
    static const auto op = c10::Dispatcher::singleton()
        .findSchemaOrThrow("rosa_soft::hard_forward", "")
        .typed<Triple(Tensor, Tensor, Tensor, int64_t)>();
    return op.call(q, k, v, W);
  }
  static const auto op = c10::Dispatcher::singleton()
      .findSchemaOrThrow("rosa_soft::hard_forward_varlen", "")
      .typed<Triple(Tensor, Tensor, Tensor, Tensor, int64_t)>();
  return op.call(q, k, v, cu, W);
}

Triple call_vjp(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, const Tensor& go,
                const Tensor& pq, const Tensor& pk, const Tensor& seed, int64_t W, double scale, double p,
                double m, int64_t mask, int64_t batch_offset, int64_t head_offset) {
  static const auto op = c10::Dispatcher::singleton()
      .findSchemaOrThrow("rosa_soft::surrogate_vjp_typed", "")
      .typed<Triple(Tensor, Tensor, Tensor, std::optional<Tensor>, Tensor, Tensor, Tensor, Tensor, int64_t,
                    double, double, double, int64_t, int64_t, int64_t)>();
  return op.call(q, k, v, cu.defined() ? std::optional<Tensor>(cu) : std::nullopt, go, pq, pk, seed, W, scale,
                 p, m, mask, batch_offset, head_offset);
}

// What the node keeps besides its differentiable inputs.
struct Controls {
  Tensor cu, seed;
  int64_t horizon, batch_offset, head_offset;
  double scale, dropout_p, mismatch_scale;
};

class HardForwardSoftVjp : public torch::autograd::Function<HardForwardSoftVjp> {
 public:
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                        const Controls& c) {
    auto [out, pq, pk] = call_forward(q, k, v, c.cu, c.horizon);
    variable_list saved = {q, k, v, pq, pk, c.seed};
    if (c.cu.defined()) saved.push_back(c.cu);
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["horizon"] = c.horizon;
    ctx->saved_data["scale"] = c.scale;
    ctx->saved_data["dropout_p"] = c.dropout_p;
    ctx->saved_data["mismatch_scale"] = c.mismatch_scale;
    ctx->saved_data["batch_offset"] = c.batch_offset;
    ctx->saved_data["head_offset"] = c.head_offset;
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    int64_t mask = 0;
    for (int x = 0; x < 3; ++x) mask |= ctx->needs_input_grad(x) ? int64_t(1) << x : 0;
    variable_list out(4);
    if (mask == 0) return out;
    // differentiable once: a second derivative raises, as torch's once_differentiable does
    const bool twice = torch::GradMode::is_enabled() && grads[0].requires_grad();
    {
      torch::AutoGradMode no_grad(false);
      auto [dq, dk, dv] = call_vjp(
          saved[0], saved[1], saved[2], saved.size() > 6 ? saved[6] : Tensor(), grads[0], saved[3], saved[4],
          saved[5], ctx->saved_data["horizon"].toInt(), ctx->saved_data["scale"].toDouble(),
          ctx->saved_data["dropout_p"].toDouble(), ctx->saved_data["mismatch_scale"].toDouble(), mask,
          ctx->saved_data["batch_offset"].toInt(), ctx->saved_data["head_offset"].toInt());
      if (mask & 1) out[0] = dq;
      if (mask & 2) out[1] = dk;
      if (mask & 4) out[2] = dv;
    }
    if (twice) {
      auto error = std::make_shared<torch::autograd::DelayedError>(
          "trying to differentiate twice a function that was marked with @once_differentiable", 3);
      variable_list wrapped;
      for (int x = 0; x < 3; ++x) {
        if (out[x].defined()) {
          Tensor fake = out[x].detach();
          fake.requires_grad_(true);
          wrapped.push_back(fake);
        } else {
          wrapped.emplace_back();
        }
      }
      wrapped = (*error)(std::move(wrapped));
      for (int x = 0; x < 3; ++x) out[x] = wrapped[x];
    }
    return out;
  }
};

bool number(PyObject* o, double* value) {   // an int or a float, exactly
  if (PyFloat_CheckExact(o)) {
    *value = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (!PyLong_CheckExact(o)) return false;
  *value = PyLong_AsDouble(o);
  if (*value == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// The call if it is plainly valid, else None: the Python form then checks the arguments one by one
// and raises, or takes what this one does not.
py::object soft(const py::object& query, const py::object& key, const py::object& value,
                const py::object& cu_seqlens, const py::object& max_suffix_length, const py::object& scale,
                const py::object& dropout_p, const py::object& mismatch_scale, int64_t batch_offset,
                int64_t head_offset) {
  const bool dense = cu_seqlens.is_none();
  if (!THPVariable_CheckExact(query.ptr()) || !THPVariable_CheckExact(key.ptr()) ||
      !THPVariable_CheckExact(value.ptr()) || (!dense && !THPVariable_CheckExact(cu_seqlens.ptr())) ||
      !PyLong_CheckExact(max_suffix_length.ptr()) ||
      c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode))
    return py::none();
  Controls c;
  int overflow = 0;
  const int64_t W = PyLong_AsLongLongAndOverflow(max_suffix_length.ptr(), &overflow);
  if (overflow != 0 || W < 1 || !number(scale.ptr(), &c.scale) || !number(dropout_p.ptr(), &c.dropout_p) ||
      !number(mismatch_scale.ptr(), &c.mismatch_scale))
    return py::none();
  const Tensor& q = THPVariable_Unpack(query.ptr());
  const Tensor& k = THPVariable_Unpack(key.ptr());
  const Tensor& v = THPVariable_Unpack(value.ptr());
  const auto type = q.scalar_type();
  const int64_t lead = dense ? 2 : 1;     // batch and sequence, or packed tokens
  if (!q.is_cuda() || q.device() != k.device() || q.device() != v.device() ||
      (type != torch::kFloat32 && type != torch::kFloat16 && type != torch::kBFloat16) ||
      k.scalar_type() != type || v.scalar_type() != type || q.dim() != lead + 2 || v.dim() != lead + 2 ||
      q.sizes() != k.sizes() || q.sizes().slice(0, lead) != v.sizes().slice(0, lead) || q.numel() == 0 ||
      v.numel() == 0 || q.size(lead) % v.size(lead) != 0 || q.size(lead + 1) > 32)
    return py::none();
  if (!dense) {
    c.cu = THPVariable_Unpack(cu_seqlens.ptr());
    if (!c.cu.is_cuda() || c.cu.device() != q.device() || c.cu.dim() != 1 || c.cu.numel() < 2 ||
        c.cu.scalar_type() != torch::kInt32)
      return py::none();
  }
  c.horizon = std::min<int64_t>(W, dense ? q.size(1) : q.size(0));
  // the float32 ranges of the controls and of the products formed from them
  const double lo = std::numeric_limits<float>::min(), hi = std::numeric_limits<float>::max();
  const double horizon = static_cast<double>(c.horizon);
  if (!(c.scale >= lo && c.scale <= hi && c.scale <= hi / horizon && c.dropout_p >= 0.0 &&
        c.dropout_p <= 1.0 - std::ldexp(1.0, -24) && c.mismatch_scale >= lo && c.mismatch_scale <= hi &&
        c.mismatch_scale <= hi / (horizon * c.scale)))
    return py::none();
  c.batch_offset = batch_offset;
  c.head_offset = head_offset;
  Tensor out;
  {
    py::gil_scoped_release no_gil;
    if (!torch::GradMode::is_enabled() || !(q.requires_grad() || k.requires_grad() || v.requires_grad())) {
      out = std::get<0>(call_forward(q, k, v, c.cu, c.horizon));
    } else {
      const auto options = q.options().dtype(torch::kInt64).requires_grad(false);
      // a seed is drawn on the device exactly when a backward with dropout will run
      c.seed = c.dropout_p != 0.0
                   ? at::randint(0, std::numeric_limits<int64_t>::max(), {}, options)
                   : at::empty({0}, options);
      out = HardForwardSoftVjp::apply(q, k, v, c);
    }
  }
  return py::reinterpret_steal<py::object>(THPVariable_Wrap(out));
}

}  // namespace

void bind_autograd(py::module_& m) { m.def("soft", &soft); }
