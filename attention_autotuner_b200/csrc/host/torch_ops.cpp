// Native operator layer between PyTorch and the C ABI of the kernel libraries: argument checks, output allocation,
// autograd nodes and the launch itself, without a Python frame in between. The Python operators
// (ops/attention_interface.py, ops/retnet_interface.py) look up which library serves a call, hand its entry point over
// as a "plan" and call one function of this module.
//
// Why: at the sizes where a kernel takes 10 to 100 us the operators were bound by the host. A forward call spent 45-50 us
// in Python (checks, tuner object, ctypes argument conversion, autograd.Function), a forward + backward 200 us. The
// reference's operators are Python as well (python/ops/attention_interface.py:8-61, python/ops/retnet_interface.py:8-58).
//
// Contract with the Python side:
//   * a function returns None when the arguments are not what the kernels take (the caller then runs the Python checks,
//     which raise with the reason) or when the plan is stale (a tuning-cache file or an environment variable it was
//     resolved from has changed); nothing has been launched in that case;
//   * a launch error raises the same exception class as the Python runtime (KernelError / AttnB200Error), in the
//     backward pass as well;
//   * plans are created once per resolution and live until the process exits. No tensor or pointer of a call outlives
//     the call except what autograd saves.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <sys/stat.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdlib>
#include <initializer_list>
#include <string>
#include <utility>
#include <vector>

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

using LastErrorFn = const char* (*)();
using AttnFwdFn = int (*)(const void*, const void*, const void*, void*, float*, int, int, int, int, float, int, void*);
using RetFwdFn = int (*)(const void*, const void*, const void*, const void*, void*, float*, int, int, int, int, float,
                         const float*, int, void*);
using RetBwdFn = int (*)(const void*, const void*, const void*, const void*, const void*, const float*, void*, void*, void*,
                         void*, int, int, int, int, float, const float*, int, void*, size_t);
using AttnBwdFn = int (*)(const void*, const void*, const void*, const void*, const void*, const float*, void*, void*, void*,
                          int, int, int, int, int, int, float, int, void*);
using ChunkBytesFn = size_t (*)(int, int, int, int, int, int);
using ChunkFwdFn = int (*)(const void*, const void*, const void*, const void*, void*, void*, size_t, int, int, int, int, int,
                           int, int, float, void*);

// ------------------------------------------------------------------------------------------------ plans
long long mtime_ns(const std::string& path) {  // -1: no such file
  struct stat st;
  if (stat(path.c_str(), &st) != 0) return -1;
  return static_cast<long long>(st.st_mtim.tv_sec) * 1000000000ll + st.st_mtim.tv_nsec;
}

// The entry point a call is served by, and what that choice was read from.
struct Plan {
  void* fn = nullptr;
  LastErrorFn last_error = nullptr;
  std::string libname;
  std::vector<std::pair<std::string, long long>> files;  // path, modification time at resolution (-1: absent)
  struct Env {
    std::string name, value;
    bool set;
  };
  std::vector<Env> env;

  // The GIL is held: assignments to os.environ call setenv under it, and getenv beside a setenv is undefined.
  bool env_unchanged() const {
    TORCH_INTERNAL_ASSERT(PyGILState_Check(), "a plan's environment is read without the GIL");
    for (const auto& e : env) {
      const char* now = getenv(e.name.c_str());
      if ((now != nullptr) != e.set || (now != nullptr && e.value != now)) return false;
    }
    return true;
  }
  // file-system calls: without the GIL where a call may
  bool files_unchanged() const {
    for (const auto& f : files)
      if (mtime_ns(f.first) != f.second) return false;
    return true;
  }
};

// The part of a plan's check that needs the GIL; its files are looked at after the GIL is released.
bool callable_now(const Plan* plan) { return plan->fn != nullptr && plan->env_unchanged(); }

constexpr const char* kPlanName = "attn_b200.plan";

// ------------------------------------------------------------------------------------------------ Python-side objects
PyObject* g_kernel_error = nullptr;    // autotuner.runtime.KernelError
PyObject* g_lib_error = nullptr;       // _lib.AttnB200Error(code, text)
PyObject* g_resolve_bwd = nullptr;     // callable: plan of a RetNet backward (may search, as the forward's lookup does)
struct {
  LastErrorFn last_error = nullptr;
  AttnBwdFn fa_bwd = nullptr;
  ChunkBytesFn chunk_bytes = nullptr;
  ChunkFwdFn chunk_fwd = nullptr;
} g_lib;

[[noreturn]] void throw_python(PyObject* exc) {  // GIL held, takes the reference; null: an error is already set
  if (exc != nullptr) {
    PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(exc)), exc);
    Py_DECREF(exc);
  }
  python_error e;
  e.persist();
  throw e;
}

void check_plan_rc(int rc, const Plan* plan) {
  if (rc == 0) return;
  const std::string text = plan->libname + ": status " + std::to_string(rc) + ": " + plan->last_error();
  py::gil_scoped_acquire gil;
  throw_python(PyObject_CallFunction(g_kernel_error, "s", text.c_str()));
}

void check_lib_rc(int rc) {
  if (rc == 0) return;
  const std::string text = g_lib.last_error();
  py::gil_scoped_acquire gil;
  throw_python(PyObject_CallFunction(g_lib_error, "is", rc, text.c_str()));
}

[[noreturn]] void raise_not_implemented(const std::string& text) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_NotImplementedError, text.c_str());
  throw_python(nullptr);
}
[[noreturn]] void raise_value_error(const std::string& text) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_ValueError, text.c_str());
  throw_python(nullptr);
}

// ------------------------------------------------------------------------------------------------ checks
// The conditions of ops/_checks.py, which words the errors: false sends the caller there.
bool qkv_ok(const Tensor& q, const Tensor& k, const Tensor& v) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return false;
  const auto dt = q.scalar_type();
  if (dt != at::kHalf && dt != at::kBFloat16) return false;
  if (k.scalar_type() != dt || v.scalar_type() != dt) return false;
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device()) return false;
  const int64_t dqk = q.size(3), dv = v.size(3);
  return k.size(0) == q.size(0) && k.size(1) == q.size(1) && v.size(0) == q.size(0) && v.size(1) == q.size(1) &&
         k.size(3) == dqk && v.size(2) == k.size(2) && q.numel() > 0 && k.numel() > 0 && v.numel() > 0 && dqk % 64 == 0 &&
         dqk <= 256 && dv % 64 == 0 && dv <= 512;
}

bool mask_decay_ok(const Tensor& q, const Tensor& k, const Tensor& mask, const Tensor& decay) {
  if (mask.defined() == decay.defined()) return false;
  if (mask.defined())
    return mask.dim() == 3 && mask.size(0) == q.size(1) && mask.size(1) == q.size(2) && mask.size(2) == k.size(2) &&
           mask.scalar_type() == q.scalar_type() && mask.device() == q.device() && k.size(2) % 8 == 0;
  return decay.numel() == q.size(1) && at::isFloatingType(decay.scalar_type());
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
int i32(int64_t x) { return static_cast<int>(x); }
std::string shape_text(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + (t.dim() == 1 ? ",)" : ")");
}

// What the engine hands a backward must match the output it is the gradient of (it may differ in dtype only if a caller
// built the graph by hand).
void check_grad(const char* op, const Tensor& dout, at::IntArrayRef shape, at::ScalarType dt, at::Device dev) {
  if (!dout.defined()) raise_value_error(std::string(op) + ": dO must be a tensor");
  if (dout.sizes() != shape) raise_value_error(std::string(op) + ": dO has shape " + shape_text(dout) + ", which is not the output's");
  if (dout.scalar_type() != dt) raise_value_error(std::string(op) + ": dO has dtype " + c10::toString(dout.scalar_type()) + ", expected " + c10::toString(dt));
  if (dout.device() != dev) raise_value_error(std::string(op) + ": dO is on " + dout.device().str() + ", expected " + dev.str());
}

// ------------------------------------------------------------------------------------------------ attention
// Forward launch; lse only when asked for.
std::pair<Tensor, Tensor> attn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Plan* plan, double scale,
                                       bool causal, bool want_lse) {
  c10::cuda::CUDAGuard guard(q.device());
  Tensor o = at::empty({q.size(0), q.size(1), q.size(2), v.size(3)}, q.options());
  Tensor lse;
  if (want_lse) lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
  check_plan_rc(reinterpret_cast<AttnFwdFn>(plan->fn)(ptr(q), ptr(k), ptr(v), ptr(o), static_cast<float*>(ptr(lse)), i32(q.size(0)),
                                                      i32(q.size(1)), i32(k.size(2)), i32(q.size(2)), static_cast<float>(scale),
                                                      causal ? 1 : 0, stream_of(q)),
                plan);
  return {o, lse};
}

struct AttnNode : public torch::autograd::Function<AttnNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, int64_t plan, double scale,
                               bool causal, bool return_lse) {
    const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
    auto [o, lse] = attn_forward(q, k, v, reinterpret_cast<const Plan*>(plan), scale, causal, true);
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    if (!return_lse) return {o};
    ctx->mark_non_differentiable({lse});
    return {o, lse};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &o = saved[3], &lse = saved[4];
    const bool causal = ctx->saved_data["causal"].toBool();
    const int64_t d = q.size(3), Lq = q.size(2), Lkv = k.size(2);
    if (!(k.size(3) == d && v.size(3) == d && (d == 64 || d == 128)))
      raise_not_implemented("attention backward needs one head dimension of 64 or 128 for q, k and v (got " + std::to_string(d) + ", " +
                            std::to_string(k.size(3)) + ", " + std::to_string(v.size(3)) + ")");
    if (causal && Lq != Lkv) raise_not_implemented("causal attention backward needs Lq == Lkv");
    check_grad("flash_attn_func backward", grads[0], o.sizes(), o.scalar_type(), o.device());
    const Tensor dout = grads[0].contiguous();
    c10::cuda::CUDAGuard guard(q.device());
    Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
    check_lib_rc(g_lib.fa_bwd(ptr(q), ptr(k), ptr(v), ptr(o), ptr(dout), static_cast<const float*>(ptr(lse)), ptr(dq), ptr(dk), ptr(dv),
                              i32(q.size(0)), i32(q.size(1)), i32(Lq), i32(Lkv), i32(d), q.scalar_type() == at::kHalf ? 0 : 1,
                              static_cast<float>(ctx->saved_data["scale"].toDouble()), causal ? 1 : 0, stream_of(q)));
    return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ RetNet, parallel form
Tensor decay_on(const Tensor& decay, const Tensor& q) {
  if (!decay.defined()) return decay;
  return decay.detach().to(q.options().dtype(at::kFloat)).contiguous().reshape({-1});
}

std::pair<Tensor, Tensor> ret_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& mask, const Tensor& decay,
                                      const Plan* plan, double scale, bool causal) {
  c10::cuda::CUDAGuard guard(q.device());
  Tensor o = at::empty({q.size(0), q.size(1), q.size(2), v.size(3)}, q.options());
  Tensor r = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
  check_plan_rc(reinterpret_cast<RetFwdFn>(plan->fn)(ptr(q), ptr(k), ptr(v), ptr(mask), ptr(o), static_cast<float*>(ptr(r)),
                                                     i32(q.size(0)), i32(q.size(1)), i32(k.size(2)), i32(q.size(2)),
                                                     static_cast<float>(scale), static_cast<const float*>(ptr(decay)), causal ? 1 : 0,
                                                     stream_of(q)),
                plan);
  return {o, r};
}

// Scratch of the backward: with a mask tensor, room for a transposed copy of it (read by rows in the dV / dK kernels).
// It takes the place of the reference's dq_accum (python/ops/retnet_interface.py:48-54).
Tensor ret_bwd_scratch(const Tensor& q, const Tensor& k, const Tensor& mask) {
  if (!mask.defined() || q.size(2) % 8 != 0) return Tensor();
  return at::empty({mask.size(0) * q.size(2) * k.size(2)}, q.options());
}

variable_list ret_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& mask, const Tensor& dout_, const Tensor& r,
                           const Tensor& decay, const Plan* plan, int64_t token, double scale, bool causal) {
  const Tensor dout = dout_.contiguous();
  c10::cuda::CUDAGuard guard(q.device());
  Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  Tensor scratch = ret_bwd_scratch(q, k, mask);
  if (plan != nullptr) {
    bool current = plan->files_unchanged();
    if (current) {
      py::gil_scoped_acquire gil;
      current = callable_now(plan);
    }
    if (!current) plan = nullptr;
  }
  if (plan == nullptr) {
    // not looked up yet (or changed since): the Python side resolves it, with these tensors should it want to search
    py::gil_scoped_acquire gil;
    auto wrap = [](const Tensor& t) { return py::reinterpret_steal<py::object>(THPVariable_Wrap(t)); };
    py::list arr;
    for (const Tensor& t : {q, k, v, mask, dout, r, dq, dk, dv, scratch}) {
      if (t.defined()) arr.append(wrap(t));
      else arr.append(py::none());
    }
    PyObject* res = PyObject_CallFunction(g_resolve_bwd, "LOdOO", static_cast<long long>(token), arr.ptr(), scale,
                                          causal ? Py_True : Py_False, decay.defined() ? wrap(decay).ptr() : Py_None);
    if (res == nullptr) throw_python(nullptr);
    plan = static_cast<const Plan*>(PyCapsule_GetPointer(res, kPlanName));
    Py_DECREF(res);  // the plan itself is never freed
    if (plan == nullptr) throw_python(nullptr);
  }
  check_plan_rc(reinterpret_cast<RetBwdFn>(plan->fn)(
                    ptr(q), ptr(k), ptr(v), ptr(mask), ptr(dout), static_cast<const float*>(ptr(r)), ptr(dq), ptr(dk), ptr(dv),
                    ptr(scratch), i32(q.size(0)), i32(q.size(1)), i32(k.size(2)), i32(q.size(2)), static_cast<float>(scale),
                    static_cast<const float*>(ptr(decay)), causal ? 1 : 0, stream_of(q),
                    scratch.defined() ? static_cast<size_t>(scratch.nbytes()) : size_t(0)),
                plan);
  return {dq, dk, dv};
}

struct RetNode : public torch::autograd::Function<RetNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_,
                               const std::optional<Tensor>& mask_, const std::optional<Tensor>& decay_, int64_t plan, int64_t bwd_plan,
                               int64_t token, double scale, bool causal) {
    const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
    const Tensor mask = mask_ ? mask_->detach().contiguous() : Tensor();
    const Tensor decay = decay_ ? decay_on(*decay_, q) : Tensor();
    auto [o, r] = ret_forward(q, k, v, mask, decay, reinterpret_cast<const Plan*>(plan), scale, causal);
    ctx->save_for_backward({q, k, v, mask, r, decay});
    ctx->saved_data["plan"] = bwd_plan;
    ctx->saved_data["token"] = token;
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    return {o};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &v = saved[2];
    check_grad("RetNetAttnFunc backward", grads[0], {q.size(0), q.size(1), q.size(2), v.size(3)}, q.scalar_type(), q.device());
    variable_list out = ret_backward(q, saved[1], v, saved[3], grads[0], saved[4], saved[5],
                                     reinterpret_cast<const Plan*>(ctx->saved_data["plan"].toInt()), ctx->saved_data["token"].toInt(),
                                     ctx->saved_data["scale"].toDouble(), ctx->saved_data["causal"].toBool());
    out.resize(10);
    return out;
  }
};

// ------------------------------------------------------------------------------------------------ Python functions
// Whether the call has to go through an autograd node: any of its tensors does, the mask or the decay as well (their gradient
// is none, but the output has a node). Forward-mode duals do too, whatever the grad mode: the node raises (there is no jvp),
// whereas the plain launch would drop the tangents.
bool any_grad(std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    if (t->defined() && (t->_fw_grad(/*level=*/0).defined() || (at::GradMode::is_enabled() && t->requires_grad()))) return true;
  return false;
}
// A tensor argument, or an undefined tensor for None; false for any other object.
bool take_tensor(PyObject* obj, Tensor& t, bool none_ok = false) {
  if (none_ok && obj == Py_None) return true;
  if (!THPVariable_Check(obj)) return false;
  t = THPVariable_Unpack(obj);
  return true;
}
Plan* take_plan(PyObject* obj) {
  if (obj == Py_None) return nullptr;
  return static_cast<Plan*>(PyCapsule_GetPointer(obj, kPlanName));
}
PyObject* none() { Py_RETURN_NONE; }
bool arg_count(Py_ssize_t n, Py_ssize_t want, const char* fn) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", fn, want, n);
  return false;
}

// attn(q, k, v, plan, scale, causal, return_lse) -> o | (o, lse) | None
PyObject* py_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 7, "attn")) return nullptr;
  Tensor q, k, v;
  if (!take_tensor(a[0], q) || !take_tensor(a[1], k) || !take_tensor(a[2], v) || !qkv_ok(q, k, v)) return none();
  Plan* plan = take_plan(a[3]);
  if (plan == nullptr) return PyErr_Occurred() ? nullptr : none();
  if (!callable_now(plan)) return none();
  const double scale = PyFloat_AsDouble(a[4]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  const int causal = PyObject_IsTrue(a[5]), ret_lse = PyObject_IsTrue(a[6]);
  if (causal < 0 || ret_lse < 0) return nullptr;
  Tensor o, lse;
  {
    py::gil_scoped_release nogil;
    if (!plan->files_unchanged()) plan = nullptr;
    else if (any_grad({&q, &k, &v})) {
      variable_list out = AttnNode::apply(q, k, v, reinterpret_cast<int64_t>(plan), scale, causal != 0, ret_lse != 0);
      o = out[0];
      if (ret_lse) lse = out[1];
    } else {
      std::tie(o, lse) = attn_forward(q.contiguous(), k.contiguous(), v.contiguous(), plan, scale, causal != 0, ret_lse != 0);
    }
  }
  if (plan == nullptr) return none();
  if (!ret_lse) return THPVariable_Wrap(std::move(o));
  PyObject* po = THPVariable_Wrap(std::move(o));
  PyObject* pl = THPVariable_Wrap(std::move(lse));
  return Py_BuildValue("(NN)", po, pl);
  END_HANDLE_TH_ERRORS
}

// retnet(q, k, v, mask | None, decay | None, plan, backward plan | None, token, scale, causal) -> o | None
PyObject* py_retnet(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 10, "retnet")) return nullptr;
  Tensor q, k, v, mask, decay;
  if (!take_tensor(a[0], q) || !take_tensor(a[1], k) || !take_tensor(a[2], v) || !take_tensor(a[3], mask, true) ||
      !take_tensor(a[4], decay, true) || !qkv_ok(q, k, v) || !mask_decay_ok(q, k, mask, decay))
    return none();
  Plan* plan = take_plan(a[5]);
  Plan* bwd = take_plan(a[6]);
  if (PyErr_Occurred()) return nullptr;
  if (plan == nullptr || !callable_now(plan)) return none();
  const long long token = PyLong_AsLongLong(a[7]);
  const double scale = PyFloat_AsDouble(a[8]);
  if (PyErr_Occurred()) return nullptr;
  const int causal = PyObject_IsTrue(a[9]);
  if (causal < 0) return nullptr;
  Tensor o;
  {
    py::gil_scoped_release nogil;
    if (!plan->files_unchanged()) plan = nullptr;
    else if (any_grad({&q, &k, &v, &mask, &decay})) {
      auto given = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
      o = RetNode::apply(q, k, v, given(mask), given(decay), reinterpret_cast<int64_t>(plan), reinterpret_cast<int64_t>(bwd),
                         static_cast<int64_t>(token), scale, causal != 0)[0];
    } else {
      o = ret_forward(q.contiguous(), k.contiguous(), v.contiguous(), mask.defined() ? mask.detach().contiguous() : mask,
                      decay_on(decay, q), plan, scale, causal != 0)
              .first;
    }
  }
  if (plan == nullptr) return none();
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// retnet_fwd_raw(q, k, v, mask | None, decay | None, plan, scale, causal) -> (o, r, mask, decay) | None; no autograd
PyObject* py_retnet_fwd_raw(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 8, "retnet_fwd_raw")) return nullptr;
  Tensor q, k, v, mask, decay;
  if (!take_tensor(a[0], q) || !take_tensor(a[1], k) || !take_tensor(a[2], v) || !take_tensor(a[3], mask, true) ||
      !take_tensor(a[4], decay, true) || !qkv_ok(q, k, v) || !mask_decay_ok(q, k, mask, decay))
    return none();
  Plan* plan = take_plan(a[5]);
  if (plan == nullptr) return PyErr_Occurred() ? nullptr : none();
  if (!callable_now(plan)) return none();
  const double scale = PyFloat_AsDouble(a[6]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  const int causal = PyObject_IsTrue(a[7]);
  if (causal < 0) return nullptr;
  Tensor o, r, m, d;
  {
    py::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    if (!plan->files_unchanged()) plan = nullptr;
    else {
      if (mask.defined()) m = mask.detach().contiguous();
      d = decay_on(decay, q);
      std::tie(o, r) = ret_forward(q.contiguous(), k.contiguous(), v.contiguous(), m, d, plan, scale, causal != 0);
    }
  }
  if (plan == nullptr) return none();
  auto wrap = [](Tensor& t) -> PyObject* {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(t));
  };
  PyObject *po = wrap(o), *pr = wrap(r), *pm = wrap(m), *pd = wrap(d);
  return Py_BuildValue("(NNNN)", po, pr, pm, pd);
  END_HANDLE_TH_ERRORS
}

// retnet_bwd_raw(q, k, v, mask | None, do, r, decay | None, plan | None, token, scale, causal) -> (dq, dk, dv); the
// arguments have been checked
PyObject* py_retnet_bwd_raw(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 11, "retnet_bwd_raw")) return nullptr;
  Tensor q, k, v, mask, dout, r, decay;
  if (!take_tensor(a[0], q) || !take_tensor(a[1], k) || !take_tensor(a[2], v) || !take_tensor(a[3], mask, true) ||
      !take_tensor(a[4], dout) || !take_tensor(a[5], r) || !take_tensor(a[6], decay, true)) {
    PyErr_SetString(PyExc_TypeError, "retnet_bwd_raw: tensors expected");
    return nullptr;
  }
  Plan* plan = take_plan(a[7]);
  const long long token = PyLong_AsLongLong(a[8]);
  const double scale = PyFloat_AsDouble(a[9]);
  if (PyErr_Occurred()) return nullptr;
  const int causal = PyObject_IsTrue(a[10]);
  if (causal < 0) return nullptr;
  variable_list out;
  {
    py::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    out = ret_backward(q.contiguous(), k.contiguous(), v.contiguous(), mask.defined() ? mask.contiguous() : mask, dout, r.contiguous(),
                       decay_on(decay, q), plan, token, scale, causal != 0);
  }
  PyObject *p0 = THPVariable_Wrap(out[0]), *p1 = THPVariable_Wrap(out[1]), *p2 = THPVariable_Wrap(out[2]);
  return Py_BuildValue("(NNN)", p0, p1, p2);
  END_HANDLE_TH_ERRORS
}

// chunkwise(q, k, v, decay, scale) -> o | None
PyObject* py_chunkwise(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 5, "chunkwise")) return nullptr;
  Tensor q, k, v, decay;
  if (!take_tensor(a[0], q) || !take_tensor(a[1], k) || !take_tensor(a[2], v) || !take_tensor(a[3], decay) || !qkv_ok(q, k, v) ||
      !mask_decay_ok(q, k, Tensor(), decay) || k.size(2) != q.size(2) || (q.size(3) != 128 && q.size(3) != 256))
    return none();
  const double scale = PyFloat_AsDouble(a[4]);
  if (scale == -1.0 && PyErr_Occurred()) return nullptr;
  Tensor o;
  {
    py::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    const Tensor qc = q.contiguous(), kc = k.contiguous(), vc = v.contiguous(), dc = decay_on(decay, q);
    c10::cuda::CUDAGuard guard(q.device());
    const int B = i32(q.size(0)), H = i32(q.size(1)), L = i32(q.size(2)), dqk = i32(q.size(3)), dv = i32(v.size(3));
    o = at::empty({B, H, L, dv}, q.options());
    const size_t bytes = g_lib.chunk_bytes(B, H, L, dqk, dv, 0);
    Tensor ws;
    if (bytes != 0) ws = at::empty({static_cast<int64_t>(bytes)}, q.options().dtype(at::kByte));
    check_lib_rc(g_lib.chunk_fwd(ptr(qc), ptr(kc), ptr(vc), ptr(dc), ptr(o), ptr(ws), bytes, 0, B, H, L, dqk, dv,
                                 q.scalar_type() == at::kHalf ? 0 : 1, static_cast<float>(scale), stream_of(q)));
  }
  return THPVariable_Wrap(std::move(o));
  END_HANDLE_TH_ERRORS
}

// make_plan(entry point, last_error, library name, [paths], [environment variables]) -> plan, stamped with the files' times
// and the variables' values of this moment. What the plan is made from is to be read after that: then a change in between
// makes the plan stale instead of being taken as seen. The entry point may follow with set_entry; a plan without one is
// declined by every function.
PyObject* py_make_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 5, "make_plan")) return nullptr;
  auto* plan = new Plan();
  plan->fn = reinterpret_cast<void*>(py::cast<uintptr_t>(py::handle(a[0])));
  plan->last_error = reinterpret_cast<LastErrorFn>(py::cast<uintptr_t>(py::handle(a[1])));
  plan->libname = py::cast<std::string>(py::handle(a[2]));
  for (auto h : py::cast<py::list>(py::handle(a[3]))) {
    const std::string path = py::cast<std::string>(h);
    plan->files.emplace_back(path, mtime_ns(path));
  }
  for (auto h : py::cast<py::list>(py::handle(a[4]))) {
    const std::string name = py::cast<std::string>(h);
    const char* now = getenv(name.c_str());
    plan->env.push_back({name, now ? now : "", now != nullptr});
  }
  return PyCapsule_New(plan, kPlanName, nullptr);
  END_HANDLE_TH_ERRORS
}

// set_entry(plan, entry point, last_error, library name); before the plan is handed to any other function
PyObject* py_set_entry(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 4, "set_entry")) return nullptr;
  Plan* plan = take_plan(a[0]);
  if (plan == nullptr) return PyErr_Occurred() ? nullptr : none();
  plan->last_error = reinterpret_cast<LastErrorFn>(py::cast<uintptr_t>(py::handle(a[2])));
  plan->libname = py::cast<std::string>(py::handle(a[3]));
  plan->fn = reinterpret_cast<void*>(py::cast<uintptr_t>(py::handle(a[1])));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* py_plan_fresh(PyObject*, PyObject* obj) {
  Plan* plan = take_plan(obj);
  if (plan == nullptr && PyErr_Occurred()) return nullptr;
  return PyBool_FromLong(plan != nullptr && plan->env_unchanged() && plan->files_unchanged());
}

// init(KernelError, AttnB200Error, resolver of backward plans, last_error, fa_bwd, chunk workspace bytes, chunk forward)
PyObject* py_init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 7, "init")) return nullptr;
  PyObject** keep[3] = {&g_kernel_error, &g_lib_error, &g_resolve_bwd};
  for (int i = 0; i < 3; ++i) {
    Py_INCREF(a[i]);
    *keep[i] = a[i];
  }
  auto addr = [&](int i) { return py::cast<uintptr_t>(py::handle(a[i])); };
  g_lib.last_error = reinterpret_cast<LastErrorFn>(addr(3));
  g_lib.fa_bwd = reinterpret_cast<AttnBwdFn>(addr(4));
  g_lib.chunk_bytes = reinterpret_cast<ChunkBytesFn>(addr(5));
  g_lib.chunk_fwd = reinterpret_cast<ChunkFwdFn>(addr(6));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

template <class F>
PyCFunction fast(F f) {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef g_methods[] = {
    {"attn", fast(py_attn), METH_FASTCALL, nullptr},
    {"retnet", fast(py_retnet), METH_FASTCALL, nullptr},
    {"retnet_fwd_raw", fast(py_retnet_fwd_raw), METH_FASTCALL, nullptr},
    {"retnet_bwd_raw", fast(py_retnet_bwd_raw), METH_FASTCALL, nullptr},
    {"chunkwise", fast(py_chunkwise), METH_FASTCALL, nullptr},
    {"make_plan", fast(py_make_plan), METH_FASTCALL, nullptr},
    {"set_entry", fast(py_set_entry), METH_FASTCALL, nullptr},
    {"plan_fresh", py_plan_fresh, METH_O, nullptr},
    {"init", fast(py_init), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torch_ops", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// build.py passes the hash of what the module is made from; ops/_native.py compares it when it loads the module
PyMODINIT_FUNC PyInit__torch_ops() {
  PyObject* module = PyModule_Create(&g_module);
  if (module != nullptr && PyModule_AddStringConstant(module, "source_hash", ATTN_B200_OPS_HASH) != 0) Py_CLEAR(module);
  return module;
}
