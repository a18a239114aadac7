// The host side of the functional surface as native code: from pytrees of torch tensors to fo_step_ex calls.
//
// tx.step() of a pytree of L leaves touches 5 L Python objects before its launches.  Walking them in Python costs
// about 1.5 us per leaf when the buffers are donated and 30 us per leaf when they are not (the ResNet-50 pytree:
// 280 us of host time for 90 us of device time).  What does not change from step to step is therefore
// compiled once into a Plan (structure of the trees, shapes and dtypes, param-group membership, launch tables), and a
// step walks the trees with the plan in hand: structure, types, devices and contiguity of every leaf are checked
// again, addresses and hyper-parameter values are filled in, results that must not overwrite their operands
// are allocated, and the launches are issued.  Anything the plan does not describe makes run() return None
// before it has had any effect, and the general path in _engine.py takes the step (and its error messages).
//
// The same walk serves reconstruct_weights / set_fp32_params, the moment codecs and the gradient norm.
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <unordered_map>
#include <vector>

#include "../../include/flashoptim_b200.h"

namespace {

// ---- the C ABI, bound by address (the library is loaded by _lib.py) ---------------------------------------------
struct Api {
  decltype(&fo_step_ex) step = nullptr;
  decltype(&fo_sq_norm_mixed) sq_norm = nullptr;
  decltype(&fo_split_many) split = nullptr;
  decltype(&fo_reconstruct_many) reconstruct = nullptr;
  decltype(&fo_quantize_momentum) quantize_m = nullptr;
  decltype(&fo_quantize_variance) quantize_v = nullptr;
  decltype(&fo_dequantize_momentum) dequantize_m = nullptr;
  decltype(&fo_dequantize_variance) dequantize_v = nullptr;
  decltype(&fo_status_string) status_string = nullptr;
  decltype(&fo_last_error) last_error = nullptr;
} api;

// _lib.check() of a status: false with a Python exception set
bool ok(int status) {
  if (status == FO_OK) return true;
  PyErr_Format(status == FO_ERR_INVALID_ARG || status == FO_ERR_UNSUPPORTED || status == FO_ERR_TOO_LARGE ? PyExc_ValueError : PyExc_RuntimeError,
               "flashoptim_b200: %s: %s", api.status_string(status), api.last_error());
  return false;
}

struct Ref {  // owning reference
  PyObject* p = nullptr;
  Ref() = default;
  explicit Ref(PyObject* owned) : p(owned) {}
  Ref(Ref&& o) noexcept : p(o.p) { o.p = nullptr; }
  Ref& operator=(Ref&& o) noexcept { std::swap(p, o.p); return *this; }
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  PyObject* release() { PyObject* q = p; p = nullptr; return q; }
  static Ref borrow(PyObject* q) { Py_XINCREF(q); return Ref(q); }
};

PyObject* quantized_type = nullptr;  // QuantizedArray
PyObject *ordered_type = nullptr, *default_type = nullptr;  // collections.OrderedDict and defaultdict

// ---- pytrees -----------------------------------------------------------------------------------------------------
// The containers of tree.py, exact types and the two dicts of the standard library that keep dict's item access (another subclass may
// redefine it: the Python walk takes those).
bool is_dict(PyObject* x) {
  PyObject* const type = (PyObject*)Py_TYPE(x);
  return PyDict_CheckExact(x) || type == ordered_type || type == default_type;
}
struct Node {
  enum Kind { kLeaf, kNone, kDict, kList, kTuple, kNamed } kind = kLeaf;
  PyTypeObject* type = nullptr;      // kNamed
  std::vector<Ref> keys;             // kDict: flattening order
  std::vector<int> seen;             // kDict: position in flattening order of the k-th item in insertion order
  std::vector<Ref> seen_keys;        // kDict: keys in insertion order
  PyTypeObject* key_type = nullptr;  // kDict: type of all its keys, if it is one
  std::vector<Node> children;
  bool nested = false;               // a child is no leaf
  int first = 0, count = 1;          // leaves
};

// A NamedTuple that is made of its items and nothing else: no __new__ or __init__ of its own (build() calls tuple.__new__), no metaclass,
// no iteration of its own.  A subclass that adds one is left to the Python walk.
bool is_named(PyObject* x) {
  if (!PyTuple_Check(x) || PyTuple_CheckExact(x)) return false;
  PyTypeObject* const type = Py_TYPE(x);
  if (!Py_IS_TYPE((PyObject*)type, &PyType_Type) || type->tp_init != PyTuple_Type.tp_init || type->tp_iter != PyTuple_Type.tp_iter || type->tp_mro == nullptr) return false;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(type->tp_mro); ++i) {
    PyObject* const d = ((PyTypeObject*)PyTuple_GET_ITEM(type->tp_mro, i))->tp_dict;
    if (d == nullptr) return false;  // (tuple itself: nothing in front of it has _fields)
    if (PyDict_GetItemString(d, "__new__") != nullptr) return PyDict_GetItemString(d, "_fields") != nullptr;
  }
  return false;
}

// A container inside itself, or nested too deeply for the stack, is a RecursionError, as in the Python walk.  (The other walks follow
// a compiled tree and go no deeper than that.)
struct Deeper {
  const bool ok = Py_EnterRecursiveCall(" while walking a pytree") == 0;
  ~Deeper() {
    if (ok) Py_LeaveRecursiveCall();
  }
};

// false: a container this walk does not take (or, with an exception set, an error)
bool compile(PyObject* x, Node& n, int& leaves) {
  const Deeper deeper;
  if (!deeper.ok) return false;
  n.first = leaves;
  if (x == Py_None) {
    n.kind = Node::kNone;
  } else if (is_dict(x)) {
    n.kind = Node::kDict;
    Ref keys(PyDict_Keys(x));
    if (keys.p == nullptr) return false;
    const Py_ssize_t size = PyList_GET_SIZE(keys.p);
    for (Py_ssize_t i = 0; i < size; ++i) n.seen_keys.push_back(Ref::borrow(PyList_GET_ITEM(keys.p, i)));
    if (PyList_Sort(keys.p) != 0) {  // keys without an order keep the dict's
      if (!PyErr_ExceptionMatches(PyExc_TypeError)) return false;
      PyErr_Clear();
      return false;  // (left to the Python walk)
    }
    n.children.resize(size);
    std::unordered_map<PyObject*, int> place;
    place.reserve(size);
    for (Py_ssize_t i = 0; i < size; ++i) {
      PyObject* k = PyList_GET_ITEM(keys.p, i);
      n.keys.push_back(Ref::borrow(k));
      PyObject* v = PyDict_GetItemWithError(x, k);
      if (v == nullptr || !compile(v, n.children[i], leaves)) return false;
      place[k] = (int)i;
    }
    for (const Ref& k : n.seen_keys) n.seen.push_back(place[k.p]);
    if (size > 0) n.key_type = Py_TYPE(n.keys[0].p);
    for (const Ref& k : n.keys)
      if (Py_TYPE(k.p) != n.key_type) n.key_type = nullptr;
  } else if (PyList_CheckExact(x) || PyTuple_CheckExact(x) || is_named(x)) {
    n.kind = PyList_CheckExact(x) ? Node::kList : PyTuple_CheckExact(x) ? Node::kTuple : Node::kNamed;
    if (n.kind == Node::kNamed) n.type = Py_TYPE(x);
    const Py_ssize_t size = n.kind == Node::kList ? PyList_GET_SIZE(x) : PyTuple_GET_SIZE(x);
    n.children.resize(size);
    for (Py_ssize_t i = 0; i < size; ++i)
      if (!compile(n.kind == Node::kList ? PyList_GET_ITEM(x, i) : PyTuple_GET_ITEM(x, i), n.children[i], leaves)) return false;
  } else if (PyDict_Check(x) || PyList_Check(x) || PyTuple_Check(x)) {
    return false;
  } else {
    ++leaves;
  }
  n.count = leaves - n.first;
  for (const Node& c : n.children) n.nested = n.nested || c.kind != Node::kLeaf;
  return true;
}

// the leaves of x (borrowed) if it has the structure of n
bool walk(const Node& n, PyObject* x, PyObject** out) {
  switch (n.kind) {
    case Node::kLeaf:
      out[n.first] = x;
      // (containers other than a QuantizedArray are no leaves; the callers check for tensors)
      return true;
    case Node::kNone:
      return x == Py_None;
    case Node::kDict: {
      if (!is_dict(x) || PyDict_GET_SIZE(x) != (Py_ssize_t)n.keys.size()) return false;
      // usually the very key objects, in the order of the parameters or (trees that were rebuilt: states, results) sorted: no look-up by hash
      Py_ssize_t pos = 0;
      PyObject *k, *v;
      size_t j = 0;
      bool same = true, sorted = false;
      while (PyDict_Next(x, &pos, &k, &v)) {
        if (j == 0) sorted = k != n.seen_keys[0].p;
        if (k != (sorted ? n.keys : n.seen_keys)[j].p) { same = false; break; }
        if (!walk(n.children[sorted ? (int)j : n.seen[j]], v, out)) return false;
        ++j;
      }
      if (same) return true;
      // Equal keys then, of the same type: 1 and True are equal, and selectors see different paths.
      pos = 0;
      while (PyDict_Next(x, &pos, &k, &v))
        if (Py_TYPE(k) != n.key_type) return false;
      for (size_t i = 0; i < n.keys.size(); ++i) {
        v = PyDict_GetItemWithError(x, n.keys[i].p);
        if (v == nullptr || !walk(n.children[i], v, out)) return false;
      }
      return true;
    }
    case Node::kList:
      if (!PyList_CheckExact(x) || PyList_GET_SIZE(x) != (Py_ssize_t)n.children.size()) return false;
      for (size_t i = 0; i < n.children.size(); ++i)
        if (!walk(n.children[i], PyList_GET_ITEM(x, i), out)) return false;
      return true;
    case Node::kTuple:
    case Node::kNamed:
      if (n.kind == Node::kTuple ? !PyTuple_CheckExact(x) : Py_TYPE(x) != n.type) return false;
      if (PyTuple_GET_SIZE(x) != (Py_ssize_t)n.children.size()) return false;
      for (size_t i = 0; i < n.children.size(); ++i)
        if (!walk(n.children[i], PyTuple_GET_ITEM(x, i), out)) return false;
      return true;
  }
  return false;
}

// is every dict of x, which walk() has taken, a dict and no subclass?
bool plain(const Node& n, PyObject* x) {
  if (n.kind == Node::kLeaf || n.kind == Node::kNone) return true;
  if (n.kind != Node::kDict) {
    for (size_t i = 0; i < n.children.size(); ++i)
      if (!plain(n.children[i], n.kind == Node::kList ? PyList_GET_ITEM(x, i) : PyTuple_GET_ITEM(x, i))) return false;
    return true;
  }
  if (!PyDict_CheckExact(x)) return false;
  if (!n.nested) return true;
  for (size_t i = 0; i < n.keys.size(); ++i)
    if (!plain(n.children[i], PyDict_GetItem(x, n.keys[i].p))) return false;
  return true;
}

PyObject* tuple_of_type(PyTypeObject* type, PyObject* items) {  // items: a tuple, stolen
  Ref hold(items);
  if (items == nullptr) return nullptr;
  if (type == nullptr) return hold.release();
  Ref args(PyTuple_Pack(1, items));
  return args.p == nullptr ? nullptr : PyTuple_Type.tp_new(type, args.p, nullptr);
}

// a tree of the structure n with the given leaves (new references are taken)
PyObject* build(const Node& n, const std::vector<Ref>& leaves) {
  switch (n.kind) {
    case Node::kLeaf: {
      PyObject* x = leaves[n.first].p;
      Py_INCREF(x);
      return x;
    }
    case Node::kNone:
      Py_RETURN_NONE;
    case Node::kDict: {
      Ref d(PyDict_New());
      if (d.p == nullptr) return nullptr;
      for (size_t i = 0; i < n.keys.size(); ++i) {
        Ref v(build(n.children[i], leaves));
        if (v.p == nullptr || PyDict_SetItem(d.p, n.keys[i].p, v.p) != 0) return nullptr;
      }
      return d.release();
    }
    default: {
      const Py_ssize_t size = (Py_ssize_t)n.children.size();
      Ref seq(n.kind == Node::kList ? PyList_New(size) : PyTuple_New(size));
      if (seq.p == nullptr) return nullptr;
      for (Py_ssize_t i = 0; i < size; ++i) {
        PyObject* v = build(n.children[i], leaves);
        if (v == nullptr) return nullptr;
        if (n.kind == Node::kList) PyList_SET_ITEM(seq.p, i, v); else PyTuple_SET_ITEM(seq.p, i, v);
      }
      return n.kind == Node::kNamed ? tuple_of_type(n.type, seq.release()) : seq.release();
    }
  }
}

// ---- tensors -----------------------------------------------------------------------------------------------------
int dtype_code(at::ScalarType t) { return t == at::kFloat ? FO_F32 : t == at::kBFloat16 ? FO_BF16 : t == at::kHalf ? FO_F16 : -1; }

const at::Tensor* plain_tensor(PyObject* x) {  // torch.Tensor or Parameter itself, strided
  if (!THPVariable_CheckExact(x)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(x);
  return t.defined() && t.layout() == at::kStrided ? &t : nullptr;
}
const at::Tensor* cuda_tensor(PyObject* x, at::ScalarType dtype, at::IntArrayRef sizes, int device) {
  const at::Tensor* t = plain_tensor(x);
  if (t == nullptr || t->scalar_type() != dtype || !t->is_cuda() || t->device().index() != device || t->sizes() != sizes || !t->is_contiguous()) return nullptr;
  return t;
}
at::Tensor empty_like_on(at::IntArrayRef sizes, at::ScalarType dtype, int device) {
  return at::Tensor(at::detail::empty_cuda(sizes, dtype, at::Device(at::kCUDA, (c10::DeviceIndex)device), std::nullopt));
}
PyObject* host_int(int32_t v) {
  at::Tensor t(at::detail::empty_cpu({}, at::kInt));
  *t.mutable_data_ptr<int32_t>() = v;
  return THPVariable_Wrap(t);
}

// Runs f (an allocation or a launch may block: no Python in it) on the device and its current stream, with the GIL released; returns f's
// status, for ok().  The caller holds references to the tensors whose addresses f uses.
template <typename F>
int on_device(int device, F f) {
  struct Released {
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  c10::cuda::OptionalCUDAGuard guard;
  if (c10::cuda::current_device() != device) guard.set_index((c10::DeviceIndex)device);
  return f(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream());
}

// ---- the compiled step ---------------------------------------------------------------------------------------------
struct LeafSpec {
  std::vector<int64_t> sizes;
  int64_t n = 0, n_scales = 0;
  at::ScalarType param, grad, ecc;   // ecc: of the buffer, when ecc_bits
  int ecc_bits = 0, state = 0, group = 0, call = 0, at = 0;
};
struct Group {
  Ref lr;      // the learning rate, unless the watched dict has one
  int dict;    // which of the watched dicts the group comes from, or -1
  float wd, b1, b2, omb1, omb2, eps;
  double beta1, beta2;  // as fp32, for the bias corrections
  uint32_t flags;
};
struct Call {
  FoStepDesc desc;
  std::vector<FoLeaf> leaves;
  std::vector<FoLeafOut> outs;
  std::vector<FoHyper> hypers;
  std::vector<int> slots;  // group of each hyper set
  bool empty = true;       // no leaf has an element: nothing is launched
  int64_t elems = 0;
};
struct Watched {  // a param-group dict as it was when the plan was made
  Ref dict;
  std::vector<Ref> keys, values;
  Ref items;        // a list of selectors: its items then
  int lr = -1;      // position of the learning rate, if it has one
};
struct Plan {
  int opt = 0, device = 0, n_states = 0;
  bool donate = false;
  Node tree;
  int n = 0;
  std::vector<LeafSpec> leaves;
  std::vector<Group> groups;
  std::vector<Call> calls;
  std::vector<int> order;          // in which they are issued
  Ref param_groups;
  std::vector<Watched> watched;
  bool dynamic = false;            // a selector that has to be asked at every step (a callable)
  Ref selectors, paths;            // per group: selector(path, leaf), or a tuple with its answer for every leaf; the leaves' paths
  std::vector<int> membership;     // of each leaf: the first group that takes it, or -1
  Ref resolve;                     // learning rate of a schedule: resolve(lr, count tensor)
  bool busy = false;               // a selector or a schedule may run Python code, and that another step
  std::vector<PyObject*> p, g;     // scratch (borrowed; run() holds references for as long as it needs them)
  std::vector<std::vector<PyObject*>> s;
};
bool is_lr(PyObject* key) { return PyUnicode_CheckExact(key) && PyUnicode_CompareWithASCIIString(key, "learning_rate") == 0; }
constexpr const char* kPlanName = "flashoptim_b200.plan";

float f32(double x) { return (float)x; }

bool num(PyObject* t, Py_ssize_t i, double& out) {
  out = PyFloat_AsDouble(PyTuple_GET_ITEM(t, i));
  return !(out == -1.0 && PyErr_Occurred());
}

// make_plan(opt, donate, device, params, n_states, leaves, groups, calls, param_groups, watched, selectors, paths, membership, resolve)
//   leaves: tuples (shape, param dtype code, grad dtype code, ecc bits, state, group size, group, call, position)
//   groups: tuples (default lr, weight decay, b1, b2, 1 - b1, 1 - b2, eps, flags, position of its dict in watched or -1)
//   calls:  tuples (param dtype code, grad dtype code, ecc bits, state, group size, (group of each hyper set))
PyObject* make_plan(PyObject*, PyObject* args) {
  PyObject *params, *leaves, *groups, *calls, *param_groups, *watched, *selectors, *paths, *membership, *resolve;
  auto plan = std::make_unique<Plan>();
  int donate;
  if (!PyArg_ParseTuple(args, "ipiOiO!O!O!OO!O!O!O!O", &plan->opt, &donate, &plan->device, &params, &plan->n_states, &PyTuple_Type, &leaves, &PyTuple_Type, &groups,
                        &PyTuple_Type, &calls, &param_groups, &PyTuple_Type, &watched, &PyTuple_Type, &selectors, &PyTuple_Type, &paths, &PyTuple_Type, &membership, &resolve))
    return nullptr;
  plan->donate = donate != 0;
  if (!compile(params, plan->tree, plan->n)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  if (plan->n != PyTuple_GET_SIZE(leaves)) Py_RETURN_NONE;
  static const at::ScalarType kDtype[3] = {at::kFloat, at::kBFloat16, at::kHalf};
  for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(calls); ++k) {
    Call c;
    std::memset(&c.desc, 0, sizeof(c.desc));
    c.desc.struct_size = sizeof(c.desc);
    c.desc.opt = plan->opt;
    PyObject* slots;
    if (!PyArg_ParseTuple(PyTuple_GET_ITEM(calls, k), "iiiiiO!", &c.desc.param_dtype, &c.desc.grad_dtype, &c.desc.ecc_bits, &c.desc.state, &c.desc.group_size, &PyTuple_Type, &slots))
      return nullptr;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(slots); ++i) c.slots.push_back((int)PyLong_AsLong(PyTuple_GET_ITEM(slots, i)));
    c.hypers.resize(c.slots.size());
    std::memset(c.hypers.data(), 0, c.hypers.size() * sizeof(FoHyper));
    plan->calls.push_back(std::move(c));
  }
  for (Py_ssize_t i = 0; i < plan->n; ++i) {
    LeafSpec l;
    PyObject* shape;
    int pd, gd, group_size, slot;
    if (!PyArg_ParseTuple(PyTuple_GET_ITEM(leaves, i), "O!iiiiiiii", &PyTuple_Type, &shape, &pd, &gd, &l.ecc_bits, &l.state, &group_size, &l.group, &l.call, &slot)) return nullptr;
    l.n = 1;
    for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(shape); ++k) {
      l.sizes.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(shape, k)));
      l.n *= l.sizes.back();
    }
    l.n_scales = (l.n + group_size - 1) / group_size;
    l.param = kDtype[pd];
    l.grad = kDtype[gd];
    l.ecc = l.ecc_bits == 8 ? at::kChar : at::kShort;
    Call& c = plan->calls[l.call];
    l.at = (int)c.leaves.size();
    FoLeaf f;
    std::memset(&f, 0, sizeof(f));
    f.n = (uint64_t)l.n;
    c.empty = c.empty && l.n == 0;
    f.hyper = (uint32_t)slot;
    c.leaves.push_back(f);
    c.outs.push_back(FoLeafOut{});
    plan->leaves.push_back(std::move(l));
  }
  if (PyErr_Occurred()) return nullptr;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(groups); ++i) {
    PyObject* t = PyTuple_GET_ITEM(groups, i);
    Group gr;
    double v[6];
    gr.lr = Ref::borrow(PyTuple_GET_ITEM(t, 0));
    for (int k = 0; k < 6; ++k)
      if (!num(t, k + 1, v[k])) return nullptr;
    gr.wd = f32(v[0]); gr.b1 = f32(v[1]); gr.b2 = f32(v[2]); gr.omb1 = f32(v[3]); gr.omb2 = f32(v[4]); gr.eps = f32(v[5]);
    gr.beta1 = (double)gr.b1; gr.beta2 = (double)gr.b2;
    gr.flags = (uint32_t)PyLong_AsUnsignedLong(PyTuple_GET_ITEM(t, 7));
    gr.dict = (int)PyLong_AsLong(PyTuple_GET_ITEM(t, 8));
    if (gr.dict >= (int)PyTuple_GET_SIZE(watched)) Py_RETURN_NONE;
    plan->groups.push_back(std::move(gr));
  }
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(watched); ++i) {
    PyObject* d = PyTuple_GET_ITEM(watched, i);
    if (!PyDict_CheckExact(d)) Py_RETURN_NONE;
    Watched w;
    w.dict = Ref::borrow(d);
    Py_ssize_t pos = 0;
    PyObject *k, *v;
    while (PyDict_Next(d, &pos, &k, &v)) {
      if (is_lr(k)) w.lr = (int)w.keys.size();
      w.keys.push_back(Ref::borrow(k));
      w.values.push_back(Ref::borrow(v));
      if ((int)w.keys.size() - 1 == w.lr) continue;
      if (PyList_CheckExact(v)) {
        if (w.items.p != nullptr) Py_RETURN_NONE;
        w.items = Ref(PyList_AsTuple(v));
      }
    }
    plan->watched.push_back(std::move(w));
  }
  if (PyErr_Occurred()) return nullptr;
  plan->param_groups = Ref::borrow(param_groups);
  if (PyTuple_GET_SIZE(paths) != plan->n || PyTuple_GET_SIZE(membership) != plan->n || PyTuple_GET_SIZE(selectors) != (Py_ssize_t)plan->watched.size()) Py_RETURN_NONE;
  for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(selectors); ++k) {
    PyObject* sel = PyTuple_GET_ITEM(selectors, k);
    if (!PyTuple_CheckExact(sel)) plan->dynamic = true;
    else if (PyTuple_GET_SIZE(sel) != plan->n) Py_RETURN_NONE;
  }
  for (int i = 0; i < plan->n; ++i) plan->membership.push_back((int)PyLong_AsLong(PyTuple_GET_ITEM(membership, i)));
  if (PyErr_Occurred()) return nullptr;
  plan->selectors = Ref::borrow(selectors);
  plan->paths = Ref::borrow(paths);
  plan->resolve = Ref::borrow(resolve);
  plan->p.resize(plan->n); plan->g.resize(plan->n);
  plan->s.assign(plan->n_states, std::vector<PyObject*>(plan->n));
  for (Call& c : plan->calls) {  // moved into place: the tables' addresses are final now
    c.desc.n_leaves = (uint32_t)c.leaves.size();
    c.desc.n_hypers = (uint32_t)c.hypers.size();
    c.desc.leaves = c.leaves.data();
    c.desc.hypers = c.hypers.data();
    plan->order.push_back((int)plan->order.size());
  }
  // The largest first: the calls work on different leaves, and the launches of the small ones fill the SMs that are done with the large one.  In front
  // of it they keep its blocks, which need an SM each, from beginning.  (ResNet-50, 25.5 M bf16 elements and 106 fp32 vectors, which the tree has first:
  // SGDW 51.9 us a step in that order and 51.0 so, AdamW 71.2 and 66.6.)
  for (const LeafSpec& l : plan->leaves) plan->calls[l.call].elems += l.n;
  std::stable_sort(plan->order.begin(), plan->order.end(), [&](int a, int b) { return plan->calls[a].elems > plan->calls[b].elems; });
  return PyCapsule_New(plan.release(), kPlanName, [](PyObject* c) { delete (Plan*)PyCapsule_GetPointer(c, kPlanName); });
}

// Are the optimizer's param_groups what they were?  (Learning rates aside: a program may write one before every step, and the
// step reads it.)
bool groups_unchanged(const Plan& plan) {
  PyObject* pg = plan.param_groups.p;
  const Py_ssize_t size = pg == Py_None ? 0 : PyList_CheckExact(pg) ? PyList_GET_SIZE(pg) : PyTuple_CheckExact(pg) ? PyTuple_GET_SIZE(pg) : -1;
  if (size != (Py_ssize_t)plan.watched.size()) return false;
  for (Py_ssize_t i = 0; i < size; ++i) {
    const Watched& w = plan.watched[i];
    if ((PyList_CheckExact(pg) ? PyList_GET_ITEM(pg, i) : PyTuple_GET_ITEM(pg, i)) != w.dict.p) return false;
    if (PyDict_GET_SIZE(w.dict.p) != (Py_ssize_t)w.keys.size()) return false;
    Py_ssize_t pos = 0;
    PyObject *k, *v;
    size_t j = 0;
    while (PyDict_Next(w.dict.p, &pos, &k, &v)) {
      if (j >= w.keys.size() || k != w.keys[j].p) return false;
      if ((int)j == w.lr) {
        ++j;
        continue;
      }
      if (v != w.values[j].p) return false;
      if (PyList_CheckExact(v)) {
        if (PyList_GET_SIZE(v) != PyTuple_GET_SIZE(w.items.p)) return false;
        for (Py_ssize_t q = 0; q < PyList_GET_SIZE(v); ++q)
          if (PyList_GET_ITEM(v, q) != PyTuple_GET_ITEM(w.items.p, q)) return false;
      }
      ++j;
    }
  }
  return true;
}

// Checks one leaf and fills its table entry.  False: not what the plan describes.
bool fill_leaf(Plan& plan, const LeafSpec& l, int i) {
  Call& c = plan.calls[l.call];
  FoLeaf& f = c.leaves[l.at];
  const at::Tensor* p = cuda_tensor(plan.p[i], l.param, l.sizes, plan.device);
  const at::Tensor* g = p == nullptr ? nullptr : cuda_tensor(plan.g[i], l.grad, l.sizes, plan.device);
  if (g == nullptr) return false;
  f.param = p->data_ptr();
  f.grad = g->const_data_ptr();
  if (l.ecc_bits != 0) {
    const at::Tensor* e = cuda_tensor(plan.s[0][i], l.ecc, l.sizes, plan.device);
    if (e == nullptr) return false;
    f.ecc = e->data_ptr();
  } else {
    const at::Tensor* e = plain_tensor(plan.s[0][i]);  // the 0-d marker of an absent buffer is handed on
    if (e == nullptr || e->dim() != 0) return false;
  }
  for (int k = 1; k < plan.n_states; ++k) {
    PyObject* m = plan.s[k][i];
    void *values = nullptr, *scales = nullptr;
    if (l.state == FO_STATE_QUANT) {
      if ((PyObject*)Py_TYPE(m) != quantized_type || PyTuple_GET_SIZE(m) != 2) return false;
      const at::Tensor* v = cuda_tensor(PyTuple_GET_ITEM(m, 0), k == 1 ? at::kChar : at::kByte, l.sizes, plan.device);
      const at::Tensor* s = v == nullptr ? nullptr : cuda_tensor(PyTuple_GET_ITEM(m, 1), at::kHalf, {l.n_scales}, plan.device);
      if (s == nullptr) return false;
      values = v->data_ptr();
      scales = s->data_ptr();
    } else if (l.state == FO_STATE_FULL) {
      const at::Tensor* v = cuda_tensor(m, at::kFloat, l.sizes, plan.device);
      if (v == nullptr) return false;
      values = v->data_ptr();
    } else {
      if (plain_tensor(m) == nullptr) return false;
    }
    if (k == 1) { f.mu = values; f.mu_scales = scales; } else { f.nu = values; f.nu_scales = scales; }
  }
  return true;
}

// The leaves of the trees into the plan's scratch.  False: not what the plan describes (or, with an exception set, an error).
bool walk_params(Plan& plan, PyObject* params, PyObject* grads) {
  return walk(plan.tree, params, plan.p.data()) && walk(plan.tree, grads, plan.g.data());
}
bool walk_states(Plan& plan, PyObject* states) {
  for (int k = 0; k < plan.n_states; ++k)
    if (!walk(plan.tree, PyTuple_GET_ITEM(states, k), plan.s[k].data())) return false;
  return true;
}
// Do parameters and gradients look like the plan's?  (What tells plans apart, asked before the user's selectors and schedules
// are called for a plan; fill_leaf checks everything.)
bool plausible(const Plan& plan) {
  for (int i = 0; i < plan.n; ++i) {
    const LeafSpec& l = plan.leaves[i];
    const at::Tensor *p = plain_tensor(plan.p[i]), *g = plain_tensor(plan.g[i]);
    if (p == nullptr || g == nullptr || p->scalar_type() != l.param || g->scalar_type() != l.grad || p->sizes() != l.sizes || g->sizes() != l.sizes || !g->is_contiguous()) return false;
  }
  return true;
}

// owning references to leaves
class Held {
  std::vector<PyObject*> v_;

 public:
  explicit Held(const Plan& plan) { v_.reserve((size_t)plan.n * (2 + plan.n_states)); }
  Held(const Held&) = delete;
  ~Held() {
    for (PyObject* x : v_) Py_DECREF(x);
  }
  void take(const std::vector<PyObject*>& leaves) {
    for (PyObject* x : leaves) Py_INCREF(x);
    v_.insert(v_.end(), leaves.begin(), leaves.end());
  }
  // are these the leaves taken first and second?
  bool are(const std::vector<PyObject*>& a, const std::vector<PyObject*>& b) const {
    return std::equal(a.begin(), a.end(), v_.begin()) && std::equal(b.begin(), b.end(), v_.begin() + (ptrdiff_t)a.size());
  }
};

// Is every leaf in the group it was in when the plan was made?  1, 0, or -1 with an exception set.  Selectors that are
// functions are called, as the general path calls them: what they answer may depend on more than the leaf.
int membership_unchanged(const Plan& plan) {
  const Py_ssize_t groups = PyTuple_GET_SIZE(plan.selectors.p);
  for (int i = 0; i < plan.n; ++i) {
    int index = -1;
    for (Py_ssize_t k = 0; k < groups && index < 0; ++k) {
      PyObject* sel = PyTuple_GET_ITEM(plan.selectors.p, k);
      if (PyTuple_CheckExact(sel)) {
        if (PyTuple_GET_ITEM(sel, i) == Py_True) index = (int)k;
        continue;
      }
      PyObject* const a[2] = {PyTuple_GET_ITEM(plan.paths.p, i), plan.p[i]};
      Ref answer(PyObject_Vectorcall(sel, a, 2, nullptr));
      const int yes = answer.p == nullptr ? -1 : PyObject_IsTrue(answer.p);
      if (yes < 0) return -1;
      if (yes) index = (int)k;
    }
    if (index != plan.membership[i]) return 0;
  }
  return 1;
}

// f(leaf, output table entry of its array k, size of that array, dtype): the arrays of a leaf that a step writes.
// (0 parameter; 1 code; 2, 3 moment 1 and its scales; 4, 5 moment 2 and its scales)
template <typename F>
void each_result(Plan& plan, F f) {
  for (int i = 0; i < plan.n; ++i) {
    const LeafSpec& l = plan.leaves[i];
    FoLeafOut& o = plan.calls[l.call].outs[l.at];
    const at::IntArrayRef sizes = l.sizes;
    f(i, 0, o.param, sizes, l.param);
    if (l.ecc_bits != 0) f(i, 1, o.ecc, sizes, l.ecc);
    for (int k = 1; k < plan.n_states; ++k) {
      void *&values = k == 1 ? o.mu : o.nu, *&scales = k == 1 ? o.mu_scales : o.nu_scales;
      if (l.state == FO_STATE_QUANT) {
        f(i, 2 * k, values, sizes, k == 1 ? at::kChar : at::kByte);
        f(i, 2 * k + 1, scales, at::IntArrayRef(l.n_scales), at::kHalf);
      } else if (l.state == FO_STATE_FULL) {
        f(i, 2 * k, values, sizes, at::kFloat);
      }
    }
  }
}
void allocate_results(Plan& plan, std::vector<at::Tensor>& made) {
  made.reserve((size_t)plan.n * 6);
  each_result(plan, [&](int, int, void*& address, at::IntArrayRef sizes, at::ScalarType dtype) {
    made.push_back(empty_like_on(sizes, dtype, plan.device));
    address = made.back().data_ptr();
  });
}
// the same arrays as Python objects, with the markers of the absent ones handed on
bool wrap_results(Plan& plan, std::vector<at::Tensor>& made, std::vector<Ref>& params, std::vector<Ref> (&states)[3]) {
  params.resize(plan.n);
  for (int k = 0; k < plan.n_states; ++k) {
    states[k].resize(plan.n);
    for (int i = 0; i < plan.n; ++i)
      if (k == 0 ? plan.leaves[i].ecc_bits == 0 : plan.leaves[i].state == FO_STATE_NONE) states[k][i] = Ref::borrow(plan.s[k][i]);
  }
  size_t at = 0;
  Ref pending;  // values, until their scales come
  bool good = true;
  each_result(plan, [&](int i, int array, void*&, at::IntArrayRef, at::ScalarType) {
    Ref t(good ? THPVariable_Wrap(std::move(made[at++])) : nullptr);
    good = good && t.p != nullptr;
    if (!good) return;
    if (array <= 1) {
      (array == 0 ? params : states[0])[i] = std::move(t);
    } else if (array & 1) {
      PyObject* pair = PyTuple_New(2);
      if (pair != nullptr) {
        PyTuple_SET_ITEM(pair, 0, pending.release());
        PyTuple_SET_ITEM(pair, 1, t.release());
      }
      states[array / 2][i] = Ref(tuple_of_type((PyTypeObject*)quantized_type, pair));
      good = states[array / 2][i].p != nullptr;
    } else if (plan.leaves[i].state == FO_STATE_QUANT) {
      pending = std::move(t);
    } else {
      states[array / 2][i] = std::move(t);
    }
  });
  return good;
}

// run(plan, params, count, states, grads, sq_norm address or 0, max_norm)
//   -> None, or (params, states, count)
PyObject* run(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 7) { PyErr_SetString(PyExc_TypeError, "run takes 7 arguments"); return nullptr; }
  Plan* plan = (Plan*)PyCapsule_GetPointer(a[0], kPlanName);
  if (plan == nullptr) return nullptr;
  if (plan->busy) Py_RETURN_NONE;  // the tables are in use (another thread, or a step inside a callback)
  struct Busy {
    bool& b;
    explicit Busy(bool& x) : b(x) { b = true; }
    ~Busy() { b = false; }
  } busy(plan->busy);
  PyObject *params = a[1], *states = a[3], *grads = a[4];
  const at::Tensor* count_t = plain_tensor(a[2]);
  if (count_t == nullptr || !count_t->is_cpu() || count_t->scalar_type() != at::kInt || count_t->dim() != 0) Py_RETURN_NONE;
  if (!walk_params(*plan, params, grads) || !groups_unchanged(*plan)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const int32_t old_count = *count_t->const_data_ptr<int32_t>();
  const double step = (double)old_count + 1.0;
  Held held(*plan);  // the leaves stay alive, whatever happens to the trees meanwhile
  held.take(plan->p);
  held.take(plan->g);

  std::vector<double> lr(plan->groups.size());
  std::vector<Ref> lr_now;
  bool call = plan->dynamic;  // code of the user's
  for (const Group& gr : plan->groups) {
    const Watched* w = gr.dict < 0 ? nullptr : &plan->watched[gr.dict];
    PyObject* value = w == nullptr || w->lr < 0 ? gr.lr.p : PyDict_GetItemWithError(w->dict.p, w->keys[w->lr].p);
    if (value == nullptr) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_NONE;
    }
    lr_now.push_back(Ref::borrow(value));
    call = call || !PyFloat_CheckExact(value);
  }
  if (call && !plausible(*plan)) Py_RETURN_NONE;
  if (plan->dynamic) {
    const int same = membership_unchanged(*plan);
    if (same < 0) return nullptr;
    if (same == 0) Py_RETURN_NONE;
  }
  for (size_t i = 0; i < lr.size(); ++i) {
    PyObject* const value = lr_now[i].p;
    if (PyFloat_CheckExact(value)) {
      lr[i] = PyFloat_AS_DOUBLE(value);
      continue;
    }
    Ref v(PyObject_CallFunctionObjArgs(plan->resolve.p, value, a[2], nullptr));  // zero-based count (adamw.py:526)
    if (v.p == nullptr) return nullptr;
    lr[i] = PyFloat_AsDouble(v.p);
    if (lr[i] == -1.0 && PyErr_Occurred()) return nullptr;
  }
  // A selector or a schedule, or another thread that ran meanwhile, may have put other tensors into the trees or other storage
  // under a tensor: addresses are taken now, and nothing is called between here and the launches.
  if ((call && (!walk_params(*plan, params, grads) || !held.are(plan->p, plan->g))) || !walk_states(*plan, states)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  for (int k = 0; k < plan->n_states; ++k) held.take(plan->s[k]);
  for (int i = 0; i < plan->n; ++i)
    if (!fill_leaf(*plan, plan->leaves[i], i)) Py_RETURN_NONE;

  // from here on the step is taken
  std::vector<FoHyper> hyper(plan->groups.size());
  for (size_t i = 0; i < plan->groups.size(); ++i) {
    const Group& gr = plan->groups[i];
    FoHyper& h = hyper[i];
    std::memset(&h, 0, sizeof(h));
    h.lr = f32(lr[i]); h.wd = gr.wd; h.b1 = gr.b1; h.b2 = gr.b2; h.one_minus_b1 = gr.omb1; h.one_minus_b2 = gr.omb2; h.eps = gr.eps;
    h.bc1 = h.bc2 = 1.0f;
    if (plan->opt == FO_OPT_ADAM) {  // as _engine.bias_correction
      h.bc1 = 1.0f - f32(std::pow(gr.beta1, step));
      h.bc2 = 1.0f - f32(std::pow(gr.beta2, step));
    }
    h.flags = gr.flags;
  }
  void* const sq = PyLong_AsVoidPtr(a[5]);
  const double max_norm = PyFloat_AsDouble(a[6]);
  if (PyErr_Occurred()) return nullptr;
  std::vector<at::Tensor> made;  // results that must not overwrite their operands, in the order of leaf, array
  const int status = on_device(plan->device, [&](cudaStream_t stream) {
    if (!plan->donate) allocate_results(*plan, made);
    uint32_t chain = 0u;
    for (const int at : plan->order) {
      Call& c = plan->calls[at];
      for (size_t k = 0; k < c.slots.size(); ++k) c.hypers[k] = hyper[c.slots[k]];
      c.desc.grad_sq_norm = (const double*)sq;
      c.desc.max_grad_norm = f32(max_norm);
      const FoStepMore more = {sizeof(FoStepMore), chain, plan->donate ? nullptr : c.outs.data()};
      const int rc = api.step(&c.desc, &more, stream);
      if (rc != FO_OK) return rc;
      if (!c.empty) chain = FO_LAUNCH_CHAINED;  // (behind a call that launches nothing the stream holds what it held before)
    }
    return (int)FO_OK;
  });
  if (!ok(status)) return nullptr;

  std::vector<Ref> out_p, out_s[3];
  Ref count(host_int(old_count + 1));
  if (count.p == nullptr) return nullptr;
  if (plan->donate) {  // every array was updated in place
    bool as_they_are = plain(plan->tree, params);
    for (int k = 0; k < plan->n_states; ++k) as_they_are = as_they_are && plain(plan->tree, PyTuple_GET_ITEM(states, k));
    if (as_they_are) return PyTuple_Pack(3, params, states, count.p);
    // plain dicts come back, as from the general path
    auto leaves = [](const std::vector<PyObject*>& x) {
      std::vector<Ref> out;
      for (PyObject* leaf : x) out.push_back(Ref::borrow(leaf));
      return out;
    };
    out_p = leaves(plan->p);
    for (int k = 0; k < plan->n_states; ++k) out_s[k] = leaves(plan->s[k]);
  } else if (!wrap_results(*plan, made, out_p, out_s)) {
    return nullptr;
  }
  Ref new_params(build(plan->tree, out_p));
  Ref new_states(PyTuple_New(plan->n_states));
  if (new_params.p == nullptr || new_states.p == nullptr) return nullptr;
  for (int k = 0; k < plan->n_states; ++k) {
    PyObject* t = build(plan->tree, out_s[k]);
    if (t == nullptr) return nullptr;
    PyTuple_SET_ITEM(new_states.p, k, t);
  }
  return PyTuple_Pack(3, new_params.p, new_states.p, count.p);
}

// ---- gradient norm -------------------------------------------------------------------------------------------------
bool collect(PyObject* x, std::vector<at::Tensor>& out) {
  const Deeper deeper;
  if (!deeper.ok) return false;
  if (x == Py_None) return true;
  if (is_dict(x)) {
    // the order of the sum is that of the flattened tree
    bool sorted = true;
    Py_ssize_t pos = 0;
    PyObject *k, *v, *before = nullptr;
    while (sorted && PyDict_Next(x, &pos, &k, &v)) {
      if (!PyUnicode_CheckExact(k)) return false;
      sorted = before == nullptr || PyUnicode_Compare(before, k) < 0;
      before = k;
    }
    if (sorted) {
      pos = 0;
      while (PyDict_Next(x, &pos, &k, &v))
        if (!collect(v, out)) return false;
      return true;
    }
    while (PyDict_Next(x, &pos, &k, &v))
      if (!PyUnicode_CheckExact(k)) return false;
    Ref keys(PyDict_Keys(x));
    if (keys.p == nullptr || PyList_Sort(keys.p) != 0) return false;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(keys.p); ++i) {
      v = PyDict_GetItemWithError(x, PyList_GET_ITEM(keys.p, i));
      if (v == nullptr || !collect(v, out)) return false;
    }
    return true;
  }
  if (PyList_CheckExact(x) || PyTuple_CheckExact(x) || is_named(x)) {
    const Py_ssize_t size = PySequence_Fast_GET_SIZE(x);
    for (Py_ssize_t i = 0; i < size; ++i)
      if (!collect(PySequence_Fast_GET_ITEM(x, i), out)) return false;
    return true;
  }
  const at::Tensor* t = plain_tensor(x);
  if (t == nullptr || !t->is_cuda() || dtype_code(t->scalar_type()) < 0 || !t->is_contiguous()) return false;
  if (!out.empty() && t->device() != out[0].device()) return false;
  out.push_back(*t);
  return true;
}

// sq_norm(tree) -> one-element float64 tensor, or None
PyObject* sq_norm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 1) { PyErr_SetString(PyExc_TypeError, "sq_norm takes 1 argument"); return nullptr; }
  std::vector<at::Tensor> t;  // (references: the GIL is released below)
  const bool taken = collect(a[0], t);
  if (PyErr_Occurred()) return nullptr;
  if (!taken || std::all_of(t.begin(), t.end(), [](const at::Tensor& x) { return x.numel() == 0; })) Py_RETURN_NONE;  // (an error, reported there)
  const int device = t[0].device().index();
  std::vector<FoArray> arrays(t.size());
  std::vector<int32_t> dtypes(t.size());
  for (size_t i = 0; i < t.size(); ++i) {
    arrays[i] = FoArray{t[i].const_data_ptr(), (uint64_t)t[i].numel()};
    dtypes[i] = dtype_code(t[i].scalar_type());
  }
  at::Tensor out;
  if (!ok(on_device(device, [&](cudaStream_t s) {
        out = empty_like_on({1}, at::kDouble, device);
        const at::Tensor workspace = empty_like_on({FO_SQ_NORM_WORKSPACE_BYTES}, at::kByte, device);  // its own: streams do not share one
        return api.sq_norm(arrays.data(), dtypes.data(), (uint32_t)arrays.size(), 0, (double*)out.data_ptr(), workspace.data_ptr(), s);
      })))
    return nullptr;
  return THPVariable_Wrap(std::move(out));
}

// ---- fp32 weights <-> (parameters, ECC) ------------------------------------------------------------------------------
struct SplitTables {  // by (dtype, ECC width)
  std::vector<FoSplitLeaf> t[3][3];
  std::vector<at::Tensor> in;  // what the tables point to
  int launch(cudaStream_t s, decltype(&fo_split_many) fn) {
    for (int d = 0; d < 3; ++d)
      for (int e = 0; e < 3; ++e)
        if (!t[d][e].empty())
          if (const int rc = fn(t[d][e].data(), (uint32_t)t[d][e].size(), d, e * 8, s)) return rc;
    return FO_OK;
  }
};
int one_device(const std::vector<PyObject*>& xs, int device) {  // index of the CUDA device all tensors are on, or -1
  for (PyObject* x : xs) {
    const at::Tensor* t = plain_tensor(x);
    if (t == nullptr || !t->is_cuda() || (device >= 0 && t->device().index() != device)) return -1;
    device = t->device().index();
  }
  return device;
}

// reconstruct(params, ecc) -> tree of fp32 tensors, or None
PyObject* reconstruct(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "reconstruct takes 2 arguments"); return nullptr; }
  Node tree;
  int n = 0;
  if (!compile(a[0], tree, n)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  std::vector<PyObject*> p(n), e(n);
  if (n == 0 || !walk(tree, a[0], p.data()) || !walk(tree, a[1], e.data())) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const int device = one_device(p, -1);
  if (device < 0) Py_RETURN_NONE;
  for (int i = 0; i < n; ++i) {
    const at::Tensor *pt = plain_tensor(p[i]), *et = plain_tensor(e[i]);
    if (et == nullptr || !pt->is_contiguous()) Py_RETURN_NONE;
    const int code = dtype_code(pt->scalar_type());
    const bool ecc = et->scalar_type() == at::kChar || et->scalar_type() == at::kShort;
    if (code == FO_F32) continue;            // handed on as it is
    if (code < 0 || !ecc) Py_RETURN_NONE;    // (a conversion by torch)
    if (!et->is_cuda() || et->device().index() != device || et->sizes() != pt->sizes() || !et->is_contiguous()) Py_RETURN_NONE;
  }
  SplitTables tables;
  for (int i = 0; i < n; ++i) {
    tables.in.push_back(*plain_tensor(p[i]));
    tables.in.push_back(*plain_tensor(e[i]));
  }
  std::vector<at::Tensor> made(n);
  if (!ok(on_device(device, [&](cudaStream_t s) {
        for (int i = 0; i < n; ++i) {
          const at::Tensor &pt = tables.in[2 * i], &et = tables.in[2 * i + 1];
          const int code = dtype_code(pt.scalar_type());
          if (code == FO_F32) continue;
          made[i] = empty_like_on(pt.sizes(), at::kFloat, device);
          tables.t[code][et.scalar_type() == at::kChar ? 1 : 2].push_back(FoSplitLeaf{(float*)made[i].data_ptr(), const_cast<void*>(pt.const_data_ptr()), const_cast<void*>(et.const_data_ptr()), (uint64_t)pt.numel()});
        }
        return tables.launch(s, api.reconstruct);
      })))
    return nullptr;
  std::vector<Ref> out(n);
  for (int i = 0; i < n; ++i) out[i] = made[i].defined() ? Ref(THPVariable_Wrap(std::move(made[i]))) : Ref(THPVariable_Wrap(tables.in[2 * i]));
  return build(tree, out);
}

// split(fp32 tree, template tree, ECC bits of 16-bit leaves) -> (params, ecc), or None
PyObject* split(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "split takes 3 arguments"); return nullptr; }
  const long ecc_bits = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  Node tree;
  int n = 0;
  if (!compile(a[0], tree, n)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  std::vector<PyObject*> w(n), like(n);
  if (n == 0 || !walk(tree, a[0], w.data()) || !walk(tree, a[1], like.data())) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const int device = one_device(w, -1);
  if (device < 0) Py_RETURN_NONE;
  for (int i = 0; i < n; ++i) {
    const at::Tensor *wt = plain_tensor(w[i]), *lt = plain_tensor(like[i]);
    if (lt == nullptr || wt->scalar_type() != at::kFloat || !wt->is_contiguous()) Py_RETURN_NONE;
    if (dtype_code(lt->scalar_type()) < 0) Py_RETURN_NONE;
  }
  SplitTables tables;
  std::vector<at::ScalarType> dtype(n);
  for (int i = 0; i < n; ++i) {
    tables.in.push_back(*plain_tensor(w[i]));
    dtype[i] = plain_tensor(like[i])->scalar_type();
  }
  std::vector<at::Tensor> lp(n), ecc(n);
  if (!ok(on_device(device, [&](cudaStream_t s) {
        std::vector<at::Tensor> markers;  // 0-d zeros in the place of an absent ECC, each with storage of its own
        for (int i = 0; i < n; ++i) {
          const at::Tensor& wt = tables.in[i];
          const int code = dtype_code(dtype[i]);
          if (code == FO_F32 || ecc_bits == 0) markers.push_back(ecc[i] = empty_like_on({}, at::kInt, device));
          if (code == FO_F32) continue;
          lp[i] = empty_like_on(wt.sizes(), dtype[i], device);
          if (ecc_bits != 0) ecc[i] = empty_like_on(wt.sizes(), ecc_bits == 8 ? at::kChar : at::kShort, device);
          tables.t[code][ecc_bits / 8].push_back(FoSplitLeaf{(float*)const_cast<void*>(wt.const_data_ptr()), lp[i].data_ptr(), ecc_bits != 0 ? ecc[i].data_ptr() : nullptr, (uint64_t)wt.numel()});
        }
        if (!markers.empty()) at::_foreach_zero_(markers);  // (one launch)
        return tables.launch(s, api.split);
      })))
    return nullptr;
  std::vector<Ref> new_p(n), new_e(n);
  for (int i = 0; i < n; ++i) {
    new_p[i] = lp[i].defined() ? Ref(THPVariable_Wrap(std::move(lp[i]))) : Ref(THPVariable_Wrap(tables.in[i]));
    new_e[i] = Ref(THPVariable_Wrap(std::move(ecc[i])));
  }
  Ref x(build(tree, new_p)), y(build(tree, new_e));
  return x.p == nullptr || y.p == nullptr ? nullptr : PyTuple_Pack(2, x.p, y.p);
}

// ---- moment codecs ---------------------------------------------------------------------------------------------------
long group_size(PyObject* x) {  // 0: not one the library's int32_t holds
  int beyond = 0;
  const long g = PyLong_AsLongAndOverflow(x, &beyond);
  return beyond != 0 || g < 0 || g > INT32_MAX ? 0 : g;
}

// quantize(x, group size, variance) -> QuantizedArray, or None
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "quantize takes 3 arguments"); return nullptr; }
  const at::Tensor* given = plain_tensor(a[0]);
  if (given == nullptr || !given->is_cuda() || given->scalar_type() != at::kFloat || !given->is_contiguous() || !PyLong_CheckExact(a[1])) Py_RETURN_NONE;
  const long g = group_size(a[1]);
  if (g < 1 || g > 1024) Py_RETURN_NONE;
  const bool variance = a[2] == Py_True;
  const at::Tensor x = *given;  // (a reference: the GIL is released below)
  const int device = x.device().index();
  const int64_t n = x.numel();
  at::Tensor values, scales;
  if (!ok(on_device(device, [&](cudaStream_t s) {
        values = empty_like_on(x.sizes(), variance ? at::kByte : at::kChar, device);
        scales = empty_like_on({(n + g - 1) / g}, at::kHalf, device);
        return variance ? api.quantize_v((const float*)x.const_data_ptr(), (uint8_t*)values.data_ptr(), scales.data_ptr(), (uint64_t)n, (int32_t)g, 0, s)
                        : api.quantize_m((const float*)x.const_data_ptr(), (int8_t*)values.data_ptr(), scales.data_ptr(), (uint64_t)n, (int32_t)g, 0, s);
      })))
    return nullptr;
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(values)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(scales)));
  return tuple_of_type((PyTypeObject*)quantized_type, t);
}

// dequantize(QuantizedArray, group size, variance) -> fp32 tensor, or None
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "dequantize takes 3 arguments"); return nullptr; }
  if ((PyObject*)Py_TYPE(a[0]) != quantized_type || PyTuple_GET_SIZE(a[0]) != 2 || !PyLong_CheckExact(a[1])) Py_RETURN_NONE;
  const at::Tensor *v = plain_tensor(PyTuple_GET_ITEM(a[0], 0)), *sc = plain_tensor(PyTuple_GET_ITEM(a[0], 1));
  const long g = group_size(a[1]);
  const bool variance = a[2] == Py_True;
  if (v == nullptr || sc == nullptr || g < 1 || !v->is_cuda() || !sc->is_cuda() || v->device() != sc->device() || v->element_size() != 1 || sc->scalar_type() != at::kHalf ||
      !v->is_contiguous() || !sc->is_contiguous() || sc->numel() < (v->numel() + g - 1) / g)
    Py_RETURN_NONE;
  const at::Tensor codes = *v, scales = *sc;  // (references: the GIL is released below)
  const int device = codes.device().index();
  at::Tensor out;
  if (!ok(on_device(device, [&](cudaStream_t s) {
        out = empty_like_on(codes.sizes(), at::kFloat, device);
        return variance ? api.dequantize_v((const uint8_t*)codes.const_data_ptr(), scales.const_data_ptr(), (float*)out.data_ptr(), (uint64_t)codes.numel(), (int32_t)g, s)
                        : api.dequantize_m((const int8_t*)codes.const_data_ptr(), scales.const_data_ptr(), (float*)out.data_ptr(), (uint64_t)codes.numel(), (int32_t)g, s);
      })))
    return nullptr;
  return THPVariable_Wrap(std::move(out));
}

// bind({name: address}, QuantizedArray)
PyObject* bind(PyObject*, PyObject* args) {
  PyObject *d, *type;
  if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &d, &type)) return nullptr;
  auto get = [&](const char* name, auto& fn) {
    PyObject* v = PyDict_GetItemString(d, name);
    if (v == nullptr) { PyErr_Format(PyExc_KeyError, "%s", name); return false; }
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(PyLong_AsVoidPtr(v));
    return PyErr_Occurred() == nullptr;
  };
  if (!get("fo_step_ex", api.step) || !get("fo_sq_norm_mixed", api.sq_norm) || !get("fo_split_many", api.split) || !get("fo_reconstruct_many", api.reconstruct) ||
      !get("fo_quantize_momentum", api.quantize_m) || !get("fo_quantize_variance", api.quantize_v) || !get("fo_dequantize_momentum", api.dequantize_m) ||
      !get("fo_dequantize_variance", api.dequantize_v) || !get("fo_status_string", api.status_string) || !get("fo_last_error", api.last_error))
    return nullptr;
  Ref collections(PyImport_ImportModule("collections"));
  Ref ordered(collections.p == nullptr ? nullptr : PyObject_GetAttrString(collections.p, "OrderedDict"));
  Ref with_default(ordered.p == nullptr ? nullptr : PyObject_GetAttrString(collections.p, "defaultdict"));
  if (with_default.p == nullptr) return nullptr;
  auto keep = [](PyObject*& slot, PyObject* x) {
    Py_INCREF(x);
    Py_XDECREF(slot);
    slot = x;
  };
  keep(quantized_type, type);
  keep(ordered_type, ordered.p);
  keep(default_type, with_default.p);
  Py_RETURN_NONE;
}

// C++ exceptions (an allocation that fails) as Python exceptions
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, a, n);
  END_HANDLE_TH_ERRORS
}
template <PyObject* (*F)(PyObject*, PyObject*)>
PyObject* guarded_args(PyObject* self, PyObject* args) {
  HANDLE_TH_ERRORS
  return F(self, args);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"bind", (PyCFunction)(void*)guarded_args<bind>, METH_VARARGS, nullptr},
    {"make_plan", (PyCFunction)(void*)guarded_args<make_plan>, METH_VARARGS, nullptr},
    {"run", (PyCFunction)(void*)guarded<run>, METH_FASTCALL, nullptr},
    {"sq_norm", (PyCFunction)(void*)guarded<sq_norm>, METH_FASTCALL, nullptr},
    {"reconstruct", (PyCFunction)(void*)guarded<reconstruct>, METH_FASTCALL, nullptr},
    {"split", (PyCFunction)(void*)guarded<split>, METH_FASTCALL, nullptr},
    {"quantize", (PyCFunction)(void*)guarded<quantize>, METH_FASTCALL, nullptr},
    {"dequantize", (PyCFunction)(void*)guarded<dequantize>, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fo_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fo_host() { return PyModule_Create(&module); }
