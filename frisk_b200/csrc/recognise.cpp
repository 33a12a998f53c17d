// The usual kernels recognised natively: a CPython module (no GPU code) with one function,
//
//   plan(kernel) -> None                                                        look with the Python recognisers
//                 | (False, S_q, S_kv, D, scale, type of q, type of o, iq, ik, iv, io)       the attention graph
//                 | (True, M, N, K, type of A, type of C, trans_a, trans_b, clear_accum, policy, ia, ib, ic,
//                    fill or None, reduce kind or None, reduce argument, reduce_clear)        one gemm, its fill and reduce
//
// Walking and verifying a built kernel op by op in Python took most of a small call (a 64 x 64 attention tile 53.1 us, 16.2 with
// this module, whose part is 8; a 512 x 384 x 256 gemm with fill and reduce 28.8 and 13.4, of which 3), and nothing may be
// remembered between calls, since every list and attribute of the IR can be changed at any time.  So the same walk and
// the checks of ir._verify and of tensor_ops.attention_plan / execute.fused_plan are made here, read off the same objects.
//
// It only ever ACCEPTS: a kernel of the classes below whose checks all hold.  Anything else, whether it is wrong or merely
// unusual (a subclass, an attribute that is missing or of another type, two types that are equal without being plainly so),
// gives None, and the Python recognisers decide and word the error.  No exception leaves this file.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstring>
#include <deque>
#include <utility>
#include <vector>

namespace {

// an owned reference, null where a look-up failed (every check below treats null as "not the usual kernel")
class Ref {
 public:
  Ref() = default;
  explicit Ref(PyObject* owned) : p_(owned) {}
  Ref(const Ref& o) : p_(Py_XNewRef(o.p_)) {}
  Ref(Ref&& o) noexcept : p_(std::exchange(o.p_, nullptr)) {}
  Ref& operator=(Ref o) noexcept {
    std::swap(p_, o.p_);
    return *this;
  }
  ~Ref() { Py_XDECREF(p_); }
  PyObject* get() const { return p_; }
  explicit operator bool() const { return p_ != nullptr; }

 private:
  PyObject* p_ = nullptr;
};

#define NAMES(X)                                                                                                          \
  X(regions) X(blocks) X(operations) X(operands) X(results) X(attrs) X(type) X(owner) X(index) X(is_arg) X(kind) X(name)  \
  X(shape) X(element) X(space) X(map) X(op_name) X(arguments) X(m) X(n) X(k) X(trans_a) X(trans_b) X(dim) X(dimensions)   \
  X(threads) X(ranges) X(srcMap) X(dstMap) X(_nsrc) X(num_dims) X(num_symbols) X(_value) X(transA) X(transB) X(M) X(N)    \
  X(K) X(policy) X(clear_accum) X(value) X(clear) X(lower) X(upper) X(step) X(function_type) X(inputs)
struct Names {
#define X(n) PyObject* n = nullptr;
  NAMES(X)
#undef X
} names;

enum Class { kOther, kEnd, kParallel, kFor, kCopy, kFill, kReduce, kGemm, kMma, kReduceTensor, kView, kStore, kUpstream, kClasses };
PyObject* classes[kClasses];  // the Python classes, in the order of Class
PyObject *type_class, *value_class, *map_class, *space_class, *policy_class;
struct {
  Py_ssize_t type, owner, index, is_arg;
} value_at;  // places of a value's slots
struct {
  Py_ssize_t operands, results, attrs, regions;
} op_at[kClasses];

Ref attr(const Ref& o, PyObject* name) {
  if (!o) return Ref();
  PyObject* v = PyObject_GetAttr(o.get(), name);
  if (!v) PyErr_Clear();
  return Ref(v);
}
// An attribute that every object of a class holds in a slot: the descriptor's place in the object, 0 if there is none.
Py_ssize_t slot_of(PyObject* cls, PyObject* name) {
  const Ref d(PyObject_GetAttr(cls, name));
  if (!d) PyErr_Clear();
  if (!d || !Py_IS_TYPE(d.get(), &PyMemberDescr_Type)) return 0;
  const PyMemberDef* member = reinterpret_cast<PyMemberDescrObject*>(d.get())->d_member;
  return member->type == T_OBJECT_EX ? member->offset : 0;
}
// Read there, without PyObject_GetAttr, which looks through the classes first: a 64 x 64 attention graph takes 8.1 us, and 10.5 in its
// first call.  (Out of the objects' instance dictionaries it took 9.3, but they have none until somebody asks: a first call of 15.7,
// 4 KB a kernel that stayed, and ir._verify 7 % slower from then on.)
Ref slot(const Ref& o, Py_ssize_t at, PyObject* name) {
  if (o && at) {
    PyObject* v = *reinterpret_cast<PyObject**>(reinterpret_cast<char*>(o.get()) + at);
    if (v) return Ref(Py_NewRef(v));
  }
  return attr(o, name);
}

// The attributes of a type.  Its constructor fills the instance's dictionary, so there is one; an attribute costs a third of
// PyObject_GetAttr there.  What is not there is asked for the usual way.
class Fields {
 public:
  explicit Fields(const Ref& o) : o_(o.get()), dict_(o ? PyObject_GenericGetDict(o.get(), nullptr) : nullptr) {
    if (o_ && !dict_) PyErr_Clear();
  }
  Ref operator()(PyObject* name) const {
    if (!o_) return Ref();
    PyObject* v = dict_ ? PyDict_GetItemWithError(dict_.get(), name) : nullptr;
    if (v) return Ref(Py_NewRef(v));
    PyErr_Clear();
    v = PyObject_GetAttr(o_, name);
    if (!v) PyErr_Clear();
    return Ref(v);
  }
  bool holds(PyObject* name) const {  // in the instance itself
    if (!dict_) return true;
    const int has = PyDict_Contains(dict_.get(), name);
    if (has < 0) PyErr_Clear();
    return has != 0;
  }

 private:
  PyObject* o_;  // (the caller keeps it)
  Ref dict_;
};
Ref key(const Ref& dict, PyObject* name) {
  if (!dict || !PyDict_CheckExact(dict.get())) return Ref();
  PyObject* v = PyDict_GetItemWithError(dict.get(), name);
  if (!v) PyErr_Clear();
  return Ref(Py_XNewRef(v));
}
Ref item(const Ref& list, Py_ssize_t i) {
  if (!list || !PyList_CheckExact(list.get()) || i >= PyList_GET_SIZE(list.get())) return Ref();
  return Ref(Py_NewRef(PyList_GET_ITEM(list.get(), i)));
}
Py_ssize_t length(const Ref& list) { return list && PyList_CheckExact(list.get()) ? PyList_GET_SIZE(list.get()) : -1; }
bool text_is(const Ref& s, const char* t) {
  if (!s || !PyUnicode_CheckExact(s.get()) || !PyUnicode_IS_COMPACT_ASCII(s.get())) return false;  // (the names are ASCII)
  const size_t n = strlen(t);
  return (size_t)PyUnicode_GET_LENGTH(s.get()) == n && memcmp(PyUnicode_DATA(s.get()), t, n) == 0;
}
bool to_int(const Ref& o, long long* out) {
  if (!o || !PyLong_CheckExact(o.get())) return false;
  int overflow = 0;
  *out = PyLong_AsLongLongAndOverflow(o.get(), &overflow);
  return overflow == 0;
}
bool to_bool(const Ref& o, bool* out) {
  if (!o || !PyBool_Check(o.get())) return false;
  *out = o.get() == Py_True;
  return true;
}
// member of an IntEnum class: its value
bool to_enum(const Ref& o, PyObject* cls, long long* out) {
  if (!o || reinterpret_cast<PyObject*>(Py_TYPE(o.get())) != cls) return false;
  int overflow = 0;
  *out = PyLong_AsLongLongAndOverflow(o.get(), &overflow);
  return overflow == 0;
}
bool is_a(const Ref& o, PyObject* cls) { return o && reinterpret_cast<PyObject*>(Py_TYPE(o.get())) == cls; }

enum Element { kNone = -1, kF16, kBF16, kF32, kF64 };
constexpr int kBits[] = {16, 16, 32, 64};

// What the checks need of a type of the IR: a memref or tensor of up to two floating extents.
struct Shaped {
  bool memref = false;
  int rank = 0;
  long long e[2] = {0, 0};
  Element element = kNone;
  long long space = -1;  // of a memref
  Ref map;
  // of one shape and element type
  bool same_tile(const Shaped& o) const { return rank == o.rank && e[0] == o.e[0] && e[1] == o.e[1] && element == o.element; }
  // the same type, plainly
  bool same(const Shaped& o) const { return memref == o.memref && same_tile(o) && space == o.space && map.get() == o.map.get(); }
};

struct Value {
  PyObject* id = nullptr;  // the value object (kept alive by the operation or block that holds it)
  Shaped t;
  Ref owner;
  long long index = 0;
  bool is_arg = false;
};

struct Values {  // up to three, which the kernel's list of known values holds
  const Value* at[3] = {nullptr, nullptr, nullptr};
  size_t n = 0;
  const Value& operator[](size_t i) const { return *at[i]; }
  size_t size() const { return n; }
  bool empty() const { return n == 0; }
};

struct Op {
  Ref op, attrs, name;  // name: op_name of an upstream op
  Class cls = kOther;
  Values in, out;
};

// What has been read in this call already (an object appears many times), and the objects it was read from.
template <typename T>
struct Known {
  std::vector<PyObject*> ids;  // looked through from the end: most operands have just been results
  std::deque<T> what;          // (does not move)
  std::vector<Ref> keep;
  Known() {
    ids.reserve(64);
    keep.reserve(64);
  }
  const T* find(PyObject* id) const {
    for (size_t j = ids.size(); j > 0; --j)
      if (ids[j - 1] == id) return &what[j - 1];
    return nullptr;
  }
  const T* add(const Ref& o, T&& t) {
    what.push_back(std::move(t));
    keep.push_back(o);
    ids.push_back(o.get());
    return &what.back();
  }
};

struct Kernel {
  std::vector<Op> ops;  // nested ones, in program order
  Ref entry;
  Known<Shaped> types;
  Known<Value> values;
  Known<Element> elements;
  bool class_has_place = false;  // the class of the types itself has a `space` or a `map`
};

bool read_element(Kernel& k, const Ref& e, Element* out) {
  if (!is_a(e, type_class)) return false;
  if (const Element* known = k.elements.find(e.get())) {
    *out = *known;
    return true;
  }
  const Fields of(e);
  if (!text_is(of(names.kind), "float")) return false;
  const Ref name = of(names.name);
  *out = text_is(name, "f16") ? kF16 : text_is(name, "bf16") ? kBF16 : text_is(name, "f32") ? kF32 : text_is(name, "f64") ? kF64 : kNone;
  if (*out == kNone) return false;
  k.elements.add(e, Element(*out));
  return true;
}

bool read_type(Kernel& k, const Ref& t, Shaped* out) {
  if (!is_a(t, type_class)) return false;
  if (const Shaped* known = k.types.find(t.get())) {
    *out = *known;
    return true;
  }
  Shaped s;
  const Fields of(t);
  const Ref kind = of(names.kind);
  s.memref = text_is(kind, "memref");
  if (!s.memref && !text_is(kind, "tensor")) return false;
  const Ref shape = of(names.shape), element = of(names.element);
  s.rank = (int)length(shape);
  if (s.rank < 1 || s.rank > 2) return false;
  for (int i = 0; i < s.rank; ++i)
    if (!to_int(item(shape, i), &s.e[i]) || s.e[i] <= 0 || s.e[i] > (1LL << 40)) return false;
  if (!read_element(k, element, &s.element)) return false;
  if (s.memref) {
    if (!to_enum(of(names.space), space_class, &s.space)) return false;
    s.map = of(names.map);
    if (!s.map) return false;
  } else if (k.class_has_place || of.holds(names.space) || of.holds(names.map)) {
    return false;  // (a tensor has neither; types are compared with them)
  }
  *out = *k.types.add(t, std::move(s));
  return true;
}

bool read_values(Kernel& k, const Ref& list, Values* out) {
  const Py_ssize_t n = length(list);
  if (n < 0 || n > 3) return false;
  out->n = (size_t)n;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const Ref v = item(list, i);
    if (!v) return false;
    if ((out->at[i] = k.values.find(v.get()))) continue;
    if (!is_a(v, value_class)) return false;
    Value x;
    if (!read_type(k, slot(v, value_at.type, names.type), &x.t) || !to_bool(slot(v, value_at.is_arg, names.is_arg), &x.is_arg) ||
        !to_int(slot(v, value_at.index, names.index), &x.index))
      return false;
    x.owner = slot(v, value_at.owner, names.owner);
    x.id = v.get();
    out->at[i] = k.values.add(v, std::move(x));
  }
  return true;
}

bool is_pow2(long long n) { return n > 0 && (n & (n - 1)) == 0; }

// a dictionary's flag that the Python side reads by its truth
bool flag(const Op& op, PyObject* name, bool* out) { return to_bool(key(op.attrs, name), out); }

// the verifiers of ir._verify
bool verify_op(const Op& op, long long n_args) {
  const auto& in = op.in;
  const auto& out = op.out;
  switch (op.cls) {
    case kEnd:
    case kFor:
      return true;
    case kParallel: {
      long long threads = 0;
      if (!to_int(key(op.attrs, names.threads), &threads)) return false;
      if (threads != 32 && threads != 64 && threads != 128 && threads != 256 && threads != 512 && threads != 1024) return false;
      const Ref ranges = key(op.attrs, names.ranges);
      const Py_ssize_t n = length(ranges);
      if (n < 1 || n != n_args) return false;
      for (Py_ssize_t i = 0; i < n; ++i) {
        long long r = 0;
        if (!to_int(item(ranges, i), &r) || r <= 0) return false;
      }
      return true;
    }
    case kCopy: {  // whole tiles: no indices, maps without inputs
      long long n_src = 0, dims = 0;
      if (in.size() != 2 || !to_int(key(op.attrs, names._nsrc), &n_src) || n_src != 0) return false;
      for (PyObject* name : {names.srcMap, names.dstMap}) {
        const Ref map = key(op.attrs, name);
        if (!is_a(map, map_class)) return false;
        if (!to_int(attr(map, names.num_dims), &dims) || dims != 0) return false;
        if (!to_int(attr(map, names.num_symbols), &dims) || dims != 0) return false;
      }
      return true;
    }
    case kFill: {
      const Ref v = key(op.attrs, names.value);
      if (in.size() != 1 || !v || !PyTuple_CheckExact(v.get()) || PyTuple_GET_SIZE(v.get()) != 2) return false;
      const Ref e(Py_NewRef(PyTuple_GET_ITEM(v.get(), 1)));
      if (!PyFloat_CheckExact(PyTuple_GET_ITEM(v.get(), 0)) || !is_a(e, type_class) || !text_is(attr(e, names.kind), "float")) return false;
      static const char* const kNames[] = {"f16", "bf16", "f32", "f64"};
      return text_is(attr(e, names.name), kNames[in[0].t.element]);
    }
    case kReduce: {
      long long dim = 0;
      if (in.size() != 2 || !to_int(key(op.attrs, names.dim), &dim) || dim != 1) return false;
      const Shaped &s = in[0].t, &d = in[1].t;
      const Ref kind = key(op.attrs, names.kind);
      return s.memref && d.memref && s.rank == 2 && d.rank == 1 && s.e[0] == d.e[0] && s.element == d.element &&
             (text_is(kind, "add") || text_is(kind, "min") || text_is(kind, "max"));
    }
    case kGemm: {
      long long m = 0, n = 0, k = 0, policy = 0;
      bool ta = false, tb = false;
      if (in.size() != 3 || !flag(op, names.transA, &ta) || !flag(op, names.transB, &tb)) return false;
      if (!to_int(key(op.attrs, names.M), &m) || !to_int(key(op.attrs, names.N), &n) || !to_int(key(op.attrs, names.K), &k)) return false;
      if (!to_enum(key(op.attrs, names.policy), policy_class, &policy) || policy < 0 || policy > 2) return false;  // 3: Auto
      const Shaped &a = in[0].t, &b = in[1].t, &c = in[2].t;
      if (!a.memref || !b.memref || !c.memref || a.rank != 2 || b.rank != 2 || c.rank != 2) return false;
      if (a.element != b.element || a.element == kF64 || (c.element != a.element && c.element != kF32)) return false;
      return a.e[ta ? 1 : 0] == m && a.e[ta ? 0 : 1] == k && b.e[tb ? 1 : 0] == k && b.e[tb ? 0 : 1] == n && c.e[0] == m && c.e[1] == n;
    }
    case kMma: {
      long long m = 0, n = 0, k = 0;
      bool ta = false, tb = false;
      if (in.size() != 3 || out.size() != 1 || !flag(op, names.trans_a, &ta) || !flag(op, names.trans_b, &tb)) return false;
      if (!to_int(key(op.attrs, names.m), &m) || !to_int(key(op.attrs, names.n), &n) || !to_int(key(op.attrs, names.k), &k)) return false;
      const Shaped &a = in[0].t, &b = in[1].t, &c = in[2].t, &r = out[0].t;
      if (m <= 0 || n <= 0 || k <= 0 || a.rank != 2 || b.rank != 2 || c.rank != 2 || r.rank != 2) return false;
      if (a.element != b.element || c.element != r.element || kBits[c.element] < kBits[a.element]) return false;
      return a.e[ta ? 1 : 0] == m && a.e[ta ? 0 : 1] == k && b.e[tb ? 1 : 0] == k && b.e[tb ? 0 : 1] == n && c.e[0] == m &&
             c.e[1] == n && r.e[0] == m && r.e[1] == n;
    }
    case kReduceTensor: {
      long long dim = 0;
      if (in.size() != 1 || out.size() != 1 || !to_int(key(op.attrs, names.dim), &dim) || dim < 0 || dim > 1) return false;
      const Shaped &s = in[0].t, &d = out[0].t;
      const Ref kind = key(op.attrs, names.kind);
      return (text_is(kind, "sum") || text_is(kind, "max") || text_is(kind, "min")) && s.rank == 2 && d.rank == 1 &&
             s.element != kF64 && s.element == d.element && is_pow2(s.e[0]) && is_pow2(s.e[1]) && d.e[0] == s.e[1 - dim];
    }
    case kView:
      return in.size() == 1 && out.size() == 1 && in[0].t.memref && out[0].t.memref && in[0].t.same_tile(out[0].t);
    case kStore:
      return in.size() == 2 && in[0].t.same_tile(in[1].t);
    case kUpstream: {
      const Ref& name = op.name;
      if (out.size() != 1) return false;
      if (text_is(name, "arith.constant") || text_is(name, "tensor.empty") || text_is(name, "memref.alloc")) return in.empty();
      if (text_is(name, "math.exp")) return in.size() == 1;
      if (text_is(name, "arith.mulf") || text_is(name, "arith.subf") || text_is(name, "arith.divf"))
        return in.size() == 2 && in[0].t.same(in[1].t) && in[0].t.same(out[0].t);
      if (text_is(name, "arith.truncf"))
        return in.size() == 1 && in[0].t.rank == out[0].t.rank && in[0].t.e[0] == out[0].t.e[0] && in[0].t.e[1] == out[0].t.e[1] &&
               kBits[out[0].t.element] < kBits[in[0].t.element];
      if (text_is(name, "linalg.broadcast")) {  // a row statistic along dim 1
        const Ref dims = key(op.attrs, names.dimensions);
        long long d = 0;
        return in.size() == 2 && length(dims) == 1 && to_int(item(dims, 0), &d) && d == 1 && in[0].t.rank == 1 && in[1].t.rank == 2 &&
               in[0].t.e[0] == in[1].t.e[0] && in[0].t.element == in[1].t.element;
      }
      return false;
    }
    default:
      return false;
  }
}

// lists and verifies what is nested in `op`; frisk.parallel and frisk.for are what may hold other ops
bool walk(Kernel& k, const Ref& op, int depth) {
  const Ref regions = attr(op, names.regions);
  if (depth > 8 || length(regions) != 1) return false;
  const Ref blocks = attr(item(regions, 0), names.blocks);
  if (length(blocks) != 1) return false;
  const Ref block = item(blocks, 0), operations = attr(block, names.operations);
  if (depth == 0) k.entry = block;
  const Py_ssize_t n = length(operations);
  if (n < 0 || n > 256) return false;
  k.ops.reserve(k.ops.size() + n);
  for (Py_ssize_t i = 0; i < n; ++i) {
    Op x;
    x.op = item(operations, i);
    if (!x.op) return false;
    for (int c = 1; c < kClasses; ++c)
      if (is_a(x.op, classes[c])) x.cls = static_cast<Class>(c);
    if (x.cls == kOther) return false;
    const auto& at = op_at[x.cls];
    x.attrs = slot(x.op, at.attrs, names.attrs);
    if (x.cls == kUpstream) x.name = attr(x.op, names.op_name);
    const bool holds = x.cls == kParallel || x.cls == kFor;
    long long n_args = 0;
    const Ref r = slot(x.op, at.regions, names.regions);
    if (length(r) != (holds ? 1 : 0)) return false;
    if (holds) n_args = length(attr(item(attr(item(r, 0), names.blocks), 0), names.arguments));
    if (!read_values(k, slot(x.op, at.operands, names.operands), &x.in) ||
        !read_values(k, slot(x.op, at.results, names.results), &x.out))
      return false;
    if (!verify_op(x, n_args)) return false;
    const Ref self = x.op;
    k.ops.push_back(std::move(x));
    if (holds && !walk(k, self, depth + 1)) return false;
  }
  return true;
}

// The plan is read off the entry block's arguments, execute checks the tensors against the function type: the same type objects
// (others that are equal are for the Python side to compare).
bool arguments_match(const Ref& kernel, const Ref& entry) {
  const Ref inputs = attr(key(attr(kernel, names.attrs), names.function_type), names.inputs), arguments = attr(entry, names.arguments);
  const Py_ssize_t n = length(inputs);
  if (n < 0 || length(arguments) != n) return false;
  for (Py_ssize_t i = 0; i < n; ++i)
    if (attr(item(arguments, i), names.type).get() != item(inputs, i).get()) return false;
  return true;
}

// ------------------------------------------------------------------------ the attention graph
struct Graph {
  const Kernel& k;
  const Op* producer(const Value& v, Class cls, const char* name = nullptr) const {
    if (v.is_arg) return nullptr;
    for (const Op& op : k.ops)
      if (op.op.get() == v.owner.get()) return op.cls == cls && (!name || text_is(op.name, name)) ? &op : nullptr;
    return nullptr;
  }
  Value strip(Value v) const {
    for (int i = 0; i < 16; ++i) {
      const Op* view = producer(v, kView);
      if (!view) break;
      v = view->in[0];
    }
    return v;
  }
  // a global kernel argument
  bool global_arg(const Value& v) const { return v.is_arg && v.owner.get() == k.entry.get() && v.t.space == 1; }  // 1: GLOBAL
  // the global kernel argument whose data a memref operand holds, staged or not, and of the operand's extents: the kernel reads
  // those from the argument's address, and a copy's verifier does not compare the two sides
  bool root(const Value& operand, Value* out) const {
    Value v = strip(operand);
    if (producer(v, kUpstream, "memref.alloc")) {
      const Op* from = nullptr;
      for (const Op& op : k.ops)
        if (op.cls == kCopy && strip(op.in[1]).id == v.id) {
          if (from) return false;
          from = &op;
        }
      if (!from) return false;
      v = strip(from->in[0]);
    }
    if (!global_arg(v) || v.t.rank != operand.t.rank || v.t.e[0] != operand.t.e[0] || v.t.e[1] != operand.t.e[1]) return false;
    *out = v;
    return true;
  }
  bool constant(const Value& v, double* out) const {
    const Op* c = producer(v, kUpstream, "arith.constant");
    const Ref x = c ? key(c->attrs, names._value) : Ref();
    if (!x || !PyFloat_CheckExact(x.get())) return false;
    *out = PyFloat_AS_DOUBLE(x.get());
    return true;
  }
  bool zero(const Value& v) const {
    double x = 0.0;
    return constant(v, &x) && x == 0.0;
  }
  const Op* statistic(const Value& v, const char* kind) const {
    const Op* b = producer(v, kUpstream, "linalg.broadcast");
    const Op* r = b ? producer(b->in[0], kReduceTensor) : nullptr;
    long long dim = 0;
    return r && text_is(key(r->attrs, names.kind), kind) && to_int(key(r->attrs, names.dim), &dim) && dim == 1 ? r : nullptr;
  }
};

PyObject* attention(const Kernel& k) {
  const Graph g{k};
  const Op* store = nullptr;
  for (const Op& op : k.ops) {
    if (op.cls == kGemm || op.cls == kFill || op.cls == kReduce) return nullptr;
    if (op.cls == kStore) {
      if (store) return nullptr;
      store = &op;
    }
  }
  Value o, v, q, key_arg;
  if (!store) return nullptr;
  o = g.strip(store->in[1]);  // (a copy INTO a buffer does not say where the buffer's contents go)
  if (!g.global_arg(o)) return nullptr;
  const Value* result = &store->in[0];
  if (const Op* t = g.producer(*result, kUpstream, "arith.truncf")) result = &t->in[0];
  const Op* pv = g.producer(*result, kMma);
  bool ta = false, tb = false;
  if (!pv || !flag(*pv, names.trans_a, &ta) || !flag(*pv, names.trans_b, &tb) || ta || tb || !g.zero(pv->in[2]) || !g.root(pv->in[1], &v)) return nullptr;
  const Op* trunc = g.producer(pv->in[0], kUpstream, "arith.truncf");
  const Op* div = trunc ? g.producer(trunc->in[0], kUpstream, "arith.divf") : nullptr;
  const Op* e = div ? g.producer(div->in[0], kUpstream, "math.exp") : nullptr;
  const Op* sum = e ? g.statistic(div->in[1], "sum") : nullptr;
  if (!sum || sum->in[0].id != e->out[0].id) return nullptr;
  const Op* sub = g.producer(e->in[0], kUpstream, "arith.subf");
  const Op* top = sub ? g.statistic(sub->in[1], "max") : nullptr;
  if (!top || top->in[0].id != sub->in[0].id) return nullptr;
  const Op* mul = g.producer(sub->in[0], kUpstream, "arith.mulf");
  if (!mul) return nullptr;
  const bool swapped = g.producer(mul->in[0], kUpstream, "arith.constant") != nullptr;
  double scale = 0.0;
  if (!g.constant(mul->in[swapped ? 0 : 1], &scale) || !(scale > 0.0)) return nullptr;
  const Op* qk = g.producer(mul->in[swapped ? 1 : 0], kMma);
  if (!qk || !flag(*qk, names.trans_a, &ta) || !flag(*qk, names.trans_b, &tb) || ta || !tb || !g.zero(qk->in[2])) return nullptr;
  if (!g.root(qk->in[0], &q) || !g.root(qk->in[1], &key_arg)) return nullptr;
  const long long n_q = qk->out[0].t.e[0], n_kv = qk->out[0].t.e[1], d = qk->in[1].t.e[1];
  if (pv->out[0].t.e[0] != n_q || pv->out[0].t.e[1] != d || pv->in[1].t.e[0] != n_kv) return nullptr;
  const Element in = q.t.element, out = o.t.element;
  if (trunc->out[0].t.element != in || key_arg.t.element != in || v.t.element != in) return nullptr;
  if ((in != kF16 && in != kBF16) || (out != kF32 && out != in) || (d != 64 && d != 128)) return nullptr;
  return Py_BuildValue("(OLLLdiiLLLL)", Py_False, n_q, n_kv, d, scale, (int)in, (int)out, q.index, key_arg.index, v.index, o.index);
}

// ------------------------------------------------------------------------ one gemm with its fill and reduce
PyObject* fused(const Kernel& k) {
  const Op *gemm = nullptr, *fill = nullptr, *reduce = nullptr;
  for (const Op& op : k.ops) {
    switch (op.cls) {
      case kEnd:
      case kParallel:
        break;
      case kFor: {  // (one iteration each: whatever encloses the gemm runs once)
        long long lower = 0, upper = 0, step = 0;
        if (!to_int(key(op.attrs, names.lower), &lower) || !to_int(key(op.attrs, names.upper), &upper) ||
            !to_int(key(op.attrs, names.step), &step))
          return nullptr;
        if (step < 1 || lower < 0 || upper <= lower || upper - lower > step) return nullptr;
        break;
      }
      case kFill:
        if (fill || gemm) return nullptr;
        fill = &op;
        break;
      case kGemm:
        if (gemm) return nullptr;
        gemm = &op;
        break;
      case kReduce:
        if (reduce || !gemm) return nullptr;
        reduce = &op;
        break;
      default:
        return nullptr;
    }
  }
  if (!gemm) return nullptr;
  const Value& c = gemm->in[2];
  if ((fill && fill->in[0].id != c.id) || (reduce && reduce->in[0].id != c.id)) return nullptr;
  auto global_arg = [&](const Value& v) { return v.is_arg && v.owner.get() == k.entry.get() && v.t.space == 1; };
  for (size_t i = 0; i < gemm->in.size(); ++i)
    if (!global_arg(gemm->in[i])) return nullptr;
  if (reduce && !global_arg(reduce->in[1])) return nullptr;
  bool ta = false, tb = false, clear = false, reduce_clear = true;
  if (!flag(*gemm, names.transA, &ta) || !flag(*gemm, names.transB, &tb) || !flag(*gemm, names.clear_accum, &clear)) return nullptr;
  if (reduce && !flag(*reduce, names.clear, &reduce_clear)) return nullptr;
  long long policy = 0;
  if (!to_enum(key(gemm->attrs, names.policy), policy_class, &policy)) return nullptr;
  const Ref value = fill ? key(fill->attrs, names.value) : Ref();
  const Ref kind = reduce ? key(reduce->attrs, names.kind) : Ref();
  return Py_BuildValue("(OLLLiiiiiLLLLOOLi)", Py_True, c.t.e[0], c.t.e[1], gemm->in[0].t.e[ta ? 0 : 1], (int)gemm->in[0].t.element,
                       (int)c.t.element, (int)ta, (int)tb, (int)clear, policy, gemm->in[0].index, gemm->in[1].index, c.index,
                       fill ? PyTuple_GET_ITEM(value.get(), 0) : Py_None, reduce ? kind.get() : Py_None,
                       reduce ? reduce->in[1].index : -1LL, (int)reduce_clear);
}

PyObject* plan(PyObject*, PyObject* arg) {
  if (!type_class) Py_RETURN_NONE;
  try {
    Kernel k;
    k.class_has_place = PyObject_HasAttr(type_class, names.space) || PyObject_HasAttr(type_class, names.map);
    const Ref kernel(Py_NewRef(arg));
    if (walk(k, kernel, 0) && arguments_match(kernel, k.entry)) {
      bool mma = false;
      for (const Op& op : k.ops) mma = mma || op.cls == kMma;
      PyObject* out = mma ? attention(k) : fused(k);
      if (out) return out;
    }
  } catch (...) {  // (no memory: the Python recognisers report it, if it lasts)
  }
  PyErr_Clear();
  Py_RETURN_NONE;
}

// classes(type, value, AffineMap, MemorySpace, GemmWarpPolicy, [op classes in the order of Class, from EndOp])
PyObject* set_classes(PyObject*, PyObject* args) {
  PyObject *t, *v, *m, *s, *p, *ops;
  if (!PyArg_ParseTuple(args, "OOOOOO!", &t, &v, &m, &s, &p, &PyList_Type, &ops)) return nullptr;
  if (PyList_GET_SIZE(ops) != kClasses - 1) {
    PyErr_SetString(PyExc_ValueError, "recognise: wrong number of classes");
    return nullptr;
  }
  for (int i = 1; i < kClasses; ++i) {
    PyObject* c = PyList_GET_ITEM(ops, i - 1);
    op_at[i] = {slot_of(c, names.operands), slot_of(c, names.results), slot_of(c, names.attrs), slot_of(c, names.regions)};
    Py_XSETREF(classes[i], Py_NewRef(c));
  }
  value_at = {slot_of(v, names.type), slot_of(v, names.owner), slot_of(v, names.index), slot_of(v, names.is_arg)};
  Py_XSETREF(value_class, Py_NewRef(v));
  Py_XSETREF(map_class, Py_NewRef(m));
  Py_XSETREF(space_class, Py_NewRef(s));
  Py_XSETREF(policy_class, Py_NewRef(p));
  Py_XSETREF(type_class, Py_NewRef(t));
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"plan", plan, METH_O, "the plan of a usual kernel, or None"},
                         {"classes", set_classes, METH_VARARGS, "tells the module the IR's classes"},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef definition = {PyModuleDef_HEAD_INIT, "_recognise", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__recognise(void) {
#define X(n) \
  if (!(names.n = PyUnicode_InternFromString(#n))) return nullptr;
  NAMES(X)
#undef X
  return PyModule_Create(&definition);
}
