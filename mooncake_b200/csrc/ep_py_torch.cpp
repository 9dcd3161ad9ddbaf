// The Python side of a call, in native code: a CPython extension over the C ABI
// (include/mcep.h) that checks the tensors, allocates the outputs and makes the
// call in one step. The package's `Buffer` / `ElasticBuffer` wrappers and
// `ep.Buffer` are thin classes over it.
//
// Why it exists: a decode-sized layer keeps the GPU busy for 10 - 15 us, while
// the same steps written in Python (about twenty assertions, five torch.empty,
// eighteen ctypes conversions per call) took 50 us per layer of host time, so
// the host bounded every small call (DeepSeek-V3-shaped decode layer, 128
// tokens: 50.2 us per layer, of which the device was busy for 14.5).
//
// The module holds no state of its own; it calls the library through the
// addresses `bind` was given, so it always drives the same libmcep.so as the
// ctypes declarations of ep.py.
#define PY_SSIZE_T_CLEAN
#include <array>
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <structmember.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <string>
#include <vector>

#include "mcep.h"

namespace {

// ---- the library ---------------------------------------------------------------------
struct Library {
    decltype(&mcep_last_error) last_error;
    decltype(&mcep_dispatch) dispatch;
    decltype(&mcep_combine) combine;
    decltype(&mcep_elastic_dispatch) elastic_dispatch;
    decltype(&mcep_elastic_dispatch_counted) elastic_dispatch_counted;
    decltype(&mcep_elastic_combine) elastic_combine;
    decltype(&mcep_buffer_next_recv_x) next_recv_x;
    decltype(&mcep_event_create) event_create;
    decltype(&mcep_event_current_stream_wait) event_wait;
    decltype(&mcep_event_synchronize) event_synchronize;
    decltype(&mcep_event_free) event_free;
    decltype(&mcep_hook_run) hook_run;
    decltype(&mcep_hook_free) hook_free;
} lib;

const char* const kSymbols[] = {"mcep_last_error", "mcep_dispatch", "mcep_combine", "mcep_elastic_dispatch",
                                "mcep_elastic_dispatch_counted", "mcep_elastic_combine", "mcep_buffer_next_recv_x", "mcep_event_create",
                                "mcep_event_current_stream_wait", "mcep_event_synchronize", "mcep_event_free",
                                "mcep_hook_run", "mcep_hook_free"};
constexpr size_t kNumSymbols = sizeof(kSymbols) / sizeof(kSymbols[0]);
static_assert(sizeof(Library) == kNumSymbols * sizeof(void*), "one address per name");

PyObject* fail() {
    PyErr_SetString(PyExc_RuntimeError, lib.last_error());
    return nullptr;
}

// bind({name: address}): where the entry points of the loaded libmcep.so are.
PyObject* py_bind(PyObject*, PyObject* table) {
    void** slots = reinterpret_cast<void**>(&lib);
    for (size_t i = 0; i < kNumSymbols; ++i) {
        PyObject* v = PyDict_GetItemString(table, kSymbols[i]);
        if (v == nullptr) return PyErr_Format(PyExc_KeyError, "%s", kSymbols[i]);
        slots[i] = PyLong_AsVoidPtr(v);
        if (PyErr_Occurred()) return nullptr;
    }
    Py_RETURN_NONE;
}

#define MCEP_FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn))

// ---- arguments -----------------------------------------------------------------------
// Positional and keyword arguments of a call into `out[0..n)` (borrowed; null = not given).
bool collect(const char* const* names, int n, int required, PyObject* const* args, Py_ssize_t nargs,
             PyObject* kwnames, PyObject** out, const char* fname) {
    if (nargs > n) {
        PyErr_Format(PyExc_TypeError, "%s() takes %d arguments (%zd given)", fname, n, nargs);
        return false;
    }
    for (Py_ssize_t i = 0; i < n; ++i) out[i] = i < nargs ? args[i] : nullptr;
    const Py_ssize_t nk = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    for (Py_ssize_t j = 0; j < nk; ++j) {
        PyObject* key = PyTuple_GET_ITEM(kwnames, j);
        int at = -1;
        for (int i = 0; i < n && at < 0; ++i)
            if (PyUnicode_CompareWithASCIIString(key, names[i]) == 0) at = i;
        if (at < 0 || out[at] != nullptr) {
            PyErr_Format(PyExc_TypeError, "%s() got an unexpected or repeated keyword argument '%U'", fname, key);
            return false;
        }
        out[at] = args[nargs + j];
    }
    for (int i = 0; i < required; ++i)
        if (out[i] == nullptr) {
            PyErr_Format(PyExc_TypeError, "%s() missing required argument: '%s'", fname, names[i]);
            return false;
        }
    return true;
}

// Reads integers, addresses and truth values; the first failure sticks.
struct Reader {
    PyObject** v;
    bool ok = true;
    long long num(int i) {
        const long long r = PyLong_AsLongLong(v[i]);
        if (r == -1 && PyErr_Occurred()) ok = false;
        return r;
    }
    int i32(int i) { return (int)num(i); }
    int flag(int i) {
        if (v[i] == Py_None) PyErr_SetString(PyExc_TypeError, "a truth value is wanted, not None");
        const int r = v[i] == Py_None ? -1 : PyObject_IsTrue(v[i]);
        if (r < 0) ok = false;
        return r > 0;
    }
    void* ptr(int i) {
        if (v[i] == Py_None) return nullptr;
        void* r = PyLong_AsVoidPtr(v[i]);
        if (r == nullptr && PyErr_Occurred()) ok = false;
        return r;
    }
};

// ---- events and hooks ------------------------------------------------------------------
struct EventObject {
    PyObject_HEAD
    mcep_event* ev;
};
PyTypeObject* event_type = nullptr;

PyObject* wrap_event(mcep_event* ev) {
    if (ev == nullptr) Py_RETURN_NONE;
    EventObject* o = PyObject_New(EventObject, event_type);
    if (o == nullptr) {
        lib.event_free(ev);
        return nullptr;
    }
    o->ev = ev;
    return reinterpret_cast<PyObject*>(o);
}

PyObject* event_new(PyTypeObject* type, PyObject* args, PyObject* kw) {
    static const char* names[] = {"stream_ptr", nullptr};
    unsigned long long stream = 0;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "|K", const_cast<char**>(names), &stream)) return nullptr;
    mcep_event* ev = nullptr;
    if (lib.event_create(stream, &ev)) return fail();
    EventObject* o = reinterpret_cast<EventObject*>(type->tp_alloc(type, 0));
    if (o == nullptr) {
        lib.event_free(ev);
        return nullptr;
    }
    o->ev = ev;
    return reinterpret_cast<PyObject*>(o);
}

void event_dealloc(PyObject* self) {
    PyTypeObject* type = Py_TYPE(self);
    lib.event_free(reinterpret_cast<EventObject*>(self)->ev);
    type->tp_free(self);
    Py_DECREF(type);
}

PyObject* event_stream_wait(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    static const char* const names[] = {"stream_ptr"};
    PyObject* stream;
    if (!collect(names, 1, 1, args, nargs, kwnames, &stream, "current_stream_wait")) return nullptr;
    const unsigned long long s = PyLong_AsUnsignedLongLong(stream);
    if (PyErr_Occurred()) return nullptr;
    if (lib.event_wait(reinterpret_cast<EventObject*>(self)->ev, s)) return fail();
    Py_RETURN_NONE;
}

PyObject* event_sync(PyObject* self, PyObject*) {
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = lib.event_synchronize(reinterpret_cast<EventObject*>(self)->ev);
    Py_END_ALLOW_THREADS if (rc) return fail();
    Py_RETURN_NONE;
}

PyMethodDef event_methods[] = {
    {"current_stream_wait", MCEP_FAST(event_stream_wait), METH_FASTCALL | METH_KEYWORDS,
     "current_stream_wait($self, stream_ptr)\n--\n\nMake the stream (a cudaStream_t as an integer) wait."},
    {"synchronize", event_sync, METH_NOARGS, "Wait for the event on the host."},
    {nullptr, nullptr, 0, nullptr}};
PyType_Slot event_slots[] = {
    {Py_tp_doc, const_cast<char*>("mooncake-ep/include/mooncake_ep_event.h:9-44: a CUDA event recorded on\n"
                                  "`stream_ptr` at construction.")},
    {Py_tp_new, reinterpret_cast<void*>(event_new)},
    {Py_tp_dealloc, reinterpret_cast<void*>(event_dealloc)},
    {Py_tp_methods, event_methods},
    {0, nullptr}};
PyType_Spec event_spec = {"mooncake_b200._mcep_torch.EventHandle", sizeof(EventObject), 0,
                          Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE, event_slots};

// The state of `EventOverlap` (mooncake_ep_buffer.py derives from it): an event and the
// tensors that must outlive it.
struct OverlapObject {
    PyObject_HEAD
    PyObject* event;
    PyObject* extra_tensors;
};
PyTypeObject* overlap_type = nullptr;  // the derived class once it has been registered

int overlap_init(PyObject* self, PyObject* args, PyObject* kw) {
    static const char* names[] = {"event", "extra_tensors", nullptr};
    PyObject *event = Py_None, *extra = Py_None;
    if (!PyArg_ParseTupleAndKeywords(args, kw, "|OO", const_cast<char**>(names), &event, &extra)) return -1;
    OverlapObject* o = reinterpret_cast<OverlapObject*>(self);
    Py_INCREF(event), Py_INCREF(extra);
    Py_XSETREF(o->event, event);
    Py_XSETREF(o->extra_tensors, extra);
    return 0;
}
int overlap_traverse(PyObject* self, visitproc visit, void* arg) {
    OverlapObject* o = reinterpret_cast<OverlapObject*>(self);
    Py_VISIT(o->event);
    Py_VISIT(o->extra_tensors);
    Py_VISIT(Py_TYPE(self));
    return 0;
}
int overlap_clear(PyObject* self) {
    OverlapObject* o = reinterpret_cast<OverlapObject*>(self);
    Py_CLEAR(o->event);
    Py_CLEAR(o->extra_tensors);
    return 0;
}
void overlap_dealloc(PyObject* self) {
    PyTypeObject* type = Py_TYPE(self);
    PyObject_GC_UnTrack(self);
    overlap_clear(self);
    type->tp_free(self);
    Py_DECREF(type);
}
PyMemberDef overlap_members[] = {
    {"event", T_OBJECT, offsetof(OverlapObject, event), 0, nullptr},
    {"extra_tensors", T_OBJECT, offsetof(OverlapObject, extra_tensors), 0, nullptr},
    {nullptr, 0, 0, 0, nullptr}};
PyType_Slot overlap_slots[] = {
    {Py_tp_doc, const_cast<char*>("An event plus the tensors that must outlive it.")},
    {Py_tp_new, reinterpret_cast<void*>(PyType_GenericNew)},
    {Py_tp_init, reinterpret_cast<void*>(overlap_init)},
    {Py_tp_traverse, reinterpret_cast<void*>(overlap_traverse)},
    {Py_tp_clear, reinterpret_cast<void*>(overlap_clear)},
    {Py_tp_dealloc, reinterpret_cast<void*>(overlap_dealloc)},
    {Py_tp_members, overlap_members},
    {0, nullptr}};
PyType_Spec overlap_spec = {"mooncake_b200._mcep_torch.EventOverlapBase", sizeof(OverlapObject), 0,
                            Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC, overlap_slots};

// Takes over the references of both; null if one of them is.
PyObject* wrap_overlap(PyObject* event, PyObject* extra) {
    PyObject* self = event && extra ? overlap_type->tp_alloc(overlap_type, 0) : nullptr;
    if (self == nullptr) {
        Py_XDECREF(event);
        Py_XDECREF(extra);
        return nullptr;
    }
    reinterpret_cast<OverlapObject*>(self)->event = event;
    reinterpret_cast<OverlapObject*>(self)->extra_tensors = extra;
    return self;
}

PyObject* py_register_overlap(PyObject*, PyObject* cls) {
    PyTypeObject* base = overlap_type;
    while (base->tp_base != nullptr && base->tp_base != &PyBaseObject_Type) base = base->tp_base;
    if (!PyType_Check(cls) || !PyType_IsSubtype(reinterpret_cast<PyTypeObject*>(cls), base))
        return PyErr_Format(PyExc_TypeError, "a class derived from EventOverlapBase is wanted");
    Py_INCREF(cls);
    overlap_type = reinterpret_cast<PyTypeObject*>(cls);
    Py_RETURN_NONE;
}

// ---- EPHandle ---------------------------------------------------------------------------
const char* const kHandleNames[] = {
    "do_expand", "num_experts", "expert_alignment", "num_max_tokens_per_rank", "num_sms", "topk_idx",
    "psum_num_recv_tokens_per_scaleup_rank", "psum_num_recv_tokens_per_expert", "num_recv_tokens_per_expert_list",
    "recv_src_metadata", "dst_buffer_slot_idx", "token_metadata_at_forward", "channel_linked_list", "native_handle",
    "num_recv_tokens"};
constexpr size_t kHandleFields = sizeof(kHandleNames) / sizeof(kHandleNames[0]);
PyObject* handle_names[kHandleFields];
PyTypeObject* handle_type = nullptr;

PyObject* py_register_handle(PyObject*, PyObject* cls) {
    if (!PyType_Check(cls)) return PyErr_Format(PyExc_TypeError, "a class is wanted");
    for (size_t i = 0; i < kHandleFields; ++i)
        if (handle_names[i] == nullptr && (handle_names[i] = PyUnicode_InternFromString(kHandleNames[i])) == nullptr)
            return nullptr;
    Py_INCREF(cls);
    handle_type = reinterpret_cast<PyTypeObject*>(cls);
    Py_RETURN_NONE;
}

// A handle made of all its fields, whose references are taken over (null: an error is set).
PyObject* wrap_handle(const std::array<PyObject*, kHandleFields>& fields) {
    PyObject* dict = PyDict_New();
    bool ok = dict != nullptr;
    for (size_t i = 0; i < kHandleFields; ++i) {
        ok = ok && fields[i] != nullptr && PyDict_SetItem(dict, handle_names[i], fields[i]) == 0;
        Py_XDECREF(fields[i]);
    }
    PyObject* none = ok ? PyTuple_New(0) : nullptr;
    PyObject* self = none ? handle_type->tp_new(handle_type, none, nullptr) : nullptr;
    Py_XDECREF(none);
    if (self != nullptr && PyObject_GenericSetDict(self, dict, nullptr) != 0) Py_CLEAR(self);
    Py_XDECREF(dict);
    return self;
}

struct HookObject {
    PyObject_HEAD
    mcep_hook* hook;
};
PyTypeObject* hook_type = nullptr;

PyObject* wrap_hook(mcep_hook* hook) {
    if (hook == nullptr) Py_RETURN_NONE;
    HookObject* o = PyObject_New(HookObject, hook_type);
    if (o == nullptr) {
        lib.hook_free(hook);
        return nullptr;
    }
    o->hook = hook;
    return reinterpret_cast<PyObject*>(o);
}

void hook_dealloc(PyObject* self) {
    PyTypeObject* type = Py_TYPE(self);
    lib.hook_free(reinterpret_cast<HookObject*>(self)->hook);
    type->tp_free(self);
    Py_DECREF(type);
}

PyObject* hook_call(PyObject* self, PyObject* args, PyObject* kw) {
    if (PyTuple_GET_SIZE(args) != 0 || (kw != nullptr && PyDict_GET_SIZE(kw) != 0))
        return PyErr_Format(PyExc_TypeError, "the receive hook takes no arguments");
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = lib.hook_run(reinterpret_cast<HookObject*>(self)->hook);
    Py_END_ALLOW_THREADS if (rc) return fail();
    Py_RETURN_NONE;
}

PyType_Slot hook_slots[] = {
    {Py_tp_doc, const_cast<char*>("The receive-phase callback (the `std::function<void()>` of the reference).")},
    {Py_tp_dealloc, reinterpret_cast<void*>(hook_dealloc)},
    {Py_tp_call, reinterpret_cast<void*>(hook_call)},
    {0, nullptr}};
PyType_Spec hook_spec = {"mooncake_b200._mcep_torch.Hook", sizeof(HookObject), 0,
                         Py_TPFLAGS_DEFAULT | Py_TPFLAGS_DISALLOW_INSTANTIATION, hook_slots};

// ---- tensors -------------------------------------------------------------------------
const at::Tensor* tensor_of(PyObject* o) { return o && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// The device can read and write it where it is: its own memory, or pinned host memory.
bool reachable(const at::Tensor* t) { return t->is_cuda() || (t->is_cpu() && t->is_pinned()); }

bool matrix(const at::Tensor* t, at::ScalarType type) {
    return t && reachable(t) && t->dim() == 2 && t->scalar_type() == type && t->is_contiguous();
}
// At least `n` entries in a row, whatever the tensor's shape.
bool entries(const at::Tensor* t, at::ScalarType type, int64_t n) {
    return t && reachable(t) && t->scalar_type() == type && t->is_contiguous() && t->numel() >= n;
}
bool usable_mask(const at::Tensor* t, int64_t ranks) {
    return t && reachable(t) && t->dim() == 1 && t->numel() == ranks && t->scalar_type() == at::kInt && t->is_contiguous();
}

// torch.empty without the way through the tensor factory (0.2 us per tensor), except where
// torch has been asked to fill what is not initialised.
at::Tensor empty(at::IntArrayRef size, at::ScalarType type, at::Device dev) {
    const at::Context& context = at::globalContext();
    if (context.deterministicAlgorithms() && context.deterministicFillUninitializedMemory())
        return at::empty(size, at::TensorOptions(type).device(dev));
    if (c10::cuda::current_device() != dev.index()) return at::detail::empty_cuda(size, type, dev, std::nullopt);
    const auto meta = c10::scalarTypeToTypeMeta(type);
    size_t bytes = meta.itemsize();
    for (const int64_t n : size) {
        TORCH_CHECK(n >= 0, "negative size");
        bytes *= (size_t)n;
    }
    c10::Allocator* allocator = c10::cuda::CUDACachingAllocator::get();
    c10::Storage storage(c10::Storage::use_byte_size_t(), bytes, allocator->allocate(bytes), allocator, true);
    at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(std::move(storage), c10::DispatchKeySet(c10::DispatchKey::CUDA), meta);
    t.unsafeGetTensorImpl()->set_sizes_contiguous(size);
    return t;
}

// Several small output tensors cut out of one allocation: the caching allocator
// is asked once (an allocation costs about as much as everything else that has
// to be done for a small tensor).
class Arena {
public:
    explicit Arena(at::Device dev) : dev_(dev) {}
    int64_t reserve(int64_t bytes) {
        const int64_t at = size_;
        size_ += (bytes + 255) / 256 * 256;
        return at;
    }
    void allocate() {
        base_ = empty({size_ ? size_ : 1}, at::kByte, dev_);
        data_ = static_cast<char*>(base_.data_ptr());
    }
    char* at(int64_t offset) const { return data_ + offset; }
    at::Tensor view(int64_t offset, at::ScalarType type, at::IntArrayRef size) const {
        const auto meta = c10::scalarTypeToTypeMeta(type);
        at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(base_.storage()), base_.key_set(), meta);
        t.unsafeGetTensorImpl()->set_storage_offset(offset / (int64_t)meta.itemsize());
        t.unsafeGetTensorImpl()->set_sizes_contiguous(size);
        return t;
    }

private:
    at::Device dev_;
    int64_t size_ = 0;
    at::Tensor base_;
    char* data_ = nullptr;
};

constexpr int64_t kScalesInArena = 32 << 20;

PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

// A new tuple that takes over the references of `items`; null if any is null.
PyObject* pack(std::initializer_list<PyObject*> items) {
    bool ok = true;
    for (PyObject* o : items) ok = ok && o != nullptr;
    PyObject* t = ok ? PyTuple_New((Py_ssize_t)items.size()) : nullptr;
    if (t == nullptr) {
        for (PyObject* o : items) Py_XDECREF(o);
        return nullptr;
    }
    Py_ssize_t i = 0;
    for (PyObject* o : items) PyTuple_SET_ITEM(t, i++, o);
    return t;
}

PyObject* new_ref(PyObject* o) {
    Py_INCREF(o);
    return o;
}

uint64_t current_stream() { return reinterpret_cast<uint64_t>(c10::cuda::getCurrentCUDAStream().stream()); }

PyObject* py_current_stream(PyObject*, PyObject*) {
    HANDLE_TH_ERRORS  // (no device, no driver)
    return PyLong_FromUnsignedLongLong(current_stream());
    END_HANDLE_TH_ERRORS
}

// ---- the runtime object -----------------------------------------------------------------
struct RuntimeObject {
    PyObject_HEAD
    mcep_buffer* buf;
    int num_ranks;
};

RuntimeObject* self_of(PyObject* o) { return reinterpret_cast<RuntimeObject*>(o); }

bool alive(RuntimeObject* s) {
    if (s->buf != nullptr) return true;
    PyErr_SetString(PyExc_RuntimeError, "the buffer has been destroyed");
    return false;
}

PyObject* runtime_adopt(PyObject* self, PyObject* args) {
    PyObject* h;
    int ranks;
    if (!PyArg_ParseTuple(args, "Oi", &h, &ranks)) return nullptr;
    self_of(self)->buf = h == Py_None ? nullptr : static_cast<mcep_buffer*>(PyLong_AsVoidPtr(h));
    self_of(self)->num_ranks = ranks;
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

int call_dispatch(mcep_buffer* b, const mcep_dispatch_args* a, mcep_event** ev, mcep_hook** hk) {
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = lib.dispatch(b, a, ev, hk);
    Py_END_ALLOW_THREADS return rc;
}
int call_combine(mcep_buffer* b, const mcep_combine_args* a, mcep_event** ev, mcep_hook** hk) {
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = lib.combine(b, a, ev, hk);
    Py_END_ALLOW_THREADS return rc;
}

const char* const kDispatchNames[] = {
    "x_ptr", "topk_idx_ptr", "active_ranks_ptr", "num_tokens", "hidden", "num_topk",
    "num_max_dispatch_tokens_per_rank", "num_experts", "timeout_us", "use_fp8", "packed_recv_x_ptr",
    "packed_recv_x_scales_ptr", "packed_recv_count_ptr", "packed_recv_src_info_ptr",
    "packed_recv_layout_range_ptr", "async_finish", "return_recv_hook", "compute_stream_ptr"};

PyObject* runtime_dispatch(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    PyObject* v[18];
    if (!collect(kDispatchNames, 18, 18, args, nargs, kwnames, v, "dispatch") || !alive(self_of(self))) return nullptr;
    Reader r{v};
    mcep_dispatch_args a = {};
    a.x = r.ptr(0), a.topk_idx = static_cast<int64_t*>(r.ptr(1)), a.active_ranks = static_cast<int32_t*>(r.ptr(2));
    a.num_tokens = r.i32(3), a.hidden = r.i32(4), a.num_topk = r.i32(5);
    a.num_max_dispatch_tokens_per_rank = r.i32(6), a.num_experts = r.i32(7), a.timeout_us = r.num(8);
    a.use_fp8 = r.flag(9), a.packed_recv_x = r.ptr(10), a.packed_recv_x_scales = static_cast<float*>(r.ptr(11));
    a.packed_recv_count = static_cast<int32_t*>(r.ptr(12)), a.packed_recv_src_info = static_cast<int32_t*>(r.ptr(13));
    a.packed_recv_layout_range = static_cast<int64_t*>(r.ptr(14));
    a.async_finish = r.flag(15), a.return_recv_hook = r.flag(16);
    a.compute_stream = (uint64_t)r.num(17);
    if (!r.ok) return nullptr;
    mcep_event* ev = nullptr;
    mcep_hook* hk = nullptr;
    if (call_dispatch(self_of(self)->buf, &a, &ev, &hk)) return fail();
    return pack({wrap_event(ev), wrap_hook(hk)});
}

const char* const kCombineNames[] = {
    "x_ptr", "topk_idx_ptr", "topk_weights_ptr", "src_info_ptr", "layout_range_ptr", "active_ranks_ptr",
    "num_local_experts", "num_combined_tokens", "hidden", "num_topk", "num_max_dispatch_tokens_per_rank",
    "num_experts", "timeout_us", "zero_copy", "combined_x_ptr", "async_finish", "return_recv_hook",
    "compute_stream_ptr"};

PyObject* runtime_combine(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    PyObject* v[18];
    if (!collect(kCombineNames, 18, 18, args, nargs, kwnames, v, "combine") || !alive(self_of(self))) return nullptr;
    Reader r{v};
    mcep_combine_args a = {};
    a.x = r.ptr(0), a.topk_idx = static_cast<int64_t*>(r.ptr(1)), a.topk_weights = static_cast<float*>(r.ptr(2));
    a.src_info = static_cast<int32_t*>(r.ptr(3)), a.layout_range = static_cast<int64_t*>(r.ptr(4));
    a.active_ranks = static_cast<int32_t*>(r.ptr(5)), a.num_local_experts = r.i32(6);
    a.num_combined_tokens = r.i32(7), a.hidden = r.i32(8), a.num_topk = r.i32(9);
    a.num_max_dispatch_tokens_per_rank = r.i32(10), a.num_experts = r.i32(11), a.timeout_us = r.num(12);
    a.zero_copy = r.flag(13), a.combined_x = r.ptr(14), a.async_finish = r.flag(15), a.return_recv_hook = r.flag(16);
    a.compute_stream = (uint64_t)r.num(17);
    if (!r.ok) return nullptr;
    mcep_event* ev = nullptr;
    mcep_hook* hk = nullptr;
    if (call_combine(self_of(self)->buf, &a, &ev, &hk)) return fail();
    return pack({wrap_event(ev), wrap_hook(hk)});
}

// next_recv_x(M, hidden, num_experts, use_fp8) -> (pointer, bytes)
PyObject* runtime_next_recv_x(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    static const char* const names[] = {"num_max_dispatch_tokens_per_rank", "hidden", "num_experts", "use_fp8"};
    PyObject* v[4];
    if (!collect(names, 4, 4, args, nargs, kwnames, v, "next_recv_x") || !alive(self_of(self))) return nullptr;
    Reader r{v};
    const int M = r.i32(0), H = r.i32(1), E = r.i32(2), fp8 = r.flag(3);
    if (!r.ok) return nullptr;
    void* p = nullptr;
    size_t n = 0;
    if (lib.next_recv_x(self_of(self)->buf, M, H, E, fp8, &p, &n)) return fail();
    return pack({PyLong_FromVoidPtr(p), PyLong_FromSize_t(n)});
}

// dispatch_tensors(x, topk_idx, active_ranks, M, E, timeout_us, use_fp8, async_finish,
//                  return_recv_hook, in_place or None)
// `in_place`(pointer, bytes, L, R*M, H, use_fp8, x) makes the tensor over the symmetric memory in
// which a group's rows land; without it, or for a single rank, the rows get a tensor of their own.
//   -> what Buffer.dispatch returns: (recv_x or (recv_x, scales), recv_count,
//       (src_info, layout_range, M, H, E), EventOverlap, hook or None),
// or None when an argument is not what the call takes (the wrapper then says which).
PyObject* runtime_dispatch_tensors(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    RuntimeObject* s = self_of(self);
    if (nargs != 10) return PyErr_Format(PyExc_TypeError, "dispatch_tensors() takes 10 arguments");
    if (!alive(s)) return nullptr;
    Reader r{const_cast<PyObject**>(args)};
    const at::Tensor *x = tensor_of(args[0]), *idx = tensor_of(args[1]), *active = tensor_of(args[2]);
    const int64_t M = r.num(3), E = r.num(4), timeout = r.num(5), R = s->num_ranks;
    const int fp8 = r.flag(6), async = r.flag(7), hooked = r.flag(8);
    if (!r.ok) return nullptr;
    if (!matrix(x, at::kBFloat16) || !x->is_cuda() || !matrix(idx, at::kLong) || !usable_mask(active, R)) Py_RETURN_NONE;
    const int64_t T = x->size(0), H = x->size(1), K = idx->size(1), RM = R * M;
    if (idx->size(0) != T || T > M || H % 128 != 0 || E < 0 || E % R != 0 || (fp8 && RM % 4 != 0)) Py_RETURN_NONE;
    const int64_t L = E / R;
    const at::Device dev = x->device();
    at::Tensor recv_x;
    PyObject* rows = nullptr;
    if (args[9] != Py_None) {
        void* p = nullptr;
        size_t n = 0;
        if (lib.next_recv_x(s->buf, (int)M, (int)H, (int)E, fp8, &p, &n)) return fail();
        if (p != nullptr) {
            rows = PyObject_CallFunction(args[9], "KKLLLOO", (unsigned long long)reinterpret_cast<uintptr_t>(p),
                                         (unsigned long long)n, (long long)L, (long long)RM, (long long)H,
                                         fp8 ? Py_True : Py_False, args[0]);
            if (rows == nullptr) return nullptr;
            recv_x = *tensor_of(rows);
        }
    }
    if (rows == nullptr) recv_x = empty({L, RM, H}, fp8 ? at::kFloat8_e4m3fn : at::kBFloat16, dev);
    Arena small(dev);
    const int64_t o_count = small.reserve(L * 4), o_range = small.reserve(L * R * 8), o_src = small.reserve(L * RM * 4);
    // The scales, too, while they are small (a thirtieth of the rows): the handle then
    // keeps their memory until combine. Larger ones are freed with their tensor.
    const bool scales_inside = fp8 && L * H / 128 * RM * 4 <= kScalesInArena;
    const int64_t o_scales = scales_inside ? small.reserve(L * H / 128 * RM * 4) : 0;
    small.allocate();
    at::Tensor scales;
    if (fp8) {  // [L, H/128, R*M] storage seen as [L, R*M, H/128]
        scales = scales_inside ? small.view(o_scales, at::kFloat, {L, H / 128, RM}) : empty({L, H / 128, RM}, at::kFloat, dev);
        const int64_t sizes[3] = {L, RM, H / 128}, strides[3] = {H / 128 * RM, 1, RM};
        scales.unsafeGetTensorImpl()->set_sizes_and_strides(at::IntArrayRef(sizes), at::IntArrayRef(strides));
    }
    mcep_dispatch_args a = {};
    a.x = x->const_data_ptr(), a.topk_idx = static_cast<const int64_t*>(idx->const_data_ptr());
    a.active_ranks = static_cast<int32_t*>(active->data_ptr());
    a.num_tokens = (int)T, a.hidden = (int)H, a.num_topk = (int)K;
    a.num_max_dispatch_tokens_per_rank = (int)M, a.num_experts = (int)E, a.use_fp8 = fp8, a.timeout_us = timeout;
    a.packed_recv_x = recv_x.data_ptr();
    a.packed_recv_x_scales = fp8 ? static_cast<float*>(scales.data_ptr()) : nullptr;
    a.packed_recv_count = reinterpret_cast<int32_t*>(small.at(o_count));
    a.packed_recv_layout_range = reinterpret_cast<int64_t*>(small.at(o_range));
    a.packed_recv_src_info = reinterpret_cast<int32_t*>(small.at(o_src));
    a.async_finish = async, a.return_recv_hook = hooked, a.compute_stream = current_stream();
    mcep_event* ev = nullptr;
    mcep_hook* hk = nullptr;
    if (call_dispatch(s->buf, &a, &ev, &hk)) {
        Py_XDECREF(rows);
        return fail();
    }
    PyObject* p_rows = rows ? rows : wrap(std::move(recv_x));
    PyObject* p_scales = fp8 ? wrap(std::move(scales)) : new_ref(Py_None);
    PyObject* p_count = wrap(small.view(o_count, at::kInt, {L}));
    PyObject* p_src = wrap(small.view(o_src, at::kInt, {L, RM}));
    PyObject* p_range = wrap(small.view(o_range, at::kLong, {L, R}));
    PyObject* keep = Py_None;
    if (async) {
        keep = PyTuple_Pack(7, args[0], args[1], p_rows, p_scales, p_count, p_src, p_range);
    } else {
        Py_INCREF(keep);
    }
    PyObject* handle = pack({p_src, p_range, new_ref(args[3]), PyLong_FromLongLong(H), new_ref(args[4])});
    PyObject* got = p_rows;
    if (fp8) {
        got = pack({p_rows, p_scales});
    } else {
        Py_DECREF(p_scales);
    }
    return pack({got, p_count, handle, wrap_overlap(wrap_event(ev), keep), wrap_hook(hk)});
    END_HANDLE_TH_ERRORS
}

// combine_tensors(x, topk_idx, topk_weights, active_ranks, timeout_us, handle, zero_copy,
//                 async_finish, return_recv_hook, out or None)
//   -> what Buffer.combine returns: (combined_x, EventOverlap, hook or None), or None (as above)
PyObject* runtime_combine_tensors(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    RuntimeObject* s = self_of(self);
    if (nargs != 10) return PyErr_Format(PyExc_TypeError, "combine_tensors() takes 10 arguments");
    if (!alive(s)) return nullptr;
    if (!PyTuple_Check(args[5]) || PyTuple_GET_SIZE(args[5]) != 5) Py_RETURN_NONE;
    PyObject* const* h = &PyTuple_GET_ITEM(args[5], 0);  // (src_info, layout_range, M, H, E)
    Reader r{const_cast<PyObject**>(args)}, hr{const_cast<PyObject**>(h)};
    const at::Tensor *x = tensor_of(args[0]), *idx = tensor_of(args[1]), *w = tensor_of(args[2]);
    const at::Tensor *active = tensor_of(args[3]), *src = tensor_of(h[0]), *range = tensor_of(h[1]);
    const int64_t timeout = r.num(4), M = hr.num(2), H = hr.num(3), E = hr.num(4), R = s->num_ranks;
    const int zero_copy = r.flag(6), async = r.flag(7), hooked = r.flag(8);
    if (!hr.ok) return nullptr;
    if (!r.ok) return nullptr;
    // (without `out` the result is where x is; with zero copy a group looks only at x's shape)
    const bool own_out = args[9] != Py_None;
    if (!(x && (x->is_cuda() || (own_out && ((zero_copy && R > 1) || reachable(x)))) && x->dim() == 3 &&
          x->scalar_type() == at::kBFloat16 && x->is_contiguous()) ||
        !matrix(idx, at::kLong) || !matrix(w, at::kFloat) || !usable_mask(active, R) || !matrix(src, at::kInt) ||
        !matrix(range, at::kLong) || E <= 0 || E % R != 0)
        Py_RETURN_NONE;
    const int64_t L = E / R, T = w->size(0), K = w->size(1);
    if (x->size(0) != L || x->size(1) != R * M || x->size(2) != H || H % 128 != 0 || idx->size(0) != T ||
        idx->size(1) != K || T > M || src->size(0) != L || range->size(0) != L || range->size(1) != R)
        Py_RETURN_NONE;
    const at::Tensor* given = tensor_of(args[9]);
    if (own_out && (!matrix(given, at::kBFloat16) || given->size(0) != T || given->size(1) != H))
        Py_RETURN_NONE;
    at::Tensor out = given ? *given : empty({T, H}, at::kBFloat16, x->device());
    mcep_combine_args a = {};
    a.x = x->const_data_ptr(), a.topk_idx = static_cast<const int64_t*>(idx->const_data_ptr());
    a.topk_weights = static_cast<const float*>(w->const_data_ptr());
    a.src_info = static_cast<const int32_t*>(src->const_data_ptr());
    a.layout_range = static_cast<const int64_t*>(range->const_data_ptr());
    a.active_ranks = static_cast<int32_t*>(active->data_ptr());
    a.num_local_experts = (int)L, a.num_combined_tokens = (int)T, a.hidden = (int)H, a.num_topk = (int)K;
    a.num_max_dispatch_tokens_per_rank = (int)M, a.num_experts = (int)E, a.timeout_us = timeout;
    a.zero_copy = zero_copy, a.combined_x = out.data_ptr(), a.async_finish = async, a.return_recv_hook = hooked;
    a.compute_stream = current_stream();
    mcep_event* ev = nullptr;
    mcep_hook* hk = nullptr;
    if (call_combine(s->buf, &a, &ev, &hk)) return fail();
    PyObject* p_out = given ? new_ref(args[9]) : wrap(std::move(out));
    PyObject* keep = Py_None;
    if (async) {
        keep = PyTuple_Pack(6, args[0], args[1], args[2], h[0], h[1], p_out);
    } else {
        Py_INCREF(keep);
    }
    return pack({p_out, wrap_overlap(wrap_event(ev), keep), wrap_hook(hk)});
    END_HANDLE_TH_ERRORS
}

// elastic_dispatch_tensors(x, topk_idx, topk_weights or None, active_ranks, kept_idx or None, E, M,
//                          alignment, do_expand, do_cpu_sync, timeout_us, async, in_place or None, num_sms)
//   -> what ElasticBuffer.dispatch returns: (recv_x, recv_topk_idx, recv_topk_weights or None, EPHandle,
//       EventOverlap), or None (as above)
// `kept_idx`: the cached handle's routing (topk_idx is then that tensor); None: a copy is made.
// psum_expert is [L + 1] with do_expand and its entries 1.. without, as the wrapper hands it out;
// With do_cpu_sync the handle has the list of tokens per local expert, and the row tensors are cut to length.
PyObject* runtime_elastic_dispatch_tensors(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    RuntimeObject* s = self_of(self);
    if (nargs != 14) return PyErr_Format(PyExc_TypeError, "elastic_dispatch_tensors() takes 14 arguments");
    if (!alive(s)) return nullptr;
    Reader r{const_cast<PyObject**>(args)};
    const at::Tensor *x = tensor_of(args[0]), *idx = tensor_of(args[1]), *w = tensor_of(args[2]);
    const at::Tensor *active = tensor_of(args[3]), *cached = tensor_of(args[4]);
    const int64_t E = r.num(5), M = r.num(6), alignment = r.num(7), timeout = r.num(10), R = s->num_ranks;
    const int expand = r.flag(8), sync = r.flag(9), async = r.flag(11);
    if (!r.ok) return nullptr;
    if (!matrix(x, at::kBFloat16) || !x->is_cuda() || !idx || idx->dim() < 2 || !usable_mask(active, R) || M < 0 ||
        R < 1 || E < 0)
        Py_RETURN_NONE;
    const int64_t T = x->size(0), H = x->size(1), K = idx->size(1), L = E / R;
    // [T][K] entries of each are read; their shapes beyond that are the caller's
    if (!entries(idx, at::kLong, T * K) || (args[2] != Py_None && !entries(w, at::kFloat, T * K))) Py_RETURN_NONE;
    const int64_t n_cap = M * R, out_cap = expand ? n_cap * K : n_cap;
    const at::Device dev = x->device();

    at::Tensor recv_x;
    if (args[12] != Py_None && !expand) {
        void* p = nullptr;
        size_t n = 0;
        if (lib.next_recv_x(s->buf, (int)M, (int)H, (int)R, 0, &p, &n)) return fail();
        if (p != nullptr) {
            PyObject* rows = PyObject_CallFunction(args[12], "KKLLO", (unsigned long long)reinterpret_cast<uintptr_t>(p),
                                                   (unsigned long long)n, (long long)n_cap, (long long)H, args[0]);
            if (rows == nullptr) return nullptr;
            recv_x = *tensor_of(rows);
            Py_DECREF(rows);
        }
    }
    const bool in_place = recv_x.defined();
    if (!in_place) recv_x = empty({out_cap, H}, at::kBFloat16, dev);
    Arena small(dev);
    const int64_t o_rank = small.reserve(R * 4), o_expert = small.reserve((L + 1) * 4), o_slot = small.reserve(T * K * 4);
    const int64_t o_idx = small.reserve(n_cap * K * 8), o_md = small.reserve(n_cap * (K + 2) * 4);
    const int64_t o_w = w ? small.reserve((expand ? out_cap : n_cap * K) * 4) : 0;
    const int64_t o_kept = cached ? 0 : small.reserve(idx->numel() * 8);
    small.allocate();

    mcep_elastic_dispatch_args a = {};
    a.x = x->const_data_ptr(), a.x_element_size = 2, a.num_tokens = (int)T, a.hidden = (int)H;
    a.topk_idx = static_cast<const int64_t*>(idx->const_data_ptr()), a.num_topk = (int)K;
    a.topk_weights = w ? static_cast<const float*>(w->const_data_ptr()) : nullptr;
    a.active_ranks = static_cast<int32_t*>(active->data_ptr());
    a.num_experts = (int)E, a.num_max_tokens_per_rank = (int)M, a.expert_alignment = (int)alignment;
    a.do_expand = expand, a.cached_mode = cached != nullptr, a.timeout_us = timeout;
    a.async_with_compute_stream = async, a.compute_stream = current_stream();
    a.psum_num_recv_tokens_per_scaleup_rank = reinterpret_cast<int32_t*>(small.at(o_rank));
    a.psum_num_recv_tokens_per_expert = reinterpret_cast<int32_t*>(small.at(o_expert));
    a.dst_buffer_slot_idx = reinterpret_cast<int32_t*>(small.at(o_slot));
    a.recv_x = recv_x.data_ptr(), a.recv_topk_idx = reinterpret_cast<int64_t*>(small.at(o_idx));
    a.recv_topk_weights = w ? reinterpret_cast<float*>(small.at(o_w)) : nullptr;
    a.recv_src_metadata = reinterpret_cast<int32_t*>(small.at(o_md));
    a.copied_topk_idx = cached ? nullptr : reinterpret_cast<int64_t*>(small.at(o_kept));
    mcep_event* ev = nullptr;
    std::vector<int32_t> host(sync ? R + L + 1 : 0);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = sync ? lib.elastic_dispatch_counted(s->buf, &a, host.data(), host.data() + R, &ev)
              : lib.elastic_dispatch(s->buf, &a, &ev);
    Py_END_ALLOW_THREADS
    if (rc) return fail();

    int64_t n = n_cap, n_out = out_cap;
    PyObject* counts = PyList_New(sync ? L : 0);
    if (counts == nullptr) return nullptr;
    if (sync) {
        const int32_t* psum = host.data() + R;
        // (never beyond what was allocated: aligned segments can end further on than the
        // expanded rows have room for, and those rows are dropped)
        n = std::min<int64_t>(host[R - 1], n_cap);
        n_out = expand ? std::min<int64_t>(L ? psum[L - 1] : 0, out_cap) : n;
        int64_t prev = 0;  // expanded: the entries are where the segments end, unaligned
        for (int64_t i = 0; i < L; ++i) {
            const int64_t c = expand ? psum[i] - (prev + alignment - 1) / alignment * alignment : psum[i + 1] - psum[i];
            prev = psum[i];
            PyList_SET_ITEM(counts, i, PyLong_FromLongLong(c));
        }
        if (n_out != recv_x.size(0)) recv_x = in_place ? recv_x.narrow(0, 0, n_out) : recv_x;
        if (!in_place) recv_x.unsafeGetTensorImpl()->set_sizes_contiguous({n_out, H});
    }
    const int64_t first = expand ? 0 : 1;
    PyObject* p_rows = wrap(std::move(recv_x));
    PyObject* p_idx = wrap(small.view(o_idx, at::kLong, {n, K}));
    PyObject* p_w = !w       ? new_ref(Py_None)
                    : expand ? wrap(small.view(o_w, at::kFloat, {n_out}))
                             : wrap(small.view(o_w, at::kFloat, {n, K}));
    PyObject* p_md = wrap(small.view(o_md, at::kInt, {n, K + 2}));
    PyObject* p_rank = wrap(small.view(o_rank, at::kInt, {R}));
    PyObject* p_expert = wrap(small.view(o_expert + 4 * first, at::kInt, {L + 1 - first}));
    PyObject* p_slot = wrap(small.view(o_slot, at::kInt, {T, K}));
    PyObject* p_kept = cached ? new_ref(args[4]) : wrap(small.view(o_kept, at::kLong, idx->sizes()));
    PyObject* keep = nullptr;
    if (!async)
        keep = new_ref(Py_None);
    else if (!p_rows || !p_idx || !p_w || !p_md || !p_rank || !p_expert || !p_slot || !p_kept)
        keep = nullptr;  // (an error is set)
    else if (w)
        keep = PyTuple_Pack(12, args[0], args[1], p_kept, args[3], p_rows, p_idx, p_rank, p_expert, p_md, p_slot, args[2], p_w);
    else
        keep = PyTuple_Pack(10, args[0], args[1], p_kept, args[3], p_rows, p_idx, p_rank, p_expert, p_md, p_slot);
    PyObject* handle = wrap_handle({new_ref(args[8]), new_ref(args[5]), new_ref(args[7]), new_ref(args[6]),
                                    new_ref(args[13]), p_kept, p_rank, p_expert, counts, p_md, p_slot, new_ref(Py_None),
                                    new_ref(Py_None), new_ref(Py_True), PyLong_FromLongLong(n)});
    return pack({p_rows, p_idx, p_w, handle, wrap_overlap(wrap_event(ev), keep)});
    END_HANDLE_TH_ERRORS
}

// elastic_combine_tensors(x, topk_idx, topk_weights or None, psum_rank, recv_src_metadata, active_ranks,
//                         E, M, do_expand, timeout_us, async)
//   -> what ElasticBuffer.combine returns: (combined_x, None, EventOverlap), or None (as above)
PyObject* runtime_elastic_combine_tensors(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    RuntimeObject* s = self_of(self);
    if (nargs != 11) return PyErr_Format(PyExc_TypeError, "elastic_combine_tensors() takes 11 arguments");
    if (!alive(s)) return nullptr;
    Reader r{const_cast<PyObject**>(args)};
    const at::Tensor *x = tensor_of(args[0]), *idx = tensor_of(args[1]), *w = tensor_of(args[2]);
    const at::Tensor *psum = tensor_of(args[3]), *md = tensor_of(args[4]), *active = tensor_of(args[5]);
    const int64_t E = r.num(6), M = r.num(7), timeout = r.num(9);
    const int expand = r.flag(8), async = r.flag(10);
    if (!r.ok) return nullptr;
    if (!matrix(x, at::kBFloat16) || !x->is_cuda() || !idx || idx->dim() < 2 || !entries(idx, at::kLong, 0) || !psum || !md ||
        !usable_mask(active, s->num_ranks) || (args[2] != Py_None && !w))
        Py_RETURN_NONE;
    const int64_t T = idx->size(0), K = idx->size(1), H = x->size(1);
    at::Tensor out = empty({T, H}, at::kBFloat16, x->device());
    mcep_elastic_combine_args a = {};
    a.x = x->const_data_ptr(), a.num_input_tokens = (int)x->size(0), a.hidden = (int)H;
    a.topk_idx = static_cast<const int64_t*>(idx->const_data_ptr());
    a.num_combined_tokens = (int)T, a.num_topk = (int)K;
    a.topk_weights = w ? static_cast<const float*>(w->const_data_ptr()) : nullptr;
    a.psum_num_recv_tokens_per_scaleup_rank = static_cast<const int32_t*>(psum->const_data_ptr());
    // (the handle's tensor by its address: it stays the same when the host cut it to length)
    a.recv_src_metadata = reinterpret_cast<const int32_t*>(static_cast<const char*>(md->storage().data()) +
                                                           md->storage_offset() * (int64_t)sizeof(int32_t));
    a.active_ranks = static_cast<int32_t*>(active->data_ptr());
    a.num_experts = (int)E, a.num_max_tokens_per_rank = (int)M, a.do_expand = expand, a.timeout_us = timeout;
    a.async_with_compute_stream = async, a.compute_stream = current_stream();
    a.combined_x = out.data_ptr();
    mcep_event* ev = nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = lib.elastic_combine(s->buf, &a, &ev);
    Py_END_ALLOW_THREADS if (rc) return fail();
    PyObject* p_out = wrap(std::move(out));
    PyObject* keep = nullptr;
    if (!async)
        keep = new_ref(Py_None);
    else if (!p_out)
        keep = nullptr;  // (an error is set)
    else if (w)
        keep = PyTuple_Pack(6, args[0], args[5], p_out, args[1], args[4], args[2]);
    else
        keep = PyTuple_Pack(5, args[0], args[5], p_out, args[1], args[4]);
    return pack({p_out, new_ref(Py_None), wrap_overlap(wrap_event(ev), keep)});
    END_HANDLE_TH_ERRORS
}

PyMethodDef runtime_methods[] = {
    {"_adopt", runtime_adopt, METH_VARARGS, "_adopt(handle or None, num_ranks): the mcep_buffer the calls go to."},
    {"dispatch", MCEP_FAST(runtime_dispatch), METH_FASTCALL | METH_KEYWORDS,
     "dispatch($self, x_ptr, topk_idx_ptr, active_ranks_ptr, num_tokens, hidden, num_topk, "
     "num_max_dispatch_tokens_per_rank, num_experts, timeout_us, use_fp8, packed_recv_x_ptr, "
     "packed_recv_x_scales_ptr, packed_recv_count_ptr, packed_recv_src_info_ptr, packed_recv_layout_range_ptr, "
     "async_finish, return_recv_hook, compute_stream_ptr)\n--\n\n"
     "mooncake-ep/include/mooncake_ep_buffer.h:116-124. Returns (event or None, hook or None)."},
    {"combine", MCEP_FAST(runtime_combine), METH_FASTCALL | METH_KEYWORDS,
     "combine($self, x_ptr, topk_idx_ptr, topk_weights_ptr, src_info_ptr, layout_range_ptr, active_ranks_ptr, "
     "num_local_experts, num_combined_tokens, hidden, num_topk, num_max_dispatch_tokens_per_rank, num_experts, "
     "timeout_us, zero_copy, combined_x_ptr, async_finish, return_recv_hook, compute_stream_ptr)\n--\n\n"
     "mooncake-ep/include/mooncake_ep_buffer.h:126-133. Returns (event or None, hook or None)."},
    {"next_recv_x", MCEP_FAST(runtime_next_recv_x), METH_FASTCALL | METH_KEYWORDS,
     "next_recv_x($self, num_max_dispatch_tokens_per_rank, hidden, num_experts, use_fp8)\n--\n\n"
     "(device pointer, bytes) of the in-place receive tensor of the next dispatch call, (0, 0) when there is\n"
     "none (include/mcep.h)."},
    {"dispatch_tensors", MCEP_FAST(runtime_dispatch_tensors), METH_FASTCALL, "Buffer.dispatch on checked tensors."},
    {"combine_tensors", MCEP_FAST(runtime_combine_tensors), METH_FASTCALL, "Buffer.combine on checked tensors."},
    {"elastic_dispatch_tensors", MCEP_FAST(runtime_elastic_dispatch_tensors), METH_FASTCALL,
     "ElasticBuffer.dispatch on checked tensors."},
    {"elastic_combine_tensors", MCEP_FAST(runtime_elastic_combine_tensors), METH_FASTCALL,
     "ElasticBuffer.combine on checked tensors."},
    {nullptr, nullptr, 0, nullptr}};
PyType_Slot runtime_slots[] = {{Py_tp_doc, const_cast<char*>("The calls of an mcep_buffer; base of ep.Buffer.")},
                               {Py_tp_methods, runtime_methods},
                               {0, nullptr}};
PyType_Spec runtime_spec = {"mooncake_b200._mcep_torch.Runtime", sizeof(RuntimeObject), 0,
                            Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE, runtime_slots};

PyObject* py_adopt_event(PyObject*, PyObject* address) {
    if (address == Py_None) Py_RETURN_NONE;
    void* p = PyLong_AsVoidPtr(address);
    if (PyErr_Occurred()) return nullptr;
    return wrap_event(static_cast<mcep_event*>(p));
}

PyMethodDef module_methods[] = {
    {"adopt_event", py_adopt_event, METH_O, "An EventHandle that owns the mcep_event at this address (None: None)."},
    {"bind", py_bind, METH_O, "bind({name: address}): the entry points of the loaded libmcep.so."},
    {"register_overlap", py_register_overlap, METH_O, "The class (derived from EventOverlapBase) that calls return."},
    {"register_handle", py_register_handle, METH_O, "The class of the handles that elastic calls return."},
    {"current_stream", py_current_stream, METH_NOARGS, "torch's current CUDA stream as an integer."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_mcep_torch", "Native binding of libmcep.so for torch tensors.",
                          -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__mcep_torch(void) {
    PyObject* m = PyModule_Create(&module_def);
    if (m == nullptr) return nullptr;
    event_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&event_spec));
    hook_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&hook_spec));
    overlap_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&overlap_spec));
    PyObject* runtime = PyType_FromSpec(&runtime_spec);
    if (!event_type || !hook_type || !overlap_type || !runtime) return nullptr;
    if (PyModule_AddObjectRef(m, "EventHandle", reinterpret_cast<PyObject*>(event_type)) < 0 ||
        PyModule_AddObjectRef(m, "EventOverlapBase", reinterpret_cast<PyObject*>(overlap_type)) < 0 ||
        PyModule_AddObjectRef(m, "Hook", reinterpret_cast<PyObject*>(hook_type)) < 0 ||
        PyModule_AddObjectRef(m, "Runtime", runtime) < 0)
        return nullptr;
    return m;
}
