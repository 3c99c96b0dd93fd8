// Native host side of the optimizer classes and of the codec functions (extension module came_b200._host).
//
// A step of a few hundred small tensors is over on the GPU before Python has looked at every parameter's gradient:
// walking 528 parameters (two data_ptr() calls, a dtype and a shape each) takes 280 us in Python, 15 us here.  What is
// here: the check that the tensor table of the previous step still stands, the new gradient addresses when only those
// moved, the hyper-parameter records, the step call itself; and the codec functions' allocation and launch.  Everything
// else (first step, changed tensors, states, errors) stays in optim.py / engine.py, to which `step` hands over by
// returning SLOW.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <memory>
#include <string>
#include <vector>

#include "came_b200.h"

namespace {

constexpr long SLOW = -1;         // the caller takes the Python path
constexpr long FAILED = -1000;    // FAILED + code: the library refused (came_b200_last_error has the message)

// Without the interpreter's lock: a launch may wait for room in the stream's queue, an allocation for the device.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};
struct Unref { void operator()(PyObject* o) const { Py_XDECREF(o); } };
using Owned = std::unique_ptr<PyObject, Unref>;

struct Param {                    // (no reference to the parameter: swap_tensors() and the garbage collector count them)
    PyObject* obj;                // borrowed from the group's list: compared with what the list holds now
    PyTypeObject* type;
    bool has_grad;
    at::ScalarType p_type, g_type;
    const void *p_ptr, *g_ptr;
    std::vector<int64_t> sizes;
    int plan, pos;                // entry of a plan's tensor table
};
struct Plan {
    int device;
    PyObject* py;                 // the DevicePlan (owned); its `handle` is read at every step, None once it is closed
    std::vector<const void*> g;   // gradient addresses in table order
};
struct StepTable {
    PyObject_HEAD
    std::vector<std::vector<Param>>* groups;
    std::vector<Plan>* plans;
    std::vector<PyObject*>* states;      // state dicts that carry a "step" count (owned)
    PyObject *k_params, *k_lr, *k_betas, *k_eps, *k_clip, *k_wd, *k_scale, *k_step, *one;
};

void table_clear(StepTable* s) {
    s->groups->clear();
    for (auto& p : *s->plans) Py_XDECREF(p.py);
    s->plans->clear();
    for (PyObject* d : *s->states) Py_XDECREF(d);
    s->states->clear();
}

PyObject* table_new(PyTypeObject* type, PyObject*, PyObject*) {
    StepTable* s = reinterpret_cast<StepTable*>(type->tp_alloc(type, 0));
    if (!s) return nullptr;
    s->groups = new std::vector<std::vector<Param>>();
    s->plans = new std::vector<Plan>();
    s->states = new std::vector<PyObject*>();
    auto key = [](const char* x) { return PyUnicode_InternFromString(x); };
    s->k_params = key("params"); s->k_lr = key("lr"); s->k_betas = key("betas"); s->k_eps = key("eps");
    s->k_clip = key("clip_threshold"); s->k_wd = key("weight_decay"); s->k_scale = key("grad_scale"); s->k_step = key("step");
    s->one = PyLong_FromLong(1);
    return reinterpret_cast<PyObject*>(s);
}
void table_dealloc(PyObject* self) {
    StepTable* s = reinterpret_cast<StepTable*>(self);
    table_clear(s);
    delete s->groups;
    delete s->plans;
    delete s->states;
    for (PyObject* k : {s->k_params, s->k_lr, s->k_betas, s->k_eps, s->k_clip, s->k_wd, s->k_scale, s->k_step, s->one}) Py_XDECREF(k);
    Py_TYPE(self)->tp_free(self);
}

// The gradient of a parameter as the table can hold it; false: the Python path copies, raises or rebuilds.
bool usable(const at::Tensor& p, const at::Tensor& g) {
    return g.layout() == at::kStrided && g.is_contiguous() && p.is_contiguous() && g.numel() == p.numel();
}

// build(param_groups, [(DevicePlan, device index, n)], [state dict]): remembers the tensors of a step that the
// Python path has just made.  Parameters with a gradient fill the plans' tables in order, by device.  False when they do not.
bool build(StepTable* s, PyObject* groups, PyObject* plans, PyObject* states) {
    table_clear(s);
    std::vector<int> expect;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(plans); ++i) {
        int device, n;
        PyObject* py;
        if (!PyArg_ParseTuple(PyList_GET_ITEM(plans, i), "Oii", &py, &device, &n)) return false;
        Py_INCREF(py);
        s->plans->push_back(Plan{device, py, {}});
        expect.push_back(n);
    }
    bool ok = true;
    for (Py_ssize_t gi = 0; ok && gi < PyList_GET_SIZE(groups); ++gi) {
        PyObject* list = PyDict_GetItemWithError(PyList_GET_ITEM(groups, gi), s->k_params);
        if (!list || !PyList_Check(list)) { ok = false; break; }
        std::vector<Param> ps;
        ps.reserve((size_t)PyList_GET_SIZE(list));
        for (Py_ssize_t i = 0; ok && i < PyList_GET_SIZE(list); ++i) {
            PyObject* obj = PyList_GET_ITEM(list, i);
            if (!THPVariable_Check(obj)) { ok = false; break; }
            Param e{obj, Py_TYPE(obj), false, at::kFloat, at::kFloat, nullptr, nullptr, {}, -1, -1};
            const at::Tensor& t = THPVariable_Unpack(obj);
            const at::Tensor& g = t.grad();
            if (g.defined()) {
                int k = 0;
                while (k < (int)s->plans->size() && (*s->plans)[k].device != t.device().index()) ++k;
                if (k == (int)s->plans->size() || !usable(t, g)) { ok = false; break; }
                Plan& plan = (*s->plans)[k];
                e.has_grad = true;
                e.p_type = t.scalar_type();
                e.g_type = g.scalar_type();
                e.p_ptr = t.const_data_ptr();
                e.g_ptr = g.const_data_ptr();
                e.sizes = t.sizes().vec();
                e.plan = k;
                e.pos = (int)plan.g.size();
                plan.g.push_back(e.g_ptr);
            }
            ps.push_back(std::move(e));
        }
        s->groups->push_back(std::move(ps));
    }
    for (size_t k = 0; k < expect.size(); ++k) ok = ok && (int)(*s->plans)[k].g.size() == expect[k];
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(states); ++i) {
        PyObject* d = PyList_GET_ITEM(states, i);
        ok = ok && PyDict_Check(d);
        Py_INCREF(d);
        s->states->push_back(d);
    }
    return ok;
}
// Every entry below: what torch throws becomes the Python exception torch has for it (END_HANDLE_TH_ERRORS).
PyObject* table_build(PyObject* self, PyObject* args) {
    HANDLE_TH_ERRORS
    StepTable* s = reinterpret_cast<StepTable*>(self);
    PyObject *groups, *plans, *states;
    if (!PyArg_ParseTuple(args, "O!O!O!", &PyList_Type, &groups, &PyList_Type, &plans, &PyList_Type, &states)) return nullptr;
    bool ok = false;
    try {
        ok = build(s, groups, plans, states);
    } catch (...) {
        table_clear(s);
        throw;
    }
    if (!ok || PyErr_Occurred()) table_clear(s);
    if (PyErr_Occurred()) return nullptr;
    return PyBool_FromLong(ok);
    END_HANDLE_TH_ERRORS
}

bool number(PyObject* dict, PyObject* key, double* out) {
    PyObject* v = PyDict_GetItemWithError(dict, key);
    if (!v) return false;
    *out = PyFloat_AsDouble(v);
    return !(*out == -1.0 && PyErr_Occurred());
}
bool numbers(PyObject* dict, PyObject* key, double* out, Py_ssize_t n) {
    PyObject* v = PyDict_GetItemWithError(dict, key);
    if (!v || !(PyTuple_Check(v) || PyList_Check(v)) || PySequence_Fast_GET_SIZE(v) != n) return false;
    for (Py_ssize_t i = 0; i < n; ++i) {
        out[i] = PyFloat_AsDouble(PySequence_Fast_GET_ITEM(v, i));
        if (out[i] == -1.0 && PyErr_Occurred()) return false;
    }
    return true;
}

// The two records of a group (engine.make_hyper): kernel-style scalars formed in fp32, Python-style ones in double.
bool hypers_of(StepTable* s, PyObject* group, CameHyper* out) {
    double lr, betas[3], eps[2], clip, wd, scale = 1.0;
    if (!number(group, s->k_lr, &lr) || !numbers(group, s->k_betas, betas, 3) || !numbers(group, s->k_eps, eps, 2) ||
        !number(group, s->k_clip, &clip) || !number(group, s->k_wd, &wd))
        return false;
    if (PyDict_GetItemWithError(group, s->k_scale) && !number(group, s->k_scale, &scale)) return false;
    for (int py = 0; py < 2; ++py) {
        CameHyper& h = out[py];
        h = CameHyper{};
        h.lr = (float)lr;
        float* b[3] = {&h.beta1, &h.beta2, &h.beta3};
        float* om[3] = {&h.om_beta1, &h.om_beta2, &h.om_beta3};
        for (int k = 0; k < 3; ++k) {
            *b[k] = (float)betas[k];
            *om[k] = py ? (float)(1.0 - betas[k]) : 1.0f - (float)betas[k];
        }
        h.wd_lr = py ? (float)(wd * lr) : (float)wd * (float)lr;
        const volatile float prod = (float)lr * (float)wd;      // (two roundings, no fused multiply-add)
        h.decay_mul = py ? (float)(1.0 - lr * wd) : 1.0f - prod;
        h.eps0 = (float)eps[0];
        h.eps1 = (float)eps[1];
        h.clip_threshold = (float)clip;
        h.weight_decay = (float)wd;
        h.grad_scale = (float)scale;
    }
    return true;
}

// The plan as it stands, null when it has been closed (PyErr set on an error)
came_plan_t* handle_of(const Plan& plan) {
    PyObject* h = PyObject_GetAttrString(plan.py, "handle");      // ctypes.c_void_p or None
    if (!h || h == Py_None) { Py_XDECREF(h); return nullptr; }
    PyObject* v = PyObject_GetAttrString(h, "value");
    Py_DECREF(h);
    void* p = v && v != Py_None ? PyLong_AsVoidPtr(v) : nullptr;
    Py_XDECREF(v);
    return static_cast<came_plan_t*>(p);
}

// step(param_groups): launches (>= 0), SLOW or FAILED + code
long step(StepTable* s, PyObject* groups) {
    if (s->plans->empty() || !PyList_Check(groups) || (size_t)PyList_GET_SIZE(groups) != s->groups->size()) return SLOW;
    const size_t n_groups = s->groups->size();
    if (2 * n_groups > 64) return SLOW;
    // (what is used without the lock below: the table may be dropped or rebuilt by another thread meanwhile)
    struct Target {
        came_plan_t* handle;
        c10::DeviceIndex device;
        Owned plan;
        std::vector<const void*> g;
    };
    std::vector<Target> targets;
    for (const Plan& plan : *s->plans) {
        came_plan_t* h = handle_of(plan);
        if (!h) return SLOW;
        Py_INCREF(plan.py);
        targets.push_back(Target{h, (c10::DeviceIndex)plan.device, Owned(plan.py), {}});
    }
    bool moved = false;
    for (size_t gi = 0; gi < n_groups; ++gi) {
        std::vector<Param>& ps = (*s->groups)[gi];
        PyObject* list = PyDict_GetItemWithError(PyList_GET_ITEM(groups, gi), s->k_params);
        if (!list || !PyList_Check(list) || (size_t)PyList_GET_SIZE(list) != ps.size()) return SLOW;
        for (size_t i = 0; i < ps.size(); ++i) {
            Param& e = ps[i];
            if (PyList_GET_ITEM(list, (Py_ssize_t)i) != e.obj || Py_TYPE(e.obj) != e.type) return SLOW;
            const at::Tensor& t = THPVariable_Unpack(e.obj);
            const at::Tensor& g = t.grad();
            if (g.defined() != e.has_grad) return SLOW;
            if (!e.has_grad) continue;
            if (!usable(t, g) || g.scalar_type() != e.g_type || t.scalar_type() != e.p_type || t.const_data_ptr() != e.p_ptr ||
                t.sizes() != at::IntArrayRef(e.sizes) || g.device() != t.device())
                return SLOW;
            const void* at = g.const_data_ptr();
            if (at != e.g_ptr) {
                moved = true;
                e.g_ptr = at;
                (*s->plans)[e.plan].g[e.pos] = at;
            }
        }
    }
    // The states' step counts go up for all or for none: what does not simply add is left to the Python path.
    for (PyObject* d : *s->states) {
        PyObject* v = PyDict_GetItemWithError(d, s->k_step);
        if (!v || !(PyLong_CheckExact(v) || PyFloat_CheckExact(v))) return SLOW;
    }
    CameHyper hyp[64];
    for (size_t gi = 0; gi < n_groups; ++gi)
        if (!hypers_of(s, PyList_GET_ITEM(groups, (Py_ssize_t)gi), hyp + 2 * gi)) {
            PyErr_Clear();      // the Python path raises what there is to raise
            return SLOW;
        }
    if (moved) {
        for (size_t k = 0; k < targets.size(); ++k) {
            if (PyObject_SetAttrString(targets[k].plan.get(), "addresses", Py_None) != 0) return SLOW;
            targets[k].g = (*s->plans)[k].g;
        }
        NoGil unlocked;
        for (const Target& t : targets) {
            c10::cuda::CUDAGuard guard(t.device);
            const int rc = came_b200_plan_set_pointers(t.handle, t.g.data(), nullptr, (int)t.g.size(),
                                                       c10::cuda::getCurrentCUDAStream(t.device).stream());
            if (rc == CAME_E_INVALID) return SLOW;      // another alignment class: a new plan
            if (rc != CAME_OK) return FAILED + rc;
        }
    }
    for (PyObject* d : *s->states) {
        PyObject* v = PyDict_GetItemWithError(d, s->k_step);
        const Owned next(v ? PyNumber_Add(v, s->one) : nullptr);
        if (!next || PyDict_SetItem(d, s->k_step, next.get()) != 0) return SLOW;
    }
    long launches = 0;
    NoGil unlocked;
    for (const Target& t : targets) {
        c10::cuda::CUDAGuard guard(t.device);
        const int rc = came_b200_step(t.handle, hyp, (int)(2 * n_groups), c10::cuda::getCurrentCUDAStream(t.device).stream());
        if (rc != CAME_OK) return FAILED + rc;
        launches += came_b200_plan_last_launches(t.handle);
    }
    return launches;
}

PyObject* table_step(PyObject* self, PyObject* groups) {
    HANDLE_TH_ERRORS
    const long r = step(reinterpret_cast<StepTable*>(self), groups);
    if (PyErr_Occurred()) return nullptr;
    return PyLong_FromLong(r);
    END_HANDLE_TH_ERRORS
}
PyObject* table_forget(PyObject* self, PyObject*) {
    table_clear(reinterpret_cast<StepTable*>(self));
    Py_RETURN_NONE;
}

PyMethodDef table_methods[] = {{"build", table_build, METH_VARARGS, "remember the tensors of a step"},
                               {"step", table_step, METH_O, "step them again; launches, -1 (slow path) or -1000 + code"},
                               {"forget", table_forget, METH_NOARGS, "drop every reference"},
                               {nullptr, nullptr, 0, nullptr}};
PyTypeObject table_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---- codec: the checks are made by the caller (quant.py) -------------------------------------------------------------
cudaStream_t stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
PyObject* status(int rc, PyObject* result) {
    if (rc == CAME_OK) return result;
    Py_XDECREF(result);
    const Owned lib(PyImport_ImportModule("came_b200._lib"));
    const Owned type(lib ? PyObject_GetAttrString(lib.get(), "CameError") : nullptr);
    return type ? PyErr_Format(type.get(), "came_b200 error %d: %s", rc, came_b200_last_error()) : nullptr;
}
const at::Tensor& tensor_of(PyObject* o) {
    if (!THPVariable_Check(o)) throw torch::TypeError(std::string("expected a tensor, got ") + Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
}
at::Tensor fp32_contiguous(const at::Tensor& t) {
    return t.scalar_type() == at::kFloat && t.is_contiguous() ? t : t.to(at::kFloat).contiguous();
}

PyObject* quantize(PyObject*, PyObject* args) {
    HANDLE_TH_ERRORS
    PyObject* obj;
    int is_signed, tile;
    if (!PyArg_ParseTuple(args, "Opp", &obj, &is_signed, &tile)) return nullptr;
    const at::Tensor in = tensor_of(obj).detach();
    at::Tensor q, a;
    int rc;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(in.device());
        const at::Tensor src = fp32_contiguous(in);
        const int64_t n = src.numel(), blocks = tile ? ((src.size(0) + 15) / 16) * ((src.size(1) + 15) / 16) : std::max<int64_t>(1, (n + 255) / 256);
        q = at::empty(src.sizes(), src.options().dtype(is_signed ? at::kChar : at::kByte));
        a = at::empty({blocks}, src.options());
        rc = tile ? came_b200_quantize_tile16(src.const_data_ptr<float>(), static_cast<int8_t*>(q.mutable_data_ptr()),
                                              a.mutable_data_ptr<float>(), src.size(0), src.size(1), stream_of(src))
                  : came_b200_quantize_blockwise(src.const_data_ptr<float>(), q.mutable_data_ptr(), a.mutable_data_ptr<float>(), n,
                                                 is_signed, stream_of(src));
    }
    return status(rc, rc == CAME_OK ? Py_BuildValue("(NN)", THPVariable_Wrap(q), THPVariable_Wrap(a)) : nullptr);
    END_HANDLE_TH_ERRORS
}

PyObject* dequantize(PyObject*, PyObject* args) {
    HANDLE_TH_ERRORS
    PyObject *qobj, *aobj;
    int is_signed, tile;
    if (!PyArg_ParseTuple(args, "OOpp", &qobj, &aobj, &is_signed, &tile)) return nullptr;
    const at::Tensor q0 = tensor_of(qobj), a0 = tensor_of(aobj);
    at::Tensor out;
    int rc;
    {
        NoGil unlocked;
        c10::cuda::CUDAGuard guard(q0.device());
        const at::Tensor q = q0.is_contiguous() ? q0 : q0.contiguous(), a = fp32_contiguous(a0);
        out = at::empty(q.sizes(), q.options().dtype(at::kFloat));
        rc = tile ? came_b200_dequantize_tile16(static_cast<const int8_t*>(q.const_data_ptr()), a.const_data_ptr<float>(),
                                                out.mutable_data_ptr<float>(), q.size(0), q.size(1), stream_of(q))
                  : came_b200_dequantize_blockwise(q.const_data_ptr(), a.const_data_ptr<float>(), out.mutable_data_ptr<float>(),
                                                   q.numel(), is_signed, stream_of(q));
    }
    return status(rc, rc == CAME_OK ? THPVariable_Wrap(out) : nullptr);
    END_HANDLE_TH_ERRORS
}

PyMethodDef module_methods[] = {{"quantize", quantize, METH_VARARGS, "(tensor, signed, tile) -> (codes, absmax)"},
                                {"dequantize", dequantize, METH_VARARGS, "(codes, absmax, signed, tile) -> fp32"},
                                {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "native host side of came_b200", -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    table_type.tp_name = "came_b200._host.StepTable";
    table_type.tp_basicsize = sizeof(StepTable);
    table_type.tp_flags = Py_TPFLAGS_DEFAULT;
    table_type.tp_new = table_new;
    table_type.tp_dealloc = table_dealloc;
    table_type.tp_methods = table_methods;
    if (PyType_Ready(&table_type) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&table_type);
    if (PyModule_AddObject(m, "StepTable", reinterpret_cast<PyObject*>(&table_type)) < 0) return nullptr;
    return m;
}
