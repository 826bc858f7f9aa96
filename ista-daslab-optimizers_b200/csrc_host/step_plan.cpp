// Host side of MicroAdam.step() in native code: walks the optimizer's parameter list, brings the descriptors of the
// fused step up to date and calls the library, without a Python statement per tensor.
//
// What bounds a step over small tensors is the host: the Python form of this walk (micro_adam.py, _refresh_entries and
// _fused_step) costs about 2 us per tensor and 20 us per call, more than the kernels of a 10 M-element list take.
// Here a tensor costs about 40 ns.  The plan is built by the Python side whenever the set of tensors to update changes;
// every step it is checked against the optimizer as it stands (same groups, same parameters, a gradient where there was
// one, the same element types, contiguous CUDA memory), and any difference hands the step back to the Python side,
// which rebuilds the plan or raises.  Learning rates, weight decays, ring positions, parameter and gradient
// addresses are read every step.  What torch throws on the way becomes the Python exception it stands for.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <exception>
#include <memory>
#include <optional>
#include <utility>
#include <vector>

#include "microadam_b200.h"

namespace {

using FusedStep = int (*)(mab_tensor*, int, const mab_step_args*, void*, int64_t, void*);

// What a parameter of the optimizer was when the plan was made.
enum class Kind { Elsewhere, NoGradient, Active };   // Elsewhere: another rank's, whatever its gradient

struct Param {
    PyObject* object;            // owned reference
    PyObject* state;             // owned reference to its state dictionary (Active only)
    Kind kind;
    at::ScalarType param_type, grad_type;
    int64_t numel, first;        // first: where the updated slice starts
};

struct Group {
    PyObject* object;            // owned reference to the group's dictionary
    std::vector<Param> params;
};

struct Plan {
    std::vector<Group> groups;
    std::vector<mab_tensor> descs;
    std::vector<PyObject*> ring_next;   // owned: the Python integer each ring position advances to
    int window = 0;
    c10::DeviceIndex device = -1;
    FusedStep fused_step = nullptr;
    void* workspace = nullptr;
    int64_t workspace_bytes = 0;
    PyObject *key_params = nullptr, *key_lr = nullptr, *key_weight_decay = nullptr, *key_index = nullptr;

    // Every reference the plan owns, for Python's collector: a group or a parameter may refer to the optimizer that holds the plan.
    template <typename F> int each_reference(F&& visit) {
        for (Group& g : groups) {
            for (Param& p : g.params) {
                if (int rc = visit(p.object)) return rc;
                if (int rc = visit(p.state)) return rc;
            }
            if (int rc = visit(g.object)) return rc;
        }
        for (PyObject*& o : ring_next) if (int rc = visit(o)) return rc;
        for (PyObject** o : {&key_params, &key_lr, &key_weight_decay, &key_index}) if (int rc = visit(*o)) return rc;
        return 0;
    }
    ~Plan() { each_reference([](PyObject*& o) { Py_CLEAR(o); return 0; }); }
};

// The Python object around a plan.
struct PlanObject {
    PyObject_HEAD
    Plan* plan;                  // nullptr once the collector has cleared it
};

PyTypeObject* g_plan_type = nullptr;     // (the module owns it as well)

int plan_traverse(PyObject* self, visitproc visit, void* arg) {
    Py_VISIT(Py_TYPE(self));
    Plan* plan = reinterpret_cast<PlanObject*>(self)->plan;
    return plan == nullptr ? 0 : plan->each_reference([&](PyObject* o) { Py_VISIT(o); return 0; });
}

int plan_clear(PyObject* self) {
    delete std::exchange(reinterpret_cast<PlanObject*>(self)->plan, nullptr);
    return 0;
}

void plan_dealloc(PyObject* self) {
    PyObject_GC_UnTrack(self);
    plan_clear(self);
    PyTypeObject* type = Py_TYPE(self);
    PyObject_GC_Del(self);
    Py_DECREF(type);
}

PyType_Slot plan_slots[] = {{Py_tp_traverse, reinterpret_cast<void*>(plan_traverse)},
                            {Py_tp_clear, reinterpret_cast<void*>(plan_clear)},
                            {Py_tp_dealloc, reinterpret_cast<void*>(plan_dealloc)},
                            {0, nullptr}};
PyType_Spec plan_spec = {"_step_plan.Plan", sizeof(PlanObject), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_DISALLOW_INSTANTIATION, plan_slots};

// A number in a group's dictionary (a float, an int, or anything float() takes, such as a tensor).
bool number(PyObject* dict, PyObject* key, double* out) {
    PyObject* v = PyDict_GetItemWithError(dict, key);
    if (v == nullptr) return false;
    if (PyFloat_CheckExact(v)) { *out = PyFloat_AS_DOUBLE(v); return true; }
    PyObject* f = PyNumber_Float(v);
    if (f == nullptr) return false;
    *out = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return true;
}

// The exception in flight (torch's errors, bad_alloc) as Python's: none may cross the interpreter's C frames.
PyObject* raise_python() {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
}

// plan_new(groups, descs_address, n_descs, m, device_index, fused_step_address, workspace_address, workspace_bytes)
//   groups: [(group dictionary, [(parameter, kind, state dictionary or None, first element of its slice), ...]), ...]
//   descs: the descriptors of the Active parameters in that order, their fixed fields filled in
PyObject* plan_new(PyObject*, PyObject* args) try {
    PyObject* groups;
    unsigned long long descs_at, fn_at, ws_at;
    long long n_descs, ws_bytes;
    int window, device;
    if (!PyArg_ParseTuple(args, "O!KLiiKKL", &PyList_Type, &groups, &descs_at, &n_descs, &window, &device, &fn_at, &ws_at, &ws_bytes))
        return nullptr;
    auto owner = std::make_unique<Plan>();
    Plan* plan = owner.get();
    const auto* d = reinterpret_cast<const mab_tensor*>(static_cast<uintptr_t>(descs_at));
    plan->descs.assign(d, d + n_descs);
    plan->window = window;
    plan->device = static_cast<c10::DeviceIndex>(device);
    plan->fused_step = reinterpret_cast<FusedStep>(static_cast<uintptr_t>(fn_at));
    plan->workspace = reinterpret_cast<void*>(static_cast<uintptr_t>(ws_at));
    plan->workspace_bytes = ws_bytes;
    plan->key_params = PyUnicode_InternFromString("params");
    plan->key_lr = PyUnicode_InternFromString("lr");
    plan->key_weight_decay = PyUnicode_InternFromString("weight_decay");
    plan->key_index = PyUnicode_InternFromString("index");
    for (int r = 0; r < window; ++r) plan->ring_next.push_back(PyLong_FromLong((r + 1) % window));
    int64_t active = 0;
    for (Py_ssize_t gi = 0; gi < PyList_GET_SIZE(groups); ++gi) {
        PyObject *dict, *list;
        if (!PyArg_ParseTuple(PyList_GET_ITEM(groups, gi), "O!O!", &PyDict_Type, &dict, &PyList_Type, &list)) return nullptr;
        plan->groups.emplace_back();
        Group& g = plan->groups.back();
        g.object = Py_NewRef(dict);
        for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
            PyObject *object, *state;
            int kind;
            long long first;
            if (!PyArg_ParseTuple(PyList_GET_ITEM(list, i), "OiOL", &object, &kind, &state, &first)) return nullptr;
            if (!THPVariable_Check(object) || kind < 0 || kind > 2 || (kind == 2 && !PyDict_Check(state))) {
                PyErr_SetString(PyExc_TypeError, "plan_new: a parameter is not a tensor, or has no state dictionary");
                return nullptr;
            }
            Param p = {};
            p.object = Py_NewRef(object);
            p.kind = static_cast<Kind>(kind);
            p.first = first;
            g.params.push_back(p);
            Param& q = g.params.back();
            if (q.kind == Kind::Active) {
                const at::Tensor& t = THPVariable_Unpack(object);
                q.state = Py_NewRef(state);
                q.param_type = t.scalar_type();
                q.grad_type = t.grad().scalar_type();
                q.numel = t.numel();
                ++active;
            }
        }
    }
    if (active != n_descs || window < 1) {
        PyErr_SetString(PyExc_ValueError, "plan_new: one descriptor per active parameter");
        return nullptr;
    }
    auto* object = PyObject_GC_New(PlanObject, g_plan_type);
    if (object == nullptr) return nullptr;
    object->plan = owner.release();
    PyObject_GC_Track(object);
    return reinterpret_cast<PyObject*>(object);
} catch (...) {
    return raise_python();
}

// Brings plan.descs up to date.  1: the optimizer no longer looks like the plan, 0: done, -1: a Python error is set.
int refresh(Plan& plan, PyObject* groups) {
    if (!PyList_Check(groups) || static_cast<size_t>(PyList_GET_SIZE(groups)) != plan.groups.size()) return 1;
    size_t at = 0;
    for (size_t gi = 0; gi < plan.groups.size(); ++gi) {
        Group& g = plan.groups[gi];
        if (PyList_GET_ITEM(groups, gi) != g.object) return 1;
        PyObject* list = PyDict_GetItemWithError(g.object, plan.key_params);
        if (list == nullptr || !PyList_Check(list) || static_cast<size_t>(PyList_GET_SIZE(list)) != g.params.size()) return PyErr_Occurred() ? -1 : 1;
        double lr, weight_decay;
        if (!number(g.object, plan.key_lr, &lr) || !number(g.object, plan.key_weight_decay, &weight_decay)) return PyErr_Occurred() ? -1 : 1;
        // (a group's numbers may be read through Python code, so the list is looked at again afterwards)
        if (PyDict_GetItemWithError(g.object, plan.key_params) != list || static_cast<size_t>(PyList_GET_SIZE(list)) != g.params.size()) return 1;
        for (size_t i = 0; i < g.params.size(); ++i) {
            const Param& p = g.params[i];
            if (PyList_GET_ITEM(list, i) != p.object) return 1;
            if (p.kind == Kind::Elsewhere) continue;
            const at::Tensor& t = THPVariable_Unpack(p.object);
            const at::Tensor& grad = t.grad();
            if (p.kind == Kind::NoGradient) {
                if (grad.defined()) return 1;
                continue;
            }
            if (!grad.defined() || grad.layout() != at::kStrided || t.scalar_type() != p.param_type || grad.scalar_type() != p.grad_type ||
                !t.is_cuda() || !grad.is_cuda() || t.numel() != p.numel || grad.numel() != p.numel || !t.is_contiguous() || !grad.is_contiguous())
                return 1;
            PyObject* index = PyDict_GetItemWithError(p.state, plan.key_index);
            if (index == nullptr || !PyLong_Check(index)) return PyErr_Occurred() ? -1 : 1;
            const long ring = PyLong_AsLong(index);
            if (ring < 0 || ring >= plan.window) { PyErr_Clear(); return 1; }
            mab_tensor& d = plan.descs[at++];
            d.param = static_cast<char*>(t.data_ptr()) + p.first * t.element_size();
            d.grad = static_cast<char*>(grad.data_ptr()) + p.first * grad.element_size();
            d.ring_index = static_cast<int32_t>(ring);
            d.lr = lr;
            d.weight_decay = weight_decay;
        }
    }
    return 0;
}

struct ReleasedInterpreter {
    PyThreadState* saved = PyEval_SaveThread();
    ~ReleasedInterpreter() { PyEval_RestoreThread(saved); }
};

// plan_step(plan, param_groups, steps, quant_block_size, alpha, beta1, beta2, eps) -> 1 stale, <= 0 the library's status
PyObject* plan_step(PyObject*, PyObject* const* args, Py_ssize_t n) try {
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "plan_step takes 8 arguments"); return nullptr; }
    if (!Py_IS_TYPE(args[0], g_plan_type)) { PyErr_SetString(PyExc_TypeError, "plan_step: not a plan"); return nullptr; }
    Plan* plan = reinterpret_cast<PlanObject*>(args[0])->plan;
    if (plan == nullptr) return PyLong_FromLong(1);
    mab_step_args a = {};
    a.steps = PyLong_AsLongLong(args[2]);
    a.m = plan->window;
    a.quant_block_size = static_cast<int32_t>(PyLong_AsLong(args[3]));
    a.alpha = static_cast<float>(PyFloat_AsDouble(args[4]));
    a.beta1 = PyFloat_AsDouble(args[5]);
    a.beta2 = PyFloat_AsDouble(args[6]);
    a.eps = PyFloat_AsDouble(args[7]);
    if (PyErr_Occurred()) return nullptr;
    const int state = refresh(*plan, args[1]);
    if (state != 0) return state < 0 ? nullptr : PyLong_FromLong(1);
    std::optional<c10::cuda::CUDAGuard> guard;           // (the calls that can fail, before anything has changed)
    if (c10::cuda::current_device() != plan->device) guard.emplace(plan->device);
    void* stream = c10::cuda::getCurrentCUDAStream(plan->device).stream();
    size_t at = 0;                                       // every position has been read: now they advance (micro_adam.py:211)
    for (Group& g : plan->groups)
        for (Param& p : g.params)
            if (p.kind == Kind::Active && PyDict_SetItem(p.state, plan->key_index, plan->ring_next[plan->descs[at++].ring_index]) < 0) return nullptr;
    long status;
    {
        const ReleasedInterpreter other_threads_run;     // the copy of the table and the launches may wait for the GPU
        status = plan->fused_step(plan->descs.data(), static_cast<int>(plan->descs.size()), &a, plan->workspace, plan->workspace_bytes, stream);
    }
    return PyLong_FromLong(status);
} catch (...) {
    return raise_python();
}

PyMethodDef methods[] = {
    {"plan_new", plan_new, METH_VARARGS, "Lays the native form of a step out."},
    {"plan_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(plan_step)), METH_FASTCALL, "One fused step: 1 = the plan is stale, else the library's status."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_step_plan", "Native host side of MicroAdam.step().", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__step_plan(void) {
    PyObject* m = PyModule_Create(&module);
    if (m == nullptr) return nullptr;
    g_plan_type = reinterpret_cast<PyTypeObject*>(PyType_FromSpec(&plan_spec));
    if (g_plan_type == nullptr || PyModule_AddObjectRef(m, "Plan", reinterpret_cast<PyObject*>(g_plan_type)) < 0) { Py_DECREF(m); return nullptr; }
    return m;
}
