/**
 * Host side of the one-kernel AdamW update (csrc/kernels/adamw.cu) for dccl_b200/parallel/zero.py, which has the same in Python for
 * where this extension is missing: the checks of a slice's
 * options and state, its step count, the launch on torch's current stream and the version counters. About forty attribute
 * look-ups and tensor calls per slice: made from Python a step of 0.4 M parameters takes 12.8 us, and 5.6 from here.
 *
 * Plain CPython functions: their arguments are borrowed and not converted. Everything that could throw is caught at this border.
 */
#include "adamw_step.hpp"
#include "../kernels/adamw.hpp"
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>

namespace {

using FlatUpdate = decltype(&dccl_adamw_flat);

/** ncclDataType_t of the parameters' types that the kernel takes, or -1. */
int flat_dtype(at::ScalarType t) { return t == at::kHalf ? 6 : t == at::kFloat ? 7 : t == at::kBFloat16 ? 9 : -1; }

/** The keys of torch's parameter groups and optimizer state, made once: a look-up then hashes nothing. */
struct Keys {
    PyObject *amsgrad, *maximize, *capturable, *differentiable, *fused, *decoupled_weight_decay, *betas, *lr, *weight_decay, *eps, *step, *exp_avg, *exp_avg_sq;
} key;

bool is_plain_tensor(PyObject* o) { return o && (PyObject*)Py_TYPE(o) == THPVariableClass; }

/** An fp32 tensor of torch's own class with `n` elements in a row on `device`. */
bool is_flat_fp32(PyObject* o, int64_t n, c10::Device device) {
    if (!is_plain_tensor(o)) return false;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.scalar_type() == at::kFloat && t.device() == device && t.numel() == n && t.is_contiguous();
}

/** A Python number (no tensor, no array scalar of another type). */
bool number(PyObject* o, double* v) {
    if (!o || !(PyFloat_Check(o) || PyLong_Check(o))) return false;
    *v = PyFloat_AsDouble(o);
    if (*v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
}

/** Whether Python takes `o` for true; what has no truth value, and a missing option, is left to torch to report (-1). */
int truth(PyObject* o) {
    if (o == Py_False || o == Py_None) return 0;
    if (o == Py_True) return 1;
    if (!o) return -1;
    const int t = PyObject_IsTrue(o);
    if (t < 0) PyErr_Clear();
    return t;
}

struct Options { double lr, weight_decay, eps, beta1, beta2; };

/** The options of a parameter group, when they are those of plain AdamW. Betas outside [0, 1), which torch refuses or fails on,
 *  are left to it. */
bool read_options(PyObject* group, Options* o) {
    for (PyObject* k : {key.amsgrad, key.maximize, key.capturable, key.differentiable, key.fused})
        if (truth(PyDict_GetItem(group, k)) != 0) return false;
    PyObject* decoupled = PyDict_GetItem(group, key.decoupled_weight_decay);
    if (decoupled && truth(decoupled) != 1) return false;
    PyObject* betas = PyDict_GetItem(group, key.betas);
    const THPObjectPtr pair(betas ? PySequence_Fast(betas, "") : nullptr);     // any two numbers in a row: an array, a list of a configuration file
    if (!pair) { PyErr_Clear(); return false; }
    return PySequence_Fast_GET_SIZE(pair.get()) == 2
           && number(PyDict_GetItem(group, key.lr), &o->lr) && number(PyDict_GetItem(group, key.weight_decay), &o->weight_decay)
           && number(PyDict_GetItem(group, key.eps), &o->eps)
           && number(PySequence_Fast_GET_ITEM(pair.get(), 0), &o->beta1) && number(PySequence_Fast_GET_ITEM(pair.get(), 1), &o->beta2)
           && o->beta1 >= 0 && o->beta1 < 1 && o->beta2 >= 0 && o->beta2 < 1;
}

/** A step count in plain memory of the host, which is read and changed in place. Anything else (another type, a subclass, an
 *  inference tensor, which torch may refuse to change) goes through torch. */
bool counts_in_place(PyObject* count, const at::Tensor& t) {
    return is_plain_tensor(count) && t.scalar_type() == at::kFloat && t.is_cpu() && t.numel() == 1 && t.layout() == at::kStrided
           && !t.is_inference() && !t.requires_grad() && !t.is_neg();
}

/** A step count of zero or more. Below zero the bias corrections divide by zero or have no square root, which torch's step reports. */
bool counts_up(PyObject* count) {
    if (counts_in_place(count, THPVariable_Unpack(count))) return *THPVariable_Unpack(count).const_data_ptr<float>() >= 0;
    const at::Tensor t = THPVariable_Unpack(count);        // a copy: item() can run Python
    return t.numel() == 1 && !t.is_complex() && t.item().toDouble() >= 0;
}

/** adamw_ready(param_group, state, master, master_grad, grad, n): whether the kernel can update this slice of n elements, now that
 *  nothing is being captured. */
PyObject* adamw_ready(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(nargs == 6, "adamw_ready takes six arguments");
    PyObject *group = args[0], *state = args[1];
    const int64_t n = PyLong_AsLongLong(args[5]);
    if (n == -1 && PyErr_Occurred()) return nullptr;
    Options o;
    if (!PyDict_Check(group) || !PyDict_Check(state) || !is_plain_tensor(args[2]) || !is_plain_tensor(args[4])) Py_RETURN_FALSE;
    const c10::Device device = THPVariable_Unpack(args[2]).device();
    if (!device.is_cuda() || flat_dtype(THPVariable_Unpack(args[4]).scalar_type()) < 0 || !read_options(group, &o)) Py_RETURN_FALSE;
    PyObject* count = PyDict_GetItem(state, key.step);
    if (!count || !THPVariable_Check(count) || THPVariable_Unpack(count).is_cuda() || !counts_up(count)) Py_RETURN_FALSE;
    for (PyObject* t : {args[2], args[3], PyDict_GetItem(state, key.exp_avg), PyDict_GetItem(state, key.exp_avg_sq)})
        if (!is_flat_fp32(t, n, device)) Py_RETURN_FALSE;
    return PyBool_FromLong(c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None);
    END_HANDLE_TH_ERRORS
}

/** Counts the step and returns its number. */
double next_step(PyObject* count) {
    const at::Tensor t = THPVariable_Unpack(count);
    if (counts_in_place(count, t)) {
        float* p = t.mutable_data_ptr<float>();
        const double now = (double)*p + 1;
        *p = (float)now;
        t.unsafeGetTensorImpl()->bump_version();
        return now;
    }
    const double now = t.item().toDouble() + 1;
    t.fill_(now);
    return now;
}

/** adamw_update(dccl_adamw_flat's address, param_group, state, master, master_grad, grad, out, n): one step of a slice that adamw_ready
 *  let through; returns what the launch returned. */
PyObject* adamw_update(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(nargs == 8, "adamw_update takes eight arguments");
    const auto update = reinterpret_cast<FlatUpdate>(PyLong_AsVoidPtr(args[0]));
    const int64_t n = PyLong_AsLongLong(args[7]);
    if (PyErr_Occurred()) return nullptr;
    Options o;
    TORCH_CHECK(update && PyDict_Check(args[1]) && PyDict_Check(args[2]) && read_options(args[1], &o), "adamw_update: options that adamw_ready refuses");
    PyObject *count = PyDict_GetItem(args[2], key.step), *exp_avg = PyDict_GetItem(args[2], key.exp_avg), *exp_avg_sq = PyDict_GetItem(args[2], key.exp_avg_sq);
    for (PyObject* x : {count, exp_avg, exp_avg_sq, args[3], args[4], args[5], args[6]}) TORCH_CHECK(x && THPVariable_Check(x), "adamw_update: no tensor");
    // copies: other threads may run Python while the kernel is launched
    const at::Tensor p = THPVariable_Unpack(args[3]), p_grad = THPVariable_Unpack(args[4]), grad = THPVariable_Unpack(args[5]), out = THPVariable_Unpack(args[6]);
    const at::Tensor m = THPVariable_Unpack(exp_avg), v = THPVariable_Unpack(exp_avg_sq);
    const double t = next_step(count);
    const int device = p.device().index(), dtype = flat_dtype(grad.scalar_type());
    void* const stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
    void *pp = p.data_ptr(), *pg = p_grad.data_ptr(), *pm = m.data_ptr(), *pv = v.data_ptr(), *po = out.data_ptr();
    const void* g = grad.data_ptr();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = update(device, dtype, (size_t)n, pp, pg, pm, pv, g, po, 1 - o.lr * o.weight_decay, 1 - o.beta1, o.beta2, 1 - o.beta2,
                o.lr / (1 - std::pow(o.beta1, t)), std::sqrt(1 - std::pow(o.beta2, t)), o.eps, stream);
    Py_END_ALLOW_THREADS
    if (rc == 0)
        for (const at::Tensor* x : {&p, &p_grad, &m, &v, &out})
            if (!x->is_inference()) x->unsafeGetTensorImpl()->bump_version();
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"adamw_ready", (PyCFunction)(void (*)())adamw_ready, METH_FASTCALL, "whether the one-kernel AdamW update can take a slice"},
    {"adamw_update", (PyCFunction)(void (*)())adamw_update, METH_FASTCALL, "one step of a slice; 0, or an error code after a message on stderr"},
    {nullptr, nullptr, 0, nullptr},
};

} // namespace

int add_adamw_step(PyObject* module) {
    const struct { PyObject** key; const char* name; } names[] = {
        {&key.amsgrad, "amsgrad"}, {&key.maximize, "maximize"}, {&key.capturable, "capturable"}, {&key.differentiable, "differentiable"},
        {&key.fused, "fused"}, {&key.decoupled_weight_decay, "decoupled_weight_decay"}, {&key.betas, "betas"}, {&key.lr, "lr"},
        {&key.weight_decay, "weight_decay"}, {&key.eps, "eps"}, {&key.step, "step"}, {&key.exp_avg, "exp_avg"}, {&key.exp_avg_sq, "exp_avg_sq"}};
    for (const auto& k : names)
        if (!(*k.key = PyUnicode_InternFromString(k.name))) return -1;
    return PyModule_AddFunctions(module, methods);
}
