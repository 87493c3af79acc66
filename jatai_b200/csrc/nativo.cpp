// Host half of the operator launcher in native code (a CPython extension): the format checks of the arguments, the allocation of the
// outputs and the call of a C-ABI entry point, which in Python cost three to five times the launch itself.  What is wrong with an
// argument is found and told by the Python checks of registro.py: these functions only say that something is.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

typedef long long A_;

inline const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

PyObject* E_memoria;      // torch.OutOfMemoryError

// in a catch block: the exception in flight as a Python error of the type that PyTorch's own functions raise for it
PyObject* erro_python() {
    try {
        throw;
    } catch (const c10::OutOfMemoryError& e) {
        PyErr_SetString(E_memoria, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    } catch (...) {
        PyErr_SetString(PyExc_RuntimeError, "unknown exception");
    }
    return nullptr;
}

// the two members of a pair that bloco_valido has passed
inline PyObject* const* par_de_args(PyObject* par) { return &PyTuple_GET_ITEM(par, 0); }

// (mantissas, exponents) of a block tensor with block length `blk`: int8, on a GPU, contiguous, exponents [R, C / blk]
bool bloco_valido(PyObject* par, int64_t blk, int64_t* R, int64_t* C) {
    if (!PyTuple_Check(par) || PyTuple_GET_SIZE(par) != 2) return false;
    const at::Tensor *m = tensor(PyTuple_GET_ITEM(par, 0)), *e = tensor(PyTuple_GET_ITEM(par, 1));
    if (!m || !e || m->scalar_type() != at::kChar || e->scalar_type() != at::kChar || !m->is_cuda() || !e->is_cuda()) return false;
    if (m->dim() != 2 || e->dim() != 2 || !m->is_contiguous() || !e->is_contiguous()) return false;
    *R = m->size(0);
    *C = m->size(1);
    return *C % blk == 0 && e->size(0) == *R && e->size(1) == *C / blk;
}

// blocos(blk, t1, t2, ...) -> (R1, C1, R2, C2, ...), or None when one of them is no block tensor
PyObject* blocos(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n < 2) { PyErr_SetString(PyExc_TypeError, "blocos(blk, tensor pair, ...)"); return nullptr; }
    const int64_t blk = PyLong_AsLongLong(args[0]);
    if (blk <= 0) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "block length"); return nullptr; }
    PyObject* r = PyTuple_New(2 * (n - 1));
    for (Py_ssize_t i = 1; r && i < n; i++) {
        int64_t R, C;
        if (!bloco_valido(args[i], blk, &R, &C)) { Py_DECREF(r); Py_RETURN_NONE; }
        PyObject *pr = PyLong_FromLongLong(R), *pc = PyLong_FromLongLong(C);
        PyTuple_SET_ITEM(r, 2 * (i - 1), pr);
        PyTuple_SET_ITEM(r, 2 * (i - 1) + 1, pc);
        if (!pr || !pc) { Py_DECREF(r); return nullptr; }
    }
    return r;
}

// cru((acc, e)) -> (R, C), or None: int32 accumulators and int16 exponents of one shape, on a GPU, contiguous, two dimensions
PyObject* cru(PyObject*, PyObject* par) {
    if (!PyTuple_Check(par) || PyTuple_GET_SIZE(par) != 2) Py_RETURN_NONE;
    const at::Tensor *a = tensor(PyTuple_GET_ITEM(par, 0)), *e = tensor(PyTuple_GET_ITEM(par, 1));
    if (!a || !e || a->scalar_type() != at::kInt || e->scalar_type() != at::kShort || !a->is_cuda() || !e->is_cuda()) Py_RETURN_NONE;
    if (a->dim() != 2 || a->sizes() != e->sizes() || !a->is_contiguous() || !e->is_contiguous()) Py_RETURN_NONE;
    return Py_BuildValue("(LL)", (long long)a->size(0), (long long)a->size(1));
}

at::Tensor vazio(at::IntArrayRef forma, at::ScalarType tipo, const at::Device& dev) { return at::detail::empty_cuda(forma, tipo, dev, c10::nullopt); }      // at::empty without the dispatcher

// a workspace; undefined where there is no memory for it (the library then takes the kernels that need none)
at::Tensor espaco(int64_t bytes, const at::Device& dev) {
    try {
        return vazio({bytes}, at::kByte, dev);
    } catch (const c10::OutOfMemoryError&) { return at::Tensor(); }
}

PyObject* par_de(at::Tensor a, at::Tensor b) {
    PyObject *pa = THPVariable_Wrap(std::move(a)), *pb = pa ? THPVariable_Wrap(std::move(b)) : nullptr;
    PyObject* r = pb ? PyTuple_Pack(2, pa, pb) : nullptr;
    Py_XDECREF(pa);
    Py_XDECREF(pb);
    return r;
}

// novo_bloco(like, R, C, blk) / novo_cru(like, R, C): uninitialised outputs on the device of the tensor `like`
PyObject* novo_bloco(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor* como = n == 4 ? tensor(args[0]) : nullptr;
    if (!como) { PyErr_SetString(PyExc_TypeError, "novo_bloco(tensor, R, C, blk)"); return nullptr; }
    const int64_t R = PyLong_AsLongLong(args[1]), C = PyLong_AsLongLong(args[2]), blk = PyLong_AsLongLong(args[3]);
    if (PyErr_Occurred()) return nullptr;
    try {
        return par_de(vazio({R, C}, at::kChar, como->device()), vazio({R, C / blk}, at::kChar, como->device()));
    } catch (...) { return erro_python(); }
}
PyObject* novo_cru(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor* como = n == 3 ? tensor(args[0]) : nullptr;
    if (!como) { PyErr_SetString(PyExc_TypeError, "novo_cru(tensor, R, C)"); return nullptr; }
    const int64_t R = PyLong_AsLongLong(args[1]), C = PyLong_AsLongLong(args[2]);
    if (PyErr_Occurred()) return nullptr;
    try {
        return par_de(vazio({R, C}, at::kInt, como->device()), vazio({R, C}, at::kShort, como->device()));
    } catch (...) { return erro_python(); }
}
// novo(like, type, d0, d1, ...): "u1" uint8, "i4" int32
PyObject* novo(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor* como = n >= 3 && n <= 6 ? tensor(args[0]) : nullptr;
    const char* t = como ? PyUnicode_AsUTF8(args[1]) : nullptr;
    if (!t) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "novo(tensor, type, d0, ...)"); return nullptr; }
    int64_t d[4];
    for (Py_ssize_t i = 2; i < n; i++) d[i - 2] = PyLong_AsLongLong(args[i]);
    if (PyErr_Occurred()) return nullptr;
    try {
        return THPVariable_Wrap(vazio(at::IntArrayRef(d, n - 2), t[0] == 'u' ? at::kByte : at::kInt, como->device()));
    } catch (...) { return erro_python(); }
}

// espaco_gemm(address of jt_gemm_ws_bytes, address of jt_stream_atual, like, M, N, K, mode) -> workspace tensor, or None where the product
// wants none.  The workspace goes back to PyTorch's allocator right after the launch, which is safe only where the library launches on the
// stream the allocator orders it by: on any other stream there is none, as where there is no memory for it, and the library takes the kernel
// that needs none.
PyObject* espaco_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    const at::Tensor* como = n == 7 ? tensor(args[2]) : nullptr;
    if (!como) { PyErr_SetString(PyExc_TypeError, "espaco_gemm(function, function, tensor, M, N, K, mode)"); return nullptr; }
    void *fb = PyLong_AsVoidPtr(args[0]), *fs = PyLong_AsVoidPtr(args[1]);
    int d[4];
    for (int i = 0; i < 4; i++) d[i] = (int)PyLong_AsLong(args[3 + i]);
    if (PyErr_Occurred()) return nullptr;
    if (!fb || !fs) Py_RETURN_NONE;
    if (reinterpret_cast<void* (*)()>(fs)() != (void*)c10::cuda::getCurrentCUDAStream(como->device().index()).stream()) Py_RETURN_NONE;
    const long long bytes = reinterpret_cast<long long (*)(int, int, int, int)>(fb)(d[0], d[1], d[2], d[3]);
    if (bytes <= 0) Py_RETURN_NONE;
    try {
        const at::Tensor ws = espaco(bytes, como->device());
        if (!ws.defined()) Py_RETURN_NONE;
        return THPVariable_Wrap(ws);
    } catch (...) { return erro_python(); }
}

// Entry points of the library take pointers and ints (long long for element counts) and return an int: every one of them is an integer
// argument of the x86-64 calling convention, passed in a 64-bit register or stack slot of which the callee reads what it declares, so one
// call through a pointer type with N 64-bit arguments serves every signature with N arguments.
int chama_ja(void* f, const A_* a, int n) {
#define C_(...) return reinterpret_cast<int (*)(__VA_ARGS__)>(f)
    switch (n) {
        case 1: C_(A_)(a[0]);
        case 2: C_(A_, A_)(a[0], a[1]);
        case 3: C_(A_, A_, A_)(a[0], a[1], a[2]);
        case 4: C_(A_, A_, A_, A_)(a[0], a[1], a[2], a[3]);
        case 5: C_(A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4]);
        case 6: C_(A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5]);
        case 7: C_(A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6]);
        case 8: C_(A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
        case 9: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8]);
        case 10: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9]);
        case 11: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10]);
        case 12: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11]);
        case 13: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12]);
        case 14: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13]);
        case 15: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14]);
        case 16: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15]);
        case 17: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16]);
        case 18: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17]);
        case 19: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17], a[18]);
        case 20: C_(A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_, A_)(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17], a[18], a[19]);
    }
#undef C_
    return -1;
}
// The call without the interpreter lock, as ctypes makes it: a launch waits while the GPU's queue is full, and other threads go on meanwhile.
int chama(void* f, const A_* a, int n) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = chama_ja(f, a, n);
    Py_END_ALLOW_THREADS
    return rc;
}

PyObject *S_op, *S_trecho, *S_entradas, *S_forma, *S_A[2], *S_B[2], *S_X[2], *S_qkv[2], *S_go[2], *S_P, *S_registra, *S_depois;

// The launch record {op, trecho, entradas, forma}: appended to a list - the registry's own - or, of anything else, given to its method
// registra(op, entradas, forma).  The launch id, or -1 with a Python error set.
Py_ssize_t anota(PyObject* reg, PyObject* op, PyObject* trecho, PyObject* entradas, PyObject* forma) {
    if (!PyList_Check(reg)) {
        PyObject* r = PyObject_CallMethodObjArgs(reg, S_registra, op, entradas, forma, nullptr);
        const Py_ssize_t kid = r ? PyLong_AsSsize_t(r) : -1;
        Py_XDECREF(r);
        if (kid < 0 && !PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "registra gave no launch id");
        return kid;
    }
    PyObject* d = PyDict_New();
    if (!d) return -1;
    const Py_ssize_t kid = PyList_GET_SIZE(reg);
    const bool certo = PyDict_SetItem(d, S_op, op) == 0 && PyDict_SetItem(d, S_trecho, trecho) == 0 && PyDict_SetItem(d, S_entradas, entradas) == 0 &&
                       PyDict_SetItem(d, S_forma, forma) == 0 && PyList_Append(reg, d) == 0;
    Py_DECREF(d);
    return certo ? kid : -1;
}
// The launch has returned `rc`: a list's owner sees to that; anything else is told, depois(launch id, rc).  False with a Python error set.
bool avisa(PyObject* reg, Py_ssize_t kid, int rc) {
    if (PyList_Check(reg)) return true;
    PyObject *k = PyLong_FromSsize_t(kid), *c = PyLong_FromLong(rc);
    PyObject* r = k && c ? PyObject_CallMethodObjArgs(reg, S_depois, k, c, nullptr) : nullptr;
    Py_XDECREF(k);
    Py_XDECREF(c);
    Py_XDECREF(r);
    return r != nullptr;
}

// lanca(function address, launch list or registry, op, section, names, tensors, ints, output shape) -> None, or (launch id, return code)
// Records the launch ({op, trecho, entradas, forma}; `names` name the first tensors, None skips one) and calls function(pointers..., ints...,
// launch id).  A None tensor is a null pointer.
PyObject* lanca(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 8 || !PyTuple_Check(args[4]) || !PyTuple_Check(args[5]) || !PyTuple_Check(args[6])) {
        PyErr_SetString(PyExc_TypeError, "lanca(function, launches, op, section, names, tensors, ints, shape)");
        return nullptr;
    }
    PyObject *lista = args[1], *nomes = args[4], *ts = args[5], *ints = args[6];
    const Py_ssize_t np = PyTuple_GET_SIZE(ts), ni = PyTuple_GET_SIZE(ints), nn = PyTuple_GET_SIZE(nomes);
    if (np + ni + 1 > 20 || nn > np) { PyErr_SetString(PyExc_ValueError, "too many arguments"); return nullptr; }
    A_ a[20];
    for (Py_ssize_t i = 0; i < np; i++) {
        PyObject* o = PyTuple_GET_ITEM(ts, i);
        if (o == Py_None) { a[i] = 0; continue; }
        const at::Tensor* t = tensor(o);
        if (!t) { PyErr_Format(PyExc_TypeError, "argument %zd is no tensor", i); return nullptr; }
        a[i] = (A_)(t->numel() ? t->data_ptr() : nullptr);
    }
    for (Py_ssize_t i = 0; i < ni; i++) a[np + i] = PyLong_AsLongLong(PyTuple_GET_ITEM(ints, i));
    void* f = PyLong_AsVoidPtr(args[0]);
    if (PyErr_Occurred()) return nullptr;
    if (!f) { PyErr_SetString(PyExc_ValueError, "null function"); return nullptr; }
    PyObject* ent = PyDict_New();
    if (!ent) return nullptr;
    for (Py_ssize_t i = 0; i < nn; i++)
        if (PyTuple_GET_ITEM(nomes, i) != Py_None && PyDict_SetItem(ent, PyTuple_GET_ITEM(nomes, i), PyTuple_GET_ITEM(ts, i)) != 0) { Py_DECREF(ent); return nullptr; }
    const Py_ssize_t kid = anota(lista, args[2], args[3], ent, args[7]);
    Py_DECREF(ent);
    if (kid < 0) return nullptr;
    a[np + ni] = (A_)kid;
    const int rc = chama(f, a, (int)(np + ni + 1));
    if (!avisa(lista, kid, rc)) return nullptr;
    if (rc == 0 || !PyList_Check(lista)) Py_RETURN_NONE;
    return Py_BuildValue("(ni)", kid, rc);
}

// gemm(address of jt_gemm_ws_bytes, of jt_stream_atual, of jt_gemm_ws, of jt_gemm_ext, blk, launch list or registry, op, section, mode, A, B, X or None, two
// outputs) -> the output (pair), or both; None where an argument is not as it should be (nothing was done), the return code where the launch
// failed.  The whole of a product in one call: checks, outputs, workspace, record, launch.
PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 13) { PyErr_SetString(PyExc_TypeError, "gemm(4 functions, blk, launches, op, section, mode, A, B, X, two)"); return nullptr; }
    void *fb = PyLong_AsVoidPtr(args[0]), *fs = PyLong_AsVoidPtr(args[1]), *fw = PyLong_AsVoidPtr(args[2]), *fe = PyLong_AsVoidPtr(args[3]);
    const int64_t blk = PyLong_AsLongLong(args[4]);
    const int modo = (int)PyLong_AsLong(args[8]), duas = PyObject_IsTrue(args[12]);
    if (PyErr_Occurred()) return nullptr;
    int64_t M, K, N, Kb, Mx, Nx;
    if (!fb || !fs || !fw || !fe || blk <= 0 || !bloco_valido(args[9], blk, &M, &K) || !bloco_valido(args[10], blk, &N, &Kb)) Py_RETURN_NONE;
    const bool tem_x = args[11] != Py_None;
    if (Kb != K || M % 64 || N % 128 || K % blk || (tem_x && (!bloco_valido(args[11], blk, &Mx, &Nx) || Mx != M || Nx != N))) Py_RETURN_NONE;
    try {
        const at::Tensor& a = *tensor(PyTuple_GET_ITEM(args[9], 0));
        const at::Device dev = a.device();
        A_ p[20] = {0};
        auto poe = [&](int i, PyObject* par) { for (int k = 0; k < 2; k++) p[i + k] = (A_)tensor(PyTuple_GET_ITEM(par, k))->data_ptr(); };
        poe(0, args[9]);
        poe(2, args[10]);
        at::Tensor m1, e1, m2, e2, ws;
        if (modo == 1) { m1 = vazio({M, N}, at::kInt, dev); e1 = vazio({M, N}, at::kShort, dev); }
        else { m1 = vazio({M, N}, at::kChar, dev); e1 = vazio({M, N / blk}, at::kChar, dev); }
        p[modo == 1 ? 6 : 4] = (A_)m1.data_ptr();
        p[modo == 1 ? 7 : 5] = (A_)e1.data_ptr();
        if (tem_x) poe(8, args[11]);
        if (duas) {
            m2 = vazio({M, N}, at::kChar, dev); e2 = vazio({M, N / blk}, at::kChar, dev);
            p[10] = (A_)m2.data_ptr(); p[11] = (A_)e2.data_ptr();
        }
        long long bytes = 0;
        if (reinterpret_cast<void* (*)()>(fs)() == (void*)c10::cuda::getCurrentCUDAStream(dev.index()).stream())
            bytes = reinterpret_cast<long long (*)(int, int, int, int)>(fb)((int)M, (int)N, (int)K, modo);
        int i = 14;                                                // (12, 13: no external row maxima)
        if (bytes > 0) ws = espaco(bytes, dev);
        if (ws.defined()) p[i++] = (A_)ws.data_ptr();
        p[i++] = M; p[i++] = N; p[i++] = K; p[i++] = modo;
        PyObject *ent = PyDict_New(), *forma = Py_BuildValue("(LL)", (long long)M, (long long)N);
        bool certo = ent && forma;
        for (int k = 0; k < 2 && certo; k++)
            certo = PyDict_SetItem(ent, S_A[k], PyTuple_GET_ITEM(args[9], k)) == 0 && PyDict_SetItem(ent, S_B[k], PyTuple_GET_ITEM(args[10], k)) == 0 &&
                    (!tem_x || PyDict_SetItem(ent, S_X[k], PyTuple_GET_ITEM(args[11], k)) == 0);
        const Py_ssize_t kid = certo ? anota(args[5], args[6], args[7], ent, forma) : -1;
        Py_XDECREF(ent);
        Py_XDECREF(forma);
        if (kid < 0) return nullptr;
        p[i++] = (A_)kid;
        const int rc = chama(ws.defined() ? fw : fe, p, i);
        if (!avisa(args[5], kid, rc)) return nullptr;
        if (rc && PyList_Check(args[5])) return PyLong_FromLong(rc);
        PyObject* r = par_de(std::move(m1), std::move(e1));
        if (!r || !duas) return r;
        PyObject* r2 = par_de(std::move(m2), std::move(e2));
        if (!r2) { Py_DECREF(r); return nullptr; }
        PyObject* dois = PyTuple_Pack(2, r, r2);
        Py_DECREF(r);
        Py_DECREF(r2);
        return dois;
    } catch (...) { return erro_python(); }
}

// atencao(address of jt_atencao_ws_bytes, of jt_stream_atual, of the entry point with a workspace, of the raw one without, blk, launch list or registry, op,
// section, QKV, dO or None, P or None, Bt, T, H, GA, limit, block outputs) -> forward: (output pair, P), backward (dO and P given): the output
// pair; None where an argument is not as it should be or there is no workspace for block outputs (nothing was done), the return code
// where the launch failed.  The whole of an attention call: checks, outputs, workspace, record, launch.
PyObject* atencao(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != 17) { PyErr_SetString(PyExc_TypeError, "atencao(4 functions, blk, launches, op, section, QKV, dO, P, Bt, T, H, GA, limit, blocks)"); return nullptr; }
    void *fb = PyLong_AsVoidPtr(args[0]), *fs = PyLong_AsVoidPtr(args[1]), *fw = PyLong_AsVoidPtr(args[2]), *fp = PyLong_AsVoidPtr(args[3]);
    const int64_t blk = PyLong_AsLongLong(args[4]), Bt = PyLong_AsLongLong(args[11]), T = PyLong_AsLongLong(args[12]), H = PyLong_AsLongLong(args[13]);
    const int GA = (int)PyLong_AsLong(args[14]), limite = (int)PyLong_AsLong(args[15]), blocos_ = PyObject_IsTrue(args[16]);
    if (PyErr_Occurred()) return nullptr;
    const bool tras = args[9] != Py_None;
    int64_t M, D3, Mg = 0, Dg = 0;
    if (!fb || !fs || !fw || !fp || blk <= 0 || Bt <= 0 || T <= 0 || H <= 0 || !bloco_valido(args[8], blk, &M, &D3)) Py_RETURN_NONE;
    const at::Tensor* P0 = tras ? tensor(args[10]) : nullptr;
    if (tras && (!P0 || !bloco_valido(args[9], blk, &Mg, &Dg))) Py_RETURN_NONE;
    const int64_t D = tras ? Dg : D3 / 3, hd = D / H;
    if (M != Bt * T || D3 != 3 * D || D != H * hd || (tras && Mg != M) || (hd != 4 && hd != 16 && hd != 64) || T % 32 || T > 1024 || Bt * H > INT32_MAX) Py_RETURN_NONE;
    try {
        PyObject* const* qkv = par_de_args(args[8]);
        PyObject* const* go = tras ? par_de_args(args[9]) : nullptr;
        const at::Tensor &q0 = *tensor(qkv[0]), &q1 = *tensor(qkv[1]);
        const at::Device dev = q0.device();
        const A_ pg = tras ? (A_)tensor(go[0])->data_ptr() : 0, pP = tras ? (A_)P0->data_ptr() : 0;
        at::Tensor ws, m, e, P;
        long long bytes = 0;
        if ((((A_)q0.data_ptr() | pg) & 7) == 0 && (pP & 15) == 0 &&
            reinterpret_cast<void* (*)()>(fs)() == (void*)c10::cuda::getCurrentCUDAStream(dev.index()).stream())
            bytes = reinterpret_cast<long long (*)(int, int, int, int, int, int)>(fb)((int)Bt, (int)T, (int)H, (int)D, GA, tras);
        if (bytes <= 0 && blocos_) Py_RETURN_NONE;
        const int64_t C = tras ? 3 * D : D;
        m = vazio({M, C}, blocos_ ? at::kChar : at::kInt, dev);
        e = vazio({M, blocos_ ? C / blk : C}, blocos_ ? at::kChar : at::kShort, dev);
        if (!tras) P = vazio({Bt * H, T, T}, at::kByte, dev);
        if (bytes > 0) ws = espaco(bytes, dev);
        const bool com_ws = ws.defined();
        if (!com_ws && blocos_) Py_RETURN_NONE;
        A_ p[20];
        int i = 0;
        if (tras) { p[i++] = pg; p[i++] = (A_)tensor(go[1])->data_ptr(); }
        p[i++] = (A_)q0.data_ptr();
        p[i++] = (A_)q1.data_ptr();
        if (tras) p[i++] = pP;
        if (com_ws && blocos_) { p[i++] = 0; p[i++] = 0; }
        p[i++] = (A_)m.data_ptr();
        p[i++] = (A_)e.data_ptr();
        if (com_ws && !blocos_) { p[i++] = 0; p[i++] = 0; }
        if (!tras) p[i++] = (A_)P.data_ptr();
        if (com_ws) p[i++] = (A_)ws.data_ptr();
        p[i++] = Bt; p[i++] = T; p[i++] = H; p[i++] = D; p[i++] = GA;
        if (tras) p[i++] = limite;
        PyObject *ent = PyDict_New(), *forma = Py_BuildValue("(LL)", (long long)M, (long long)C);
        bool certo = ent && forma;
        for (int k = 0; k < 2 && certo; k++) {
            certo = PyDict_SetItem(ent, S_qkv[k], qkv[k]) == 0;
            if (tras) certo = certo && PyDict_SetItem(ent, S_go[k], go[k]) == 0;
        }
        if (tras) certo = certo && PyDict_SetItem(ent, S_P, args[10]) == 0;
        const Py_ssize_t kid = certo ? anota(args[5], args[6], args[7], ent, forma) : -1;
        Py_XDECREF(ent);
        Py_XDECREF(forma);
        if (kid < 0) return nullptr;
        p[i++] = (A_)kid;
        const int rc = chama(com_ws ? fw : fp, p, i);
        if (!avisa(args[5], kid, rc)) return nullptr;
        if (rc && PyList_Check(args[5])) return PyLong_FromLong(rc);
        PyObject* r = par_de(std::move(m), std::move(e));
        if (!r || tras) return r;
        PyObject* Po = THPVariable_Wrap(std::move(P));
        PyObject* dois = Po ? PyTuple_Pack(2, r, Po) : nullptr;
        Py_DECREF(r);
        Py_XDECREF(Po);
        return dois;
    } catch (...) { return erro_python(); }
}

PyMethodDef metodos[] = {
    {"blocos", (PyCFunction)(void (*)(void))blocos, METH_FASTCALL, "shapes of block tensors, or None"},
    {"cru", cru, METH_O, "shape of a raw tensor, or None"},
    {"novo_bloco", (PyCFunction)(void (*)(void))novo_bloco, METH_FASTCALL, "uninitialised block tensor"},
    {"novo_cru", (PyCFunction)(void (*)(void))novo_cru, METH_FASTCALL, "uninitialised raw tensor"},
    {"novo", (PyCFunction)(void (*)(void))novo, METH_FASTCALL, "uninitialised tensor"},
    {"espaco_gemm", (PyCFunction)(void (*)(void))espaco_gemm, METH_FASTCALL, "workspace of a product, or None"},
    {"gemm", (PyCFunction)(void (*)(void))gemm, METH_FASTCALL, "a product: checks, outputs, workspace, record, launch"},
    {"atencao", (PyCFunction)(void (*)(void))atencao, METH_FASTCALL, "an attention call: checks, outputs, workspace, record, launch"},
    {"lanca", (PyCFunction)(void (*)(void))lanca, METH_FASTCALL, "records and performs a launch; None, or (launch id, error code)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef modulo = {PyModuleDef_HEAD_INIT, "_nativo", "host half of the operator launcher", -1, metodos, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__nativo(void) {
    PyObject* torch = PyImport_ImportModule("torch");
    E_memoria = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    Py_XDECREF(torch);
    if (!E_memoria) return nullptr;
    bool certo = true;
    auto nome = [&](PyObject*& d, const char* t) { certo = certo && (d = PyUnicode_InternFromString(t)) != nullptr; };
    nome(S_op, "op");
    nome(S_trecho, "trecho");
    nome(S_entradas, "entradas");
    nome(S_forma, "forma");
    for (int k = 0; k < 2; k++) {
        nome(S_A[k], k ? "EA" : "A");
        nome(S_B[k], k ? "EB" : "B");
        nome(S_X[k], k ? "XE" : "X");
        nome(S_qkv[k], k ? "qkvE" : "qkv");
        nome(S_go[k], k ? "goE" : "go");
    }
    nome(S_P, "P");
    nome(S_registra, "registra");
    nome(S_depois, "depois");
    PyObject* m = certo ? PyModule_Create(&modulo) : nullptr;
    if (m && PyModule_AddStringConstant(m, "MARCA", JT_MARCA) != 0) { Py_DECREF(m); return nullptr; }      // the versions it was built against
    return m;
}
