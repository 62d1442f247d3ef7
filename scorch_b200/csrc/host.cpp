// Native front end of the small calls: one CPython call checks the tensors, allocates the result
// and the workspace from torch's allocator and calls the C ABI.
//
// Why: a product over a small matrix is a few microseconds of GPU work, and the Python path to it
// (argument checks, torch.empty, a device guard and a 17-argument ctypes call) costs 20 to 30.  The
// functions here return None for any operand that is not in the plain form (CUDA, contiguous,
// matching types and sizes); the caller then takes the Python path, which converts or raises, so
// every check and message lives in one place.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <dlfcn.h>
#include <stdlib.h>

#include <ATen/ATen.h>
#include <ATen/SparseCsrTensorUtils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "scorch_b200.h"

namespace {

struct Abi {
  decltype(&sb_last_error) last_error;
  decltype(&sb_spmm_csr_once_workspace_bytes) spmm_once_bytes;
  decltype(&sb_spmm_csr_once) spmm_once;
  decltype(&sb_spmm_wide_select) spmm_wide_select;
  decltype(&sb_spmv_csr_tiled_scratch_bytes) spmv_bytes;
  decltype(&sb_spmv_csr_tiled) spmv;
  decltype(&sb_sddmm_coo_f32) sddmm_coo;
  decltype(&sb_sddmm_csr_f32) sddmm_csr;
  decltype(&sb_sparse_attention_scratch_bytes) attention_bytes;
  decltype(&sb_sparse_attention_csr_f32) attention_csr;
  decltype(&sb_sparse_attention_band_f32) attention_band;
  decltype(&sb_spgemm_workspace_bytes) spgemm_bytes;
  decltype(&sb_spgemm_begin) spgemm_begin;
  decltype(&sb_spgemm_rows) spgemm_rows;
  decltype(&sb_spgemm_finish) spgemm_finish;
} abi;
bool bound = false;
PyObject *error_class = nullptr, *oom_class = nullptr;

// A tensor argument, or null when the object is not a torch.Tensor.
const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

bool plain(const at::Tensor& t, at::ScalarType type) {
  return t.is_cuda() && t.layout() == at::kStrided && t.scalar_type() == type && t.is_contiguous();
}
bool indices(const at::Tensor& t) { return plain(t, at::kInt) && t.dim() == 1; }

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SB_F32;
    case at::kDouble: return SB_F64;
    case at::kInt: return SB_I32;
    case at::kLong: return SB_I64;
    default: return -1;
  }
}

PyObject* fail(int rc) {
  PyObject* args = Py_BuildValue("(is)", rc, abi.last_error());
  if (args) {
    PyObject* e = PyObject_CallObject(error_class, args);
    Py_DECREF(args);
    if (e) {
      PyErr_SetObject(error_class, e);
      Py_DECREF(e);
    }
  }
  return nullptr;
}

// The caller asked for every operand to be checked: the Python path does that.
bool checking() {
  const char* v = getenv("SCORCH_B200_VALIDATE");
  return v && v[0] == '1' && v[1] == 0;
}

at::Tensor workspace(size_t bytes, const at::Tensor& like) {
  return at::empty({(int64_t)(bytes > 16 ? bytes : 16)}, like.options().dtype(at::kByte));
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// C++ exceptions (the allocator out of memory, ...) as Python ones; None = not in the plain form.
template <typename F>
PyObject* guarded(F&& f) {
  if (!bound) Py_RETURN_NONE;
  try {
    return f();
  } catch (const c10::OutOfMemoryError& e) {
    PyErr_SetString(oom_class, e.what());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// The interpreter is free for other threads while one of these lives: around calls that wait for the
// device.  Nothing of Python is touched meanwhile.
class Unlocked {
  PyThreadState* const state = PyEval_SaveThread();

 public:
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  Unlocked& operator=(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// pos, crd, val of a matrix times B (rows x k): the common part of the entry points below.
PyObject* spmm(const at::Tensor& pos, const at::Tensor& crd, const at::Tensor& val, const at::Tensor& B,
               const at::Tensor* bias, bool relu, int64_t n) {
  const int code = dtype_code(val.scalar_type());
  if (code < 0 || !indices(pos) || !indices(crd) || !plain(val, val.scalar_type()) || val.dim() != 1 ||
      B.dim() != 2 || !plain(B, val.scalar_type()) || val.numel() != crd.numel() || pos.numel() < 1 ||
      (n >= 0 && n != B.size(0)) || checking())
    Py_RETURN_NONE;
  const int64_t m = pos.numel() - 1, k = B.size(1), nnz = crd.numel();
  if (bias && (code != SB_F32 || !plain(*bias, at::kFloat) || bias->numel() != k)) Py_RETURN_NONE;
  if (code == SB_F32 ? (k >= 512 && abi.spmm_wide_select(-1) == 1) : (k > 65535 * 32 || relu)) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard device(B.device());
  at::Tensor out = at::empty({m, k}, val.options());
  const size_t bytes = abi.spmm_once_bytes(code, k, nnz);
  at::Tensor ws = workspace(bytes, out);
  const int rc = abi.spmm_once(code, m, B.size(0), k, nnz, pos.const_data_ptr<int>(), crd.const_data_ptr<int>(),
                               val.const_data_ptr(), B.const_data_ptr(), k, bias ? bias->const_data_ptr() : nullptr,
                               relu, 0, out.data_ptr(), k, ws.data_ptr(), bytes > 16 ? bytes : 16, stream_of(B));
  return rc == SB_OK ? THPVariable_Wrap(std::move(out)) : fail(rc);
}

PyObject* spmv(const at::Tensor& pos, const at::Tensor& crd, const at::Tensor& val, const at::Tensor& x) {
  const int code = dtype_code(val.scalar_type());
  if (code < 0 || !indices(pos) || !indices(crd) || !plain(val, val.scalar_type()) || val.dim() != 1 ||
      x.dim() != 1 || !plain(x, val.scalar_type()) || val.numel() != crd.numel() || pos.numel() < 1 || checking())
    Py_RETURN_NONE;
  const int64_t m = pos.numel() - 1, nnz = crd.numel();
  const c10::cuda::CUDAGuard device(x.device());
  at::Tensor y = at::empty({m}, val.options());
  const size_t bytes = abi.spmv_bytes(code, nnz);
  at::Tensor ws = workspace(bytes, y);
  const int rc = abi.spmv(code, m, x.numel(), nnz, pos.const_data_ptr<int>(), crd.const_data_ptr<int>(),
                          val.const_data_ptr(), x.const_data_ptr(), y.data_ptr(), ws.data_ptr(), bytes, stream_of(x));
  return rc == SB_OK ? THPVariable_Wrap(std::move(y)) : fail(rc);
}

// ---- Python functions ---------------------------------------------------------------------------
// bind(path of libscorch_b200.so, class of ABI errors, class of allocation errors)
PyObject* py_bind(PyObject*, PyObject* args) {
  const char* path;
  PyObject *cls, *oom;
  if (!PyArg_ParseTuple(args, "sOO", &path, &cls, &oom)) return nullptr;
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!lib) return PyErr_Format(PyExc_ImportError, "%s", dlerror());
  bool ok = true;
  auto find = [&](auto& f, const char* name) {
    f = reinterpret_cast<std::decay_t<decltype(f)>>(dlsym(lib, name));
    ok = ok && f;
  };
  find(abi.last_error, "sb_last_error");
  find(abi.spmm_once_bytes, "sb_spmm_csr_once_workspace_bytes");
  find(abi.spmm_once, "sb_spmm_csr_once");
  find(abi.spmm_wide_select, "sb_spmm_wide_select");
  find(abi.spmv_bytes, "sb_spmv_csr_tiled_scratch_bytes");
  find(abi.spmv, "sb_spmv_csr_tiled");
  find(abi.sddmm_coo, "sb_sddmm_coo_f32");
  find(abi.sddmm_csr, "sb_sddmm_csr_f32");
  find(abi.attention_bytes, "sb_sparse_attention_scratch_bytes");
  find(abi.attention_csr, "sb_sparse_attention_csr_f32");
  find(abi.attention_band, "sb_sparse_attention_band_f32");
  find(abi.spgemm_bytes, "sb_spgemm_workspace_bytes");
  find(abi.spgemm_begin, "sb_spgemm_begin");
  find(abi.spgemm_rows, "sb_spgemm_rows");
  find(abi.spgemm_finish, "sb_spgemm_finish");
  if (!ok) return PyErr_Format(PyExc_ImportError, "%s lacks a symbol of the C ABI", path);
  Py_INCREF(cls);
  Py_INCREF(oom);
  Py_XDECREF(error_class);
  Py_XDECREF(oom_class);
  error_class = cls;
  oom_class = oom;
  bound = true;
  Py_RETURN_NONE;
}

// spmm(pos, crd, val, B, bias | None, relu, n | -1) -> (m, k) tensor or None
PyObject* py_spmm(PyObject*, PyObject* const* a, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 7) Py_RETURN_NONE;
    const at::Tensor *pos = tensor(a[0]), *crd = tensor(a[1]), *val = tensor(a[2]), *B = tensor(a[3]);
    const at::Tensor* bias = a[4] == Py_None ? nullptr : tensor(a[4]);
    if (!pos || !crd || !val || !B || (a[4] != Py_None && !bias)) Py_RETURN_NONE;
    const int relu = PyObject_IsTrue(a[5]);
    const long long n = PyLong_AsLongLong(a[6]);
    if (relu < 0 || (n == -1 && PyErr_Occurred())) return nullptr;
    return spmm(*pos, *crd, *val, *B, bias, relu == 1, n);
  });
}

PyObject* py_spmv(PyObject*, PyObject* const* a, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 4) Py_RETURN_NONE;
    const at::Tensor *pos = tensor(a[0]), *crd = tensor(a[1]), *val = tensor(a[2]), *x = tensor(a[3]);
    if (!pos || !crd || !val || !x) Py_RETURN_NONE;
    return spmv(*pos, *crd, *val, *x);
  });
}

// matmul_csr(A torch CSR, B dense matrix or vector) -> tensor or None
PyObject* py_matmul_csr(PyObject*, PyObject* const* a, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 2) Py_RETURN_NONE;
    const at::Tensor *A = tensor(a[0]), *B = tensor(a[1]);
    if (!A || !B || A->layout() != at::kSparseCsr || A->dim() != 2 || B->layout() != at::kStrided || B->dim() < 1)
      Py_RETURN_NONE;
    const auto* csr = at::sparse_csr::get_sparse_csr_impl(*A);
    const at::Tensor &pos = csr->compressed_indices(), &crd = csr->plain_indices(), &val = csr->values();
    if (B->dim() == 1) return spmv(pos, crd, val, *B);
    return spmm(pos, crd, val, *B, nullptr, false, -1);
  });
}

// sddmm(row or pos, col, mask_val, Q, K, csr) -> values, or (values, row, col) for a CSR mask, or None
PyObject* py_sddmm(PyObject*, PyObject* const* a, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 6) Py_RETURN_NONE;
    const at::Tensor *row = tensor(a[0]), *col = tensor(a[1]), *val = tensor(a[2]), *Q = tensor(a[3]), *K = tensor(a[4]);
    const int csr = PyObject_IsTrue(a[5]);
    if (csr < 0) return nullptr;
    if (!row || !col || !val || !Q || !K || !indices(*row) || !indices(*col) || !plain(*val, at::kFloat) ||
        !plain(*Q, at::kFloat) || !plain(*K, at::kFloat) || Q->dim() != 2 || K->dim() != 2 ||
        Q->size(1) != K->size(1) || val->numel() != col->numel() ||
        (csr ? row->numel() != Q->size(0) + 1 : row->numel() != col->numel()) || checking())
      Py_RETURN_NONE;
    const int64_t m = Q->size(0), n = K->size(0), d = Q->size(1), nnz = col->numel();
    const c10::cuda::CUDAGuard device(Q->device());
    at::Tensor out = at::empty({nnz}, Q->options());
    int rc;
    if (!csr) {
      rc = abi.sddmm_coo(m, n, d, nnz, row->const_data_ptr<int>(), col->const_data_ptr<int>(),
                         val->const_data_ptr<float>(), Q->const_data_ptr<float>(), d, K->const_data_ptr<float>(), d,
                         out.data_ptr<float>(), 1, 0, 0, 0, stream_of(*Q));
      return rc == SB_OK ? THPVariable_Wrap(std::move(out)) : fail(rc);
    }
    at::Tensor orow = at::empty({nnz}, row->options()), ocol = at::empty({nnz}, row->options());
    rc = abi.sddmm_csr(m, n, d, nnz, row->const_data_ptr<int>(), col->const_data_ptr<int>(),
                       val->const_data_ptr<float>(), Q->const_data_ptr<float>(), d, K->const_data_ptr<float>(), d,
                       out.data_ptr<float>(), orow.data_ptr<int>(), ocol.data_ptr<int>(), 1, 0, 0, 0, stream_of(*Q));
    if (rc != SB_OK) return fail(rc);
    return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(out)), THPVariable_Wrap(std::move(orow)),
                         THPVariable_Wrap(std::move(ocol)));
  });
}

// attention(pos, crd, mask_val | None, Q, K, V, scale, plan buffer, plan rows, plan columns, blocks | -1
// (band plan), entries outside) -> O or None
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 12) Py_RETURN_NONE;
    const at::Tensor *pos = tensor(a[0]), *crd = tensor(a[1]), *Q = tensor(a[3]), *K = tensor(a[4]), *V = tensor(a[5]),
                     *plan = tensor(a[7]);
    const at::Tensor* val = a[2] == Py_None ? nullptr : tensor(a[2]);
    if (!pos || !crd || !Q || !K || !V || !plan || (a[2] != Py_None && !val)) Py_RETURN_NONE;
    const double scale = PyFloat_AsDouble(a[6]);
    const long long pm = PyLong_AsLongLong(a[8]), pn = PyLong_AsLongLong(a[9]), blocks = PyLong_AsLongLong(a[10]),
                    rem = PyLong_AsLongLong(a[11]);
    if (PyErr_Occurred()) return nullptr;
    if (!indices(*pos) || !indices(*crd) || (val && (!plain(*val, at::kFloat) || val->numel() != crd->numel())) ||
        !plain(*Q, at::kFloat) || !plain(*K, at::kFloat) || !plain(*V, at::kFloat) || Q->dim() < 2 || Q->dim() > 3 ||
        K->dim() != Q->dim() || K->sizes() != V->sizes() || checking())
      Py_RETURN_NONE;
    const bool batched = Q->dim() == 3;
    const int64_t m = Q->size(-2), d = Q->size(-1), n = K->size(-2), nnz = crd->numel(), batch = batched ? Q->size(0) : 1;
    if (pos->numel() != m + 1 || pm != m || pn != n || K->size(-1) != d || (batched && K->size(0) != batch) ||
        (blocks < 0 ? d != 64 : (d != 32 && d != 64)))
      Py_RETURN_NONE;
    const c10::cuda::CUDAGuard device(Q->device());
    at::Tensor out = at::empty(Q->sizes(), Q->options());
    const size_t bytes = abi.attention_bytes(m, rem, batch);
    at::Tensor ws = workspace(bytes, out);
    const int *p = pos->const_data_ptr<int>(), *c = crd->const_data_ptr<int>();
    const float *w = val ? val->const_data_ptr<float>() : nullptr, *q = Q->const_data_ptr<float>(),
                *k = K->const_data_ptr<float>(), *v = V->const_data_ptr<float>();
    const int rc =
        blocks < 0
            ? abi.attention_band(m, n, d, nnz, p, c, w, q, d, k, d, v, d, (float)scale, out.data_ptr<float>(), d, batch,
                                 m * d, n * d, n * d, m * d, plan->const_data_ptr(), rem, ws.data_ptr(), bytes,
                                 SB_ATTN_ALL_STAGES, stream_of(*Q))
            : abi.attention_csr(m, n, d, nnz, p, c, w, q, d, k, d, v, d, (float)scale, out.data_ptr<float>(), d, batch,
                                m * d, n * d, n * d, m * d, plan->const_data_ptr(), blocks, rem, ws.data_ptr(), bytes,
                                SB_ATTN_ALL_STAGES, stream_of(*Q));
    return rc == SB_OK ? THPVariable_Wrap(std::move(out)) : fail(rc);
  });
}

// C = A B in one pass; kTwoPhases where the products need more memory than that form may take.
constexpr int64_t kOnePassBytes = (int64_t)16 << 30;
constexpr int kTwoPhases = -1;

int spgemm(int code, const at::Tensor& apos, const at::Tensor& acrd, const at::Tensor& aval, const at::Tensor& bpos,
           const at::Tensor& bcrd, const at::Tensor& bval, int64_t n, at::Tensor& cpos, at::Tensor& ccrd,
           at::Tensor& cval) {
  const int64_t m = apos.numel() - 1, kb = bpos.numel() - 1, size = aval.element_size();
  const c10::cuda::CUDAGuard device(aval.device());
  void* stream = stream_of(aval);
  const size_t bytes = abi.spgemm_bytes(m, n, code);
  at::Tensor ws = workspace(bytes, aval), off = at::empty({m + 1}, apos.options());
  int64_t counts[5], products = 0, total = 0;
  const int *ap = apos.const_data_ptr<int>(), *ac = acrd.const_data_ptr<int>();
  const int *bp = bpos.const_data_ptr<int>(), *bc = bcrd.const_data_ptr<int>();
  int rc = abi.spgemm_begin(m, kb, n, ap, ac, bp, off.data_ptr<int>(), counts, &products, ws.data_ptr(), bytes, stream);
  if (rc != SB_OK) return rc;
  if (products > INT32_MAX || products * (4 + size) > kOnePassBytes) return kTwoPhases;
  cpos = at::empty({m + 1}, apos.options());
  at::Tensor tcrd, tval;
  try {
    tcrd = at::empty({products}, apos.options());
    tval = at::empty({products}, aval.options());
  } catch (const c10::OutOfMemoryError&) {
    return kTwoPhases;
  }
  rc = abi.spgemm_rows(code, m, kb, n, ap, ac, aval.const_data_ptr(), bp, bc, bval.const_data_ptr(),
                       off.data_ptr<int>(), counts, tcrd.data_ptr<int>(), tval.data_ptr(), cpos.data_ptr<int>(), &total,
                       ws.data_ptr(), bytes, stream);
  if (rc != SB_OK) return rc;
  if (total == products) {     // no two products met: the rows are in place already
    ccrd = tcrd;
    cval = tval;
    return SB_OK;
  }
  try {
    ccrd = at::empty({total}, apos.options());
    cval = at::empty({total}, aval.options());
  } catch (const c10::OutOfMemoryError&) {
    return kTwoPhases;
  }
  return abi.spgemm_finish(code, m, total, off.data_ptr<int>(), tcrd.data_ptr<int>(), tval.data_ptr(),
                           cpos.data_ptr<int>(), ccrd.data_ptr<int>(), cval.data_ptr(), stream);
}

// spgemm(Apos, Acrd, Aval, Bpos, Bcrd, Bval, n) -> (Cpos, Ccrd, Cval), or None: not in the plain
// form, or more products than the one-pass form has memory for
PyObject* py_spgemm(PyObject*, PyObject* const* a, Py_ssize_t count) {
  return guarded([&]() -> PyObject* {
    if (count != 7) Py_RETURN_NONE;
    const at::Tensor* t[6];
    for (int i = 0; i < 6; i++)
      if (!(t[i] = tensor(a[i]))) Py_RETURN_NONE;
    const long long n = PyLong_AsLongLong(a[6]);
    if (n == -1 && PyErr_Occurred()) return nullptr;
    // (copies: the wait for the device lets other threads run)
    const at::Tensor apos = *t[0], acrd = *t[1], aval = *t[2], bpos = *t[3], bcrd = *t[4], bval = *t[5];
    const int code = dtype_code(aval.scalar_type());
    if (code < 0 || !indices(apos) || !indices(acrd) || !indices(bpos) || !indices(bcrd) ||
        !plain(aval, aval.scalar_type()) || !plain(bval, aval.scalar_type()) || aval.dim() != 1 || bval.dim() != 1 ||
        aval.numel() != acrd.numel() || bval.numel() != bcrd.numel() || apos.numel() < 1 || bpos.numel() < 1 ||
        checking())
      Py_RETURN_NONE;
    at::Tensor cpos, ccrd, cval;
    int rc;
    {
      const Unlocked unlocked;
      rc = spgemm(code, apos, acrd, aval, bpos, bcrd, bval, n, cpos, ccrd, cval);
    }
    if (rc == kTwoPhases) Py_RETURN_NONE;
    if (rc != SB_OK) return fail(rc);
    return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(cpos)), THPVariable_Wrap(std::move(ccrd)),
                         THPVariable_Wrap(std::move(cval)));
  });
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, "bind(path, error_class, oom_class): resolve the C ABI"},
    {"spmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_spmm)), METH_FASTCALL,
     "spmm(pos, crd, val, B, bias, relu, n) -> tensor, or None for the general path"},
    {"spmv", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_spmv)), METH_FASTCALL,
     "spmv(pos, crd, val, x) -> tensor, or None for the general path"},
    {"matmul_csr", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_matmul_csr)), METH_FASTCALL,
     "matmul_csr(A, B) for a torch CSR tensor A -> tensor, or None for the general path"},
    {"sddmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sddmm)), METH_FASTCALL,
     "sddmm(row_or_pos, col, mask_val, Q, K, csr) -> tensor(s), or None for the general path"},
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL,
     "attention(pos, crd, mask_val, Q, K, V, scale, plan, m, n, blocks, rem) -> tensor, or None for the general path"},
    {"spgemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_spgemm)), METH_FASTCALL,
     "spgemm(Apos, Acrd, Aval, Bpos, Bcrd, Bval, n) -> (Cpos, Ccrd, Cval), or None for the two-phase path"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
