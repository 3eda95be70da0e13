// CPython binding of the device-tensor calls: the whole host path of one call -- argument checks, the result tensor, the
// current stream, the C-ABI entry -- in one native function.
//
// A decode GEMV is on the device for 4 to 10 microseconds.  The same path in Python (tensor attribute reads, torch.empty, a
// device context manager, ctypes) took 17 us a call, so every small launch was bound by it; here it takes 3 to 4 us, most of it
// the kernel launch itself.
//
// Each function takes its arguments by position and returns the result, or None when a call is not one it serves: a CPU
// tensor, a tensor subclass, a type, shape or layout that the Python wrapper converts or refuses.  The wrapper then takes its
// own path, which raises the error or does the conversion; nothing has been enqueued by then.  A non-zero return code of the
// C ABI raises the wrapper's RuntimeError.
//
// The C-ABI functions are reached through addresses handed over by bind(), so both bindings use the one loaded library.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "../../include/quactlize_b200.h"

namespace {

// ---- k-quant geometry (formats.py holds the same table for the Python side) ---------------------------------------------
struct Geo { int block, gs, lo, hi, sb_per_unit, unit; };
bool geometry(long q, Geo& g) {
  switch (q) {
    case 10: g = {84, 16, 2, 0, 1, 20}; return true;
    case 11: g = {110, 16, 2, 1, 2, 28}; return true;
    case 12: g = {144, 32, 4, 0, 1, 16}; return true;
    case 13: g = {176, 32, 4, 1, 1, 16}; return true;
    case 14: g = {210, 16, 4, 2, 2, 36}; return true;
    default: return false;
  }
}

// ---- the C ABI ------------------------------------------------------------------------------------------------------------
#define QB_ENTRIES(X)                                                                                                       \
  X(quactlize_ppu_vecdot_dense_dev_v1) X(quactlize_b200_vecdot_rows_dev_v1) X(quactlize_b200_vecdot_dense2_dev_v1)          \
  X(quactlize_b200_vecdot_moe_dev_v1) X(quactlize_b200_vecdot_moe_clamped_dev_v1)                                           \
  X(quactlize_b200_dequantize_dev_v1) X(quactlize_ppu_bc_gemv_dev_v1) X(quactlize_ppu_gemv_lowbit_dev_v1)                   \
  X(quactlize_b200_gemv_plane_dev_v1) X(quactlize_b200_gemm_plane_dev_v1)                                                   \
  X(quactlize_ppu_dense_fully_quantized_workspace_bytes_v1) X(quactlize_ppu_dense_fully_quantized_dev_v1)
struct Api {
#define X(name) decltype(&::name) name = nullptr;
  QB_ENTRIES(X)
#undef X
} api;

// ---- argument access ------------------------------------------------------------------------------------------------------
using T = at::Tensor;

// a plain (not subclassed) tensor, or nullptr
inline T const* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
inline bool integer(PyObject* o, int64_t& v) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0 && v >= INT32_MIN && v <= INT32_MAX;
}
inline bool on_cuda(T const& t) { return t.is_cuda() && t.is_contiguous() && !t.is_conj() && !t.is_neg(); }
inline bool same(T const& a, T const& b) { return a.get_device() == b.get_device(); }
inline bool bytes(T const* t, int64_t dim) { return t && on_cuda(*t) && t->scalar_type() == at::kByte && t->dim() == dim; }
inline bool halves(T const* t, int64_t dim) { return t && on_cuda(*t) && t->scalar_type() == at::kHalf && t->dim() == dim; }
inline bool halves_as(T const* t, int64_t a, int64_t b, int64_t c) {
  return halves(t, 3) && t->size(0) == a && t->size(1) == b && t->size(2) == c;
}
inline T empty(at::IntArrayRef shape, at::ScalarType dtype, T const& like) {
  return T(at::detail::empty_cuda(shape, dtype, like.device(), std::nullopt));
}
inline uint16_t const* u16(T const& t) { return static_cast<uint16_t const*>(t.const_data_ptr()); }
inline uint8_t const* u8(T const& t) { return static_cast<uint8_t const*>(t.const_data_ptr()); }
inline uint8_t const* u8_or_null(T const* t) { return t && t->numel() ? u8(*t) : nullptr; }

// `device` is made current for the call (a no-op when it is already), the GIL is dropped around the enqueue
struct Scope {
  c10::cuda::CUDAGuard guard;
  void* stream;
  explicit Scope(T const& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.get_device()).stream()) {}
};

PyObject* answer(int rc, char const* what, T&& out) {
  if (rc == 0) return THPVariable_Wrap(std::move(out));
  PyErr_Format(PyExc_RuntimeError, "%s failed in libquactlize_b200 (rc=%d%s)", what, rc,
               rc == 41 ? "; runtime failure, see stderr" : "");
  return nullptr;
}

#define QB_CALL(rc, expr)                                                   \
  int rc;                                                                   \
  { Py_BEGIN_ALLOW_THREADS rc = (expr); Py_END_ALLOW_THREADS }

// the GIL dropped for a scope that may throw
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// exceptions of torch (out of memory, ...) leave as Python exceptions
template <class F>
PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  return f();
  END_HANDLE_TH_ERRORS
}

// ---- raw blocks -----------------------------------------------------------------------------------------------------------
// (blocks, x, n, k, qtype): one activation row
PyObject* vecdot_dense(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t n, k, q;
    Geo g;
    T const *b = nargs == 5 ? tensor(a[0]) : nullptr, *x = b ? tensor(a[1]) : nullptr;
    if (!x || !integer(a[2], n) || !integer(a[3], k) || !integer(a[4], q) || !geometry(q, g) || n <= 0 || k <= 0 || k % 256 ||
        !bytes(b, 2) || b->size(1) != g.block || b->size(0) != n * (k / 256) ||
        !halves(x, 2) || x->size(0) != 1 || x->size(1) != k || !same(*b, *x)) Py_RETURN_NONE;
    Scope s(*b);
    T out = empty({1, n}, at::kFloat, *b);
    QB_CALL(rc, api.quactlize_ppu_vecdot_dense_dev_v1(u8(*b), g.block, u16(*x), static_cast<float*>(out.data_ptr()), int(n),
                                                      int(k / 256), int(q), s.stream));
    return answer(rc, "gguf_vecdot_dense", std::move(out));
  });
}

// (blocks, x, n, k, qtype, force_generic): m activation rows
PyObject* vecdot_rows(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t n, k, q, generic;
    Geo g;
    T const *b = nargs == 6 ? tensor(a[0]) : nullptr, *x = b ? tensor(a[1]) : nullptr;
    if (!x || !integer(a[2], n) || !integer(a[3], k) || !integer(a[4], q) || !integer(a[5], generic) || !geometry(q, g) || n <= 0 ||
        k <= 0 || k % 256 || !bytes(b, 2) || b->size(1) != g.block || b->size(0) != n * (k / 256) ||
        !halves(x, 2) || x->size(0) < 1 || x->size(1) != k || !same(*b, *x)) Py_RETURN_NONE;
    int64_t const m = x->size(0);
    Scope s(*b);
    T out = empty({m, n}, at::kFloat, *b);
    QB_CALL(rc, api.quactlize_b200_vecdot_rows_dev_v1(u8(*b), g.block, u16(*x), static_cast<float*>(out.data_ptr()), int(m), int(n),
                                                      int(k / 256), int(q), int(generic), s.stream));
    return answer(rc, "gguf_vecdot_rows", std::move(out));
  });
}

// (blocks, x, row_offsets, qtype).  The offsets are read back and checked, as in the wrapper.  The kernel that clamps offsets to
// the rows there are is enqueued while the copy is on its way, so the check costs the device nothing (3 tokens, 8 experts,
// 4096 -> 14336 Q4_K: 59 us a call with the check first, kernel 40); bad offsets raise after a launch whose result is dropped.
PyObject* vecdot_moe(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t q;
    Geo g;
    T const *b = nargs == 4 ? tensor(a[0]) : nullptr, *x = b ? tensor(a[1]) : nullptr, *off = x ? tensor(a[2]) : nullptr;
    if (!off || !integer(a[3], q) || !geometry(q, g) || !bytes(b, 3) || b->size(2) != g.block || !halves(x, 2) || !same(*b, *x) ||
        !on_cuda(*off) || !same(*x, *off) || off->scalar_type() != at::kInt || off->dim() != 1) Py_RETURN_NONE;
    int64_t const e = b->size(0), k = x->size(1), rows = x->size(0);
    if (e <= 0 || k <= 0 || k % 256 || rows <= 0 || b->size(1) <= 0 || b->size(1) % (k / 256) || off->numel() != e + 1) Py_RETURN_NONE;
    int64_t const n = b->size(1) / (k / 256);
    Scope s(*b);
    // a capture refuses the read-back: the wrapper says so
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) Py_RETURN_NONE;
    T out = empty({rows, n}, at::kFloat, *b);
    T host = at::empty({e + 1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    int most = 0, rc;
    bool good;
    {
      NoGil free;
      int const* dev = static_cast<int const*>(off->const_data_ptr());
      int* o = host.mutable_data_ptr<int>();
      auto const stream = c10::cuda::getCurrentCUDAStream(b->get_device());
      C10_CUDA_CHECK(cudaMemcpyAsync(o, dev, size_t(e + 1) * 4, cudaMemcpyDeviceToHost, stream));
      at::cuda::CUDAEvent arrived;
      arrived.record(stream);
      rc = api.quactlize_b200_vecdot_moe_clamped_dev_v1(u8(*b), g.block, u16(*x), dev, static_cast<float*>(out.data_ptr()), int(n),
                                                        int(k / 256), int(e), int(rows), int(q), s.stream);
      arrived.synchronize();
      good = o[0] == 0 && o[e] == rows;
      for (int64_t i = 0; good && i < e; ++i) {
        good = o[i + 1] >= o[i];
        most = std::max(most, o[i + 1] - o[i]);
      }
      if (good && rc == 40)                                            // a form that kernel does not cover
        rc = api.quactlize_b200_vecdot_moe_dev_v1(u8(*b), g.block, u16(*x), dev, static_cast<float*>(out.data_ptr()), int(n), int(k / 256),
                                                  int(e), int(rows), most, int(q), s.stream);
    }
    if (!good) Py_RETURN_NONE;
    return answer(rc, "gguf_vecdot_moe", std::move(out));
  });
}

// (blocks_a, blocks_b, x, n_a, n_b, k, qtype) -> (out_a, out_b)
PyObject* vecdot_dense2(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t na, nb, k, q;
    Geo g;
    T const *b0 = nargs == 7 ? tensor(a[0]) : nullptr, *b1 = b0 ? tensor(a[1]) : nullptr, *x = b1 ? tensor(a[2]) : nullptr;
    if (!x || !integer(a[3], na) || !integer(a[4], nb) || !integer(a[5], k) || !integer(a[6], q) || !geometry(q, g) || na <= 0 ||
        nb <= 0 || k <= 0 || k % 256 || !bytes(b0, 2) || !bytes(b1, 2) || b0->size(1) != g.block || b1->size(1) != g.block ||
        b0->size(0) != na * (k / 256) || b1->size(0) != nb * (k / 256) || !halves(x, 2) || x->size(0) != 1 || x->size(1) != k ||
        !same(*b0, *x) || !same(*b0, *b1)) Py_RETURN_NONE;
    Scope s(*b0);
    T oa = empty({1, na}, at::kFloat, *b0), ob = empty({1, nb}, at::kFloat, *b0);
    QB_CALL(rc, api.quactlize_b200_vecdot_dense2_dev_v1(u8(*b0), int(na), u8(*b1), int(nb), g.block, u16(*x),
                                                        static_cast<float*>(oa.data_ptr()), static_cast<float*>(ob.data_ptr()),
                                                        int(k / 256), int(q), s.stream));
    PyObject* pa = answer(rc, "gguf_vecdot_dense2", std::move(oa));
    if (!pa) return nullptr;
    PyObject* pb = THPVariable_Wrap(std::move(ob));
    PyObject* t = pb ? PyTuple_Pack(2, pa, pb) : nullptr;
    Py_DECREF(pa);
    Py_XDECREF(pb);
    return t;
  });
}

// (blocks, qtype) -> fp16 [rows, 256]
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t q;
    Geo g;
    T const* b = nargs == 2 ? tensor(a[0]) : nullptr;
    if (!b || !integer(a[1], q) || !geometry(q, g) || !bytes(b, 2) || b->size(1) != g.block || b->size(0) < 1 || b->size(0) > INT32_MAX) Py_RETURN_NONE;
    Scope s(*b);
    T out = empty({b->size(0), 256}, at::kHalf, *b);
    QB_CALL(rc, api.quactlize_b200_dequantize_dev_v1(u8(*b), g.block, static_cast<uint16_t*>(out.data_ptr()), int(b->size(0)), int(q), s.stream));
    return answer(rc, "gguf_dequantize", std::move(out));
  });
}

// ---- planes ---------------------------------------------------------------------------------------------------------------
// low [e,n,..], high of the format beside it (absent: None or empty); false = not served here
bool planes(T const* x, PyObject* low_o, PyObject* high_o, int lo, int hi, T const*& low, T const*& high, int64_t& e, int64_t& n, int64_t& k) {
  low = tensor(low_o);
  high = high_o == Py_None ? nullptr : tensor(high_o);
  if (high_o != Py_None && !high) return false;
  if (!x || !on_cuda(*x) || x->dim() != 2 || !bytes(low, 3) || !same(*x, *low)) return false;
  k = x->size(1); e = low->size(0); n = low->size(1);
  if (x->size(0) < 1 || e < 1 || n < 1 || n > INT32_MAX || k <= 0 || k % 256 || k > INT32_MAX || x->size(0) > INT32_MAX ||
      low->size(2) != k * lo / 8) return false;
  if (!hi) return !high || high->numel() == 0;
  return bytes(high, 3) && same(*x, *high) && high->size(0) == e && high->size(1) == n && high->size(2) == k * hi / 8;
}

// (a, low, high, units, qtype): dense merged artifact, one row
PyObject* gemv_bc(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t q, e, n, k;
    Geo g;
    T const *x = nargs == 5 ? tensor(a[0]) : nullptr, *low, *high, *u = x ? tensor(a[3]) : nullptr;
    if (!u || !integer(a[4], q) || !geometry(q, g) || !planes(x, a[1], a[2], g.lo, g.hi, low, high, e, n, k) || !halves(x, 2) ||
        x->size(0) != 1 || e != 1 || n % 256 || k % (256 * g.sb_per_unit) || !bytes(u, 3) || !same(*x, *u) ||
        u->size(0) != k / 256 / g.sb_per_unit || u->size(1) != n || u->size(2) != g.unit) Py_RETURN_NONE;
    Scope s(*x);
    T out = empty({1, n}, at::kFloat, *x);
    QB_CALL(rc, api.quactlize_ppu_bc_gemv_dev_v1(u16(*x), u8(*low), u8_or_null(high), u8(*u), nullptr, static_cast<float*>(out.data_ptr()),
                                                 1, int(n), int(k), 0, 1, int(q), s.stream));
    return answer(rc, "BC GEMV", std::move(out));
  });
}

// (a, low, high, scale, zero, qtype): dense scale-first artifact
PyObject* gemv_scale_first(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t q, e, n, k;
    Geo g;
    T const *x = nargs == 6 ? tensor(a[0]) : nullptr, *low, *high, *sc = x ? tensor(a[3]) : nullptr, *ze = sc ? tensor(a[4]) : nullptr;
    if (!ze || !integer(a[5], q) || !geometry(q, g) || !planes(x, a[1], a[2], g.lo, g.hi, low, high, e, n, k) || !halves(x, 2) ||
        e != 1 || n % 256 || !halves_as(sc, 1, k / g.gs, n) || !halves_as(ze, 1, k / g.gs, n) || !same(*x, *sc) || !same(*x, *ze)) Py_RETURN_NONE;
    int64_t const m = x->size(0);
    Scope s(*x);
    T out = empty({m, n}, at::kHalf, *x);
    QB_CALL(rc, api.quactlize_ppu_gemv_lowbit_dev_v1(u16(*x), u8(*low), u8_or_null(high), u16(*sc), u16(*ze), static_cast<uint16_t*>(out.data_ptr()),
                                                     int(m), int(n), int(k), g.gs, int(q), s.stream, nullptr));
    return answer(rc, "scale-first GEMV", std::move(out));
  });
}

// What gemv_plane and gemm_plane share: (a, low, high, scale, zero, bits_lo, bits_hi, group_size, code_offset, row_offsets, ...).
struct PlaneCall {
  T const *x, *low, *high, *sc, *ze, *off;
  int64_t e, n, k, m, lo, hi, gs, shift;
  bool bf16;
  bool read(PyObject* const* a) {
    x = tensor(a[0]);
    sc = x ? tensor(a[3]) : nullptr;
    ze = off = nullptr;
    if (!sc || !integer(a[5], lo) || !integer(a[6], hi) || !integer(a[7], gs) || !integer(a[8], shift)) return false;
    if (!(lo == 1 || lo == 2 || lo == 4) || hi < 0 || hi > 2 || gs <= 0) return false;
    if (!planes(x, a[1], hi ? a[2] : Py_None, int(lo), int(hi), low, high, e, n, k) || k % gs || !same(*x, *sc) || !halves_as(sc, e, k / gs, n)) return false;
    if (a[4] != Py_None && (!(ze = tensor(a[4])) || !halves_as(ze, e, k / gs, n) || !same(*x, *ze))) return false;
    if (a[9] != Py_None) {
      off = tensor(a[9]);
      if (!off || !on_cuda(*off) || !same(*x, *off) || off->scalar_type() != at::kInt || off->dim() != 1 || off->numel() != e + 1) return false;
    } else if (e != 1) {
      return false;
    }
    auto const t = x->scalar_type();
    if (t != at::kHalf && t != at::kBFloat16) return false;
    bf16 = t == at::kBFloat16;
    m = x->size(0);
    return true;
  }
};

// (..., out_dtype or None, max_rows or None)
PyObject* gemv_plane(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    PlaneCall c;
    // offsets without a row bound have to be read back first: the Python wrapper does that
    if (nargs != 12 || !c.read(a) || a[10] != Py_None || (c.off && a[11] == Py_None)) Py_RETURN_NONE;
    int64_t bound = c.m;
    if (c.off && (!integer(a[11], bound) || bound <= 0 || bound > std::max<int64_t>(c.m, 1))) Py_RETURN_NONE;
    Scope s(*c.x);
    T out = empty({c.m, c.n}, c.x->scalar_type(), *c.x);
    QB_CALL(rc, api.quactlize_b200_gemv_plane_dev_v1(c.x->const_data_ptr(), u8(*c.low), u8_or_null(c.high), u16(*c.sc), c.ze ? u16(*c.ze) : nullptr,
                                                     out.data_ptr(), int(c.m), int(c.n), int(c.k), int(c.lo), int(c.hi), int(c.gs), int(c.shift),
                                                     c.bf16 ? 1 : 0, c.bf16 ? 2 : 0, c.off ? int(c.e) : 0,
                                                     c.off ? static_cast<int const*>(c.off->const_data_ptr()) : nullptr, int(bound), s.stream));
    return answer(rc, "plane GEMV", std::move(out));
  });
}

PyObject* gemm_plane(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    PlaneCall c;
    if (nargs != 10 || !c.read(a)) Py_RETURN_NONE;
    Scope s(*c.x);
    T out = empty({c.m, c.n}, c.x->scalar_type(), *c.x);
    QB_CALL(rc, api.quactlize_b200_gemm_plane_dev_v1(c.x->const_data_ptr(), u8(*c.low), u8_or_null(c.high), u16(*c.sc), c.ze ? u16(*c.ze) : nullptr,
                                                     out.data_ptr(), int(c.m), int(c.n), int(c.k), int(c.lo), int(c.hi), int(c.gs), int(c.shift),
                                                     c.bf16 ? 1 : 0, c.off ? int(c.e) : 0,
                                                     c.off ? static_cast<int const*>(c.off->const_data_ptr()) : nullptr, s.stream));
    return answer(rc, "plane GEMM", std::move(out));
  });
}

// (a, low, high, units, qtype)
PyObject* dense_fully_quantized(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject* {
    int64_t q, e, n, k;
    Geo g;
    T const *x = nargs == 5 ? tensor(a[0]) : nullptr, *low, *high, *u = x ? tensor(a[3]) : nullptr;
    if (!u || !integer(a[4], q) || !geometry(q, g) || !planes(x, a[1], a[2], g.lo, g.hi, low, high, e, n, k) || !halves(x, 2) || e != 1 ||
        n % 256 || k % (256 * g.sb_per_unit) || !bytes(u, 3) || !same(*x, *u) || u->size(0) != k / 256 / g.sb_per_unit ||
        u->size(1) != n || u->size(2) != g.unit) Py_RETURN_NONE;
    int const m = int(x->size(0));
    int64_t const need = api.quactlize_ppu_dense_fully_quantized_workspace_bytes_v1(m, int(n), int(k), int(q));
    if (need < 0) Py_RETURN_NONE;
    Scope s(*x);
    T out = empty({m, n}, at::kHalf, *x), ws = empty({need}, at::kByte, *x);
    QB_CALL(rc, api.quactlize_ppu_dense_fully_quantized_dev_v1(u16(*x), u8(*low), u8_or_null(high), u8(*u), static_cast<uint16_t*>(out.data_ptr()), m,
                                                               int(n), int(k), int(q), ws.data_ptr(), need, s.stream));
    return answer(rc, "fully-quantized dense GEMM", std::move(out));
  });
}

// bind({name: address, ...}): the entries of the loaded library
PyObject* bind(PyObject*, PyObject* table) {
  if (!PyDict_Check(table)) { PyErr_SetString(PyExc_TypeError, "bind takes a dict of addresses"); return nullptr; }
#define X(name)                                                                                    \
  {                                                                                                \
    PyObject* v = PyDict_GetItemString(table, #name);                                              \
    if (!v) { PyErr_SetString(PyExc_KeyError, #name); return nullptr; }                            \
    void* p = PyLong_AsVoidPtr(v);                                                                 \
    if (!p) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, #name); return nullptr; }   \
    api.name = reinterpret_cast<decltype(api.name)>(p);                                            \
  }
  QB_ENTRIES(X)
#undef X
  Py_RETURN_NONE;
}

// entries(): the names bind() wants
PyObject* entries(PyObject*, PyObject*) {
#define X(name) #name,
  static char const* const names[] = {QB_ENTRIES(X)};
#undef X
  Py_ssize_t const count = Py_ssize_t(sizeof(names) / sizeof(names[0]));
  PyObject* t = PyTuple_New(count);
  for (Py_ssize_t i = 0; t && i < count; ++i) PyTuple_SET_ITEM(t, i, PyUnicode_FromString(names[i]));
  return t;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    FAST(vecdot_dense), FAST(vecdot_rows), FAST(vecdot_dense2), FAST(vecdot_moe), FAST(dequantize), FAST(gemv_bc), FAST(gemv_scale_first),
    FAST(gemv_plane), FAST(gemm_plane), FAST(dense_fully_quantized),
    {"bind", &bind, METH_O, nullptr}, {"entries", &entries, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
