// Native form of the host launchers' regular path: reads shape, dtype, device and address of the torch tensors in C++ and
// calls the C entry point, where the Python launchers (kernels.py) spend several microseconds per call on attribute
// reads and ctypes argument conversion. Loaded as x17ai_b200._hostcall; the entry points' addresses come from
// the library that _lib.py has loaded.
//
// Every function returns None after a launch, the diagnostic's address (int) where the entry point returned one, and
// False where an argument is not exactly what the launch expects: the caller then runs the Python checks, which
// name the argument.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdint>

#include "../../include/x17ai_b200.h"

namespace {

#define X17_ENTRIES(X)               \
	X(x17ai_b200_attn_fwd_i8)        \
	X(x17ai_b200_attn_fwd_pv_fp8)    \
	X(x17ai_b200_attn_fwd_i8_scaled) \
	X(x17ai_b200_attn_decode_i8)     \
	X(x17ai_b200_attn_decode_i8_noalloc) \
	X(x17ai_b200_gemm_fwd)           \
	X(x17ai_b200_qkvg_fwd_i8)        \
	X(x17ai_b200_rms_norm)

#define X17_DECL(name) decltype(&name) p_##name = nullptr;
X17_ENTRIES(X17_DECL)
#undef X17_DECL

using at::Tensor;

constexpr int64_t ANY = -1;

enum Kind { I8, E4M3, BF16, F32, I32_OUT, U32_IN };

bool dtype_is(Tensor const &t, Kind k) {
	switch (t.scalar_type()) {
	case at::kChar: return k == I8;
	case at::kByte:
	case at::kFloat8_e4m3fn: return k == E4M3;
	case at::kBFloat16: return k == BF16;
	case at::kFloat: return k == F32;
	case at::kInt: return k == I32_OUT || k == U32_IN;
	case at::kUInt32: return k == U32_IN;
	default: return false;
	}
}
// X17AI_DTYPE_* of a GEMM operand
bool dtype_is(Tensor const &t, int32_t code) {
	switch (code) {
	case X17AI_DTYPE_INT8: return dtype_is(t, I8);
	case X17AI_DTYPE_E4M3: return dtype_is(t, E4M3);
	case X17AI_DTYPE_I32_RAW: return dtype_is(t, I32_OUT);
	default: return false;
	}
}

// A regular device tensor: contiguous, on the GPU, no empty dimension.
struct Arg {
	Tensor const *t = nullptr;
	bool ok = true;   // an absent (None) argument is fine where the caller allows it
	explicit Arg(PyObject *o, bool may_be_none = false) {
		if (may_be_none && o == Py_None) return;
		ok = THPVariable_Check(o);
		if (!ok) return;
		t = &THPVariable_Unpack(o);
		ok = t->is_cuda() && t->is_contiguous() && t->numel() > 0;
	}
	bool none() const { return t == nullptr; }
	void *ptr() const { return t == nullptr ? nullptr : t->data_ptr(); }
	template <typename K>
	bool is2(int64_t rows, int64_t cols, K kind) const {
		return ok && t->dim() == 2 && (rows == ANY || t->size(0) == rows) && (cols == ANY || t->size(1) == cols) && dtype_is(*t, kind);
	}
	// [rows, cols], or [batch, rows, cols]
	bool is2or3(int64_t batch, int64_t rows, int64_t cols, Kind kind) const {
		if (!ok || !dtype_is(*t, kind)) return false;
		int64_t const d = t->dim();
		if (d == 3) return t->size(0) == batch && t->size(1) == rows && t->size(2) == cols;
		return d == 2 && batch == 1 && t->size(0) == rows && t->size(1) == cols;
	}
	bool is_vec(int64_t n, Kind kind) const {
		return ok && dtype_is(*t, kind) && ((t->dim() == 1 && t->size(0) == n) || (t->dim() == 2 && t->size(0) == n && t->size(1) == 1));
	}
};

bool to_size(PyObject *o, size_t &v) {
	if (!PyLong_Check(o)) return false;
	v = PyLong_AsSize_t(o);
	if (v == size_t(-1) && PyErr_Occurred()) {
		PyErr_Clear();
		return false;
	}
	return true;
}
x17ai_CudaStreamHandle *to_stream(PyObject *o) {
	size_t v = 0;
	return to_size(o, v) ? reinterpret_cast<x17ai_CudaStreamHandle *>(v) : nullptr;   // null: not a regular call
}
template <typename T>
T const *to_config(PyObject *o) {
	size_t v = 0;
	return to_size(o, v) ? reinterpret_cast<T const *>(v) : nullptr;
}

template <typename F>
PyObject *launch(F &&call) {
	x17ai_DiagnosticBuffer *d = nullptr;
	bool regular = true;
	Py_BEGIN_ALLOW_THREADS
	try {
		d = call();
	} catch (...) {   // a tensor without storage: its address cannot be read
		regular = false;
	}
	Py_END_ALLOW_THREADS
	if (!regular) {
		PyErr_Clear();
		Py_RETURN_FALSE;
	}
	if (d != nullptr) return PyLong_FromVoidPtr(d);
	Py_RETURN_NONE;
}

// The arguments that every prefill form shares; false where one is irregular.
struct AttnArgs {
	x17ai_AttnConfig const *c = nullptr;
	x17ai_CudaStreamHandle *stream = nullptr;
	int64_t batch = 1, seq = 0;
	bool read(PyObject *cfg, PyObject *st, Arg const &q, Arg const &kv, Arg const &sk, Arg const &sv, Kind sv_kind, Arg const &temp,
			  Arg const &out, Kind out_kind, Arg const &l) {
		c = to_config<x17ai_AttnConfig>(cfg);
		stream = to_stream(st);
		if (c == nullptr || stream == nullptr || !q.ok || !l.ok) return false;
		int64_t const d = q.t->dim();
		if (d != 2 && d != 3) return false;
		batch = d == 3 ? q.t->size(0) : 1;
		seq = q.t->size(d - 2);
		int64_t const heads = int64_t(c->n_heads), hd = int64_t(c->head_dim);
		return q.is2or3(batch, seq, int64_t(c->q_stride), I8) && kv.is2or3(batch, seq, int64_t(c->kv_stride), I8)
			   && q.t->dim() == kv.t->dim() && sk.is2(heads, hd, I8) && sv.is2(heads, hd, sv_kind) && temp.is_vec(heads, F32)
			   && out.is2or3(batch, seq, int64_t(c->o_stride), out_kind) && out.t->dim() == d
			   && (l.none() || (l.is2or3(batch, heads, seq, F32) && l.t->dim() == d));
	}
};

// attn(config, stream, q, kv, sink_k, sink_v, temperature, out, l, window)
PyObject *attn(PyObject *, PyObject *const *a, Py_ssize_t n) {
	if (n != 10) Py_RETURN_FALSE;
	Arg q(a[2]), kv(a[3]), sk(a[4]), sv(a[5]), temp(a[6]), out(a[7]), l(a[8], true);
	AttnArgs s;
	size_t window;
	if (!s.read(a[0], a[1], q, kv, sk, sv, I8, temp, out, I8, l) || !to_size(a[9], window)) Py_RETURN_FALSE;
	return launch([&] {
		return p_x17ai_b200_attn_fwd_i8(s.stream, s.c, size_t(s.batch), size_t(s.seq), (int8_t const *)q.ptr(), (int8_t const *)kv.ptr(),
										(int8_t const *)sk.ptr(), (int8_t const *)sv.ptr(), (float const *)temp.ptr(),
										(int8_t *)out.ptr(), (float *)l.ptr(), window);
	});
}

// attn_pv_fp8(config, stream, q, kv, sink_k, sink_v, temperature, v_scale, out, l, window)
PyObject *attn_pv_fp8(PyObject *, PyObject *const *a, Py_ssize_t n) {
	if (n != 11) Py_RETURN_FALSE;
	Arg q(a[2]), kv(a[3]), sk(a[4]), sv(a[5]), temp(a[6]), vs(a[7]), out(a[8]), l(a[9], true);
	AttnArgs s;
	size_t window;
	if (!s.read(a[0], a[1], q, kv, sk, sv, E4M3, temp, out, BF16, l) || !vs.is_vec(int64_t(s.c->n_heads), F32) || !to_size(a[10], window)) {
		Py_RETURN_FALSE;
	}
	return launch([&] {
		return p_x17ai_b200_attn_fwd_pv_fp8(s.stream, s.c, size_t(s.batch), size_t(s.seq), (int8_t const *)q.ptr(),
											(uint8_t const *)kv.ptr(), (int8_t const *)sk.ptr(), (uint8_t const *)sv.ptr(),
											(float const *)temp.ptr(), (float const *)vs.ptr(), (uint16_t *)out.ptr(), (float *)l.ptr(),
											window);
	});
}

// attn_scaled(config, stream, q, q_scale, kv, k_scale, v_scale, sink_k, sink_v, temperature, out, l, window)
PyObject *attn_scaled(PyObject *, PyObject *const *a, Py_ssize_t n) {
	if (n != 13) Py_RETURN_FALSE;
	Arg q(a[2]), qs(a[3]), kv(a[4]), ks(a[5]), vs(a[6]), sk(a[7]), sv(a[8]), temp(a[9]), out(a[10]), l(a[11], true);
	AttnArgs s;
	size_t window;
	if (!s.read(a[0], a[1], q, kv, sk, sv, I8, temp, out, BF16, l) || !to_size(a[12], window)) Py_RETURN_FALSE;
	int64_t const heads = int64_t(s.c->n_heads);
	for (Arg const *x : {&qs, &ks, &vs}) {
		if (!x->is2or3(s.batch, heads, s.seq, F32)) Py_RETURN_FALSE;
	}
	return launch([&] {
		return p_x17ai_b200_attn_fwd_i8_scaled(s.stream, s.c, size_t(s.batch), size_t(s.seq), (int8_t const *)q.ptr(),
											   (float const *)qs.ptr(), (int8_t const *)kv.ptr(), (float const *)ks.ptr(),
											   (float const *)vs.ptr(), (int8_t const *)sk.ptr(), (int8_t const *)sv.ptr(),
											   (float const *)temp.ptr(), (uint16_t *)out.ptr(), (float *)l.ptr(), window);
	});
}

// decode(config, stream, q, kv_cache, kv_len, sink_k, sink_v, temperature, out, l, window, kv_lens, n_splits, no_alloc)
PyObject *decode(PyObject *, PyObject *const *a, Py_ssize_t n) {
	if (n != 14) Py_RETURN_FALSE;
	auto const *c = to_config<x17ai_AttnConfig>(a[0]);
	auto *stream = to_stream(a[1]);
	Arg q(a[2]), kv(a[3]), sk(a[5]), sv(a[6]), temp(a[7]), out(a[8]), l(a[9], true), lens(a[11], true);
	size_t kv_len, window, splits;
	if (c == nullptr || stream == nullptr || !q.ok || !kv.ok || !l.ok || !lens.ok || !to_size(a[4], kv_len) || !to_size(a[10], window)
		|| !to_size(a[12], splits) || (a[13] != Py_True && a[13] != Py_False)) {
		Py_RETURN_FALSE;
	}
	int64_t const heads = int64_t(c->n_heads), hd = int64_t(c->head_dim);
	if (!q.is2(ANY, int64_t(c->q_stride), I8) || kv.t->dim() != 3) Py_RETURN_FALSE;
	int64_t const batch = q.t->size(0);
	if (kv.t->size(0) != batch || kv.t->size(2) != int64_t(c->kv_stride) || !dtype_is(*kv.t, I8) || !sk.is2(heads, hd, I8)
		|| !sv.is2(heads, hd, I8) || !temp.is_vec(heads, F32) || !out.is2(batch, int64_t(c->o_stride), I8)
		|| (!l.none() && !l.is2(batch, heads, F32))
		|| (!lens.none() && !(lens.t->dim() == 1 && lens.t->size(0) == batch && dtype_is(*lens.t, U32_IN)))) {
		Py_RETURN_FALSE;
	}
	auto const entry = a[13] == Py_True ? p_x17ai_b200_attn_decode_i8_noalloc : p_x17ai_b200_attn_decode_i8;
	return launch([&] {
		return entry(stream, c, size_t(batch), (int8_t const *)q.ptr(), (int8_t const *)kv.ptr(), size_t(kv.t->size(1)), kv_len,
					 (uint32_t const *)lens.ptr(), (int8_t const *)sk.ptr(), (int8_t const *)sv.ptr(), (float const *)temp.ptr(),
					 (int8_t *)out.ptr(), (float *)l.ptr(), window, splits);
	});
}

// gemm(config, stream, a, b, c, rrms, residual)
PyObject *gemm(PyObject *, PyObject *const *v, Py_ssize_t n) {
	if (n != 7) Py_RETURN_FALSE;
	auto const *g = to_config<x17ai_GemmConfig>(v[0]);
	auto *stream = to_stream(v[1]);
	Arg a(v[2]), b(v[3]), c(v[4]), rr(v[5], true), res(v[6], true);
	if (g == nullptr || stream == nullptr || !rr.ok || !res.ok) Py_RETURN_FALSE;
	int64_t const k = int64_t(g->a_cols), rows = int64_t(g->b_rows);
	bool const split = g->a_dtype == X17AI_DTYPE_E4M3 && g->b_dtype == X17AI_DTYPE_INT8;
	bool const whole = g->epilogue == X17AI_EPILOGUE_SCALE || g->epilogue == X17AI_EPILOGUE_RMS_NORM;
	if (!a.is2(ANY, k, g->a_dtype) || !b.is2(rows, split ? 2 * k : k, split ? int32_t(X17AI_DTYPE_E4M3) : g->b_dtype)) Py_RETURN_FALSE;
	int64_t const m = a.t->size(0);
	if (!c.is2(m, whole ? rows : rows / 2, g->c_dtype)) Py_RETURN_FALSE;
	if (g->epilogue == X17AI_EPILOGUE_RMS_NORM && (g->head_dim == 0 || rr.none() || !rr.is2(m, rows / (2 * int64_t(g->head_dim)), F32))) Py_RETURN_FALSE;
	if (g->epilogue == X17AI_EPILOGUE_RESIDUAL && (res.none() || !res.is2(m, rows / 2, I8))) Py_RETURN_FALSE;
	return launch([&] {
		return p_x17ai_b200_gemm_fwd(stream, g, a.ptr(), size_t(m), b.ptr(), g->b_rows, c.ptr(), (float *)rr.ptr(),
									 (int8_t const *)res.ptr());
	});
}

// qkvg(stream, x, w, n_heads, head_dim, q, kv, k_rrms, g, eps)
PyObject *qkvg(PyObject *, PyObject *const *v, Py_ssize_t n) {
	if (n != 10) Py_RETURN_FALSE;
	auto *stream = to_stream(v[0]);
	Arg x(v[1]), w(v[2]), q(v[5]), kv(v[6]), rr(v[7]), g(v[8], true);
	size_t heads, hd;
	if (stream == nullptr || !to_size(v[3], heads) || !to_size(v[4], hd) || !g.ok || !PyFloat_Check(v[9]) || !x.is2(ANY, ANY, I8)) {
		Py_RETURN_FALSE;
	}
	if (heads == 0 || heads > 65535 || hd == 0 || hd > 128) Py_RETURN_FALSE;   // the entry point names what is wrong
	int64_t const rows = x.t->size(0), dim = x.t->size(1), width = int64_t(heads * hd);
	if (!g.none() && !g.is2(rows, ANY, I8)) Py_RETURN_FALSE;
	int64_t const gate = g.none() ? 0 : g.t->size(1);
	if (!w.is2(3 * width + gate, dim, I8) || !q.is2(rows, width, I8) || !kv.is2(rows, 2 * width, I8) || !rr.is2(rows, int64_t(heads), F32)) {
		Py_RETURN_FALSE;
	}
	// the projection's scale with the operations of kernels.py (sqrt, reciprocal, divide)
	double const scale = 1.0 / std::sqrt(double(dim)) / 64.0;
	x17ai_QkvgConfig cfg{size_t(dim), heads, hd, size_t(gate), scale, 8.0, PyFloat_AS_DOUBLE(v[9])};
	return launch([&] {
		return p_x17ai_b200_qkvg_fwd_i8(stream, &cfg, (int8_t const *)x.ptr(), size_t(rows), (int8_t const *)w.ptr(), (int8_t *)q.ptr(),
										(int8_t *)kv.ptr(), (float *)rr.ptr(), (int8_t *)g.ptr());
	});
}

// rms_norm(stream, mode, inp, out, row_scale, eps)
PyObject *rms_norm(PyObject *, PyObject *const *v, Py_ssize_t n) {
	if (n != 6) Py_RETURN_FALSE;
	auto *stream = to_stream(v[0]);
	size_t mode;
	Arg inp(v[2]), out(v[3]), scale(v[4], true);
	if (stream == nullptr || !to_size(v[1], mode) || mode > 2 || !scale.ok || !PyFloat_Check(v[5])) Py_RETURN_FALSE;
	if (!inp.is2(ANY, ANY, mode == X17AI_RMS_E4M3_FIXED ? E4M3 : BF16)) Py_RETURN_FALSE;
	int64_t const rows = inp.t->size(0), cols = inp.t->size(1);
	if (!out.is2(rows, cols, I8)) Py_RETURN_FALSE;
	if (mode == X17AI_RMS_BF16_ROWSCALE && (scale.none() || !scale.is_vec(rows, F32))) Py_RETURN_FALSE;
	return launch([&] {
		return p_x17ai_b200_rms_norm(stream, int32_t(mode), inp.ptr(), size_t(rows), size_t(cols), (int8_t *)out.ptr(),
									 (float *)scale.ptr(), PyFloat_AS_DOUBLE(v[5]));
	});
}

// init({name: address}): the entry points of the loaded library
PyObject *init(PyObject *, PyObject *addresses) {
	if (!PyDict_Check(addresses)) {
		PyErr_SetString(PyExc_TypeError, "init() takes a dict of addresses");
		return nullptr;
	}
#define X17_TAKE(name)                                                              \
	{                                                                               \
		PyObject *o = PyDict_GetItemString(addresses, #name);                       \
		size_t v = 0;                                                               \
		if (o == nullptr || !to_size(o, v) || v == 0) {                             \
			PyErr_SetString(PyExc_KeyError, #name);                                 \
			return nullptr;                                                         \
		}                                                                           \
		p_##name = reinterpret_cast<decltype(&name)>(v);                            \
	}
	X17_ENTRIES(X17_TAKE)
#undef X17_TAKE
	Py_RETURN_NONE;
}

// Reading an argument can throw (a layout without strides, a subclass that answers from Python): no C++ exception leaves a C
// callback, the answer is False and the Python checks raise what there is to raise.
template <PyObject *(*F)(PyObject *, PyObject *const *, Py_ssize_t)>
PyObject *guarded(PyObject *self, PyObject *const *a, Py_ssize_t n) noexcept {
	try {
		return F(self, a, n);
	} catch (...) {
	}
	PyErr_Clear();
	Py_RETURN_FALSE;
}

#define X17_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
	{"init", init, METH_O, nullptr},
	{"entries", [](PyObject *, PyObject *) -> PyObject * {
#define X17_NAME(name) #name,
		char const *const names[] = {X17_ENTRIES(X17_NAME)};
#undef X17_NAME
		PyObject *t = PyTuple_New(Py_ssize_t(sizeof(names) / sizeof(names[0])));
		for (size_t i = 0; t != nullptr && i < sizeof(names) / sizeof(names[0]); ++i) PyTuple_SET_ITEM(t, Py_ssize_t(i), PyUnicode_FromString(names[i]));
		return t;
	}, METH_NOARGS, nullptr},
	X17_FAST(attn),
	X17_FAST(attn_pv_fp8),
	X17_FAST(attn_scaled),
	X17_FAST(decode),
	X17_FAST(gemm),
	X17_FAST(qkvg),
	X17_FAST(rms_norm),
	{nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_hostcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__hostcall() {
	PyObject *m = PyModule_Create(&module_def);
	// the version of torch whose objects this reads
	if (m != nullptr && PyModule_AddStringConstant(m, "built_for", X17_BUILT_FOR) != 0) Py_CLEAR(m);
	return m;
}
