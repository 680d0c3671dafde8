// CPython binding of the calls a program makes once per layer or more often.
//
// The package talks to libdgb200.so through its C ABI.  For calls made now and then ctypes does that; for the operators
// its marshalling costs more than the call: on a B200 host a dense GEMM that the GPU finishes in 5 us took 9.4 us per call,
// 4.5 of them in Python building four ctypes structures, and a quantise call another 6 us for its two result tensors.  Here
// the same arguments are read straight from the Python objects and tensors, and result tensors come from torch's C++
// allocator.  The library is not linked: bind() takes the handle the package loaded (an alternative build included).
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/dgb200.h"

namespace {

// Every library function the binding calls.
#define DG_BOUND_FUNCTIONS(X)                                                                                                    \
    X(dg_last_error) X(dg_fp8_fp4_gemm) X(dg_bf16_gemm) X(dg_m_grouped_fp8_fp4_gemm_contiguous)                                  \
    X(dg_m_grouped_fp8_fp4_gemm_contiguous_ends) X(dg_m_grouped_fp8_fp4_gemm_masked) X(dg_fp8_fp4_bmm) X(dg_fp8_gemm_nt)         \
    X(dg_m_grouped_fp8_gemm_nt_contiguous) X(dg_m_grouped_fp8_gemm_nt_masked) X(dg_fp8_bmm_nt) X(dg_sf_words)                    \
    X(dg_cast_bf16_to_fp8_sf) X(dg_cast_bf16_to_fp4_packed_sf) X(dg_silu_mul_cast_fp8_sf) X(dg_transform_sf) X(dg_ep_count)      \
    X(dg_ep_layout) X(dg_ep_dispatch) X(dg_ep_combine)

struct Library {
#define X(name) decltype(&::name) name = nullptr;
    DG_BOUND_FUNCTIONS(X)
#undef X
} lib;
PyObject* g_error = nullptr;     // DgError(code, message)

// attribute names, interned once
struct Names {
    PyObject *addr, *ordinal, *data, *sf, *rows, *k, *ld, *bits, *gran_k, *major_mn, *kind, *buf, *sfd, *alpha, *accumulate, *tc_util,
        *data_ptr, *numel, *element_size;
} names;

// Marks a Python exception that is already set.
struct PythonError {};

struct Ref {
    PyObject* p;
    explicit Ref(PyObject* o) : p(o) { if (p == nullptr) throw PythonError(); }
    ~Ref() { Py_DECREF(p); }
    Ref(const Ref&) = delete;
    Ref& operator=(const Ref&) = delete;
};

uint64_t as_u64(PyObject* o) {
    const uint64_t v = PyLong_AsUnsignedLongLongMask(o);
    if (v == static_cast<uint64_t>(-1) && PyErr_Occurred()) throw PythonError();
    return v;
}
uint32_t as_u32(PyObject* o) { return static_cast<uint32_t>(as_u64(o)); }
uint64_t attr_u64(PyObject* o, PyObject* name) { Ref v(PyObject_GetAttr(o, name)); return as_u64(v.p); }
uint32_t attr_u32(PyObject* o, PyObject* name) { return static_cast<uint32_t>(attr_u64(o, name)); }
bool truth(PyObject* o) {
    const int t = PyObject_IsTrue(o);
    if (t < 0) throw PythonError();
    return t != 0;
}
bool attr_truth(PyObject* o, PyObject* name) { Ref v(PyObject_GetAttr(o, name)); return truth(v.p); }

uint64_t call_u64(PyObject* o, PyObject* method) { Ref v(PyObject_CallMethodNoArgs(o, method)); return as_u64(v.p); }

// Device address of a tensor (or of any object with torch's data_ptr()).
void* ptr(PyObject* o) {
    if (THPVariable_Check(o)) return THPVariable_Unpack(o).data_ptr();
    return reinterpret_cast<void*>(call_u64(o, names.data_ptr));
}
void* ptr_or_null(PyObject* o) { return o == Py_None ? nullptr : ptr(o); }
size_t elements(PyObject* o) {
    return THPVariable_Check(o) ? static_cast<size_t>(THPVariable_Unpack(o).numel()) : static_cast<size_t>(call_u64(o, names.numel));
}
size_t bytes(PyObject* o) {
    if (THPVariable_Check(o)) {
        const at::Tensor& t = THPVariable_Unpack(o);
        return static_cast<size_t>(t.numel()) * t.element_size();
    }
    return static_cast<size_t>(call_u64(o, names.numel) * call_u64(o, names.element_size));
}

dg_ctx* context(PyObject* o) { return reinterpret_cast<dg_ctx*>(attr_u64(o, names.addr)); }

dg_lp_operand operand(PyObject* o) {
    dg_lp_operand c;
    Ref data(PyObject_GetAttr(o, names.data)), sf(PyObject_GetAttr(o, names.sf));
    c.data = ptr(data.p);
    c.sf = static_cast<uint32_t*>(ptr(sf.p));
    c.rows = attr_u32(o, names.rows);
    c.k = attr_u32(o, names.k);
    c.ld = attr_u32(o, names.ld);
    c.bits = attr_u32(o, names.bits);
    c.gran_k = attr_u32(o, names.gran_k);
    c.major_mn = attr_truth(o, names.major_mn) ? 1 : 0;
    c.data_len = bytes(data.p);
    c.sf_len = elements(sf.p);
    return c;
}
dg_out output(PyObject* o) {
    dg_out c;
    Ref buf(PyObject_GetAttr(o, names.buf)), sfd(PyObject_GetAttr(o, names.sfd));
    c.kind = static_cast<int>(attr_u64(o, names.kind));
    c.buf = ptr(buf.p);
    c.ld = attr_u32(o, names.ld);
    c.sfd = static_cast<uint32_t*>(ptr_or_null(sfd.p));
    c.buf_len = elements(buf.p);
    c.sfd_len = sfd.p == Py_None ? 0 : elements(sfd.p);
    return c;
}
dg_epilogue epilogue(PyObject* o) {
    dg_epilogue c = {1.0f, 0, 0, 100};
    if (o == Py_None) return c;
    Ref alpha(PyObject_GetAttr(o, names.alpha));
    if (alpha.p != Py_None) {
        const double v = PyFloat_AsDouble(alpha.p);
        if (v == -1.0 && PyErr_Occurred()) throw PythonError();
        c.alpha = static_cast<float>(v);
        c.has_alpha = 1;
    }
    c.accumulate = attr_truth(o, names.accumulate) ? 1 : 0;
    c.tc_util = attr_u32(o, names.tc_util);
    return c;
}

void check(int rc) {
    if (rc == 0) return;
    Ref args(Py_BuildValue("is", rc, lib.dg_last_error()));
    Ref error(PyObject_CallObject(g_error, args.p));
    PyErr_SetObject(g_error, error.p);
    throw PythonError();
}

// Runs a library call without the interpreter lock: a full launch queue makes it wait for the GPU.
template <typename Call>
void launch(Call&& call) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = call();
    Py_END_ALLOW_THREADS
    check(rc);
}

at::Tensor new_tensor(at::IntArrayRef size, at::ScalarType type, at::Device device) {
    return at::empty(size, at::TensorOptions().dtype(type).device(device));
}
at::Device device_of(PyObject* o) {
    if (!THPVariable_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "expected a torch tensor");
        throw PythonError();
    }
    return THPVariable_Unpack(o).device();
}
at::Device context_device(PyObject* ctx) { return at::Device(at::kCUDA, static_cast<at::DeviceIndex>(attr_u64(ctx, names.ordinal))); }

PyObject* pair(const at::Tensor& a, const at::Tensor& b) {
    Ref x(THPVariable_Wrap(a)), y(THPVariable_Wrap(b));
    return PyTuple_Pack(2, x.p, y.p);
}

using Args = PyObject* const*;

PyObject* none() { Py_RETURN_NONE; }

// ------------------------------------------------------------------------------------------------ the bound calls
PyObject* gemm(Args v) {      // ctx, a, b, out, epi
    dg_ctx* ctx = context(v[0]);
    const dg_lp_operand a = operand(v[1]), b = operand(v[2]);
    const dg_out out = output(v[3]);
    const dg_epilogue epi = epilogue(v[4]);
    launch([&] { return lib.dg_fp8_fp4_gemm(ctx, &a, &b, &out, &epi); });
    return none();
}
PyObject* bf16_gemm(Args v) { // ctx, a, a_ld, m, b, b_ld, n, k, out, epi
    dg_ctx* ctx = context(v[0]);
    const uint16_t *a = static_cast<const uint16_t*>(ptr(v[1])), *b = static_cast<const uint16_t*>(ptr(v[4]));
    const uint32_t a_ld = as_u32(v[2]), m = as_u32(v[3]), b_ld = as_u32(v[5]), n = as_u32(v[6]), k = as_u32(v[7]);
    const dg_out out = output(v[8]);
    const dg_epilogue epi = epilogue(v[9]);
    launch([&] { return lib.dg_bf16_gemm(ctx, a, a_ld, m, b, b_ld, n, k, &out, &epi); });
    return none();
}
PyObject* gemm_contiguous(Args v) {       // ctx, a, m_indices, b, out, num_groups, epi
    dg_ctx* ctx = context(v[0]);
    const dg_lp_operand a = operand(v[1]), b = operand(v[3]);
    const int32_t* idx = static_cast<const int32_t*>(ptr(v[2]));
    const dg_out out = output(v[4]);
    const uint32_t groups = as_u32(v[5]);
    const dg_epilogue epi = epilogue(v[6]);
    launch([&] { return lib.dg_m_grouped_fp8_fp4_gemm_contiguous(ctx, &a, idx, &b, &out, groups, &epi); });
    return none();
}
PyObject* gemm_contiguous_ends(Args v) {  // ctx, a, group_ends, b, out, num_groups, epi
    dg_ctx* ctx = context(v[0]);
    const dg_lp_operand a = operand(v[1]), b = operand(v[3]);
    const uint32_t* ends = static_cast<const uint32_t*>(ptr(v[2]));
    const dg_out out = output(v[4]);
    const uint32_t groups = as_u32(v[5]);
    const dg_epilogue epi = epilogue(v[6]);
    launch([&] { return lib.dg_m_grouped_fp8_fp4_gemm_contiguous_ends(ctx, &a, ends, &b, &out, groups, &epi); });
    return none();
}
PyObject* gemm_masked(Args v) {           // ctx, a, masked_m, b, out, num_groups, expected_m, epi
    dg_ctx* ctx = context(v[0]);
    const dg_lp_operand a = operand(v[1]), b = operand(v[3]);
    const int32_t* masked = static_cast<const int32_t*>(ptr(v[2]));
    const dg_out out = output(v[4]);
    const uint32_t groups = as_u32(v[5]), expected = as_u32(v[6]);
    const dg_epilogue epi = epilogue(v[7]);
    launch([&] { return lib.dg_m_grouped_fp8_fp4_gemm_masked(ctx, &a, masked, &b, &out, groups, expected, &epi); });
    return none();
}
PyObject* bmm(Args v) {                   // ctx, a, b, out, num_groups, epi
    dg_ctx* ctx = context(v[0]);
    const dg_lp_operand a = operand(v[1]), b = operand(v[2]);
    const dg_out out = output(v[3]);
    const uint32_t groups = as_u32(v[4]);
    const dg_epilogue epi = epilogue(v[5]);
    launch([&] { return lib.dg_fp8_fp4_bmm(ctx, &a, &b, &out, groups, &epi); });
    return none();
}

// The f32-scale calls share their first arguments: ctx, a, a_sf_t, b, sfb, m, n, out, out_ld (a and b: Fp8Tensor)
struct F32Args {
    dg_ctx* ctx;
    const uint8_t *a, *b;
    const float *sfa, *sfb;
    uint32_t a_ld, b_ld, m, n, k, out_ld;
    uint16_t* out;
    explicit F32Args(Args v) {
        ctx = context(v[0]);
        Ref ad(PyObject_GetAttr(v[1], names.data)), bd(PyObject_GetAttr(v[3], names.data));
        a = static_cast<const uint8_t*>(ptr(ad.p));
        b = static_cast<const uint8_t*>(ptr(bd.p));
        a_ld = attr_u32(v[1], names.ld);
        b_ld = attr_u32(v[3], names.ld);
        k = attr_u32(v[1], names.k);
        sfa = static_cast<const float*>(ptr(v[2]));
        sfb = static_cast<const float*>(ptr(v[4]));
        m = as_u32(v[5]);
        n = as_u32(v[6]);
        out = static_cast<uint16_t*>(ptr(v[7]));
        out_ld = as_u32(v[8]);
    }
};
PyObject* f32_gemm(Args v) {
    const F32Args f(v);
    launch([&] { return lib.dg_fp8_gemm_nt(f.ctx, f.a, f.a_ld, f.sfa, f.b, f.b_ld, f.sfb, f.m, f.n, f.k, f.out, f.out_ld); });
    return none();
}
PyObject* f32_gemm_contiguous(Args v) {   // ..., m_indices, num_groups
    const F32Args f(v);
    const int32_t* idx = static_cast<const int32_t*>(ptr(v[9]));
    const uint32_t groups = as_u32(v[10]);
    launch([&] {
        return lib.dg_m_grouped_fp8_gemm_nt_contiguous(f.ctx, f.a, f.a_ld, f.sfa, f.b, f.b_ld, f.sfb, f.m, f.n, f.k, f.out, f.out_ld, idx, groups);
    });
    return none();
}
PyObject* f32_gemm_masked(Args v) {       // ..., masked_m, num_groups, expected_m
    const F32Args f(v);
    const int32_t* masked = static_cast<const int32_t*>(ptr(v[9]));
    const uint32_t groups = as_u32(v[10]), expected = as_u32(v[11]);
    launch([&] {
        return lib.dg_m_grouped_fp8_gemm_nt_masked(f.ctx, f.a, f.a_ld, f.sfa, f.b, f.b_ld, f.sfb, f.m, f.n, f.k, f.out, f.out_ld, masked, groups, expected);
    });
    return none();
}
PyObject* f32_bmm(Args v) {               // ..., num_groups
    const F32Args f(v);
    const uint32_t groups = as_u32(v[9]);
    launch([&] { return lib.dg_fp8_bmm_nt(f.ctx, f.a, f.a_ld, f.sfa, f.b, f.b_ld, f.sfb, f.m, f.n, f.k, f.out, f.out_ld, groups); });
    return none();
}

// Scale words a quantiser call returns.  The kernels write every word of the packed layout, alignment padding included.
at::Tensor new_scale_words(PyObject* ctx, uint32_t rows, uint32_t k, uint32_t gran, uint32_t groups) {
    return new_tensor({static_cast<int64_t>(lib.dg_sf_words(rows, k, gran, groups > 1 ? groups : 1))}, at::kInt, context_device(ctx));
}
PyObject* cast_fp8(Args v) {  // ctx, src, src_ld, rows, k, gran_k, num_groups
    dg_ctx* ctx = context(v[0]);
    const uint16_t* src = static_cast<const uint16_t*>(ptr(v[1]));
    const uint32_t ld = as_u32(v[2]), rows = as_u32(v[3]), k = as_u32(v[4]), gran = as_u32(v[5]), groups = as_u32(v[6]);
    const at::Tensor dst = new_tensor({rows, k}, at::kByte, device_of(v[1])), sf = new_scale_words(v[0], rows, k, gran, groups);
    uint8_t* d = static_cast<uint8_t*>(dst.data_ptr());
    uint32_t* s = static_cast<uint32_t*>(sf.data_ptr());
    launch([&] { return lib.dg_cast_bf16_to_fp8_sf(ctx, src, ld, rows, k, gran, groups, d, s); });
    return pair(dst, sf);
}
PyObject* cast_fp4(Args v) {  // ctx, src, src_ld, rows, k, num_groups, sf_rule
    dg_ctx* ctx = context(v[0]);
    const uint16_t* src = static_cast<const uint16_t*>(ptr(v[1]));
    const uint32_t ld = as_u32(v[2]), rows = as_u32(v[3]), k = as_u32(v[4]), groups = as_u32(v[5]);
    const int rule = static_cast<int>(as_u64(v[6]));
    const at::Tensor dst = new_tensor({rows, k / 2}, at::kByte, device_of(v[1])), sf = new_scale_words(v[0], rows, k, 32, groups);
    uint8_t* d = static_cast<uint8_t*>(dst.data_ptr());
    uint32_t* s = static_cast<uint32_t*>(sf.data_ptr());
    launch([&] { return lib.dg_cast_bf16_to_fp4_packed_sf(ctx, src, ld, rows, k, groups, rule, d, s); });
    return pair(dst, sf);
}
PyObject* silu_cast(Args v) { // ctx, gate_up, src_ld, rows, n, gran_k, num_groups, live_rows, dst, sf
    dg_ctx* ctx = context(v[0]);
    const uint16_t* src = static_cast<const uint16_t*>(ptr(v[1]));
    const uint32_t ld = as_u32(v[2]), rows = as_u32(v[3]), n = as_u32(v[4]), gran = as_u32(v[5]), groups = as_u32(v[6]);
    const uint32_t* live = static_cast<const uint32_t*>(ptr_or_null(v[7]));
    uint8_t* d = static_cast<uint8_t*>(ptr(v[8]));
    uint32_t* s = static_cast<uint32_t*>(ptr(v[9]));
    launch([&] { return lib.dg_silu_mul_cast_fp8_sf(ctx, src, ld, rows, n, gran, groups, d, s, live); });
    return none();
}
PyObject* transform_sf(Args v) {          // ctx, sf, mn, sf_k, num_batches
    dg_ctx* ctx = context(v[0]);
    const float* sf = static_cast<const float*>(ptr(v[1]));
    const uint32_t mn = as_u32(v[2]), sf_k = as_u32(v[3]), batches = as_u32(v[4]);
    const at::Tensor dst = new_tensor({static_cast<int64_t>(batches) * sf_k, (static_cast<int64_t>(mn) + 3) / 4 * 4}, at::kFloat, device_of(v[1]));
    float* d = static_cast<float*>(dst.data_ptr());
    launch([&] { return lib.dg_transform_sf(ctx, sf, mn, sf_k, batches, d); });
    return THPVariable_Wrap(dst);
}

PyObject* ep_count(Args v) {  // ctx, expert_of_pair, pairs, num_experts, local_rank, block_hist, counts
    dg_ctx* ctx = context(v[0]);
    const int32_t* experts = static_cast<const int32_t*>(ptr(v[1]));
    const uint32_t pairs = as_u32(v[2]), num_experts = as_u32(v[3]);
    int32_t* rank = static_cast<int32_t*>(ptr(v[4]));
    uint32_t *hist = static_cast<uint32_t*>(ptr(v[5])), *counts = static_cast<uint32_t*>(ptr(v[6]));
    launch([&] { return lib.dg_ep_count(ctx, experts, pairs, num_experts, rank, hist, counts); });
    return none();
}
PyObject* ep_layout(Args v) { // ctx, all_counts, world, rank, num_experts, alignment, capacity, slot_rows, pair_base, group_ends, totals
    dg_ctx* ctx = context(v[0]);
    const uint32_t* counts = static_cast<const uint32_t*>(ptr(v[1]));
    const uint32_t world = as_u32(v[2]), rank = as_u32(v[3]), experts = as_u32(v[4]), alignment = as_u32(v[5]), capacity = as_u32(v[6]), slot = as_u32(v[7]);
    uint32_t *base = static_cast<uint32_t*>(ptr(v[8])), *ends = static_cast<uint32_t*>(ptr(v[9])), *totals = static_cast<uint32_t*>(ptr(v[10]));
    launch([&] { return lib.dg_ep_layout(ctx, counts, world, rank, experts, alignment, capacity, slot, base, ends, totals); });
    return none();
}
// ctx, expert_of_pair, local_rank, block_base, pair_base, pairs, topk, num_experts, world, data, k, sf, sf_stride, sf_cols, peer_data, peer_sf,
// peer_sf_stride, capacity, slot_rows, pos_of_pair, max_blocks
PyObject* ep_dispatch(Args v) {
    dg_ctx* ctx = context(v[0]);
    const int32_t *experts = static_cast<const int32_t*>(ptr(v[1])), *rank = static_cast<const int32_t*>(ptr(v[2]));
    const uint32_t *block_base = static_cast<const uint32_t*>(ptr(v[3])), *pair_base = static_cast<const uint32_t*>(ptr(v[4]));
    const uint32_t pairs = as_u32(v[5]), topk = as_u32(v[6]), num_experts = as_u32(v[7]), world = as_u32(v[8]);
    const uint8_t* data = static_cast<const uint8_t*>(ptr(v[9]));
    const uint32_t k = as_u32(v[10]), sf_stride = as_u32(v[12]), sf_cols = as_u32(v[13]);
    const uint32_t* sf = static_cast<const uint32_t*>(ptr(v[11]));
    void* const *peer_data = static_cast<void* const*>(ptr(v[14])), *const *peer_sf = static_cast<void* const*>(ptr(v[15]));
    const uint32_t peer_stride = as_u32(v[16]), capacity = as_u32(v[17]), slot = as_u32(v[18]), max_blocks = as_u32(v[20]);
    int32_t* pos = static_cast<int32_t*>(ptr(v[19]));
    launch([&] {
        return lib.dg_ep_dispatch(ctx, experts, rank, block_base, pair_base, pairs, topk, num_experts, world, data, k, sf, sf_stride, sf_cols, peer_data,
                                  peer_sf, peer_stride, capacity, slot, pos, max_blocks);
    });
    return none();
}
// ctx, expert_of_pair, pos_of_pair, weights, tokens, topk, num_experts, world, peer_rows, pitch, n, out, out_pitch, max_blocks
PyObject* ep_combine(Args v) {
    dg_ctx* ctx = context(v[0]);
    const int32_t *experts = static_cast<const int32_t*>(ptr(v[1])), *pos = static_cast<const int32_t*>(ptr(v[2]));
    const float* weights = static_cast<const float*>(ptr(v[3]));
    const uint32_t tokens = as_u32(v[4]), topk = as_u32(v[5]), num_experts = as_u32(v[6]), world = as_u32(v[7]);
    const void* const* rows = static_cast<const void* const*>(ptr(v[8]));
    const size_t pitch = as_u64(v[9]), out_pitch = as_u64(v[12]);
    const uint32_t n = as_u32(v[10]), max_blocks = as_u32(v[13]);
    uint16_t* out = static_cast<uint16_t*>(ptr(v[11]));
    launch([&] { return lib.dg_ep_combine(ctx, experts, pos, weights, tokens, topk, num_experts, world, rows, pitch, n, out, out_pitch, max_blocks); });
    return none();
}

// ------------------------------------------------------------------------------------------------------ plumbing
template <PyObject* (*kCall)(Args), Py_ssize_t kCount>
PyObject* entry(PyObject*, Args args, Py_ssize_t count) {
    HANDLE_TH_ERRORS
    if (count != kCount) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", kCount, count);
        return nullptr;
    }
    try {
        return kCall(args);
    } catch (const PythonError&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyObject* bind(PyObject*, Args args, Py_ssize_t count) {   // library handle, DgError
    if (count != 2) {
        PyErr_SetString(PyExc_TypeError, "bind takes the library handle and the error class");
        return nullptr;
    }
    void* handle = PyLong_AsVoidPtr(args[0]);
    if (handle == nullptr && PyErr_Occurred()) return nullptr;
#define X(name)                                                                                        \
    lib.name = reinterpret_cast<decltype(&::name)>(dlsym(handle, #name));                              \
    if (lib.name == nullptr) {                                                                         \
        PyErr_SetString(PyExc_ImportError, "the library does not export " #name);                      \
        return nullptr;                                                                                \
    }
    DG_BOUND_FUNCTIONS(X)
#undef X
    Py_INCREF(args[1]);
    Py_XDECREF(g_error);
    g_error = args[1];
    Py_RETURN_NONE;
}

#define DG_METHOD(call, count) {#call, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<call, count>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&bind)), METH_FASTCALL, nullptr},
    DG_METHOD(gemm, 5), DG_METHOD(bf16_gemm, 10), DG_METHOD(gemm_contiguous, 7), DG_METHOD(gemm_contiguous_ends, 7), DG_METHOD(gemm_masked, 8),
    DG_METHOD(bmm, 6), DG_METHOD(f32_gemm, 9), DG_METHOD(f32_gemm_contiguous, 11), DG_METHOD(f32_gemm_masked, 12), DG_METHOD(f32_bmm, 10),
    DG_METHOD(cast_fp8, 7), DG_METHOD(cast_fp4, 7), DG_METHOD(silu_cast, 10), DG_METHOD(transform_sf, 5), DG_METHOD(ep_count, 7),
    DG_METHOD(ep_layout, 11), DG_METHOD(ep_dispatch, 21), DG_METHOD(ep_combine, 14),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dg_binding", "Operator calls of libdgb200.so without ctypes marshalling.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dg_binding(void) {
    struct { PyObject** slot; const char* text; } const all[] = {
        {&names.addr, "_addr"}, {&names.ordinal, "ordinal"}, {&names.data, "data"}, {&names.sf, "sf"}, {&names.rows, "rows"}, {&names.k, "k"},
        {&names.ld, "ld"}, {&names.bits, "bits"}, {&names.gran_k, "gran_k"}, {&names.major_mn, "major_mn"}, {&names.kind, "kind"},
        {&names.buf, "buf"}, {&names.sfd, "sfd"}, {&names.alpha, "alpha"}, {&names.accumulate, "accumulate"}, {&names.tc_util, "tc_util"},
        {&names.data_ptr, "data_ptr"}, {&names.numel, "numel"}, {&names.element_size, "element_size"}};
    for (const auto& n : all)
        if ((*n.slot = PyUnicode_InternFromString(n.text)) == nullptr) return nullptr;
    return PyModule_Create(&module);
}
