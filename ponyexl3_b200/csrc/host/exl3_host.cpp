// Host path of the module calls: argument checks, output allocation and the C ABI call in one native
// function per call.  Through ctypes and torch's Python API the same steps take about 15 us, longer than
// a small layer's kernel; here they take about 4, most of it the launch.
//
// The entry points of libexl3b200.so come in as addresses (bind), so that the library chosen by
// ponyexl3_b200._lib is the one that is called.  Nothing is kept between calls but the address and size of
// each device's workspace, which ponyexl3_b200.ops.Workspace owns and registers (set_workspace).
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "../../../include/exl3_b200.h"
#include "../exl3_moe_plan.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr int kGemvMaxRows = 16;      // what the streamed GEMV can do
constexpr int kMaxMembers = 8;        // of exl3_gemm_members

#define EXL3_FN(name) decltype(&::name) name = nullptr
struct Api {
    EXL3_FN(exl3_workspace_bytes);
    EXL3_FN(exl3_gemm_workspace_bytes);
    EXL3_FN(exl3_gemv);
    EXL3_FN(exl3_gemm);
    EXL3_FN(exl3_gemm_members);
    EXL3_FN(exl3_gemv_blocks);
    EXL3_FN(exl3_gemm_tiles);
    EXL3_FN(exl3_moe_decode_tables);
    EXL3_FN(exl3_moe_prefill_tables);
} api;
#undef EXL3_FN

struct Workspace {
    void* ptr = nullptr;
    size_t bytes = 0;
} workspaces[kMaxDevices];

PyObject* check_fn = nullptr;         // ponyexl3_b200._lib.check
PyObject* grow_fn = nullptr;          // grows and registers the workspace of a device: (device index, bytes)

struct PyError {};                    // a Python exception is set

[[noreturn]] void fail(PyObject* type, const std::string& msg)
{
    PyErr_SetString(type, msg.c_str());
    throw PyError();
}

void check(int rc, const char* what)
{
    if (rc == 0) return;
    PyObject* r = PyObject_CallFunction(check_fn, "is", rc, what);     // raises
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, what);
    throw PyError();
}

// Allocations, copies and launches run without the interpreter's lock, as PyTorch's own do: a launch waits while
// the stream's queue is full, and what the GPU waits for may be another Python thread's work.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

// One library call.  The calls of a device's threads go one at a time: the launches of one call use the workspace
// one after the other, and another call's may not come in between on the same stream.
std::mutex launching[kMaxDevices];
template <typename F> void launch(int dev, const char* what, F&& call)
{
    if (dev < 0 || dev >= kMaxDevices) fail(PyExc_ValueError, "device index out of range");
    int rc;
    {
        const NoGil unlocked;
        const std::lock_guard<std::mutex> one(launching[dev]);
        rc = call();
    }
    check(rc, what);
}

const at::Tensor& tensor(PyObject* o, const char* name)
{
    if (!THPVariable_Check(o)) fail(PyExc_TypeError, std::string(name) + " must be a tensor");
    return THPVariable_Unpack(o);
}

const at::Tensor& cuda_tensor(PyObject* o, const char* name)
{
    const at::Tensor& t = tensor(o, name);
    if (!t.is_cuda())
        fail(PyExc_RuntimeError, std::string(name) + " must be a CUDA tensor: the EXL3 path has no CPU implementation");
    return t;
}

template <typename T> T* ptr_or_null(PyObject* o, const char* name)
{
    return o == Py_None ? nullptr : static_cast<T*>(tensor(o, name).data_ptr());
}

int64_t integer(PyObject* o)
{
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyError();
    return v;
}

int dtype_code(const at::Tensor& t)
{
    switch (t.scalar_type()) {
        case at::kHalf: return EXL3_DT_F16;
        case at::kBFloat16: return EXL3_DT_BF16;
        case at::kFloat: return EXL3_DT_F32;
        default: fail(PyExc_ValueError, std::string("unsupported dtype torch.") +
                      (t.scalar_type() == at::kDouble ? "float64" : c10::toString(t.scalar_type())));
    }
}

Workspace workspace(int dev, size_t need)
{
    if (dev < 0 || dev >= kMaxDevices) fail(PyExc_ValueError, "device index out of range");
    if (!workspaces[dev].ptr || workspaces[dev].bytes < need) {
        PyObject* r = PyObject_CallFunction(grow_fn, "in", dev, (Py_ssize_t)need);
        if (!r) throw PyError();
        Py_DECREF(r);
        if (!workspaces[dev].ptr || workspaces[dev].bytes < need) fail(PyExc_RuntimeError, "the workspace did not grow");
    }
    return workspaces[dev];
}

at::Tensor empty_half(at::IntArrayRef sizes, const at::Device& d)
{
    const NoGil unlocked;
    return at::empty(sizes, at::TensorOptions().dtype(at::kHalf).device(d));
}
at::Tensor empty_int(int64_t n, const at::Device& d)
{
    const NoGil unlocked;
    return at::empty({n}, at::TensorOptions().dtype(at::kInt).device(d));
}
at::Tensor dense(const at::Tensor& t)
{
    if (t.is_contiguous()) return t;
    const NoGil unlocked;
    return t.contiguous();
}

struct Weights {
    const uint16_t* trellis;
    int64_t t_in, t_out;
};
Weights weights(PyObject* o)
{
    const at::Tensor& t = tensor(o, "trellis");
    return {static_cast<const uint16_t*>(t.data_ptr()), t.size(0), t.size(1)};
}

// Activations as rows of unit column stride.
struct Rows {
    at::Tensor t;          // what holds them
    int64_t rows, stride;
    int dtype;
};
Rows rows_of(const at::Tensor& x, int64_t features)
{
    Rows r;
    r.dtype = dtype_code(x);
    if (x.dim() == 2) {
        r.t = x.stride(1) == 1 ? x : dense(x);
        r.rows = x.size(0);
        r.stride = r.t.stride(0);
    } else {
        r.rows = features > 0 ? x.numel() / features : 0;
        r.stride = features;
        if (x.is_contiguous()) {
            r.t = x;
        } else {                                       // a view where the leading dimensions fold into one, else a copy
            const NoGil unlocked;
            r.t = x.reshape({r.rows, features});
            if (r.t.stride(1) != 1) r.t = r.t.contiguous();
            r.stride = r.t.stride(0);
        }
    }
    // the stride of a single row means nothing (views may carry any number there)
    if (r.rows == 1 && r.stride < features) r.stride = features;
    return r;
}

void gemv(const Rows& x, int64_t rows, const Weights& w, int k, int cb, const uint16_t* suh, const uint16_t* svh,
          const uint16_t* bias, uint16_t* y, int64_t y_stride, unsigned flags, int dev, cudaStream_t s)
{
    const Workspace ws = workspace(dev, api.exl3_workspace_bytes(rows, 16 * w.t_in));
    launch(dev, "exl3_gemv", [&] {
        return api.exl3_gemv(x.t.data_ptr(), x.dtype, (int)rows, x.stride, w.trellis, w.t_in, w.t_out, k, cb, suh,
                             svh, bias, y, y_stride, ws.ptr, ws.bytes, flags, (exl3_stream_t)s);
    });
}

void gemm(const Rows& x, int64_t rows, const Weights& w, int k, int cb, const uint16_t* suh, const uint16_t* svh,
          const uint16_t* bias, uint16_t* y, int64_t y_stride, int dev, cudaStream_t s)
{
    const Workspace ws = workspace(dev, api.exl3_gemm_workspace_bytes(rows, 16 * w.t_in));
    launch(dev, "exl3_gemm", [&] {
        return api.exl3_gemm(x.t.data_ptr(), x.dtype, rows, x.stride, w.trellis, w.t_in, w.t_out, k, cb, suh, svh,
                             bias, y, y_stride, ws.ptr, ws.bytes, 0, (exl3_stream_t)s);
    });
}

// GEMV or GEMM.  Nine to sixteen rows take a second MMA and a rotation kernel in the GEMV, and the GEMM is as
// quick or quicker: us at 16 rows, GEMV / GEMM, K = 4: 4096 x 4096 16.8 / 15.1, 5120 x 17408 38.5 / 34.0,
// 17408 x 5120 39.1 / 38.3, 512 x 512 9.5 / 8.9 (at 8 rows 12.7 / 14.6, 32.0 / 32.5, 33.7 / 37.9, 6.9 / 8.8);
// the other way round only for long inputs at K = 2 and 3, by up to 4 %.  The GEMM asks for 16-byte
// alignment where the GEMV takes 8.
bool use_gemv(int64_t rows, const uint16_t* svh, const uint16_t* bias, const uint16_t* y, int64_t y_stride)
{
    if (rows <= kGemvMaxRows / 2 || rows > kGemvMaxRows) return rows <= kGemvMaxRows;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(svh) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(y);
    return bits % 16 != 0 || y_stride % 8 != 0;
}

uint16_t* u16(const at::Tensor& t) { return static_cast<uint16_t*>(t.data_ptr()); }

// ---- linear(x, trellis, k, cb, suh, svh, bias, flags, out) ---------------------------------------------------
PyObject* linear(PyObject* const* arg)
{
    const at::Tensor& x = tensor(arg[0], "x");
    const Weights w = weights(arg[1]);
    const int k = (int)integer(arg[2]), cb = (int)integer(arg[3]);
    const int64_t in = 16 * w.t_in, out_features = 16 * w.t_out;
    if (x.dim() < 1 || x.size(-1) != in)
        fail(PyExc_ValueError, "expected last dim " + std::to_string(in) + ", got " + std::to_string(x.dim() < 1 ? 0 : x.size(-1)));
    const int64_t rows = x.numel() / in;
    c10::SmallVector<int64_t, 5> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = out_features;
    if (rows == 0) return THPVariable_Wrap(empty_half(shape, x.device()));
    at::Tensor y;
    if (arg[8] != Py_None) {
        const at::Tensor& o = tensor(arg[8], "out");
        if (o.dim() != 2 || o.size(0) != rows || o.size(1) != out_features || o.scalar_type() != at::kHalf || o.stride(1) != 1)
            fail(PyExc_ValueError, "out must be a (rows, out_features) fp16 tensor with unit column stride");
        y = o;
    }
    cuda_tensor(arg[0], "x");
    const Rows r = rows_of(x, in);
    const int dev = x.device().index();
    const c10::cuda::CUDAGuard guard(x.device());
    const cudaStream_t s = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    int64_t y_stride = out_features;
    if (y.defined()) y_stride = y.stride(0) < out_features && rows == 1 ? out_features : y.stride(0);
    else y = empty_half(shape, x.device());
    const uint16_t* suh = ptr_or_null<uint16_t>(arg[4], "suh");
    const uint16_t* svh = ptr_or_null<uint16_t>(arg[5], "svh");
    const uint16_t* bias = ptr_or_null<uint16_t>(arg[6], "bias");
    if (use_gemv(rows, svh, bias, u16(y), y_stride))
        gemv(r, rows, w, k, cb, suh, svh, bias, u16(y), y_stride, (unsigned)integer(arg[7]), dev, s);
    else
        gemm(r, rows, w, k, cb, suh, svh, bias, u16(y), y_stride, dev, s);
    if (arg[8] != Py_None && x.dim() != 2) return THPVariable_Wrap(y.reshape(shape));
    return THPVariable_Wrap(std::move(y));
}

// ---- sibling groups --------------------------------------------------------------------------------------------
// Everything a group or an MLP hands over about its members:
// (trellis, k, cb, suh_stack, svh_cat, members, total)
struct Group {
    Weights w;
    int k, cb;
    const uint16_t *suh, *svh;
    int64_t members, total;
};
Group group_of(PyObject* const* arg)
{
    Group g;
    g.w = weights(arg[0]);
    g.k = (int)integer(arg[1]);
    g.cb = (int)integer(arg[2]);
    g.suh = ptr_or_null<uint16_t>(arg[3], "suh_stack");
    g.svh = ptr_or_null<uint16_t>(arg[4], "svh_cat");
    g.members = integer(arg[5]);
    g.total = integer(arg[6]);
    return g;
}
// A Python object that this frame owns.
struct Owned {
    PyObject* p;
    ~Owned() { Py_XDECREF(p); }
};
// table: FusedEXL3Group._table, which makes and keeps the block table of a row count: (blocks, row_src, suh_row).
// Only this path needs one.
void group_gemv(const Rows& x, int64_t rows, const Group& g, PyObject* table, PyObject* x_object, const at::Tensor& y,
                unsigned flags, int dev, cudaStream_t s)
{
    const Owned device{PyObject_GetAttrString(x_object, "device")};
    if (!device.p) throw PyError();
    const Owned t{PyObject_CallFunction(table, "LO", (long long)rows, device.p)};
    if (!t.p) throw PyError();
    if (!PyTuple_Check(t.p) || PyTuple_GET_SIZE(t.p) != 3) fail(PyExc_TypeError, "a table of three tensors is expected");
    const at::Tensor& b = tensor(PyTuple_GET_ITEM(t.p, 0), "blocks");
    const int32_t* row_src = ptr_or_null<int32_t>(PyTuple_GET_ITEM(t.p, 1), "row_src");
    const int32_t* suh_row = ptr_or_null<int32_t>(PyTuple_GET_ITEM(t.p, 2), "suh_row");
    const int32_t* blocks = static_cast<const int32_t*>(b.data_ptr());
    const Workspace ws = workspace(dev, api.exl3_workspace_bytes(rows * g.members, 16 * g.w.t_in));
    launch(dev, "exl3_gemv_blocks", [&] {
        return api.exl3_gemv_blocks(x.t.data_ptr(), x.dtype, x.stride, rows * g.members, row_src, g.suh, suh_row,
                                    g.w.trellis, g.w.t_in, g.w.t_out, g.k, g.cb, blocks, b.size(0), (int)rows, g.svh,
                                    nullptr, u16(y), g.total, 0, ws.ptr, ws.bytes, flags, (exl3_stream_t)s);
    });
}
// All members into the columns of one (rows, total) matrix (packed), or one matrix each.
void group_gemm(const Rows& x, int64_t rows, const Group& g, const int64_t* widths, const uint64_t* y, const int64_t* strides,
                int dev, cudaStream_t s)
{
    const Workspace ws = workspace(dev, api.exl3_gemm_workspace_bytes(rows * g.members, 16 * g.w.t_in));
    launch(dev, "exl3_gemm_members", [&] {
        return api.exl3_gemm_members(x.t.data_ptr(), x.dtype, rows, x.stride, g.w.trellis, g.w.t_in, g.w.t_out, g.k,
                                     g.cb, g.suh, g.svh, (int)g.members, widths, y, strides, ws.ptr, ws.bytes, 0,
                                     (exl3_stream_t)s);
    });
}

// All members side by side in one (rows, total) matrix.
void group_gemm_packed(const Rows& x, const Group& g, PyObject* width_tuple, const at::Tensor& y, int dev, cudaStream_t s)
{
    c10::SmallVector<int64_t, 4> widths, strides;
    c10::SmallVector<uint64_t, 4> ptrs;
    uint64_t at = reinterpret_cast<uint64_t>(y.data_ptr());
    for (int64_t i = 0; i < g.members; i++) {
        widths.push_back(integer(PyTuple_GET_ITEM(width_tuple, i)));
        strides.push_back(g.total);
        ptrs.push_back(at);
        at += 2 * (uint64_t)widths.back();
    }
    group_gemm(x, x.rows, g, widths.data(), ptrs.data(), strides.data(), dev, s);
}

// group_packed(x2d, group..., table, flags, widths) -> (rows, total), rows <= 16
PyObject* group_packed(PyObject* const* arg)
{
    const at::Tensor& x = cuda_tensor(arg[0], "x");
    const Group g = group_of(arg + 1);
    const int64_t in = 16 * g.w.t_in;
    if (x.dim() != 2 || x.size(1) != in)
        fail(PyExc_ValueError, "x has " + std::to_string(x.size(-1)) + " features, layer expects " + std::to_string(in));
    const Rows r = rows_of(x, in);
    const c10::cuda::CUDAGuard guard(x.device());
    const int dev = x.device().index();
    at::Tensor y = empty_half({r.rows, g.total}, x.device());
    const cudaStream_t s = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    if (g.members > kMaxMembers || use_gemv(r.rows, g.svh, nullptr, u16(y), g.total))
        group_gemv(r, r.rows, g, arg[8], arg[0], y, (unsigned)integer(arg[9]), dev, s);
    else
        group_gemm_packed(r, g, arg[10], y, dev, s);
    return THPVariable_Wrap(std::move(y));
}

// group_prefill(x2d, group..., widths) -> one (rows, width) tensor per member
PyObject* group_prefill(PyObject* const* arg)
{
    const at::Tensor& x = cuda_tensor(arg[0], "x");
    const Group g = group_of(arg + 1);
    const Rows r = rows_of(x, 16 * g.w.t_in);
    const c10::cuda::CUDAGuard guard(x.device());
    const int dev = x.device().index();
    c10::SmallVector<at::Tensor, 4> outs;
    c10::SmallVector<int64_t, 4> widths;
    c10::SmallVector<uint64_t, 4> ptrs;
    for (int64_t i = 0; i < g.members; i++) {
        widths.push_back(integer(PyTuple_GET_ITEM(arg[8], i)));
        outs.push_back(empty_half({r.rows, widths.back()}, x.device()));
        ptrs.push_back(reinterpret_cast<uint64_t>(outs.back().data_ptr()));
    }
    group_gemm(r, r.rows, g, widths.data(), ptrs.data(), widths.data(), dev,
               c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream());
    PyObject* t = PyTuple_New(g.members);
    if (!t) throw PyError();
    for (int64_t i = 0; i < g.members; i++) PyTuple_SET_ITEM(t, i, THPVariable_Wrap(std::move(outs[i])));
    return t;
}

// mlp(x2d, group..., table, down trellis, k, cb, suh, svh, bias, group flags, down flags)
// -> (rows, out): gate|up, then down with the GLU (part of the down flags) applied while it loads.
PyObject* mlp(PyObject* const* arg)
{
    const at::Tensor& x = cuda_tensor(arg[0], "x");
    const Group g = group_of(arg + 1);
    const Weights d = weights(arg[9]);
    const Rows r = rows_of(x, 16 * g.w.t_in);
    const c10::cuda::CUDAGuard guard(x.device());
    const int dev = x.device().index();
    const cudaStream_t s = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    const int dk = (int)integer(arg[10]), dcb = (int)integer(arg[11]);
    const uint16_t* suh = ptr_or_null<uint16_t>(arg[12], "suh");
    const uint16_t* svh = ptr_or_null<uint16_t>(arg[13], "svh");
    const uint16_t* bias = ptr_or_null<uint16_t>(arg[14], "bias");
    const unsigned gflags = (unsigned)integer(arg[15]), dflags = (unsigned)integer(arg[16]);
    const at::Tensor gu = empty_half({r.rows, g.total}, x.device());
    at::Tensor y = empty_half({r.rows, 16 * d.t_out}, x.device());
    const Rows h{gu, r.rows, g.total, EXL3_DT_F16};
    if (use_gemv(r.rows, svh, bias, g.svh, 0)) {
        group_gemv(r, r.rows, g, arg[8], arg[0], gu, gflags, dev, s);
        gemv(h, r.rows, d, dk, dcb, suh, svh, bias, u16(y), 16 * d.t_out, dflags, dev, s);
    } else {
        const int64_t half = g.total / 2, widths[2] = {half, half}, strides[2] = {g.total, g.total};
        const uint64_t base = reinterpret_cast<uint64_t>(gu.data_ptr()), ptrs[2] = {base, base + 2 * (uint64_t)half};
        group_gemm(r, r.rows, g, widths, ptrs, strides, dev, s);
        const Workspace ws = workspace(dev, api.exl3_gemm_workspace_bytes(r.rows, 16 * d.t_in));
        launch(dev, "exl3_gemm", [&] {
            return api.exl3_gemm(gu.data_ptr(), EXL3_DT_F16, r.rows, g.total, d.trellis, d.t_in, d.t_out, dk, dcb,
                                 suh, svh, bias, u16(y), 16 * d.t_out, ws.ptr, ws.bytes, dflags, (exl3_stream_t)s);
        });
    }
    return THPVariable_Wrap(std::move(y));
}

// ---- stacked-expert SwitchGLU ---------------------------------------------------------------------------------
// Few tokens by expert instead of by pairs (exl3_moe_plan.h), remembered for the shapes seen last: some us to find out, 0.02 to look up.
// The tile kernel wants the output scales on 16 bytes, where the GEMV takes 8.
bool by_expert(int64_t pairs, int64_t experts, int64_t d, int64_t h, int k, const uint16_t* gu_svh, const uint16_t* dn_svh)
{
    if ((reinterpret_cast<uintptr_t>(gu_svh) | reinterpret_cast<uintptr_t>(dn_svh)) % 16) return false;
    struct Slot { int64_t pairs, experts, d, h; int k; bool answer; };
    static thread_local Slot memo[16] = {};
    Slot& m = memo[((uint64_t)pairs * 0x9E3779B97F4A7C15u ^ (uint64_t)k * 0xC2B2AE3D27D4EB4Fu) >> 60];
    if (m.pairs != pairs || m.experts != experts || m.d != d || m.h != h || m.k != k)
        m = Slot{pairs, experts, d, h, k, exl3::moe_by_expert(pairs, experts, d, h, k)};
    return m.answer;
}

// switch_glu(x2d, indices (R, k), gu_trellis, gu_suh, gu_svh, dn_trellis, dn_suh, dn_svh, experts, hidden, k, cb,
//            glu flag, flags, decode) -> (R, k, D)
PyObject* switch_glu(PyObject* const* arg)
{
    const at::Tensor& x = cuda_tensor(arg[0], "x");
    at::Tensor idx = cuda_tensor(arg[1], "indices");
    const Weights gu = weights(arg[2]), dn = weights(arg[5]);
    const uint16_t *gu_suh = ptr_or_null<uint16_t>(arg[3], "gu_suh"), *gu_svh = ptr_or_null<uint16_t>(arg[4], "gu_svh");
    const uint16_t *dn_suh = ptr_or_null<uint16_t>(arg[6], "dn_suh"), *dn_svh = ptr_or_null<uint16_t>(arg[7], "dn_svh");
    const int64_t E = integer(arg[8]), H = integer(arg[9]), D = 16 * gu.t_in;
    const int k = (int)integer(arg[10]), cb = (int)integer(arg[11]);
    const unsigned glu = (unsigned)integer(arg[12]), flags = (unsigned)integer(arg[13]);
    if (idx.scalar_type() != at::kInt && idx.scalar_type() != at::kLong) {
        const NoGil unlocked;
        idx = idx.to(at::kLong);
    }
    idx = dense(idx);
    const int64_t R = idx.size(0), kk = idx.size(1), n = R * kk;
    const int bytes = idx.scalar_type() == at::kInt ? 4 : 8;
    const Rows r = rows_of(x, D);
    const at::Device device = x.device();
    const c10::cuda::CUDAGuard guard(device);
    const int dev = device.index();
    const cudaStream_t s = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    const exl3_stream_t es = (exl3_stream_t)s;
    const at::Tensor ygu = empty_half({n, 2 * H}, device);
    at::Tensor y = empty_half({R, kk, D}, device);
    if (n == 0) return THPVariable_Wrap(std::move(y));
    if (PyObject_IsTrue(arg[14]) && !by_expert(n, E, D, H, k, gu_svh, dn_svh)) {
        // tables, gate|up, down with the GLU on load
        const int64_t gb = H / 128, db = D / 128, n_gu = n * 2 * gb, n_dn = n * db;
        const at::Tensor tab = empty_int(4 * (n_gu + n_dn) + 5 * n, device);
        int32_t* blocks_gu = static_cast<int32_t*>(tab.data_ptr());
        int32_t *blocks_dn = blocks_gu + 4 * n_gu, *row_src = blocks_dn + 4 * n_dn, *suh_row = row_src + 2 * n, *sel = suh_row + 2 * n;
        launch(dev, "exl3_moe_decode_tables", [&] {
            return api.exl3_moe_decode_tables(idx.data_ptr(), bytes, (int)n, (int)kk, (int)E, D, H, blocks_gu,
                                              row_src, suh_row, blocks_dn, sel, flags, es);
        });
        Workspace ws = workspace(dev, api.exl3_workspace_bytes(2 * n, D));
        launch(dev, "exl3_gemv_blocks", [&] {
            return api.exl3_gemv_blocks(r.t.data_ptr(), r.dtype, r.stride, 2 * n, row_src, gu_suh, suh_row,
                                        gu.trellis, gu.t_in, gu.t_out, k, cb, blocks_gu, n_gu, 1, gu_svh, nullptr,
                                        u16(ygu), 2 * H, 0, ws.ptr, ws.bytes, flags, es);
        });
        ws = workspace(dev, api.exl3_workspace_bytes(n, H));
        launch(dev, "exl3_gemv_blocks", [&] {
            return api.exl3_gemv_blocks(ygu.data_ptr(), EXL3_DT_F16, 2 * H, n, nullptr, dn_suh, sel, dn.trellis,
                                        dn.t_in, dn.t_out, k, cb, blocks_dn, n_dn, 1, dn_svh, nullptr, u16(y), D, 0,
                                        ws.ptr, ws.bytes, flags | glu, es);
        });
    } else {
        // tables, rotation, gate|up, rotation with the GLU on load, down stored back into pair order
        const int64_t slots = n / 256 + E, ct_h = (H + 255) / 256, ct_d = (D + 255) / 256;
        const int64_t n_gu = 2 * slots * ct_h, n_dn = slots * ct_d;
        const at::Tensor tab = empty_int(8 * (n_gu + n_dn) + 6 * n, device);
        int32_t* tiles_gu = static_cast<int32_t*>(tab.data_ptr());
        int32_t *tiles_dn = tiles_gu + 8 * n_gu, *order = tiles_dn + 8 * n_dn, *row_src = order + n, *suh_gu = row_src + 2 * n,
                *suh_dn = suh_gu + 2 * n;
        launch(dev, "exl3_moe_prefill_tables", [&] {
            return api.exl3_moe_prefill_tables(idx.data_ptr(), bytes, (int)n, (int)kk, (int)E, D, H, order, row_src,
                                               suh_gu, suh_dn, tiles_gu, tiles_dn, EXL3_FLAG_ROW_PAIRS, es);
        });
        const unsigned hint = (unsigned)std::max<int64_t>(1, std::min<int64_t>(n / E, 0xFFFF)) << 16;      // rows of an expert
        const unsigned wide = PyObject_IsTrue(arg[14]) ? EXL3_FLAG_WIDE_SCALES : 0u;      // few tokens: what the GEMV would give
        // The tile kernel keeps nothing but the rotated rows in the workspace.  Few tokens ask for what their way by pairs does, so
        // that a call which fits the workspace (one that is captured behind a warm-up of other sizes) does not make it grow.
        auto scratch = [&](int64_t rows, int64_t in) { return wide ? api.exl3_workspace_bytes(rows, in) : api.exl3_gemm_workspace_bytes(rows, in); };
        Workspace ws = workspace(dev, scratch(2 * n, D));
        launch(dev, "exl3_gemm_tiles", [&] {
            return api.exl3_gemm_tiles(r.t.data_ptr(), r.dtype, r.stride, 2 * n, row_src, gu_suh, suh_gu,
                                       gu.trellis, gu.t_in, gu.t_out, k, cb, tiles_gu, n_gu, gu_svh, u16(ygu), 2 *
                                       H, nullptr, ws.ptr, ws.bytes, hint | wide | EXL3_FLAG_ROW_PAIRS, es);
        });
        ws = workspace(dev, scratch(n, H));
        launch(dev, "exl3_gemm_tiles", [&] {
            return api.exl3_gemm_tiles(ygu.data_ptr(), EXL3_DT_F16, 2 * H, n, nullptr, dn_suh, suh_dn, dn.trellis,
                                       dn.t_in, dn.t_out, k, cb, tiles_dn, n_dn, dn_svh, u16(y), D, order, ws.ptr,
                                       ws.bytes, glu | hint | wide, es);
        });
    }
    return THPVariable_Wrap(std::move(y));
}

// ---- the module ------------------------------------------------------------------------------------------------
// bind({name: address}, check, grow)
PyObject* bind(PyObject* const* arg)
{
    if (!PyDict_Check(arg[0])) fail(PyExc_TypeError, "a dict of addresses is expected");
#define EXL3_BIND(name)                                                                  \
    {                                                                                    \
        PyObject* v = PyDict_GetItemString(arg[0], #name);                               \
        if (!v) fail(PyExc_KeyError, #name);                                             \
        api.name = reinterpret_cast<decltype(api.name)>(PyLong_AsVoidPtr(v));            \
        if (PyErr_Occurred()) throw PyError();                                           \
    }
    EXL3_BIND(exl3_workspace_bytes)
    EXL3_BIND(exl3_gemm_workspace_bytes)
    EXL3_BIND(exl3_gemv)
    EXL3_BIND(exl3_gemm)
    EXL3_BIND(exl3_gemm_members)
    EXL3_BIND(exl3_gemv_blocks)
    EXL3_BIND(exl3_gemm_tiles)
    EXL3_BIND(exl3_moe_decode_tables)
    EXL3_BIND(exl3_moe_prefill_tables)
#undef EXL3_BIND
    Py_XSETREF(check_fn, Py_NewRef(arg[1]));
    Py_XSETREF(grow_fn, Py_NewRef(arg[2]));
    Py_RETURN_NONE;
}

// set_workspace(device index, address, bytes)
PyObject* set_workspace(PyObject* const* arg)
{
    const int64_t dev = integer(arg[0]);
    if (dev < 0 || dev >= kMaxDevices) fail(PyExc_ValueError, "device index out of range");
    workspaces[dev].ptr = PyLong_AsVoidPtr(arg[1]);
    if (PyErr_Occurred()) throw PyError();
    workspaces[dev].bytes = (size_t)integer(arg[2]);
    Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject* const*), int N> PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    HANDLE_TH_ERRORS
    if (nargs != N) {
        PyErr_Format(PyExc_TypeError, "%d arguments expected, got %zd", N, nargs);
        return nullptr;
    }
    try {
        return F(args);
    } catch (const PyError&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

#define EXL3_METHOD(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(call<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    EXL3_METHOD(bind, 3),
    EXL3_METHOD(set_workspace, 3),
    EXL3_METHOD(linear, 9),
    EXL3_METHOD(group_packed, 11),
    EXL3_METHOD(group_prefill, 9),
    EXL3_METHOD(mlp, 17),
    EXL3_METHOD(switch_glu, 15),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_exl3_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__exl3_host(void) { return PyModule_Create(&module_def); }
