// Host side of the attention operators: argument checks, output allocation and the library call without the interpreter in
// between.  Done in Python these cost 10 to 15 us per operator (attribute look-ups, shape and stride tuples, ctypes
// conversions), which is what bounded the operators of a single image: 8 us of kernel time each.
//
// The library's functions are bound at run time (bind), so that one copy of the library -- whichever the process chose --
// serves both this module and ctypes.  Everything runs on the inputs' device and torch's current stream there.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "../../include/clusten_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

struct Library {
    decltype(&clusten_status_string) status_string;
    decltype(&clusten_qk_forward_views) qk_forward;
    decltype(&clusten_av_forward_views) av_forward;
    decltype(&clusten_qk_backward_views) qk_backward;
    decltype(&clusten_av_backward_views) av_backward;
    decltype(&clusten_local_attention_forward) local_attention;
    decltype(&clusten_groups_bytes) groups_bytes;
    decltype(&clusten_groups_build) groups_build;
} lib;

void bind(const std::vector<unsigned long long>& a) {
    TORCH_CHECK(a.size() == 8, "clusten: eight functions to bind");
    lib.status_string = reinterpret_cast<decltype(lib.status_string)>(a[0]);
    lib.qk_forward = reinterpret_cast<decltype(lib.qk_forward)>(a[1]);
    lib.av_forward = reinterpret_cast<decltype(lib.av_forward)>(a[2]);
    lib.qk_backward = reinterpret_cast<decltype(lib.qk_backward)>(a[3]);
    lib.av_backward = reinterpret_cast<decltype(lib.av_backward)>(a[4]);
    lib.local_attention = reinterpret_cast<decltype(lib.local_attention)>(a[5]);
    lib.groups_bytes = reinterpret_cast<decltype(lib.groups_bytes)>(a[6]);
    lib.groups_build = reinterpret_cast<decltype(lib.groups_build)>(a[7]);
}

struct Strides {                                 // of a [b, h, n, .] tensor, in elements
    long long v[3];
    explicit Strides(const Tensor& t) : v{t.stride(0), t.stride(1), t.stride(2)} {}
};

int dtype_of(const Tensor& t) {                  // -1: not one of the kernels' types
    switch (t.scalar_type()) {
        case at::kFloat: return CLUSTEN_F32;
        case at::kHalf: return CLUSTEN_F16;
        case at::kBFloat16: return CLUSTEN_BF16;
        default: return -1;
    }
}

void fail(int status) {
    throw std::runtime_error(std::string("clusten: ") + lib.status_string(status) + " (status " + std::to_string(status) + ")");
}
void require(bool ok, const char* what) {
    if (!ok) throw std::runtime_error(std::string("clusten: ") + what);
}

// fn(..., stream) on t's device; the interpreter may run other threads meanwhile
template <typename F> int launch(const Tensor& t, F&& fn) {
    py::gil_scoped_release release;
    c10::cuda::CUDAGuard guard(t.device());
    return fn(c10::cuda::getCurrentCUDAStream(t.get_device()).stream());
}

// [b, h, n, 32] that the kernels read in place: rows contiguous, the other strides and the base address multiples of 16 bytes
bool row_view(const Tensor& t) {
    if (!t.is_cuda() || t.dim() != 4 || t.size(3) != 32 || t.stride(3) != 1) return false;
    const int64_t per = 16 / (int64_t)t.element_size();
    for (int i = 0; i < 3; ++i)
        if (t.stride(i) <= 0 || t.stride(i) % per != 0) return false;
    return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
}
// [b, h, n, m]: rows contiguous, anywhere
bool rows(const Tensor& t) {
    return t.is_cuda() && t.dim() == 4 && (t.stride(3) == 1 || t.size(3) == 1) && t.stride(0) >= 0 && t.stride(1) >= 0 && t.stride(2) > 0;
}
// the table of rows of width 1 .. 64 (fp32: 48);  its sizes are checked separately (what is no table at all the caller's checks name)
bool table(const Tensor& first, const Tensor& second, const Tensor& idx) {
    return first.scalar_type() == second.scalar_type() && (first.scalar_type() == at::kFloat || first.scalar_type() == at::kHalf || first.scalar_type() == at::kBFloat16) &&
           idx.is_cuda() && idx.dim() == 3 && idx.scalar_type() == at::kLong && idx.size(2) >= 1 && idx.size(2) <= (first.scalar_type() == at::kFloat ? 48 : 64) && idx.is_contiguous();
}
bool table_of(const Tensor& idx, const Tensor& like, int64_t b, int64_t n, int64_t m) {
    return idx.dim() == 3 && idx.size(0) == b && idx.size(1) == n && idx.size(2) == m && idx.scalar_type() == at::kLong && idx.device() == like.device();
}
const void* ptr(const OptTensor& t) { return t ? t->const_data_ptr() : nullptr; }
const int64_t* i64(const Tensor& t) { return static_cast<const int64_t*>(t.const_data_ptr()); }

// Do the kernels take these arguments as they are?  (No: the caller makes them contiguous.)  Sizes that do not fit raise.
bool qk_takes(const Tensor& q, const Tensor& k, const Tensor& idx) {
    if (!row_view(q) || !row_view(k) || !table(q, k, idx)) return false;
    require(k.sizes() == q.sizes() && k.device() == q.device() && table_of(idx, q, q.size(0), q.size(2), idx.size(2)), "QK shape mismatch");
    return true;
}
bool av_takes(const Tensor& a, const Tensor& v, const Tensor& idx) {
    if (!rows(a) || !row_view(v) || !table(a, v, idx)) return false;
    require(v.size(0) == a.size(0) && v.size(1) == a.size(1) && v.size(2) == a.size(2) && v.device() == a.device() &&
                table_of(idx, a, a.size(0), a.size(2), a.size(3)), "AV shape mismatch");
    return true;
}
bool qk_backward_takes(const Tensor& g, const Tensor& q, const Tensor& k, const Tensor& idx) {
    if (!rows(g) || g.scalar_type() != q.scalar_type() || !row_view(q) || !row_view(k) || !table(q, k, idx)) return false;
    require(g.size(0) == q.size(0) && g.size(1) == q.size(1) && g.size(2) == q.size(2) && g.size(3) == idx.size(2) && g.device() == q.device() &&
                k.sizes() == q.sizes() && k.device() == q.device() && table_of(idx, q, q.size(0), q.size(2), idx.size(2)),
            "QK backward shape mismatch");
    return true;
}
bool av_backward_takes(const Tensor& g, const Tensor& a, const Tensor& v, const Tensor& idx) {
    if (!row_view(g) || g.scalar_type() != a.scalar_type() || !rows(a) || !row_view(v) || !table(a, v, idx)) return false;
    require(g.sizes() == v.sizes() && g.device() == a.device() && v.size(0) == a.size(0) && v.size(1) == a.size(1) && v.size(2) == a.size(2) &&
                v.device() == a.device() && table_of(idx, a, a.size(0), a.size(2), a.size(3)), "AV backward shape mismatch");
    return true;
}

// Records of a table (clusten_groups_build) for one forward call.  They are made from the indices as they are now and never kept
// for a later forward call: a table can change without a trace that could be checked (a replayed graph, another library's kernel),
// and a buffer of another stream or of a capture need not have been written yet.
// When they pay within the call -- QK / AV, us with the build against without: not for rows of 48, which the kernels analyse at compile-time
// sizes.  With two heads nothing is gained (b128 h2 n3136 bf16 93 / 94 against 91 / 93, tables shared by a cluster 112 / 93 against 99 / 83);
// with eight it depends on what the host does not know: whole clusters gain in 16 bits (b32 h8 n1843 47 / 49 against 56 / 58, b64 h8 n784 36 / 37
// against 42 / 50, b128 h8 n196 22 / 24 against 23 / 27), shared tables lose (60 / 48 against 55 / 45, 45 / 37 against 46 / 41, 23 / 24 against
// 23 / 25).  Other rows from 2 M scores on (b256 h16 n49 m49 bf16 38 / 37 against 46 / 42, b64 h8 n784 m24 whole clusters bf16 38 / 42 against 41 / 45,
// fp32 75 / 73 against 82 / 74, shared 64 / 63 against 79 / 57, b64 h2 n3136 m40 shared bf16 70 / 65 against 69 / 63; below: b4 h8 n784 m24 bf16
// 9 / 10 against 8 / 9).
constexpr int64_t kRecordsMinScores = int64_t(1) << 21;
OptTensor records(const Tensor& idx, int heads, int n, bool wanted, int& status) {
    status = CLUSTEN_OK;
    const int b = idx.size(0), rows = idx.size(1), m = idx.size(2);
    if (!wanted && (m == 48 || idx.numel() * heads < kRecordsMinScores)) return std::nullopt;
    const size_t bytes = lib.groups_bytes(b, rows, m, n);
    if (bytes == 0) return std::nullopt;
    Tensor groups = at::empty({(int64_t)(bytes / 4)}, idx.options().dtype(at::kInt));
    status = launch(idx, [&](void* s) { return lib.groups_build(i64(idx), b, rows, m, n, groups.data_ptr(), bytes, s); });
    return groups;
}

// The calls: arguments that *_takes accepted, groups and inverse from their builds.  None: sizes without a kernel.
// Forward: (result, records or None);  wanted: a backward pass will need the records.
py::object qk_forward(const Tensor& q, const Tensor& k, const Tensor& idx, bool wanted) {
    const int b = q.size(0), h = q.size(1), n = q.size(2), m = idx.size(2);
    int st;
    const OptTensor groups = records(idx, h, n, wanted, st);
    if (st != CLUSTEN_OK) fail(st);
    Tensor out = at::empty({b, h, n, m}, q.options());
    st = launch(q, [&](void* s) {
        return lib.qk_forward(q.const_data_ptr(), Strides(q).v, k.const_data_ptr(), Strides(k).v, i64(idx), ptr(groups), out.data_ptr(), b, h, n, m,
                              32, dtype_of(q), s);
    });
    if (st == CLUSTEN_ERR_UNSUPPORTED) return py::none();
    if (st != CLUSTEN_OK) fail(st);
    return py::make_tuple(out, groups);
}
py::object av_forward(const Tensor& a, const Tensor& v, const Tensor& idx, bool wanted) {
    const int b = a.size(0), h = a.size(1), n = a.size(2), m = a.size(3);
    int st;
    const OptTensor groups = records(idx, h, n, wanted, st);
    if (st != CLUSTEN_OK) fail(st);
    Tensor out = at::empty({b, h, n, 32}, a.options());
    st = launch(a, [&](void* s) {
        return lib.av_forward(a.const_data_ptr(), Strides(a).v, v.const_data_ptr(), Strides(v).v, i64(idx), ptr(groups), out.data_ptr(), b, h, n, m,
                              32, dtype_of(a), s);
    });
    if (st == CLUSTEN_ERR_UNSUPPORTED) return py::none();
    if (st != CLUSTEN_OK) fail(st);
    return py::make_tuple(out, groups);
}
py::object qk_backward(const Tensor& g, const Tensor& q, const Tensor& k, const Tensor& idx, const Tensor& groups, const Tensor& inverse) {
    const int b = q.size(0), h = q.size(1), n = q.size(2), m = idx.size(2);
    Tensor dq = at::empty({b, h, n, 32}, q.options()), dk = at::empty({b, h, n, 32}, q.options());
    const int st = launch(q, [&](void* s) {
        return lib.qk_backward(g.const_data_ptr(), Strides(g).v, q.const_data_ptr(), Strides(q).v, k.const_data_ptr(), Strides(k).v, i64(idx),
                               groups.const_data_ptr(), inverse.const_data_ptr(), dq.data_ptr(), dk.data_ptr(), b, h, n, m, 32, dtype_of(q), s);
    });
    if (st == CLUSTEN_ERR_UNSUPPORTED) return py::none();
    if (st != CLUSTEN_OK) fail(st);
    return py::make_tuple(dq, dk);
}
py::object av_backward(const Tensor& g, const Tensor& a, const Tensor& v, const Tensor& idx, const Tensor& groups, const Tensor& inverse) {
    const int b = a.size(0), h = a.size(1), n = a.size(2), m = a.size(3);
    Tensor da = at::empty({b, h, n, m}, a.options()), dv = at::empty({b, h, n, 32}, a.options());
    const int st = launch(a, [&](void* s) {
        return lib.av_backward(g.const_data_ptr(), Strides(g).v, a.const_data_ptr(), Strides(a).v, v.const_data_ptr(), Strides(v).v, i64(idx),
                               groups.const_data_ptr(), inverse.const_data_ptr(), da.data_ptr(), dv.data_ptr(), b, h, n, m, 32, dtype_of(a), s);
    });
    if (st == CLUSTEN_ERR_UNSUPPORTED) return py::none();
    if (st != CLUSTEN_OK) fail(st);
    return py::make_tuple(da, dv);
}

// An ordinary tensor that no derivative is asked of: the call needs nothing of autograd's machinery
bool ordinary(const Tensor& t) {
    using c10::DispatchKey;
    return !t._fw_grad(0).defined() && !t.key_set().has_any(c10::DispatchKeySet({DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchGradWrapper,
                                                                                 DispatchKey::Functionalize, DispatchKey::Python, DispatchKey::Negative}));
}
// (a trace sees the operator by its node only)
bool without_grad(const Tensor& a, const Tensor& b, const Tensor& idx) {
    return !torch::jit::tracer::isTracing() && (!at::GradMode::is_enabled() || (!a.requires_grad() && !b.requires_grad())) && ordinary(a) && ordinary(b) && ordinary(idx);
}

bool dense(const OptTensor& t, const Tensor& like, at::ScalarType type, at::IntArrayRef shape) {
    return !t || (t->device() == like.device() && t->is_contiguous() && t->scalar_type() == type && t->sizes() == shape);
}
// None: some argument is not as the kernel takes it (the caller finds out which)
py::object local_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const OptTensor& bias, const OptTensor& pe_table,
                           const OptTensor& pe_idx, const OptTensor& mask, const OptTensor& blank_k, const OptTensor& blank_v) {
    const int dt = dtype_of(q);
    const auto type = q.scalar_type();
    if (dt < 0 || !row_view(q) || !row_view(k) || !row_view(v) || k.strides() != v.strides() || k.scalar_type() != type || v.scalar_type() != type ||
        k.sizes() != q.sizes() || v.sizes() != q.sizes() || k.device() != q.device() || v.device() != q.device())
        return py::none();
    if (idx.dim() != 3 || !idx.is_contiguous() || !table_of(idx, q, q.size(0), q.size(2), idx.size(2))) return py::none();
    const int b = q.size(0), h = q.size(1), n = q.size(2), m = idx.size(2);
    if (!dense(bias, q, type, {b, h, n, m}) || !dense(pe_idx, q, at::kLong, {b, n, m}) || !dense(mask, q, at::kLong, {b, n, m}) ||
        !dense(blank_k, q, type, {h, 32}) || !dense(blank_v, q, type, {h, 32}))
        return py::none();
    if (pe_table && (!pe_idx || pe_table->device() != q.device() || !pe_table->is_contiguous() || pe_table->dim() != 2 || pe_table->size(1) != h ||
                     pe_table->scalar_type() != type))
        return py::none();
    Tensor out = at::empty({b, h, n, 32}, q.options());
    const int st = launch(q, [&](void* s) {
        return lib.local_attention(q.const_data_ptr(), Strides(q).v, k.const_data_ptr(), v.const_data_ptr(), Strides(k).v, i64(idx), ptr(bias),
                                   ptr(pe_table), static_cast<const int64_t*>(ptr(pe_idx)), pe_table ? (int)pe_table->size(0) : 0,
                                   static_cast<const int64_t*>(ptr(mask)), ptr(blank_k), ptr(blank_v), out.data_ptr(), b, h, n, m, 32, dt, s);
    });
    if (st != CLUSTEN_OK) fail(st);
    return py::cast(out);
}

}  // namespace

PYBIND11_MODULE(_host, m) {
    m.def("bind", &bind);
    m.def("qk_takes", &qk_takes);
    m.def("av_takes", &av_takes);
    m.def("qk_backward_takes", &qk_backward_takes);
    m.def("av_backward_takes", &av_backward_takes);
    m.def("qk_forward", &qk_forward);
    m.def("av_forward", &av_forward);
    m.def("qk_backward", &qk_backward);
    m.def("av_backward", &av_backward);
    m.def("without_grad", &without_grad);
    m.def("local_attention", &local_attention);
}
