// The host side of an ordinary eager call, in C++: argument checks, output allocation, workspace, the autograd
// node and the call into libplx_sm100.so.
//
// Everything here is a SHORT CUT of the Python path (train.py / decode.py over the torch custom ops of ops.py),
// which stays the definition of the API: each function returns None, with nothing enqueued that shows, for any
// call that is not plainly an eager one on well-formed CUDA tensors -- a tensor subclass, a torch function or
// dispatch mode, functorch or forward-mode differentiation, tracing, shapes, strides or types that need a copy or an
// error message -- and the caller then takes the Python path, which handles it or raises.  decode, extend and step also
// leave a stream that is being captured to it; train and extend a device error waiting to be reported (the ops
// of a single-token step do not look at it either).  decode and extend find a length out of range after their launch,
// whose result is then dropped.
//
// Measured per call, Python path -> here: decode at B = 1, H = 8, 1024 keys 52 -> 6.4 us; training forward and backward
// at B = 2, H = 8, L = 1024 303 -> 100 us (24 us of host time forward; 70 us backward, 28 of them in Train::backward).
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <array>
#include <cmath>
#include <cstdlib>
#include <list>
#include <map>
#include <memory>
#include <mutex>
#include <optional>

#include "../../include/plx_abi.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using Tensors = std::initializer_list<const Tensor *>;
using Values = std::vector<c10::IValue>;   // what a profiler is shown of a call, under the name of the op it stands for

enum Layout { kBHLD = 0, kBTHD = 1 };

// entry points of the loaded libplx_sm100.so (the one ops.py calls; set once by bind())
struct Api {
    decltype(&plx_device_error_peek) device_error_peek;
    decltype(&plx_train_workspace_bytes) train_workspace_bytes;
    decltype(&plx_train_fwd) train_fwd;
    decltype(&plx_train_bwd) train_bwd;
    decltype(&plx_train_extend) train_extend;
    decltype(&plx_decode_choose_splits_gqa) decode_choose_splits_gqa;
    decltype(&plx_decode_workspace_bytes) decode_workspace_bytes;
    decltype(&plx_decode) decode;
    decltype(&plx_decode_stage) decode_stage;
    decltype(&plx_decode_step) decode_step;
};
Api api;

template <typename F>
void bind_one(F &slot, const py::dict &addresses, const char *name) {
    slot = reinterpret_cast<F>(addresses[name].cast<uintptr_t>());
}
void bind(const py::dict &addresses) {
    bind_one(api.device_error_peek, addresses, "plx_device_error_peek");
    bind_one(api.train_workspace_bytes, addresses, "plx_train_workspace_bytes");
    bind_one(api.train_fwd, addresses, "plx_train_fwd");
    bind_one(api.train_bwd, addresses, "plx_train_bwd");
    bind_one(api.train_extend, addresses, "plx_train_extend");
    bind_one(api.decode_choose_splits_gqa, addresses, "plx_decode_choose_splits_gqa");
    bind_one(api.decode_workspace_bytes, addresses, "plx_decode_workspace_bytes");
    bind_one(api.decode, addresses, "plx_decode");
    bind_one(api.decode_stage, addresses, "plx_decode_stage");
    bind_one(api.decode_step, addresses, "plx_decode_step");
}

// ------------------------------------------------------------------------- //
// what counts as a plain call
// ------------------------------------------------------------------------- //
// exactly a Tensor or a Parameter, and no torch function mode
bool plain_object(PyObject *o) {
    return (reinterpret_cast<PyObject *>(Py_TYPE(o)) == THPVariableClass || reinterpret_cast<PyObject *>(Py_TYPE(o)) == ParameterClass) &&
           !at::impl::torch_function_mode_enabled();
}

// The tensor of a plain Python object; `ok` is cleared for anything else.
Tensor take(const py::object &o, bool &ok) {
    if (!plain_object(o.ptr())) {
        ok = false;
        return Tensor();
    }
    return THPVariable_Unpack(o.ptr());
}
OptTensor take_optional(const py::object &o, bool &ok) {
    if (o.is_none()) return std::nullopt;
    return take(o, ok);
}
// qk_scale (None: head_dim ** -0.5) and the window as plain Python numbers
bool take_scale(const py::object &o, int64_t head_dim, double &scale) {
    if (o.is_none()) scale = 1.0 / std::sqrt(static_cast<double>(head_dim));
    else if (PyFloat_CheckExact(o.ptr())) scale = PyFloat_AS_DOUBLE(o.ptr());
    else return false;
    return true;
}
bool take_window(const py::object &o, int64_t &window) {
    if (!PyLong_CheckExact(o.ptr())) return false;
    int overflow = 0;
    window = PyLong_AsLongLongAndOverflow(o.ptr(), &overflow);
    return overflow == 0 && window >= -1 && window <= INT32_MAX;
}

// No dispatch key beyond those of an ordinary dense CUDA tensor and its autograd, and no forward-mode tangent.
bool plain_tensor(const Tensor &t) {
    static const c10::DispatchKeySet usual =
        c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                             c10::DispatchKey::AutocastCUDA});
    return t.is_cuda() && (t.key_set().raw_repr() & ~usual.raw_repr()) == 0 && !t._fw_grad(0).defined();
}
bool plain_thread() {
    static const c10::DispatchKeySet usual =
        c10::DispatchKeySet({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView}) | c10::autocast_dispatch_keyset;
    return (c10::impl::tls_local_dispatch_key_set().included_.raw_repr() & ~usual.raw_repr()) == 0;
}

bool capturing() { return at::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

bool device_error_waiting() {
    int32_t v = 0;
    return api.device_error_peek(&v, 0) != PLX_OK || v != 0;
}

int dtype_code(const Tensor &t) {
    return t.scalar_type() == at::kBFloat16 ? PLX_BF16 : t.scalar_type() == at::kHalf ? PLX_FP16 : -1;
}
bool aligned16(const Tensor &t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }

// train.kernel_ready without the copy: last axis contiguous, the other strides multiples of 8 elements, the base
// 16-byte aligned, no gaps or overlap in some axis order.
bool kernel_ready(const Tensor &t) {
    if (t.stride(3) != 1 || !aligned16(t)) return false;
    for (int i = 0; i < 3; ++i)
        if (t.stride(i) % 8 != 0) return false;
    return t.is_non_overlapping_and_dense();
}

const int32_t *int_ptr(const OptTensor &t) { return t ? static_cast<const int32_t *>(t->data_ptr()) : nullptr; }

bool recorded(Tensors tensors) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor *t : tensors)
        if (t->requires_grad()) return true;
    return false;
}

// ------------------------------------------------------------------------- //
// training
// ------------------------------------------------------------------------- //
plx_train_problem train_problem(const Tensor &q, const Tensor &k, const Tensor &stats, double scale, int64_t window, int64_t layout,
                                const OptTensor &cu) {
    const int h = layout == kBHLD ? 1 : 2, l = layout == kBHLD ? 2 : 1;
    plx_train_problem p{};
    p.dtype = dtype_code(q);
    p.batch = static_cast<int32_t>(q.size(0));
    p.heads_q = static_cast<int32_t>(q.size(h));
    p.heads_kv = static_cast<int32_t>(k.size(h));
    p.len_q = static_cast<int32_t>(q.size(l));
    p.len_k = static_cast<int32_t>(k.size(l));
    p.head_dim = static_cast<int32_t>(q.size(3));
    p.window_left = static_cast<int32_t>(window);
    p.qk_scale = static_cast<float>(scale);
    p.q_stride_b = q.stride(0); p.q_stride_h = q.stride(h); p.q_stride_t = q.stride(l);
    p.kv_stride_b = k.stride(0); p.kv_stride_h = k.stride(h); p.kv_stride_t = k.stride(l);
    if (stats.defined()) {
        p.st_stride_b = stats.stride(0); p.st_stride_h = stats.stride(h); p.st_stride_t = stats.stride(l);
    }
    if (cu) {
        p.cu_seqlens = int_ptr(cu);
        p.n_seqs = static_cast<int32_t>(cu->numel() - 1);
    }
    return p;
}

struct Refused {};   // a status of the library that the Python path has to report

// One node for forward and backward, as the custom op plx::train_fwd registers it.
struct Train : torch::autograd::Function<Train> {
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext *ctx, const Tensor &q, const Tensor &r, const Tensor &k, const Tensor &v,
                          double scale, int64_t window, int64_t layout, const OptTensor &cu) {
        at::AutoDispatchBelowADInplaceOrView below;
        const c10::cuda::CUDAGuard device(q.device());
        Tensor o = at::empty_like(q), barv = at::empty_like(q);
        const auto stat = [&] { return at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat)); };
        Tensor d1 = stat(), bart = stat(), m = stat();
        const plx_train_problem p = train_problem(q, k, d1, scale, window, layout, cu);
        if (api.train_fwd(&p, q.data_ptr(), r.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), barv.data_ptr(),
                          d1.data_ptr<float>(), bart.data_ptr<float>(), m.data_ptr<float>(), c10::cuda::getCurrentCUDAStream().stream()) != PLX_OK)
            throw Refused();
        ctx->save_for_backward({q, r, k, v, o, barv, d1, bart, m, cu ? *cu : Tensor()});
        ctx->set_materialize_grads(false);   // gradients of barv and the statistics are not looked at
        ctx->saved_data["scale"] = scale;
        ctx->saved_data["window"] = window;
        ctx->saved_data["layout"] = layout;
        return {o, barv, d1, bart, m};
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &q = saved[0], &r = saved[1], &k = saved[2], &v = saved[3], &o = saved[4], &barv = saved[5], &d1 = saved[6],
                     &bart = saved[7], &m = saved[8];
        const OptTensor cu = saved[9].defined() ? OptTensor(saved[9]) : std::nullopt;
        const double scale = ctx->saved_data["scale"].toDouble();
        const int64_t window = ctx->saved_data["window"].toInt(), layout = ctx->saved_data["layout"].toInt();
        Tensor go = grads[0].defined() ? grads[0] : at::zeros_like(o);
        if (go.strides() != q.strides()) go = at::empty_like(q).copy_(go);   // one stride set for all q-like tensors
        Tensor dq, dr, dk, dv;
        bool done = false;
        // A backward that is itself recorded, traced or transformed goes through the dispatcher, and so does one on
        // saved tensors that a hook has brought back in another form.
        bool plain = !at::GradMode::is_enabled() && plain_thread() && !at::impl::torch_function_mode_enabled();
        for (const Tensor *t : Tensors{&go, &q, &r, &k, &v, &o, &barv, &d1, &bart, &m}) plain = plain && plain_tensor(*t);
        for (const Tensor *t : Tensors{&d1, &bart, &m}) plain = plain && t->is_contiguous();
        for (const Tensor *t : Tensors{&go, &r, &o, &barv}) plain = plain && t->strides() == q.strides() && t->scalar_type() == q.scalar_type();
        plain = plain && v.strides() == k.strides();
        // gradients are written by the strides of q and k, which empty_like reproduces for tensors without gaps only
        plain = plain && q.is_non_overlapping_and_dense() && k.is_non_overlapping_and_dense();
        if (plain) {
            RECORD_FUNCTION("plx::train_bwd", Values({q, r, k, v, o, barv, d1, bart, m, go}));
            at::AutoDispatchBelowADInplaceOrView below;
            const c10::cuda::CUDAGuard device(q.device());
            const plx_train_problem p = train_problem(q, k, d1, scale, window, layout, cu);
            size_t need = 0;
            if (!device_error_waiting() && api.train_workspace_bytes(&p, &need) == PLX_OK) {
                dq = at::empty_like(q);
                dr = at::empty_like(q);
                dk = at::empty_like(k);
                dv = at::empty_like(k);
                const Tensor ws = at::empty({static_cast<int64_t>(need)}, q.options().dtype(at::kByte));
                done = api.train_bwd(&p, q.data_ptr(), r.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), barv.data_ptr(),
                                     d1.data_ptr<float>(), bart.data_ptr<float>(), m.data_ptr<float>(), go.data_ptr(), dq.data_ptr(), dr.data_ptr(), dk.data_ptr(), dv.data_ptr(), ws.data_ptr(), need,
                                     c10::cuda::getCurrentCUDAStream().stream()) == PLX_OK;
            }
        }
        if (!done) {
            static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("plx::train_bwd", "")
                .typed<std::tuple<Tensor, Tensor, Tensor, Tensor>(const Tensor &, const Tensor &, const Tensor &, const Tensor &,
                    const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, double, int64_t, int64_t,
                    const OptTensor &)>();
            std::tie(dq, dr, dk, dv) = op.call(q, r, k, v, o, barv, d1, bart, m, go, scale, window, layout, cu);
        }
        return {dq, dr, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// four tensors that the kernels can address as they are, and whose shapes fit together
bool train_tensors_ok(const Tensor &q, const Tensor &r, const Tensor &k, const Tensor &v, int64_t layout) {
    for (const Tensor *t : Tensors{&q, &r, &k, &v})
        if (!plain_tensor(*t) || t->dim() != 4 || t->scalar_type() != q.scalar_type() || t->device() != q.device() || t->numel() == 0 ||
            !kernel_ready(*t))
            return false;
    const int h = layout == kBHLD ? 1 : 2;
    return dtype_code(q) >= 0 && r.sizes() == q.sizes() && r.strides() == q.strides() && v.sizes() == k.sizes() && v.strides() == k.strides() &&
           k.size(0) == q.size(0) && k.size(3) == q.size(3) && q.size(h) % k.size(h) == 0;
}

bool train_ready(const py::object &q_, const py::object &r_, const py::object &k_, const py::object &v_, int64_t layout) {
    bool ok = true;
    const Tensor q = take(q_, ok), r = take(r_, ok), k = take(k_, ok), v = take(v_, ok);
    return ok && train_tensors_ok(q, r, k, v, layout);
}

// o, barv, d1, bart, m
py::object train(const py::object &q_, const py::object &r_, const py::object &k_, const py::object &v_, const py::object &scale_,
                 const py::object &window_, int64_t layout, const py::object &cu_) {
    bool ok = true;
    const Tensor q = take(q_, ok), r = take(r_, ok), k = take(k_, ok), v = take(v_, ok);
    const OptTensor cu = take_optional(cu_, ok);
    if (!ok || !plain_thread() || !train_tensors_ok(q, r, k, v, layout)) return py::none();
    if (cu && (!plain_tensor(*cu) || cu->scalar_type() != at::kInt || cu->dim() != 1 || !cu->is_contiguous() || cu->device() != q.device() ||
               q.size(0) != 1 || cu->numel() < 2))
        return py::none();
    double scale;
    int64_t window;
    if (!take_scale(scale_, q.size(3), scale) || !take_window(window_, window)) return py::none();
    const c10::cuda::CUDAGuard device(q.device());
    if (device_error_waiting()) return py::none();
    torch::autograd::variable_list res;
    RECORD_FUNCTION("plx::train_fwd", Values({q, r, k, v}));
    try {
        py::gil_scoped_release nogil;
        res = Train::apply(q, r, k, v, scale, window, static_cast<int64_t>(layout), cu);
    } catch (const Refused &) {
        return py::none();
    }
    py::tuple t(res.size());
    for (size_t i = 0; i < res.size(); ++i) t[i] = py::reinterpret_steal<py::object>(THPVariable_Wrap(res[i]));
    return t;
}

// ------------------------------------------------------------------------- //
// decode
// ------------------------------------------------------------------------- //
// Split-KV scratch of eager calls: one per (device, stream, problem shape), zero-filled when made; a launch leaves
// its arrival counters at zero.  At most kMax are kept, the least recently used going back to the allocator: a
// workspace is only ever used on the stream it was allocated on, so the allocator reuses its memory in stream order.
class Workspaces {
public:
    Tensor get(const c10::cuda::CUDAStream &stream, const Tensor &q, int n_splits, int64_t floats) {
        const Key key{q.get_device(), static_cast<int64_t>(reinterpret_cast<uintptr_t>(stream.stream())), q.size(0), q.size(2), q.size(3), n_splits};
        std::lock_guard<std::mutex> lock(mu_);
        for (auto it = list_.begin(); it != list_.end(); ++it)
            if (it->first == key) {
                list_.splice(list_.begin(), list_, it);
                return it->second;
            }
        list_.emplace_front(key, at::zeros({floats}, q.options().dtype(at::kFloat)));
        if (list_.size() > kMax) list_.pop_back();
        return list_.front().second;
    }

private:
    using Key = std::array<int64_t, 6>;
    static constexpr size_t kMax = 32;
    std::mutex mu_;
    std::list<std::pair<Key, Tensor>> list_;
};
Workspaces &workspaces() {
    static Workspaces *w = new Workspaces;   // not destroyed at exit, when the CUDA context may be gone
    return *w;
}

// A stream of this library beside one of the caller's, for small copies that must not stand between two kernels there, and
// the two events of the way there and back (to make and drop two per call was 1 us of it).  Threads that share the caller's stream
// share these: an event that another thread has recorded again is one that comes later on the same stream.
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t ready = nullptr, copied = nullptr;
    SideStream() = default;
    SideStream(const SideStream &) = delete;
    bool make() {
        return cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) == cudaSuccess &&
               cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) == cudaSuccess &&
               cudaEventCreateWithFlags(&copied, cudaEventDisableTiming) == cudaSuccess;
    }
    ~SideStream() {
        if (copied) (void)cudaEventDestroy(copied);
        if (ready) (void)cudaEventDestroy(ready);
        if (stream) (void)cudaStreamDestroy(stream);
    }
};

// One per stream, so that no copy waits for work of a stream that it has nothing to do with; at most kMax per device, which is
// as many as PyTorch hands out at a priority.  A stream beyond them takes the place of one that none of the last kStale
// calls on the device was for, if there is one; else there is none to spare.  (Calls that went round 40 streams, with the least
// recently used one dropped each time: 150 us each, 37 with the copies on their own streams.)  One that is dropped lives
// on until its last user has waited for its copy.
class SideStreams {
public:
    using Handle = std::shared_ptr<SideStream>;
    // null: none to spare
    Handle get(const c10::cuda::CUDAStream &main) {
        std::lock_guard<std::mutex> lock(mu_);
        PerDevice &d = devices_[main.device_index()];
        const int64_t now = ++d.calls;
        for (auto it = d.list.begin(); it != d.list.end(); ++it)
            if (it->main == main.stream()) {
                it->used = now;
                d.list.splice(d.list.begin(), d.list, it);
                return it->side;
            }
        if (d.list.size() >= kMax) {
            if (now - d.list.back().used < kStale) return nullptr;
            d.list.pop_back();
        }
        Handle side = std::make_shared<SideStream>();
        if (!side->make()) {
            (void)cudaGetLastError();
            return nullptr;
        }
        ++made_;
        d.list.push_front(Entry{main.stream(), side, now});
        return side;
    }
    int64_t made() {
        std::lock_guard<std::mutex> lock(mu_);
        return made_;
    }

private:
    struct Entry {
        cudaStream_t main;
        Handle side;
        int64_t used;
    };
    struct PerDevice {
        std::list<Entry> list;     // the last used one first
        int64_t calls = 0;
    };
    static constexpr size_t kMax = 32;
    static constexpr int64_t kStale = 1024;
    std::mutex mu_;
    std::map<int64_t, PerDevice> devices_;
    int64_t made_ = 0;
};
SideStreams &side_streams() {
    static SideStreams *s = new SideStreams;   // not destroyed at exit, when the CUDA context may be gone
    return *s;
}

// The lengths of the rows on their way to the host.  The copy is queued before the launch they belong to and waited for
// after it, so reading them does not leave the GPU idle; in a launch that lasts (`beside`) it runs beside the launch, behind
// what the stream held before it, and is no gap between two launches either.  Launching on lengths that turn out to be out
// of range is harmless: the kernels clamp them (and page numbers) to the buffers, and the result is dropped.
class LengthCheck {
public:
    LengthCheck(const OptTensor &lens, const c10::cuda::CUDAStream &stream, bool beside) {
        if (!lens) return;
        host_ = at::empty({lens->numel()}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
        cudaStream_t on = stream.stream();
        if (beside) side_ = side_streams().get(stream);
        if (side_) {
            C10_CUDA_CHECK(cudaEventRecord(side_->ready, on));
            on = side_->stream;
            C10_CUDA_CHECK(cudaStreamWaitEvent(on, side_->ready, 0));
        }
        C10_CUDA_CHECK(cudaMemcpyAsync(host_.data_ptr(), lens->data_ptr(), sizeof(int32_t) * lens->numel(), cudaMemcpyDeviceToHost, on));
        if (side_) C10_CUDA_CHECK(cudaEventRecord(side_->copied, on));
        else copied_.record(stream);
    }
    ~LengthCheck() {
        if (host_.defined() && !waited_) (void)cudaEventSynchronize(copied());   // the copy still writes to host_
    }
    bool within(int64_t lo, int64_t hi) {
        if (!host_.defined()) return true;
        {
            py::gil_scoped_release nogil;
            C10_CUDA_CHECK(cudaEventSynchronize(copied()));
        }
        waited_ = true;
        const int32_t *n = host_.data_ptr<int32_t>();
        for (int64_t i = 0; i < host_.numel(); ++i)
            if (n[i] < lo || n[i] > hi) return false;
        return true;
    }

private:
    cudaEvent_t copied() const { return side_ ? side_->copied : copied_.event(); }
    Tensor host_;
    SideStreams::Handle side_;
    at::cuda::CUDAEvent copied_{cudaEventDisableTiming};
    bool waited_ = false;
};

// What lasts: a decode launch by the bytes of its keys and values, a prefill launch by the keys that an item goes through or by its
// products, all at the cache ceiling (the lengths themselves are on the device).  Where the launch does not last after all, as with
// short rows in a large cache, the way over a second stream takes the host 0.2 to 0.3 us more per call (16 rows of 50 in 8192 keys in
// pages, 32 : 8 heads, 14.9 us either way).  Copy before the launch against beside it, us per call: 32 : 8 heads, 1 MB 15.2 / 15.5, 2 MB
// 15.7 / 15.6, 4 MB 20.7 / 15.8, 17 MB 22.1 / 16.6, 67 MB 29.0 / 22.8; 8 : 8 heads, 8 MB 15.3 / 15.4, 17 MB 16.5 / 15.8 and 15.3 / 15.5,
// 34 MB 26.8 / 17.3, 67 MB 27.8 / 22.1; prefill, 32 : 8 heads, 1 row of 8 or 46 tokens, 190 keys 15.3 / 15.4, 256 15.5 / 15.6, 320 16.1 / 15.7,
// 512 22.6 / 16.4, 1000 27.6 / 22.5; 4 of 32, 190 keys (0.8 GFLOP) 15.3 / 15.6, 320 16.8 / 15.7; 8 of 64, 64 keys (1.1 GFLOP) 16.7 / 15.6, 190 27.2 / 17.7.
bool decode_lasts(const Tensor &q, const Tensor &k, int64_t n_keys) {
    return 4. * q.size(0) * n_keys * k.size(2) * q.size(3) >= (q.size(2) > k.size(2) ? 2e6 : 16e6);
}
bool prefill_lasts(const Tensor &q, int64_t ceiling) { return ceiling > 256 || 8. * q.numel() * ceiling >= 1e9; }

bool int32_vector(const OptTensor &t, int64_t n, const at::Device &device) {
    return !t || (plain_tensor(*t) && t->scalar_type() == at::kInt && t->dim() == 1 && t->size(0) == n && t->is_contiguous() && t->device() == device);
}
bool page_table_ok(const OptTensor &t, int64_t batch, int64_t page, const at::Device &device) {
    return !t || (plain_tensor(*t) && t->scalar_type() == at::kInt && t->dim() == 2 && t->size(0) == batch && t->size(1) > 0 && t->is_contiguous() &&
                  t->device() == device && page > 0 && (page & (page - 1)) == 0);
}
bool kv_ok(const Tensor &k, const Tensor &v) {
    for (int i = 0; i < 3; ++i)
        if (k.stride(i) % 8 != 0) return false;
    return k.stride(3) == 1 && aligned16(k) && aligned16(v) && v.strides() == k.strides();
}
// what decode and extend ask of their tensors alike: q, r (B, L_q, H, D) contiguous, k, v in the cache layout
bool cache_call_ok(const Tensor &q, const Tensor &r, const Tensor &k, const Tensor &v, const OptTensor &lens, const OptTensor &table) {
    for (const Tensor *t : Tensors{&q, &r, &k, &v})
        if (!plain_tensor(*t) || t->dim() != 4 || t->scalar_type() != q.scalar_type() || t->device() != q.device() || t->numel() == 0)
            return false;
    if (dtype_code(q) < 0 || r.sizes() != q.sizes() || !q.is_contiguous() || !r.is_contiguous() || !aligned16(q) || !aligned16(r)) return false;
    if (v.sizes() != k.sizes() || k.size(3) != q.size(3) || (!table && k.size(0) != q.size(0)) || q.size(2) % k.size(2) != 0 || !kv_ok(k, v)) return false;
    if (q.size(3) != 64 && q.size(3) != 128) return false;
    return int32_vector(lens, q.size(0), q.device()) && page_table_ok(table, q.size(0), k.size(1), q.device()) && !recorded({&q, &r, &k, &v});
}

plx_decode_problem decode_problem(const Tensor &q, const Tensor &k, int64_t ceiling, const OptTensor &table, double scale, int64_t window,
                                  int32_t n_splits) {
    plx_decode_problem p{};
    p.dtype = dtype_code(q);
    p.batch = static_cast<int32_t>(q.size(0));
    p.heads_q = static_cast<int32_t>(q.size(2));
    p.heads_kv = static_cast<int32_t>(k.size(2));
    p.head_dim = static_cast<int32_t>(q.size(3));
    p.cache_len = static_cast<int32_t>(ceiling);
    p.window_left = static_cast<int32_t>(window);
    p.qk_scale = static_cast<float>(scale);
    p.n_splits = n_splits;
    p.kv_stride_b = k.stride(0);
    p.kv_stride_t = k.stride(1);
    p.kv_stride_h = k.stride(2);
    if (table) {
        p.page_table = int_ptr(table);
        p.page_size = static_cast<int32_t>(k.size(1));
        p.pages_per_seq = static_cast<int32_t>(table->size(1));
        p.n_pages = static_cast<int32_t>(k.size(0));
    }
    return p;
}

py::object decode(const py::object &q_, const py::object &r_, const py::object &k_, const py::object &v_, const py::object &scale_,
                  const py::object &window_, const py::object &lens_, const py::object &start_, const py::object &table_) {
    bool ok = true;
    const Tensor q = take(q_, ok), r = take(r_, ok), k = take(k_, ok), v = take(v_, ok);
    const OptTensor lens = take_optional(lens_, ok), start = take_optional(start_, ok), table = take_optional(table_, ok);
    if (!ok || !plain_thread() || !cache_call_ok(q, r, k, v, lens, table) || q.size(1) != 1 || !int32_vector(start, q.size(0), q.device()) ||
        std::getenv("PLX_DECODE_SPLITS"))
        return py::none();
    double scale;
    int64_t window;
    const int64_t ceiling = table ? table->size(1) * k.size(1) : k.size(1);
    if (!take_scale(scale_, q.size(3), scale) || !take_window(window_, window) || ceiling > INT32_MAX) return py::none();
    at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard device(q.device());
    if (capturing()) return py::none();
    RECORD_FUNCTION("plx::decode_out", Values({q, r, k, v}));
    const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
    plx_decode_problem p = decode_problem(q, k, ceiling, table, scale, window, 1);
    const int32_t n_keys = window < 0 ? p.cache_len : std::max(1, std::min(p.cache_len, p.window_left));
    p.n_splits = api.decode_choose_splits_gqa(p.batch, p.heads_q, p.heads_kv, n_keys, at::cuda::getDeviceProperties(q.get_device())->multiProcessorCount);
    size_t need = 0;
    if (api.decode_workspace_bytes(&p, &need) != PLX_OK) return py::none();
    const Tensor ws = workspaces().get(stream, q, p.n_splits, static_cast<int64_t>(need / sizeof(float)));
    Tensor out = at::empty(q.sizes(), q.options());
    LengthCheck check(lens, stream, decode_lasts(q, k, n_keys));
    if (api.decode(&p, q.data_ptr(), r.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), int_ptr(lens), int_ptr(start), ws.data_ptr(), need,
                   stream.stream()) != PLX_OK ||
        !check.within(1, ceiling))
        return py::none();
    return py::reinterpret_steal<py::object>(THPVariable_Wrap(out));
}

// L_q > 1: one launch of the training forward kernel against the cache.
py::object extend(const py::object &q_, const py::object &r_, const py::object &k_, const py::object &v_, const py::object &scale_,
                  const py::object &window_, const py::object &lens_, const py::object &table_) {
    bool ok = true;
    const Tensor q = take(q_, ok), r = take(r_, ok), k = take(k_, ok), v = take(v_, ok);
    const OptTensor lens = take_optional(lens_, ok), table = take_optional(table_, ok);
    if (!ok || !plain_thread() || !cache_call_ok(q, r, k, v, lens, table)) return py::none();
    double scale;
    int64_t window;
    const int64_t ceiling = table ? table->size(1) * k.size(1) : k.size(1);
    if (!take_scale(scale_, q.size(3), scale) || !take_window(window_, window) || ceiling > INT32_MAX || q.size(1) > ceiling) return py::none();
    at::AutoDispatchBelowADInplaceOrView below;
    const c10::cuda::CUDAGuard device(q.device());
    if (capturing() || device_error_waiting()) return py::none();
    RECORD_FUNCTION("plx::train_extend", Values({q, r, k, v}));
    const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
    plx_train_problem p = train_problem(q, k, Tensor(), scale, window, kBTHD, std::nullopt);
    p.len_k = static_cast<int32_t>(ceiling);
    Tensor out = at::empty(q.sizes(), q.options());
    LengthCheck check(lens, stream, prefill_lasts(q, ceiling));
    if (api.train_extend(&p, q.data_ptr(), r.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), int_ptr(lens), int_ptr(table),
                         table ? static_cast<int32_t>(k.size(1)) : 0, table ? static_cast<int32_t>(table->size(1)) : 0,
                         table ? static_cast<int32_t>(k.size(0)) : 0, stream.stream()) != PLX_OK ||
        !check.within(q.size(1), ceiling))
        return py::none();
    return py::reinterpret_steal<py::object>(THPVariable_Wrap(out));
}

py::object attend(const py::object &q, const py::object &r, const py::object &k, const py::object &v, const py::object &scale,
                  const py::object &window, const py::object &lens, const py::object &table) {
    if (!plain_object(q.ptr())) return py::none();
    const Tensor &t = THPVariable_Unpack(q.ptr());
    return t.dim() == 4 && t.size(1) == 1 ? decode(q, r, k, v, scale, window, lens, py::none(), table) : extend(q, r, k, v, scale, window, lens, table);
}

// No address of the sources (tensors or None) lies in one of the buffers; false where that cannot be told.
bool apart(const py::tuple &sources, const py::tuple &buffers) {
    const auto span = [](const Tensor &t) {
        int64_t last = t.numel() > 0 ? 1 : 0;
        for (int64_t i = 0; i < t.dim() && last > 0; ++i) last += (t.size(i) - 1) * t.stride(i);
        const auto at = reinterpret_cast<uintptr_t>(t.data_ptr());
        return std::pair<uintptr_t, uintptr_t>(at, at + last * t.element_size());
    };
    bool ok = true;
    for (const py::handle &s : sources) {
        const OptTensor src = take_optional(py::reinterpret_borrow<py::object>(s), ok);
        if (!ok) return false;
        if (!src || src->is_cpu()) continue;
        if (!plain_tensor(*src)) return false;
        const auto x = span(*src);
        for (const py::handle &b : buffers) {
            const Tensor buffer = take(py::reinterpret_borrow<py::object>(b), ok);
            if (!ok || !plain_tensor(buffer)) return false;
            const auto y = span(buffer);
            if (x.first < y.second && y.first < x.second) return false;
        }
    }
    return true;
}

// A GraphedDecode step: q, r and the lengths into its buffers, and the launch that its graph holds, on the same buffers and
// scratch, in one (up to PLX_DECODE_STEP_ROWS rows, inputs that lie apart from what it writes; else only the inputs are put in place).  kNothing, having done nothing, for
// anything but tensors like the buffers and lengths given as Python integers in [1, most].
// 8 : 8 heads, a launch that puts the inputs in place and the graph behind it against one launch, us: 4 rows of up to 4096 keys
// 20.5 / 14.1, 64 rows of up to 512 34.9 / 28.1.  (64: the lengths are launch parameters of every decode kernel, 4 bytes a row; more
// rows were not measured.)
enum Step { kNothing = 0, kStaged = 1, kDone = 2 };
int step(const py::object &q_, const py::object &q_src_, const py::object &r_, const py::object &r_src_, const py::object &lens_,
         const py::object &lens_src, int64_t most, const py::object &k_, const py::object &v_, const py::object &out_, const py::object &ws_,
         double scale, int64_t window, int64_t n_splits) {
    bool ok = true;
    const Tensor q = take(q_, ok), r = take(r_, ok);
    const OptTensor q_src = take_optional(q_src_, ok), r_src = take_optional(r_src_, ok), lens = take_optional(lens_, ok);
    if (!ok || !plain_thread() || !plain_tensor(q) || !plain_tensor(r) || !q.is_contiguous() || !r.is_contiguous() || q.numel() != r.numel() ||
        !aligned16(q) || !aligned16(r) || recorded({&q, &r}))
        return kNothing;
    for (const OptTensor *src : {&q_src, &r_src})
        if (*src && (!plain_tensor(**src) || (*src)->sizes() != q.sizes() || (*src)->scalar_type() != q.scalar_type() ||
                     (*src)->device() != q.device() || !(*src)->is_contiguous() || !aligned16(**src) || recorded({&**src})))
            return kNothing;
    int32_t values[PLX_DECODE_STAGE_LENS];
    int64_t n = 0;
    if (!lens_src.is_none()) {
        if (!lens || !int32_vector(lens, q.size(0), q.device()) || lens->numel() > PLX_DECODE_STAGE_LENS) return kNothing;
        n = lens->numel();
        const bool list = PyList_CheckExact(lens_src.ptr());
        if (list ? PyList_GET_SIZE(lens_src.ptr()) != n : !PyLong_CheckExact(lens_src.ptr())) return kNothing;
        for (int64_t i = 0; i < n; ++i) {
            PyObject *x = list ? PyList_GET_ITEM(lens_src.ptr(), i) : lens_src.ptr();
            int overflow = 0;
            const long long len = PyLong_CheckExact(x) ? PyLong_AsLongLongAndOverflow(x, &overflow) : 0;
            if (overflow || len < 1 || len > most) return kNothing;
            values[i] = static_cast<int32_t>(len);
        }
    }
    const c10::cuda::CUDAGuard device(q.device());
    if (capturing()) return kNothing;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    const void *q_from = q_src ? q_src->data_ptr() : nullptr, *r_from = r_src ? r_src->data_ptr() : nullptr;
    int32_t *lens_to = lens ? static_cast<int32_t *>(lens->data_ptr()) : nullptr;
    const Tensor k = take(k_, ok), v = take(v_, ok), out = take(out_, ok), ws = take(ws_, ok);
    if (ok && q.dim() == 4 && q.size(0) <= PLX_DECODE_STEP_ROWS && cache_call_ok(q, r, k, v, lens, std::nullopt) && plain_tensor(out) && plain_tensor(ws) &&
        out.sizes() == q.sizes() && out.scalar_type() == q.scalar_type() && out.device() == q.device() && out.is_contiguous()) {
        const plx_decode_problem p = decode_problem(q, k, k.size(1), std::nullopt, scale, window, static_cast<int32_t>(n_splits));
        if (api.decode_step(&p, q.data_ptr(), q_from, r.data_ptr(), r_from, k.data_ptr(), v.data_ptr(), out.data_ptr(), lens_to, n ? values : nullptr,
                            ws.data_ptr(), ws.nbytes(), stream) == PLX_OK)
            return kDone;
    }
    return api.decode_stage(q.data_ptr(), q_from, r.data_ptr(), r_from, q.nbytes(), lens_to, n ? values : nullptr, static_cast<int32_t>(n), stream) == PLX_OK
               ? kStaged : kNothing;
}

}  // namespace

PYBIND11_MODULE(_plx_host, m) {
    m.attr("abi_version") = PLX_ABI_VERSION;
    m.def("bind", &bind);
    m.def("train_ready", &train_ready);
    m.def("train", &train);
    m.def("decode", &decode);
    m.def("attend", &attend);
    m.def("apart", &apart);
    m.def("step", &step);
    m.def("side_streams_made", [] { return side_streams().made(); });
}
