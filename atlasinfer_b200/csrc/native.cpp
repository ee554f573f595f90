// Host path of the quantized linear, of its weight layouts and of the quantizer: argument checks, allocations and launches in one native call.
//
// A decode step of a small model is bound by the host, not the GPU: a linear takes 3 to 15 us on the device, and the
// same checks, allocations and argument marshalling cost 15 us a call in Python.  Semantics and errors are those of the
// Python functions that call this (integration/atlas_wrappers.py, quant/adaptive_quantizer.py); the kernels are reached
// through the C ABI of include/atlas_b200.h, as everywhere.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>

#include <algorithm>
#include <atomic>
#include <memory>
#include <mutex>

#include "atlas_b200.h"

namespace py = pybind11;

namespace {

// raises what the Python package raises for a status of the C ABI
void check(int status, const char *what) {
    if (status == ATLAS_OK) return;
    py::gil_scoped_acquire gil;
    py::module_::import("atlasinfer_b200._capi").attr("check")(status, what);
}

const void *ptr_or_null(const at::Tensor &t) { return t.numel() ? t.data_ptr() : nullptr; }

// The layouts that one stream writes: an event that is recorded again behind every further one, so that one look at it settles
// all of them (an event of each layout's own costs the first pass after loading a query and a destruction per launch).  A use
// on another stream may wait for later layouts of that stream too.
struct StreamLayouts {
    const int device;
    const unsigned long long id;   // of the stream, for the life of the process (a handle may be used again)
    cudaEvent_t event = nullptr;
    std::mutex lock;               // the event, and what it stands behind
    uint64_t enqueued = 0;         // layouts; the event stands behind the last
    std::atomic<uint64_t> final{0};   // of them known to be final

    StreamLayouts(int device, unsigned long long id) : device(device), id(id) {
        C10_CUDA_CHECK(cudaEventCreateWithFlags(&event, cudaEventDisableTiming));
    }
    ~StreamLayouts() { cudaEventDestroy(event); }
    StreamLayouts(const StreamLayouts &) = delete;

    void settle(uint64_t upto) {
        uint64_t was = final.load(std::memory_order_relaxed);
        while (was < upto && !final.compare_exchange_weak(was, upto, std::memory_order_release, std::memory_order_relaxed)) {}
    }
    // The host waits for all layouts enqueued so far.
    cudaError_t synchronize() {
        uint64_t upto;
        {
            const std::lock_guard<std::mutex> held(lock);
            upto = enqueued;
        }
        const cudaError_t e = cudaEventSynchronize(event);
        if (e == cudaSuccess) settle(upto);
        return e;
    }
    // cudaSuccess: all layouts enqueued so far are final; cudaErrorNotReady: not yet.
    cudaError_t look() {
        const std::lock_guard<std::mutex> held(lock);
        const cudaError_t e = cudaEventQuery(event);
        if (e == cudaSuccess) settle(enqueued);
        return e;
    }
};

// The current stream's.  Those of streams that no layout looks at any more are given back once there are more than 16.
std::shared_ptr<StreamLayouts> stream_layouts(int device, cudaStream_t stream) {
    static std::mutex lock;
    static auto *known = new std::vector<std::shared_ptr<StreamLayouts>>;   // (never destroyed: the driver may be gone by then)
    unsigned long long id = 0;
    C10_CUDA_CHECK(cudaStreamGetId(stream, &id));
    const std::lock_guard<std::mutex> held(lock);
    for (const auto &s : *known)
        if (s->device == device && s->id == id) return s;
    if (known->size() >= 16)
        known->erase(std::remove_if(known->begin(), known->end(), [](const auto &s) { return s.use_count() == 1; }), known->end());
    known->push_back(std::make_shared<StreamLayouts>(device, id));
    return known->back();
}

// Stands for a layout that may still be written by the stream it was enqueued on.  The linear kernels read weights before
// the stream's earlier work has completed (programmatic dependent launch): a dependent starts once the kernel in front has
// ended, but sees its stores for certain only behind griddepcontrol.wait.  Until the layout is known to be final, a linear
// on that stream is therefore launched plainly; a use on another stream, or in a capture, whose kernels run who knows where,
// waits on the host, once.
class LayoutReady {
   public:
    LayoutReady() {
        const int device = at::cuda::current_device();
        const cudaStream_t stream = at::cuda::getCurrentCUDAStream(device).stream();
        on_ = stream_layouts(device, stream);
        const std::lock_guard<std::mutex> held(on_->lock);
        C10_CUDA_CHECK(cudaEventRecord(on_->event, stream));
        number_ = ++on_->enqueued;
    }
    LayoutReady(const LayoutReady &) = delete;
    // True once the layout is final.  False: not yet, but what is launched plainly on the current stream comes after it.
    bool wait() {
        if (is_final()) return true;
        const cudaStream_t stream = at::cuda::getCurrentCUDAStream(on_->device).stream();
        const CaptureUntouched scope;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        unsigned long long id = on_->id;
        C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &capture));
        if (capture == cudaStreamCaptureStatusNone) C10_CUDA_CHECK(cudaStreamGetId(stream, &id));   // (refused in a capture)
        if (id == on_->id && capture == cudaStreamCaptureStatusNone) {
            const cudaError_t e = on_->look();
            if (e == cudaErrorNotReady) (void)cudaGetLastError();
            else C10_CUDA_CHECK(e);
            return e == cudaSuccess;
        }
        C10_CUDA_CHECK(on_->synchronize());
        return true;
    }
    // Whether it is final, whatever stream is current.
    bool done() {
        if (is_final()) return true;
        const CaptureUntouched scope;
        const cudaError_t e = on_->look();
        if (e == cudaErrorNotReady) (void)cudaGetLastError();
        else C10_CUDA_CHECK(e);
        return e == cudaSuccess;
    }
    std::pair<int, unsigned long long> stream() const { return {on_->device, on_->id}; }
    // Returns once the layout is final, for uses whose order this cannot see (copies, other libraries' kernels).
    void finish() {
        if (is_final()) return;
        const CaptureUntouched scope;
        C10_CUDA_CHECK(on_->synchronize());
    }

   private:
    // None of the calls in its scope touches a capture of this or another thread.
    struct CaptureUntouched {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CaptureUntouched() { C10_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode)); }
        ~CaptureUntouched() { cudaThreadExchangeStreamCaptureMode(&mode); }
    };
    bool is_final() const { return on_->final.load(std::memory_order_acquire) >= number_; }

    std::shared_ptr<StreamLayouts> on_;
    uint64_t number_ = 0;
};

// The linears of this scope are launched plainly (`on`), or as the thread has it.
class PlainLaunch {
   public:
    explicit PlainLaunch(bool on) : on_(on) { if (on_) was_ = atlas_qlinear_plain_launch(1); }
    ~PlainLaunch() { if (on_) atlas_qlinear_plain_launch(was_); }
    PlainLaunch(const PlainLaunch &) = delete;

   private:
    bool on_;
    int was_ = 0;
};

// x @ W^T + bias for a kernel layout; `gemv` chooses the per-strip kernel, else the tcgen05 kernels.  `pending`: the stream's
// earlier work may still write the layout.
at::Tensor linear(const at::Tensor &x, const at::Tensor &tiles, const at::Tensor &scales, const at::Tensor &chunk_ptr,
                  const at::Tensor &entries, const at::Tensor &vals, int64_t n, int64_t k, int64_t bs,
                  const std::optional<at::Tensor> &bias, const at::Tensor &status, int64_t gemv_max_rows, bool pending) {
    const int dtype = x.scalar_type() == at::kHalf ? ATLAS_DTYPE_F16 : ATLAS_DTYPE_BF16;   // (the caller has looked)
    if (x.dim() < 1 || x.size(-1) != k)
        throw std::runtime_error("QuantizedLinear: input has " + std::to_string(x.dim() ? x.size(-1) : 0) + " features, weight expects " + std::to_string(k));
    at::Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, k});
    if (x2.stride(1) != 1 || (x2.size(0) > 1 && x2.stride(0) < k)) x2 = x2.contiguous();
    const int64_t m = x2.size(0), ldx = m > 1 ? x2.stride(0) : k;
    const c10::cuda::CUDAGuard guard(x.device());
    at::Tensor y;
    if (x.dim() == 2) {
        y = at::empty({m, n}, x.options());
    } else {
        std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
        shape.back() = n;
        y = at::empty(shape, x.options());
    }
    if (m == 0) return y;
    at::Tensor b;
    if (bias.has_value()) b = bias->to(at::kHalf).contiguous();
    // (a bias converted just now is written by the kernel in front)
    const PlainLaunch plain(pending || (b.defined() && !b.is_same(*bias)));
    void *stream = at::cuda::getCurrentCUDAStream(x.get_device()).stream();
    const void *bp = b.defined() ? ptr_or_null(b) : nullptr;
    if (m <= gemv_max_rows) {
        check(atlas_qlinear_gemv(x2.data_ptr(), dtype, m, ldx, (const uint8_t *)tiles.data_ptr(), scales.data_ptr(),
                                 (const int32_t *)chunk_ptr.data_ptr(), (const uint32_t *)ptr_or_null(entries), ptr_or_null(vals), n, k,
                                 (int)bs, bp, y.data_ptr(), n, (int32_t *)status.data_ptr(), stream), "atlas_qlinear_gemv");
    } else {
        const size_t bytes = atlas_qlinear_gemm_workspace_bytes(m, n, k);
        at::Tensor ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
        check(atlas_qlinear_gemm(x2.data_ptr(), dtype, m, ldx, (const uint8_t *)tiles.data_ptr(), scales.data_ptr(),
                                 (const int32_t *)chunk_ptr.data_ptr(), (const uint32_t *)ptr_or_null(entries), ptr_or_null(vals), n, k,
                                 (int)bs, bp, y.data_ptr(), n, ws.data_ptr(), bytes, (int32_t *)status.data_ptr(), stream), "atlas_qlinear_gemm");
    }
    return y;
}

// What a tensor's streams are written to: codes and scales of their final length (codes: nearly), the outliers roomy.
struct Job {
    at::Tensor codes, scales;
    int64_t capacity, padded;
    AtlasQuantizeItem item;
};

Job make_job(const at::Tensor &flat, int64_t bs, int64_t capacity, void *ovals, void *oidx, int64_t *counts) {
    Job j;
    const int64_t blocks = (flat.numel() + bs - 1) / bs;
    j.padded = blocks * bs;
    j.capacity = capacity;
    j.codes = at::empty({j.padded}, flat.options().dtype(at::kChar));
    j.scales = at::empty({blocks}, flat.options().dtype(at::kHalf));
    j.item = {flat.data_ptr(), flat.numel(), (int8_t *)j.codes.data_ptr(), ovals, (int64_t *)oidx, capacity, j.scales.data_ptr(), counts};
    return j;
}

int64_t up16(int64_t v) { return (v + 15) / 16 * 16; }

// The four streams of every flat fp16 tensor (all on one device): one launch (block sizes of the fast kernel; up to 16
// tensors), one device-to-host copy for the stream lengths of all, one launch that takes the outliers to buffers of their
// own length.
std::vector<std::array<at::Tensor, 4>> quantize_many(const std::vector<at::Tensor> &flats, int64_t bs, double z) {
    const c10::cuda::CUDAGuard guard(flats[0].device());
    void *stream = at::cuda::getCurrentCUDAStream(flats[0].get_device()).stream();
    const auto bytes_opt = flats[0].options().dtype(at::kByte);
    const size_t n = flats.size();
    std::vector<int64_t> capacity(n);
    int64_t workspace_bytes = 0;
    for (size_t i = 0; i < n; ++i) {
        // |z| > t bounds the outliers of a block by (block_size - 1) / t^2, but weight-like data has well under
        // 1 %: start with 1/32 of the tensor and retry with full capacity in the rare case that is short
        const int64_t padded = (flats[i].numel() + bs - 1) / bs * bs;
        capacity[i] = std::min(padded, padded / 32 + 1024);
        workspace_bytes += atlas_quantize_workspace_bytes(flats[i].numel(), (int)bs);
    }
    // counts, and behind them the workspace: cleared together
    at::Tensor scratch = at::empty({(int64_t)n * 32 + workspace_bytes}, bytes_opt);
    int64_t *counts = (int64_t *)scratch.data_ptr();
    std::vector<Job> jobs;
    std::vector<AtlasQuantizeItem> items;
    // (a buffer per tensor: one for all of them is the largest block of the call, which the caching allocator then cuts up
    // for the next caller's tensors)
    std::vector<at::Tensor> held;   // until the copies are enqueued
    for (size_t i = 0; i < n; ++i) {
        held.push_back(at::empty({up16(capacity[i] * 8) + up16(capacity[i] * 2)}, bytes_opt));
        char *at_byte = (char *)held[i].data_ptr();
        jobs.push_back(make_job(flats[i], bs, capacity[i], at_byte + up16(capacity[i] * 8), at_byte, counts + 4 * i));
        items.push_back(jobs[i].item);
    }
    check(atlas_quantize_many((int)n, items.data(), (int)bs, z, counts + 4 * n, (size_t)workspace_bytes, stream), "atlas_quantize");
    const at::Tensor host = scratch.narrow(0, 0, (int64_t)n * 32).cpu();   // the one synchronisation
    const int64_t *c = (const int64_t *)host.data_ptr();
    std::vector<std::array<at::Tensor, 4>> out;
    std::vector<AtlasCopyItem> copies;
    for (size_t i = 0; i < n; ++i) {
        int64_t n_codes = c[4 * i], n_out = c[4 * i + 1], timed_out = c[4 * i + 2];
        Job &j = jobs[i];
        if (!timed_out && n_out > j.capacity) {   // rare: more outliers than the first buffer holds
            const size_t ws = atlas_quantize_workspace_bytes(flats[i].numel(), (int)bs);
            const at::Tensor again = at::empty({32 + (int64_t)ws}, bytes_opt), roomy = at::empty({j.padded * 10}, bytes_opt);
            held.push_back(roomy);
            int64_t *own = (int64_t *)again.data_ptr();
            j = make_job(flats[i], bs, j.padded, (char *)roomy.data_ptr() + j.padded * 8, roomy.data_ptr(), own);
            check(atlas_quantize_many(1, &j.item, (int)bs, z, own + 4, ws, stream), "atlas_quantize");
            const at::Tensor second = again.narrow(0, 0, 32).cpu();
            const int64_t *s = (const int64_t *)second.data_ptr();
            n_codes = s[0], n_out = s[1], timed_out = s[2];
        }
        if (timed_out) check(ATLAS_ERR_TIMEOUT, "atlas_quantize: device-side wait timed out");
        // codes: a view (the buffer is 0.3 % longer than the stream)
        const at::Tensor ovals = at::empty({n_out}, flats[i].options().dtype(at::kHalf)), oidx = at::empty({n_out}, flats[i].options().dtype(at::kLong));
        if (n_out) {
            copies.push_back({ovals.data_ptr(), j.item.outlier_vals, n_out * 2});
            copies.push_back({oidx.data_ptr(), j.item.outlier_idx, n_out * 8});
        }
        out.push_back({j.codes.narrow(0, 0, n_codes), ovals, oidx, j.scales});
    }
    check(atlas_copy_many((int)copies.size(), copies.data(), stream), "atlas_copy_many");
    return out;
}

// The kernel layouts of `members` (codes, outlier values, outlier positions, scales, rows; one device, K and block size) as
// the rows of one layout: tiles, scales, CSR row pointers (of a single tensor), chunk pointers, entries, values.  Enqueued,
// not waited for.
std::array<at::Tensor, 6> build_layout(const std::vector<std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor, int64_t>> &members,
                                       int64_t k, int64_t bs) {
    const at::Tensor &first = std::get<0>(members[0]);
    const c10::cuda::CUDAGuard guard(first.device());
    const c10::cuda::CUDAStream stream = at::cuda::getCurrentCUDAStream(first.get_device());
    int64_t rows_padded = 0, n_out = 0;
    for (const auto &m : members) {
        rows_padded += (std::get<4>(m) + 127) / 128 * 128;
        n_out += std::get<2>(m).numel();
    }
    const int64_t chunks = k / 64 + 1;
    const auto opt = first.options();
    at::Tensor tiles = at::empty({rows_padded * k}, opt.dtype(at::kByte)), scales = at::empty({rows_padded * (k / bs)}, opt.dtype(at::kHalf));
    at::Tensor row_ptr = at::empty({members.size() == 1 ? std::get<4>(members[0]) + 1 : 0}, opt.dtype(at::kInt));
    at::Tensor chunk_ptr = at::empty({rows_padded / 16 * chunks}, opt.dtype(at::kInt));
    at::Tensor entries = at::empty({n_out}, opt.dtype(at::kInt)), vals = at::empty({n_out}, opt.dtype(at::kHalf));
    std::vector<AtlasRepackItem> items;
    std::vector<at::Tensor> held;   // alive until the kernel is enqueued
    int64_t row = 0, entry = 0;
    for (const auto &m : members) {
        const at::Tensor codes = std::get<0>(m).contiguous(), ovals = std::get<1>(m).contiguous(), oidx = std::get<2>(m).contiguous(),
                         sc = std::get<3>(m).contiguous();
        const int64_t n = std::get<4>(m);
        AtlasRepackItem item = {};
        item.codes = (const int8_t *)ptr_or_null(codes);
        item.n_codes = codes.numel();
        item.outlier_vals = ptr_or_null(ovals);
        item.outlier_idx = (const int64_t *)ptr_or_null(oidx);
        item.n_outliers = oidx.numel();
        item.scales = sc.data_ptr();
        item.n_rows = n;
        item.n_cols = k;
        item.block_size = bs;
        item.tiles = (uint8_t *)tiles.data_ptr() + row * k;
        item.scales_tiled = (char *)scales.data_ptr() + row * (k / bs) * 2;
        item.outlier_row_ptr = members.size() == 1 ? (int32_t *)row_ptr.data_ptr() : nullptr;
        item.outlier_chunk_ptr = (int32_t *)chunk_ptr.data_ptr() + row / 16 * chunks;
        if (n_out) {
            item.outlier_entries = (uint32_t *)entries.data_ptr() + entry;
            item.outlier_vals_sorted = (char *)vals.data_ptr() + entry * 2;
        }
        item.entry_base = entry;
        items.push_back(item);
        // the streams may be freed, by another stream's owner too, before the kernel has read them
        for (const at::Tensor &t : {codes, ovals, oidx, sc}) {
            if (t.numel()) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), stream);
            held.push_back(t);
        }
        row += (n + 127) / 128 * 128;
        entry += oidx.numel();
    }
    check(atlas_repack_many((int)items.size(), items.data(), stream.stream()), "atlas_repack");
    return {tiles, scales, row_ptr, chunk_ptr, entries, vals};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    py::class_<LayoutReady, std::shared_ptr<LayoutReady>>(m, "LayoutReady")
        .def(py::init<>())
        .def("wait", &LayoutReady::wait, py::call_guard<py::gil_scoped_release>())
        .def("done", &LayoutReady::done, py::call_guard<py::gil_scoped_release>())
        .def_property_readonly("stream", &LayoutReady::stream)
        .def("finish", &LayoutReady::finish, py::call_guard<py::gil_scoped_release>());
    m.def("build_layout", &build_layout, py::call_guard<py::gil_scoped_release>());
    m.def("quantize_many", &quantize_many, py::call_guard<py::gil_scoped_release>());
    m.def("linear", &linear, py::call_guard<py::gil_scoped_release>());
}
