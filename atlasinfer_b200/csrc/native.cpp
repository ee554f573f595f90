// Host path of the quantized linear and of the quantizer: argument checks, allocations and launches in one native call.
//
// A decode step of a small model is bound by the host, not the GPU: a linear takes 3 to 15 us on the device, and the
// same checks, allocations and argument marshalling cost 15 us a call in Python.  Semantics and errors are those of the
// Python functions that call this (integration/atlas_wrappers.py, quant/adaptive_quantizer.py); the kernels are reached
// through the C ABI of include/atlas_b200.h, as everywhere.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

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

// x @ W^T + bias for a kernel layout; `gemv` chooses the per-strip kernel, else the tcgen05 kernels.
at::Tensor linear(const at::Tensor &x, const at::Tensor &tiles, const at::Tensor &scales, const at::Tensor &chunk_ptr,
                  const at::Tensor &entries, const at::Tensor &vals, int64_t n, int64_t k, int64_t bs,
                  const std::optional<at::Tensor> &bias, const at::Tensor &status, int64_t gemv_max_rows) {
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

struct Job {
    at::Tensor codes, scales, workspace, ovals, oidx;
    int64_t capacity = 0, padded = 0;
};

Job launch_quantize(const at::Tensor &flat, int64_t bs, double z, int64_t *counts, int64_t capacity, void *stream) {
    Job j;
    const int64_t numel = flat.numel(), blocks = (numel + bs - 1) / bs;
    j.padded = blocks * bs;
    j.capacity = capacity;
    const size_t ws = atlas_quantize_workspace_bytes(numel, (int)bs);
    const auto opt = flat.options();
    j.codes = at::empty({j.padded}, opt.dtype(at::kChar));
    j.scales = at::empty({blocks}, opt.dtype(at::kHalf));
    j.workspace = at::empty({(int64_t)ws}, opt.dtype(at::kByte));
    j.ovals = at::empty({capacity}, opt.dtype(at::kHalf));
    j.oidx = at::empty({capacity}, opt.dtype(at::kLong));
    check(atlas_quantize(flat.data_ptr(), numel, (int)bs, z, (int8_t *)j.codes.data_ptr(), j.ovals.data_ptr(), (int64_t *)j.oidx.data_ptr(),
                         capacity, j.scales.data_ptr(), counts, j.workspace.data_ptr(), ws, stream), "atlas_quantize");
    return j;
}

// The four streams of every flat fp16 tensor (all on one device): all kernels are enqueued first, the stream lengths of
// all of them come back in one device-to-host copy.
std::vector<std::array<at::Tensor, 4>> quantize_many(const std::vector<at::Tensor> &flats, int64_t bs, double z) {
    const c10::cuda::CUDAGuard guard(flats[0].device());
    void *stream = at::cuda::getCurrentCUDAStream(flats[0].get_device()).stream();
    at::Tensor counts = at::empty({(int64_t)flats.size(), 4}, flats[0].options().dtype(at::kLong));
    int64_t *dev_counts = counts.data_ptr<int64_t>();
    std::vector<Job> jobs;
    for (size_t i = 0; i < flats.size(); ++i) {
        // |z| > t bounds the outliers of a block by (block_size - 1) / t^2, but weight-like data has well under
        // 1 %: start with 1/32 of the tensor and retry with full capacity in the rare case that is short
        const int64_t padded = (flats[i].numel() + bs - 1) / bs * bs;
        jobs.push_back(launch_quantize(flats[i], bs, z, dev_counts + 4 * i, std::min(padded, padded / 32 + 1024), stream));
    }
    at::Tensor host = counts.cpu();   // the one synchronisation
    std::vector<std::array<at::Tensor, 4>> out;
    for (size_t i = 0; i < flats.size(); ++i) {
        const int64_t *c = host.data_ptr<int64_t>() + 4 * i;
        int64_t n_codes = c[0], n_out = c[1], timed_out = c[2];
        Job &j = jobs[i];
        if (!timed_out && n_out > j.capacity) {   // rare: more outliers than the first buffer holds
            j = launch_quantize(flats[i], bs, z, dev_counts + 4 * i, j.padded, stream);
            const at::Tensor again = counts.cpu();
            c = again.data_ptr<int64_t>() + 4 * i;
            n_codes = c[0], n_out = c[1], timed_out = c[2];
        }
        if (timed_out) check(ATLAS_ERR_TIMEOUT, "atlas_quantize: device-side wait timed out");
        // codes: a view (the buffer is 0.3 % longer than the stream); outliers: copied out of their roomy buffers
        out.push_back({j.codes.narrow(0, 0, n_codes), j.ovals.narrow(0, 0, n_out).clone(), j.oidx.narrow(0, 0, n_out).clone(), j.scales});
    }
    return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("quantize_many", &quantize_many, py::call_guard<py::gil_scoped_release>());
    m.def("linear", &linear, py::call_guard<py::gil_scoped_release>());
}
