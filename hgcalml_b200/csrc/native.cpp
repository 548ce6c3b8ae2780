// Host side of the ops that are called most: output allocation, workspace and the C ABI call in one step.  The Python
// mirrors check and convert their arguments and call these with dense CUDA tensors of the right types; the status code
// of the C ABI comes back as the last element.  A call costs the host about 15 us less than the same steps through
// ctypes (of 52 us for a search of nine launches).
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/ops/empty.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <optional>

#include "../../include/hgcalml_b200.h"

namespace hgc { int sm_count(); }  // of the library

namespace {

using at::Tensor;
typedef std::optional<Tensor> MaybeTensor;

template <typename T> T *data(const Tensor &t) { return static_cast<T *>(t.data_ptr()); }
template <typename T> T *data(const MaybeTensor &t) { return t.has_value() ? static_cast<T *>(t->data_ptr()) : nullptr; }

bool aligned16(const Tensor &t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }

hgc_stream_t stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

Tensor like(const Tensor &t, at::IntArrayRef sizes, at::ScalarType type) { return at::empty(sizes, t.options().dtype(type)); }

Tensor workspace(const Tensor &t, size_t bytes) { return like(t, {(int64_t)(bytes < 256 ? 256 : bytes)}, at::kByte); }

// (indices, distances, sorting, status)
std::tuple<Tensor, Tensor, Tensor, int> select_knn(const Tensor &coords, const Tensor &row_splits, const MaybeTensor &direction,
                                                   int K, int n_bins, int max_bin_dims, bool tf_compat)
{
    const int n = (int)coords.size(0), c = (int)coords.size(1), n_rs = (int)row_splits.size(0);
    Tensor idx = like(coords, {n, K}, at::kInt), dist = like(coords, {n, K}, at::kFloat), sorting = like(coords, {n}, at::kInt);
    const size_t bytes = hgc_binned_select_knn_ragged_workspace_bytes(n, K, c, n_rs, n_bins, max_bin_dims);
    if (bytes == 0) return {idx, dist, sorting, HGC_ERR_UNSUPPORTED};
    Tensor ws = workspace(coords, bytes);
    const int rc = hgc_binned_select_knn_ragged(
            data<float>(coords), data<int>(row_splits), data<int>(direction), data<int>(idx), data<float>(dist),
            data<int>(sorting), n, K, c, n_rs, n_bins, max_bin_dims, tf_compat, direction.has_value(), ws.data_ptr(),
            (size_t)ws.numel(), stream_of(coords));
    return {idx, dist, sorting, rc};
}

// (features, arg-max indices or None, status)
std::tuple<Tensor, MaybeTensor, int> accumulate(const Tensor &weights, const Tensor &features, const Tensor &indices,
                                                const MaybeTensor &order, bool mean_and_max, bool with_arg, bool exponential,
                                                float scale)
{
    const int n = (int)indices.size(0), k = (int)indices.size(1), f = (int)features.size(1);
    const int n_out = mean_and_max ? 2 * f : f;
    Tensor out = like(features, {n, n_out}, at::kFloat);
    MaybeTensor arg;
    if (with_arg) {
        arg = like(features, {n, f}, at::kInt);
        if (!mean_and_max) arg->zero_();
    }
    const hgc_stream_t stream = stream_of(features);
    const int rc = exponential
            ? hgc_accumulate_knn_exp(data<float>(weights), data<float>(features), data<int>(indices), data<float>(out),
                                     data<int>(arg), n, k, f, n_out, mean_and_max, scale, data<int>(order), stream)
            : hgc_accumulate_knn_ordered(data<float>(weights), data<float>(features), data<int>(indices), data<float>(out),
                                         data<int>(arg), n, k, f, n_out, 0, mean_and_max, data<int>(order), stream);
    return {out, arg, rc};
}

// (gradient of the weights, gradient of the features, workspace, status)
std::tuple<Tensor, Tensor, Tensor, int> accumulate_grad(const Tensor &grad, const Tensor &weights, const Tensor &features,
                                                        const Tensor &indices, const MaybeTensor &max_idx,
                                                        const MaybeTensor &order)
{
    const int n = (int)indices.size(0), k = (int)indices.size(1), f = (int)features.size(1), g = (int)grad.size(1);
    Tensor gw = like(features, {n, k}, at::kFloat), gf = like(features, {n, f}, at::kFloat);
    Tensor ws = workspace(features, aligned16(grad) ? hgc_accumulate_knn_grad_workspace_bytes(n, k, f, g > f) : hgc_knn_grad_workspace_bytes(n, k));
    const int rc = hgc_accumulate_knn_grad_ordered(
            data<float>(grad), data<float>(weights), data<float>(features), data<int>(max_idx), data<int>(indices),
            data<float>(gw), data<float>(gf), n, k, f, g, 0, g > f, data<int>(order), ws.data_ptr(), (size_t)ws.numel(),
            stream_of(features));
    return {gw, gf, ws, rc};
}

// (gradient of the coordinates, status); `lists`: the workspace that accumulate_grad left for the same table
std::tuple<Tensor, int> select_knn_grad(const Tensor &grad, const Tensor &indices, const Tensor &coords,
                                        const MaybeTensor &order, const MaybeTensor &lists)
{
    const int n = (int)indices.size(0), k = (int)indices.size(1), c = (int)coords.size(1);
    Tensor out = like(coords, coords.sizes(), at::kFloat);
    const Tensor ws = lists.has_value() ? *lists : workspace(coords, hgc_select_knn_grad_workspace_bytes(n, k));
    const auto run = lists.has_value() ? hgc_select_knn_grad_after : hgc_select_knn_grad_ordered;
    const int rc = run(data<float>(grad), data<int>(indices), nullptr, data<float>(coords), data<float>(out), n, k, c,
                       data<int>(order), ws.data_ptr(), (size_t)ws.numel(), stream_of(coords));
    return {out, rc};
}

// (squared distances, status)
std::tuple<Tensor, int> local_distance(const Tensor &indices, const Tensor &coords)
{
    Tensor out = like(coords, indices.sizes(), at::kFloat);
    const int rc = hgc_local_distance(data<int>(indices), data<float>(coords), data<float>(out), (int)coords.size(1),
                                      (int)coords.size(0), (int)indices.size(0), (int)indices.size(1), stream_of(coords));
    return {out, rc};
}

// (features, status)
std::tuple<Tensor, int> push_knn(const Tensor &weights, const Tensor &features, const Tensor &indices, const MaybeTensor &order)
{
    const int n = (int)indices.size(0), k = (int)indices.size(1), f = (int)features.size(1);
    Tensor out = like(features, features.sizes(), at::kFloat);
    Tensor ws = workspace(features, aligned16(features) ? hgc_push_knn_workspace_bytes(n, k, f) : hgc_knn_grad_workspace_bytes(n, k));
    const int rc = hgc_push_knn_ordered(data<float>(weights), data<float>(features), data<int>(indices), data<float>(out), n, k, f,
                                        data<int>(order), ws.data_ptr(), (size_t)ws.numel(), stream_of(features));
    return {out, rc};
}

// (gradient of the weights, gradient of the features, status)
std::tuple<Tensor, Tensor, int> push_knn_grad(const Tensor &grad, const Tensor &weights, const Tensor &features,
                                              const Tensor &indices, const MaybeTensor &order)
{
    const int n = (int)indices.size(0), k = (int)indices.size(1), f = (int)features.size(1);
    Tensor gw = like(weights, weights.sizes(), at::kFloat), gf = like(features, features.sizes(), at::kFloat);
    const int rc = hgc_push_knn_grad_ordered(data<float>(grad), data<float>(weights), data<float>(features), data<int>(indices),
                                             data<float>(gf), data<float>(gw), n, k, f, data<int>(order), stream_of(features));
    return {gw, gf, rc};
}

// status; `out`: the columns that take the collected features
int collect(const Tensor &dist, const Tensor &indices, int first_slot, int k, const Tensor &features, const Tensor &out,
            const MaybeTensor &max_idx, float scale, bool subtract_self, const MaybeTensor &order)
{
    const int n = (int)indices.size(0);
    return hgc_gravnet_collect(data<float>(dist), data<int>(indices), (int)indices.size(1), first_slot, k, data<float>(features),
                               n > 0 ? data<float>(out) : nullptr, (int)out.stride(0), data<int>(max_idx), n, (int)features.size(1),
                               scale, subtract_self, data<int>(order), stream_of(features));
}

Tensor host_int()  // page-locked, so that the copy that fills it needs no staging
{
    return at::empty({1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
}

// (assignment, association, condensates, flags, condensates before every event, number of condensates or -1, status); with
// `counted` the call waits for the number
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, int, int> condensates(const Tensor &coords, const Tensor &betas, const Tensor &dist,
                                                                         const MaybeTensor &mask, const Tensor &row_splits,
                                                                         double beta_threshold, double distance_threshold,
                                                                         bool by_max_beta, int nbin_dims, bool counted)
{
    const int n = (int)coords.size(0), dims = (int)coords.size(1), n_rs = (int)row_splits.size(0);
    Tensor assignment = like(coords, {n}, at::kInt), association = like(coords, {n}, at::kInt), alpha = like(coords, {n}, at::kInt);
    Tensor flags = like(coords, {n}, at::kBool), counts = like(coords, {n_rs}, at::kInt);
    Tensor ws = workspace(coords, hgc_build_and_assign_condensates_workspace_bytes(n, dims, n_rs, nbin_dims));
    Tensor n_alpha;
    if (counted) n_alpha = host_int();
    const int rc = hgc_build_and_assign_condensates(
            data<float>(coords), data<float>(betas), data<float>(dist), data<int>(mask), data<int>(row_splits), data<int>(assignment),
            data<int>(association), data<int>(alpha), static_cast<unsigned char *>(flags.data_ptr()), data<int>(counts),
            counted ? data<int>(n_alpha) : nullptr, n, dims, n_rs, (float)beta_threshold, (float)distance_threshold, by_max_beta,
            nbin_dims, ws.data_ptr(), (size_t)ws.numel(), stream_of(coords));
    return {assignment, association, alpha, flags, counts, counted && rc == HGC_OK ? *data<int>(n_alpha) : -1, rc};
}

// (assignment, association, and condensates, rows of one tensor; flags; condensates before every event; their number, status).
// `alpha` may be longer than the list of condensates.
std::tuple<Tensor, Tensor, Tensor, int, int> merge_noise(const Tensor &assignment, const Tensor &association, const Tensor &alpha,
                                                         const Tensor &flags, const Tensor &counts, const Tensor &row_splits)
{
    const int64_t n = assignment.size(0);
    const int n_rs = (int)row_splits.size(0);
    Tensor all = like(assignment, {4, n}, at::kInt);  // the condensates take up to two rows
    Tensor new_flags = like(assignment, {n}, at::kBool), new_counts = like(assignment, {n_rs}, at::kInt), n_alpha = host_int();
    Tensor ws = workspace(assignment, hgc_merge_noise_workspace_bytes((int)n, n_rs));
    int *rows = data<int>(all);
    const int rc = hgc_merge_noise(
            data<int>(assignment), data<int>(association), alpha.numel() > 0 ? data<int>(alpha) : rows,
            static_cast<unsigned char *>(flags.data_ptr()), data<int>(counts), data<int>(row_splits), rows, rows + n, rows + 2 * n,
            static_cast<unsigned char *>(new_flags.data_ptr()), data<int>(new_counts), data<int>(n_alpha), (int)n, n_rs, ws.data_ptr(),
            (size_t)ws.numel(), stream_of(assignment));
    return {all, new_flags, new_counts, rc == HGC_OK ? *data<int>(n_alpha) : 0, rc};
}

// Whether a kernel on raw pointers may stand in for a tensor operation: no function transform, dispatch mode or trace is
// to see the operation ..
bool operations_are_seen()
{
    using c10::DispatchKey;
    return c10::impl::dispatch_mode_enabled() ||
           c10::impl::tls_is_dispatch_key_included(DispatchKey::FuncTorchDynamicLayerFrontMode) ||
           c10::impl::tls_is_dispatch_key_included(DispatchKey::Functionalize) ||
           c10::impl::tls_is_dispatch_key_included(DispatchKey::Tracer);
}
// .. and the tensor is a plain one on the current device, of which nothing but the values counts.
bool values_only(const Tensor &t)
{
    return t.is_cuda() && t.get_device() == c10::cuda::current_device() && t.scalar_type() == at::kFloat && t.layout() == at::kStrided && !t.is_neg() &&
           !t.unsafeGetTensorImpl()->is_python_dispatch() && !(t.requires_grad() && c10::GradMode::is_enabled()) &&
           !t._fw_grad(0).defined();
}

constexpr int kNotTaken = 1;

// Where hgc_dense is at least as fast as the library's GEMM with the bias and activation kernel behind it: time over the library's
// (float32, 24 batches of 1 to 1M rows for each of 30 shapes).
//   up to 8 columns: 0.33 to 0.9; at 60k rows 256 x 8 1.06, so that long rows of more than four columns start above that
//   9 to 32: 0.44 to 0.95; 128 x 24 and 128 x 12 1.04 and 1.06 at 49k
//   33 to 64: up to 64 inputs 0.44 to 1.00, but 64 x 48 1.06 at 80k, where blocks of 128 rows leave a second round of the chip nearly
//     empty; likewise at 160k in the third round 192 x 64 1.06 and 128 x 48 1.05 (128 x 64 0.98); else 128 x 64 0.88 to 0.93,
//     192 x 64 0.93 to 0.98, 128 x 48 0.93 to 0.98, 192 x 48 1.00 to 1.04, from 131k on
//   65 to 128, 64 at a time: 64 x 72 and 64 x 96 below 1.00, 96 x 96 0.90 to 1.00, 128 x 120 and 128 x 128 0.93 to 0.99; 96 x 80 1.03,
//     128 x 72 and 128 x 96 1.02 to 1.14, 128 x 104 1.02
bool dense_is_faster(int64_t n, int64_t n_in, int64_t n_out)
{
    if (n < 1 || n > 0x7fffffff || n_in < 4 || n_out < 1) return false;
    if (n_out <= 8) return n_in <= 32 || (n_in <= 64 && n >= 10000) || (n_in <= 256 && n >= (n_in > 128 && n_out > 4 ? 65536 : 32768));
    if (n_out <= 32) return n_in <= 96 || (n_in <= 128 && n >= 57344);
    if (n_out <= 64) {
        const int64_t blocks = (n + 127) / 128, round = 4 * (int64_t)hgc::sm_count(), last = blocks % round;
        const bool tail = blocks > round && blocks < 3 * round && last > 0 && last * 6 < round;
        if (n_in <= 64) return n_in <= 32 || n_out > 56 || !tail || blocks > 2 * round;
        return n >= 131072 && (n_out > 56 ? n_in <= 128 || (n_in <= 192 && !tail) : n_in <= 128 && !tail);
    }
    return n_out <= 128 && n_in <= (n_out > 112 ? 128 : n_out > 88 ? 96 : 64) && n >= 131072;
}

// y = act(y + bias) in place; kNotTaken where the tensor operations would do more than that
int bias_act(const Tensor &y, const Tensor &bias, bool relu)
{
    if (operations_are_seen() || !values_only(y) || !values_only(bias) || y.dim() != 2 || !y.is_contiguous() ||
        bias.dim() != 1 || bias.size(0) != y.size(1) || !bias.is_contiguous())
        return kNotTaken;
    return hgc_bias_act(data<float>(y), data<float>(bias), (int)y.size(0), (int)y.size(1), relu, stream_of(y));
}

// Products of float32 in float32.  (allowTF32CuBLAS() asks the same, but throws where the caller chose the precision through
// torch.backends.fp32_precision or torch.backends.cuda.matmul.fp32_precision.)
bool full_precision()
{
    const at::Float32Precision p = at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL);
    return p == at::Float32Precision::NONE || p == at::Float32Precision::IEEE;
}

// (act(x kernel + bias), status) in one kernel; kNotTaken where the tensor operations would do more than that, hgc_dense does not
// take the rows (whole 16-byte vectors) or the library's GEMM is the faster one
std::tuple<MaybeTensor, int> dense(const Tensor &x, const Tensor &kernel, const MaybeTensor &bias, bool relu)
{
    const std::tuple<MaybeTensor, int> not_taken{std::nullopt, kNotTaken};
    if (operations_are_seen() || at::impl::torch_function_mode_enabled() ||
        at::autocast::is_autocast_enabled(at::kCUDA) ||
        !values_only(x) || !values_only(kernel) || x.dim() != 2 || kernel.dim() != 2 || !x.is_contiguous() ||
        !kernel.is_contiguous() || x.size(1) != kernel.size(0) || !full_precision())
        return not_taken;
    if (bias.has_value() && (!values_only(*bias) || bias->dim() != 1 || bias->size(0) != kernel.size(1) || !bias->is_contiguous()))
        return not_taken;
    const int64_t n = x.size(0), n_in = x.size(1), n_out = kernel.size(1);
    if (n_in % 4 != 0 || !aligned16(x) || !dense_is_faster(n, n_in, n_out)) return not_taken;
    Tensor y = like(x, {n, n_out}, at::kFloat);
    const int rc = hgc_dense(data<float>(x), data<float>(kernel), data<float>(bias), data<float>(y), (int)n, (int)n_in, (int)n_out, relu,
                             stream_of(x));
    return {y, rc};
}

// out[:, column:] = x, likewise
int copy_columns(const Tensor &x, const Tensor &out, int column)
{
    if (operations_are_seen() || x.requires_grad() || !values_only(x) || !values_only(out) || x.dim() != 2 || out.dim() != 2 ||
        !x.is_contiguous() || out.stride(1) != 1 || column < 0 || x.size(0) != out.size(0) ||
        x.size(1) != out.size(1) - column)
        return kNotTaken;
    return hgc_copy_columns(data<float>(x), data<float>(out) + column, (int)out.stride(0), (int)x.size(0), (int)x.size(1),
                            stream_of(x));
}

}  // namespace

PYBIND11_MODULE(_native, m)
{
    // what goes wrong inside torch (memory that runs out, say) keeps its Python type
    pybind11::register_local_exception_translator([](std::exception_ptr p) {
        if (p) torch::translate_exception_to_python(p);
    });
    // other Python threads run while a call enqueues, as they do during a ctypes call
    const auto unlocked = pybind11::call_guard<pybind11::gil_scoped_release>();
    m.def("select_knn", &select_knn, unlocked);
    m.def("accumulate", &accumulate, unlocked);
    m.def("accumulate_grad", &accumulate_grad, unlocked);
    m.def("select_knn_grad", &select_knn_grad, unlocked);
    m.def("local_distance", &local_distance, unlocked);
    m.def("push_knn", &push_knn, unlocked);
    m.def("push_knn_grad", &push_knn_grad, unlocked);
    m.def("collect", &collect, unlocked);
    m.def("condensates", &condensates, unlocked);
    m.def("merge_noise", &merge_noise, unlocked);
    m.def("dense", &dense, unlocked);
    m.def("bias_act", &bias_act, unlocked);
    m.def("copy_columns", &copy_columns, unlocked);
}
