// PyTorch extension `spatha`: the same module name, function name, positional arguments and return
// shape as the reference's extension (end2end/spatha_mod/block_sparse/api/spatha.cu:41-65 ->
// spmm_cuda, end2end/spatha_mod/block_sparse/spmm/blockwise_library.cu:294-386), implemented as a
// thin pybind wrapper over the C ABI of libvenom_b200.  Differences, all deliberate:
//   * runs on torch's current CUDA stream (the reference launches on the legacy default stream);
//   * V is a run-time argument (the reference needs a separate -DV_64 build);
//   * arguments are checked and errors raise RuntimeError (the reference checks nothing);
//   * `bias` may be an undefined / empty tensor (the reference dereferences it unconditionally);
//   * the reference-format arrays are re-packed once per distinct (values, metadata, indices) triple and the
//     prepared operand is cached.  An entry is tied to the three tensors' storages through weak references:
//     once any of them has been freed (even if a new tensor later lands on the same address) the entry is
//     dead, its device copy is released and the operand is re-packed.  In-place edits bump the tensors'
//     version counters, which are part of the key (the copies of earlier versions go with the tensors, or with clear_cache()).
//   * an operand is held in each form (gather, dense-B) that a call has wanted, at most two copies; `form` holds it in one.
#include <torch/extension.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/python_numbers.h>

#include <map>
#include <mutex>
#include <tuple>

#include "../../include/venom_b200.h"

namespace {

struct Key {
    const void *values, *meta, *idx;
    int M, K, V, n, m, device;
    uint32_t ver_v, ver_m, ver_i;
    bool operator<(const Key &o) const
    {
        return std::tie(values, meta, idx, M, K, V, n, m, device, ver_v, ver_m, ver_i) <
               std::tie(o.values, o.meta, o.idx, o.M, o.K, o.V, o.n, o.m, o.device, o.ver_v, o.ver_m, o.ver_i);
    }
};

using WeakStorage = c10::weak_intrusive_ptr<c10::StorageImpl>;

struct Entry {
    // the operand re-packed per form (0: gather, 1: dense-B), each when a call first wants it
    vnm_handle_t handle[2];
    int last_n, last_t, last_form;   // the form of the last shape of call
    int64_t nv, nm, nc;              // sizes of the three arrays
    WeakStorage values, meta, idx;   // the storages the operand was re-packed from
    void release()
    {
        for (vnm_handle_t &h : handle) { vnm_destroy(h); h = nullptr; }
    }
    bool alive() const { return !values.expired() && !meta.expired() && !idx.expired(); }
};

std::map<Key, Entry> g_cache;
std::mutex g_mutex;

WeakStorage weak_of(const torch::Tensor &t)
{
    return WeakStorage(t.storage().getWeakStorageImpl());
}

bool same_storage(const WeakStorage &w, const torch::Tensor &t)
{
    return !w.expired() && w._unsafe_get_target() == t.storage().unsafeGetStorageImpl();
}

// Releases the device copies of operands whose source tensors no longer exist.
void sweep_dead_entries()
{
    for (auto it = g_cache.begin(); it != g_cache.end();) {
        if (!it->second.alive()) {
            it->second.release();
            it = g_cache.erase(it);
        } else {
            ++it;
        }
    }
}

// torch::empty on the device of `like`, without the dispatcher (0.4 us a call)
torch::Tensor device_empty(at::IntArrayRef shape, c10::ScalarType type, const torch::Tensor &like)
{
    return at::detail::empty_cuda(shape, type, like.device(), c10::nullopt);
}

void check(int rc, const char *what)
{
    TORCH_CHECK(rc == 0, what, " failed (", rc, "): ", vnm_last_error_string());
}

void check_sizes(const torch::Tensor &A_metadata, const torch::Tensor &A_indices, const torch::Tensor &A_values, int64_t nv, int64_t nm, int64_t nc)
{
    TORCH_CHECK(A_values.numel() == nv && A_metadata.numel() == nm && A_indices.numel() == nc, "spatha.spmm: array sizes do not match the format (values ",
                nv, ", metadata ", nm, ", indices ", nc, ")");
}

// The handle that multiplies N columns: looked up in (or added to) the cache, in the form `form` (VNM_STRATEGY_*), or for AUTO in
// the one estimated to be the faster for this number of columns and the layout of the activation.  `dense_b` receives that form.
vnm_handle_t operand_for(const torch::Tensor &A_metadata, const torch::Tensor &A_indices, const torch::Tensor &A_values, int M, int K, int V, int n, int m,
                         int device, int N, bool in_place, int form, cudaStream_t stream, int *dense_b)
{
    TORCH_CHECK(form == VNM_STRATEGY_AUTO || form == VNM_STRATEGY_GATHER || form == VNM_STRATEGY_DENSE_B, "spatha.spmm: unknown form ", form);
    Key key{A_values.data_ptr(), A_metadata.data_ptr(), A_indices.data_ptr(), M, K, V, n, m, device,
            (uint32_t)A_values._version(), (uint32_t)A_metadata._version(), (uint32_t)A_indices._version()};
    std::lock_guard<std::mutex> lock(g_mutex);
    auto it = g_cache.find(key);
    if (it != g_cache.end() && !(same_storage(it->second.values, A_values) && same_storage(it->second.meta, A_metadata) &&
                                 same_storage(it->second.idx, A_indices))) {
        // same addresses, different (or freed) tensors: the cached copy belongs to an operand that is gone
        it->second.release();
        g_cache.erase(it);
        it = g_cache.end();
    }
    if (it == g_cache.end()) {
        int64_t ksp = 0, nv = 0, nm = 0, nc = 0;
        check(vnm_sizes(M, K, V, n, m, &ksp, &nv, &nm, &nc), "vnm_sizes");
        check_sizes(A_metadata, A_indices, A_values, nv, nm, nc);
        sweep_dead_entries();
        it = g_cache.emplace(key, Entry{{nullptr, nullptr}, -1, 0, 0, nv, nm, nc, weak_of(A_values), weak_of(A_metadata), weak_of(A_indices)}).first;
    }
    check_sizes(A_metadata, A_indices, A_values, it->second.nv, it->second.nm, it->second.nc);
    // Dense-B form or gather form: by the estimate for this number of columns and the layout of the activation (a
    // transposed [tokens, features] view is read in place by the dense-B form and transposed for the gather form).
    Entry &e = it->second;
    if (form != VNM_STRATEGY_AUTO) {
        *dense_b = form == VNM_STRATEGY_DENSE_B && m % 4 == 0 && K % m == 0;   // else there is only the gather form
    } else {
        if (e.last_n != N || e.last_t != (int)in_place) {
            int strategy = 0;
            check(vnm_choose_form(M, K, V, n, m, N, in_place ? 1 : 0, &strategy), "vnm_choose_form");
            e.last_form = strategy == VNM_STRATEGY_DENSE_B ? 1 : 0;
            e.last_n = N;
            e.last_t = in_place;
        }
        *dense_b = e.last_form;
        // A graph that is being captured uses the form that is there: re-packing is work for outside of it.
        if (!e.handle[*dense_b] && e.handle[1 - *dense_b] && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) *dense_b = 1 - *dense_b;
    }
    if (!e.handle[*dense_b]) {
        const int rc = vnm_prepare_as(A_values.data_ptr(), (const uint32_t *)A_metadata.data_ptr(), (const uint32_t *)A_indices.data_ptr(), M, K, V, n, m,
                                      *dense_b ? VNM_STRATEGY_DENSE_B : VNM_STRATEGY_GATHER, &e.handle[*dense_b], stream);
        if (rc == VNM_ERR_CUDA && form == VNM_STRATEGY_AUTO && e.handle[1 - *dense_b]) e.last_form = *dense_b = 1 - *dense_b;   // no memory for a second form
        else check(rc, "vnm_prepare_as");
    }
    return e.handle[*dense_b];
}

void check_arrays(const torch::Tensor &A_metadata, const torch::Tensor &A_indices, const torch::Tensor &A_values, const torch::Tensor &rhs)
{
    TORCH_CHECK(A_values.is_cuda() && A_metadata.is_cuda() && A_indices.is_cuda() && rhs.is_cuda(), "spatha.spmm: CUDA tensors expected");
    TORCH_CHECK(A_values.scalar_type() == torch::kFloat16 && rhs.scalar_type() == torch::kFloat16, "spatha.spmm: fp16 values / rhs expected");
    TORCH_CHECK(A_metadata.scalar_type() == torch::kInt32 && A_indices.scalar_type() == torch::kInt32, "spatha.spmm: int32 metadata / indices expected");
    TORCH_CHECK(A_values.is_contiguous() && A_metadata.is_contiguous() && A_indices.is_contiguous(), "spatha.spmm: contiguous sparse arrays expected");
}

// The bias as a pointer, null if there is none.
const void *bias_pointer(const c10::optional<torch::Tensor> &bias, int M)
{
    if (!(bias.has_value() && bias->defined() && bias->numel() > 0)) return nullptr;
    TORCH_CHECK(bias->is_cuda() && bias->scalar_type() == torch::kFloat16 && bias->numel() == M && bias->is_contiguous(), "spatha.spmm: bias must be fp16 [A_num_rows]");
    return bias->data_ptr();
}

// out [N, M] = (A * B).T + bias for an activation that lies as [N, K] rows of stride `ld` (16-byte aligned).
void product_nk(vnm_handle_t h, int dense_b, const torch::Tensor &act, int64_t ld, int K, int N, int M, const void *bias, torch::Tensor &out, cudaStream_t stream)
{
    torch::Tensor ws;
    if (!dense_b) ws = device_empty({K, N}, torch::kFloat16, act);
    check(vnm_spmm_f16_nk_ws(h, act.data_ptr(), ld, N, bias, out.data_ptr(), M, VNM_LAYOUT_NM, dense_b ? out.data_ptr() : ws.data_ptr(), stream),
          "vnm_spmm_f16_nk");
}

}  // namespace

torch::Tensor spmm(torch::Tensor A_metadata, torch::Tensor A_indices, torch::Tensor A_values, torch::Tensor rhs_matrix,
                   c10::optional<torch::Tensor> bias, int64_t A_num_rows, int64_t A_num_cols, int64_t B_num_cols,
                   int64_t vec_length, int64_t n, int64_t m, int64_t nnz, int64_t seed, int64_t mbrow, int64_t brow, int64_t form)
{
    (void)seed;
    check_arrays(A_metadata, A_indices, A_values, rhs_matrix);
    TORCH_CHECK(mbrow == 32 && brow == 4, "spatha.spmm: the storage format is defined for mbrow = 32, brow = 4");
    const int M = (int)A_num_rows, K = (int)A_num_cols, N = (int)B_num_cols, V = (int)vec_length;
    int64_t ksp = 0, nv = 0, nm = 0, nc = 0;
    check(vnm_sizes(M, K, V, (int)n, (int)m, &ksp, &nv, &nm, &nc), "vnm_sizes");
    TORCH_CHECK(nnz == nv, "spatha.spmm: nnz must be A_num_rows * padded compressed columns (", nv, ")");
    TORCH_CHECK(rhs_matrix.dim() == 2 && rhs_matrix.size(0) == K && rhs_matrix.size(1) == N, "spatha.spmm: rhs_matrix must be [A_num_cols, B_num_cols]");
    // A transposed view of a [B_num_cols, A_num_cols] activation (what `flattened_input.T` is) is consumed as it lies;
    // any other non-contiguous rhs is copied like the reference does.
    const bool rhs_is_t_view = rhs_matrix.stride(0) == 1 && rhs_matrix.stride(1) >= K && N > 1;
    const void *bias_ptr = bias_pointer(bias, M);

    c10::cuda::CUDAGuard guard(rhs_matrix.device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    int dense_b = 0;
    const bool in_place = rhs_is_t_view && rhs_matrix.stride(1) % 8 == 0 && (reinterpret_cast<uintptr_t>(rhs_matrix.data_ptr()) & 15) == 0;
    vnm_handle_t h = operand_for(A_metadata, A_indices, A_values, M, K, V, (int)n, (int)m, (int)rhs_matrix.device().index(), N, in_place, (int)form, stream, &dense_b);
    auto out = device_empty({N, M}, torch::kFloat16, rhs_matrix);
    if (in_place) {
        product_nk(h, dense_b, rhs_matrix, rhs_matrix.stride(1), K, N, M, bias_ptr, out, stream);
        return out;
    }
    torch::Tensor rhs = rhs_matrix.stride(1) == 1 ? rhs_matrix : rhs_matrix.contiguous();
    check(vnm_spmm_f16(h, rhs.data_ptr(), rhs.stride(0), N, bias_ptr, out.data_ptr(), M, VNM_LAYOUT_NM, stream), "vnm_spmm_f16");
    return out;
}

// A layer's forward in one call: input [..., A_num_cols] -> [..., A_num_rows], as spmm() on the flattened input's transpose gives
// it, without the views that call needs (each a trip through the dispatcher; at decoding sizes these and the interpreter's
// share of the call took longer than the product: measured 12.2 us a call before, 6.3 after, for a kernel of 5 us).  An undefined
// result (None) means: an input that is not read in place -- take spmm().
c10::optional<torch::Tensor> linear(const torch::Tensor &input, const torch::Tensor &A_metadata, const torch::Tensor &A_indices, const torch::Tensor &A_values,
                                    const c10::optional<torch::Tensor> &bias, int64_t A_num_rows, int64_t A_num_cols, int64_t vec_length, int64_t n, int64_t m, int64_t form)
{
    const int M = (int)A_num_rows, K = (int)A_num_cols;
    const int64_t dims = input.dim();
    if (dims < 2 || K <= 0 || K % 8 != 0 || input.size(-1) != K || !input.is_contiguous()) return c10::nullopt;
    const int64_t N = input.numel() / K;
    if (N <= 1 || N > INT32_MAX || (reinterpret_cast<uintptr_t>(input.data_ptr()) & 15) != 0) return c10::nullopt;
    check_arrays(A_metadata, A_indices, A_values, input);
    const void *bias_ptr = bias_pointer(bias, M);
    c10::cuda::CUDAGuard guard(input.device());
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    int dense_b = 0;
    vnm_handle_t h = operand_for(A_metadata, A_indices, A_values, M, K, (int)vec_length, (int)n, (int)m, (int)input.device().index(), (int)N, true, (int)form, stream, &dense_b);
    c10::SmallVector<int64_t, 6> shape(input.sizes().begin(), input.sizes().end());
    shape.back() = M;
    auto out = device_empty(shape, torch::kFloat16, input);
    product_nk(h, dense_b, input, K, K, (int)N, M, bias_ptr, out, stream);
    return out;
}

// capi.Prepared.spmm's call of vnm_spmm_f16 with its allocation, without the interpreter's share (attribute reads, argument
// boxing, and 3.4 us for torch.cuda.current_stream alone).  None: not the plain case, or an error that the caller's own path reports.
c10::optional<torch::Tensor> product(int64_t handle, const torch::Tensor &B, const c10::optional<torch::Tensor> &bias, int64_t M, int64_t K, int64_t layout)
{
    if (!handle || !B.is_cuda() || B.scalar_type() != torch::kFloat16 || B.dim() != 2 || B.size(0) != K || B.stride(1) != 1) return c10::nullopt;
    if (bias.has_value() && (!bias->defined() || !bias->is_cuda() || bias->scalar_type() != torch::kFloat16 || bias->numel() != M || !bias->is_contiguous()))
        return c10::nullopt;
    if ((layout != VNM_LAYOUT_MN && layout != VNM_LAYOUT_NM) || B.device().index() != c10::cuda::current_device()) return c10::nullopt;
    const int64_t N = B.size(1);
    if (N <= 0 || N > INT32_MAX) return c10::nullopt;
    auto out = layout == VNM_LAYOUT_MN ? device_empty({M, N}, torch::kFloat16, B) : device_empty({N, M}, torch::kFloat16, B);
    if (vnm_spmm_f16(reinterpret_cast<vnm_handle_t>(handle), B.data_ptr(), B.stride(0), (int)N, bias.has_value() ? bias->data_ptr() : nullptr, out.data_ptr(),
                     out.stride(0), (int)layout, c10::cuda::getCurrentCUDAStream().stream()) != 0)
        return c10::nullopt;
    return out;
}

// The format conversions of capi with their allocations, without the interpreter's share.  None: not the plain case, or an error
// that the caller's own path reports.

// A page-locked word per thread that a violation count is copied to: a copy to pageable memory goes through a staging buffer.
class HostWord {
public:
    ~HostWord() { if (p_) (void)cudaFreeHost(p_); }
    unsigned long long *get()
    {
        if (!p_ && cudaHostAlloc(reinterpret_cast<void **>(&p_), sizeof(*p_), cudaHostAllocPortable) != cudaSuccess) { (void)cudaGetLastError(); p_ = nullptr; }
        return p_;
    }
private:
    unsigned long long *p_ = nullptr;
};
thread_local HostWord t_count;

// Violations counted in `dev` by the work queued so far (waits for it); -1 if they cannot be read.
int64_t read_count(const torch::Tensor &dev, cudaStream_t stream)
{
    unsigned long long *host = t_count.get();
    if (!host || cudaMemcpyAsync(host, dev.data_ptr(), sizeof(*host), cudaMemcpyDeviceToHost, stream) != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess) return -1;
    return (int64_t)*host;
}

torch::Tensor new_count(const torch::Tensor &like, cudaStream_t stream)
{
    auto t = device_empty({1}, torch::kInt64, like);
    TORCH_CHECK(cudaMemsetAsync(t.data_ptr(), 0, 8, stream) == cudaSuccess, "cudaMemsetAsync failed");
    return t;
}

bool on_current_device(const torch::Tensor &t) { return t.is_cuda() && t.device().index() == c10::cuda::current_device(); }

using Compressed = std::tuple<torch::Tensor, torch::Tensor, c10::optional<int64_t>>;
c10::optional<Compressed> compress(const torch::Tensor &dense, const torch::Tensor &colloc, int64_t V, int64_t m, int64_t n, bool count)
{
    if (!on_current_device(dense) || !on_current_device(colloc) || dense.scalar_type() != torch::kFloat16 || dense.dim() != 2 || dense.stride(1) != 1) return c10::nullopt;
    const int64_t M = dense.size(0), K = dense.size(1);
    int64_t ksp = 0, nv = 0, nm = 0, nc = 0;
    if (M <= 0 || K <= 0 || M > INT32_MAX || K > INT32_MAX || vnm_sizes((int)M, (int)K, (int)V, (int)n, (int)m, &ksp, &nv, &nm, &nc) != 0) return c10::nullopt;
    if (colloc.numel() != nc || colloc.element_size() != 4 || !colloc.is_contiguous()) return c10::nullopt;
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    auto values = device_empty({nv}, torch::kFloat16, dense);
    auto meta = device_empty({nm}, torch::kInt32, dense);
    torch::Tensor viol;
    if (count) viol = new_count(dense, stream);
    if (vnm_compress_f16(dense.data_ptr(), dense.stride(0), nullptr, (const uint32_t *)colloc.data_ptr(), (int)M, (int)K, (int)V, (int)n, (int)m, values.data_ptr(),
                         (uint32_t *)meta.data_ptr(), count ? (unsigned long long *)viol.data_ptr() : nullptr, stream) != 0)
        return c10::nullopt;
    c10::optional<int64_t> bad;
    if (count) {
        bad = read_count(viol, stream);
        if (*bad < 0) return c10::nullopt;
    }
    return Compressed(values, meta, bad);
}

using Sparsified = std::tuple<torch::Tensor, torch::Tensor, torch::Tensor, int64_t>;
c10::optional<Sparsified> sparsify(const torch::Tensor &w, int64_t V, int64_t m, int64_t n)
{
    const bool half = w.scalar_type() == torch::kFloat16;
    if (!on_current_device(w) || (!half && w.scalar_type() != torch::kFloat32) || w.dim() != 2 || w.stride(1) != 1) return c10::nullopt;
    const int64_t M = w.size(0), K = w.size(1);
    int64_t ksp = 0, nv = 0, nm = 0, nc = 0;
    if (M <= 0 || K <= 0 || M > INT32_MAX || K > INT32_MAX || vnm_sizes((int)M, (int)K, (int)V, (int)n, (int)m, &ksp, &nv, &nm, &nc) != 0) return c10::nullopt;
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    auto values = device_empty({nv}, torch::kFloat16, w);
    auto meta = device_empty({nm}, torch::kInt32, w), cols = device_empty({nc}, torch::kInt32, w), viol = new_count(w, stream);
    if (vnm_sparsify_magnitude(w.data_ptr(), half ? VNM_F16 : VNM_F32, w.stride(0), (int)M, (int)K, (int)V, (int)n, (int)m, values.data_ptr(), (uint32_t *)meta.data_ptr(),
                               (uint32_t *)cols.data_ptr(), (unsigned long long *)viol.data_ptr(), stream) != 0)
        return c10::nullopt;
    const int64_t bad = read_count(viol, stream);
    if (bad < 0) return c10::nullopt;
    return Sparsified(values, meta, cols, bad);
}

c10::optional<torch::Tensor> decompress(const torch::Tensor &values, const torch::Tensor &meta, const torch::Tensor &colloc, int64_t M, int64_t K, int64_t V, int64_t m, int64_t n)
{
    if (!on_current_device(values) || !on_current_device(meta) || !on_current_device(colloc) || M <= 0 || K <= 0 || M > INT32_MAX || K > INT32_MAX) return c10::nullopt;
    auto dense = device_empty({M, K}, torch::kFloat16, values);
    if (vnm_decompress_f16(values.data_ptr(), (const uint32_t *)meta.data_ptr(), (const uint32_t *)colloc.data_ptr(), (int)M, (int)K, (int)V, (int)n, (int)m, dense.data_ptr(),
                           K, c10::cuda::getCurrentCUDAStream().stream()) != 0)
        return c10::nullopt;
    return dense;
}

void clear_cache()
{
    std::lock_guard<std::mutex> lock(g_mutex);
    for (auto &kv : g_cache) kv.second.release();
    g_cache.clear();
}

int64_t cache_size()
{
    std::lock_guard<std::mutex> lock(g_mutex);
    return (int64_t)g_cache.size();
}

int64_t cached_copies()
{
    std::lock_guard<std::mutex> lock(g_mutex);
    int64_t n = 0;
    for (const auto &kv : g_cache)
        for (vnm_handle_t h : kv.second.handle) n += h != nullptr;
    return n;
}

// linear() and product() as plain C functions of the module: pybind11's conversion of their arguments took 0.4 us a call.
namespace {

const at::Tensor &tensor_of(PyObject *o)
{
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor");
    return THPVariable_Unpack(o);
}

c10::optional<torch::Tensor> tensor_or_none(PyObject *o)
{
    if (o == Py_None) return c10::nullopt;
    return tensor_of(o);
}

PyObject *wrapped(c10::optional<torch::Tensor> &t)
{
    if (!t.has_value()) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(*t));
}

PyObject *py_linear(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n == 10 || n == 11, "linear(input, A_metadata, A_indices, A_values, bias, A_num_rows, A_num_cols, vec_length, n, m, form=0)");
    const at::Tensor &input = tensor_of(args[0]), &meta = tensor_of(args[1]), &idx = tensor_of(args[2]), &values = tensor_of(args[3]);
    const c10::optional<torch::Tensor> bias = tensor_or_none(args[4]);
    int64_t v[6] = {0, 0, 0, 0, 0, VNM_STRATEGY_AUTO};
    for (int i = 0; i < (int)n - 5; i++) v[i] = THPUtils_unpackLong(args[5 + i]);
    c10::optional<torch::Tensor> out;
    {
        pybind11::gil_scoped_release no_gil;
        out = linear(input, meta, idx, values, bias, v[0], v[1], v[2], v[3], v[4], v[5]);
    }
    return wrapped(out);
    END_HANDLE_TH_ERRORS
}

PyObject *py_product(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n == 6, "product(handle, B, bias, M, K, layout)");
    const int64_t handle = THPUtils_unpackLong(args[0]);
    const at::Tensor &B = tensor_of(args[1]);
    const c10::optional<torch::Tensor> bias = tensor_or_none(args[2]);
    int64_t v[3];
    for (int i = 0; i < 3; i++) v[i] = THPUtils_unpackLong(args[3 + i]);
    c10::optional<torch::Tensor> out;
    {
        pybind11::gil_scoped_release no_gil;
        out = product(handle, B, bias, v[0], v[1], v[2]);
    }
    return wrapped(out);
    END_HANDLE_TH_ERRORS
}

PyMethodDef fast_calls[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&py_linear)), METH_FASTCALL, "A layer's forward: [..., A_num_cols] -> [..., A_num_rows], or None"},
    {"product", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&py_product)), METH_FASTCALL, "vnm_spmm_f16 with its allocation, or None"},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, mod)
{
    mod.def("spmm", &spmm, "V:N:M sparse x dense product (returns [B_num_cols, A_num_rows])", pybind11::arg("A_metadata"), pybind11::arg("A_indices"),
            pybind11::arg("A_values"), pybind11::arg("rhs_matrix"), pybind11::arg("bias"), pybind11::arg("A_num_rows"), pybind11::arg("A_num_cols"),
            pybind11::arg("B_num_cols"), pybind11::arg("vec_length"), pybind11::arg("n"), pybind11::arg("m"), pybind11::arg("nnz"),
            pybind11::arg("seed"), pybind11::arg("mbrow"), pybind11::arg("brow"), pybind11::arg("form") = (int64_t)VNM_STRATEGY_AUTO);
    if (PyModule_AddFunctions(mod.ptr(), fast_calls) != 0) throw pybind11::error_already_set();
    mod.def("compress", &compress, "vnm_compress_f16 with its allocations, or None", pybind11::call_guard<pybind11::gil_scoped_release>());
    mod.def("sparsify", &sparsify, "vnm_sparsify_magnitude with its allocations, or None", pybind11::call_guard<pybind11::gil_scoped_release>());
    mod.def("decompress", &decompress, "vnm_decompress_f16 with its allocation, or None", pybind11::call_guard<pybind11::gil_scoped_release>());
    mod.def("clear_cache", &clear_cache, "Drop every cached prepared operand");
    mod.def("cache_size", &cache_size, "Cached operands");
    mod.def("cached_copies", &cached_copies, "Device copies they hold: one or two (gather form, dense-B form) each");
}
