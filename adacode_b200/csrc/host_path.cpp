// The host side of the calls that a decode step or a pack is made of, as a Python extension module (`_native`): outputs are
// allocated, launches described and views made here instead of object by object in Python.  The launches
// themselves are those of include/adacode.h; tensors go through the dispatcher (so autograd, inference mode and version
// counters see what they see of the same calls from Python).
//
// These calls were bound by the interpreter, not by the GPU.  On one B200's host, in Python and now: keys and values of one
// block through pack_pair, 13 us of kernels, 95 -> 57 us; an update of one token, 10 us of kernels, 62 -> 33 us.
#include <torch/csrc/python_headers.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/GradMode.h>
#include <c10/core/InferenceMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "adacode.h"

namespace {

using at::Tensor;

// Leave with the Python exception that is set.
[[noreturn]] void fail() {
    python_error e;
    e.persist();
    throw e;
}

// A call into the library that failed raises what the same call from Python does (adacode_b200._lib.check).
void check(int rc, const char *what) {
    if (rc == ADACODE_OK) return;
    if (PyObject *lib = PyImport_ImportModule("adacode_b200._lib")) {
        Py_XDECREF(PyObject_CallMethod(lib, "check", "is", rc, what));
        Py_DECREF(lib);
        if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s: %d", what, rc);
    }
    fail();
}

// References that are dropped when a function ends early.
struct Owned {
    PyObject *p;
    explicit Owned(PyObject *o = nullptr) : p(o) {}
    Owned(Owned &&o) noexcept : p(o.p) { o.p = nullptr; }
    Owned(const Owned &) = delete;
    ~Owned() { Py_XDECREF(p); }
    PyObject *release() {
        PyObject *o = p;
        p = nullptr;
        return o;
    }
};

const Tensor &tensor(PyObject *o) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor");
    return THPVariable_Unpack(o);
}

int64_t integer(PyObject *o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) fail();
    return v;
}

// This thread's page-locked bytes that packs report into: they grow with the largest report (of a MiB at most) and go
// with the thread.  A token never comes twice while the bytes live: they are cleared before the tokens start over.
struct ReportBox {
    void *host = nullptr;
    size_t bytes = 0;
    uint32_t token = 0;
    uint32_t next_token() {
        if (token == 0xFFFFFFFFu) memset(host, 0, bytes), token = 0;
        return ++token;
    }
    ~ReportBox() {
        if (host) (void)cudaFreeHost(host);
    }
    void reserve(size_t need) {
        if (need <= bytes) return;
        if (host) (void)cudaFreeHost(host);
        host = nullptr, bytes = 0;
        const size_t n = need < (1 << 14) ? (1 << 14) : 2 * need;
        C10_CUDA_CHECK(cudaHostAlloc(&host, n, cudaHostAllocPortable | cudaHostAllocMapped));
        bytes = n;
        memset(host, 0, n);
    }
};

ReportBox &report_box() {
    static thread_local ReportBox box;
    return box;
}

// pack(tensors, rights, nbits, seq_tile, capacities, need_hist, workspace)
//   -> (((sign_mant, codes, escapes, tile_base, seg_offsets, histogram or None, offsets, status), ...), hist bytes or None)
// Tensors that follow each other and share shape and code length go through one launch; all launches are under way before the
// first is waited for.  They are plain bf16 [B, H, S, D] on one CUDA device, strides as the library wants them:
// the caller has seen to that, and to a workspace for the largest launch.  need_hist may be one tensor's histogram to
// add to.  Nothing is trimmed or run again here; `status` is the launch's status word.
PyObject *pack(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n_args == 7 && PyTuple_Check(args[0]) && PyTuple_Check(args[1]) && PyTuple_Check(args[2]) && PyTuple_Check(args[4]),
                     "pack: arguments");
    constexpr int kMost = 8;
    const int n = (int)PyTuple_GET_SIZE(args[0]);
    TORCH_CHECK(n >= 1 && n <= kMost && PyTuple_GET_SIZE(args[1]) == n && PyTuple_GET_SIZE(args[2]) == n && PyTuple_GET_SIZE(args[4]) == n,
                "pack: one to eight tensors");
    const int64_t T = integer(args[3]);
    const Tensor given_hist = THPVariable_Check(args[5]) ? THPVariable_Unpack(args[5]) : Tensor();
    TORCH_CHECK(!given_hist.defined() || (n == 1 && given_hist.scalar_type() == at::kInt && given_hist.numel() == 256 &&
                                          given_hist.is_contiguous() && given_hist.is_cuda()),
                "pack: a histogram is 256 contiguous int32 on the GPU");
    const bool need_hist = !given_hist.defined() && PyObject_IsTrue(args[5]) == 1;
    const Tensor &ws = tensor(args[6]);
    const Tensor &x0 = tensor(PyTuple_GET_ITEM(args[0], 0));
    TORCH_CHECK(x0.is_cuda() && T > 0, "pack: tensors on a GPU, whole blocks");
    const c10::cuda::CUDAGuard on(x0.device());
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x0.device().index()).stream();
    const auto bytes = at::TensorOptions().device(x0.device()).dtype(at::kByte);

    adacode_pack_job jobs[kMost];
    Tensor sm[kMost], cd[kMost], esc[kMost], base[kMost];
    struct Launch {
        int first, n, nbits;
        int64_t B, H, D, elems, offs, words;                      // [segment offsets of its tensors | status | 128 words of histogram each]
        Tensor mail;
        size_t at;                                         // where its report begins
        uint32_t token;
    } launch[kMost];
    int n_launches = 0;
    for (int j = 0; j < n; ++j) {
        const Tensor &x = tensor(PyTuple_GET_ITEM(args[0], j));
        TORCH_CHECK(x.dim() == 4 && x.scalar_type() == at::kBFloat16 && x.device() == x0.device() && x.stride(3) == 1 && x.size(2) % T == 0,
                    "pack: [B, H, S, D] bf16 tensors of one device, whole blocks");
        const int nbits = (int)integer(PyTuple_GET_ITEM(args[2], j));
        const int64_t cap = integer(PyTuple_GET_ITEM(args[4], j));
        TORCH_CHECK(cap >= 0 && nbits >= 1 && nbits <= 4, "pack: capacity, code length");
        // (a launch covers fewer than 2**31 elements)
        const bool joins = j > 0 && launch[n_launches - 1].nbits == nbits && tensor(PyTuple_GET_ITEM(args[0], j - 1)).sizes() == x.sizes() &&
                           launch[n_launches - 1].elems + x.numel() < (1ll << 31);
        if (!joins) launch[n_launches++] = Launch{j, 0, nbits, x.size(0), x.size(1), x.size(3), 0, x.size(2) / T + 1, 0, Tensor(), 0, 0};
        Launch &l = launch[n_launches - 1];
        ++l.n, l.elems += x.numel();
        const int64_t n_blocks = l.offs - 1, plane = l.B * l.H * T * l.D;
        sm[j] = at::empty({n_blocks, plane}, bytes);
        cd[j] = at::empty({n_blocks, plane * nbits / 8}, bytes);
        esc[j] = at::empty({cap}, bytes);
        base[j] = at::empty({n_blocks, l.B * l.H}, bytes.dtype(at::kInt));
        adacode_pack_job &b = jobs[j];
        b.src_bf16 = x.const_data_ptr(), b.stride_b = x.stride(0), b.stride_h = x.stride(1), b.stride_s = x.stride(2);
        b.n_blocks = (int)n_blocks, b.right = (int)integer(PyTuple_GET_ITEM(args[1], j));
        b.sign_mant = (uint8_t *)sm[j].mutable_data_ptr(), b.codes = (uint8_t *)cd[j].mutable_data_ptr();
        b.escapes = (uint8_t *)esc[j].mutable_data_ptr(), b.escapes_capacity = cap;
        b.tile_base = (int32_t *)base[j].mutable_data_ptr();
    }
    size_t host_bytes = 0;
    for (int i = 0; i < n_launches; ++i) {
        Launch &l = launch[i];
        l.words = l.n * l.offs + 1 + (need_hist ? 128 * l.n : 0);
        l.mail = at::empty({l.words}, bytes.dtype(at::kLong));
        int64_t *const m = l.mail.mutable_data_ptr<int64_t>();
        for (int j = l.first; j < l.first + l.n; ++j) {
            jobs[j].seg_escape_offsets = m + (j - l.first) * l.offs;
            jobs[j].hist256 = need_hist              ? (int32_t *)(m + l.n * l.offs + 1) + 256 * (j - l.first)
                              : given_hist.defined() ? (int32_t *)given_hist.mutable_data_ptr()
                                                     : nullptr;
        }
        l.at = host_bytes;
        host_bytes += (size_t)l.words * 8;
    }
    // a report holds a MiB at most; more offsets than that are fetched by a copy
    const bool reports = host_bytes <= (1 << 20);
    ReportBox &box = report_box();
    if (reports) box.reserve(2 * host_bytes);
    std::vector<uint8_t> fetched(host_bytes);
    uint8_t *const host = fetched.data();
    const char *what = "adacode_pack_jobs";
    int rc = ADACODE_OK;
    {
        pybind11::gil_scoped_release waits;
        for (int i = 0; i < n_launches && rc == ADACODE_OK; ++i) {
            Launch &l = launch[i];
            int64_t *const m = l.mail.mutable_data_ptr<int64_t>();
            int32_t *const status = (int32_t *)(m + l.n * l.offs);
            const size_t report = (size_t)l.words * 8;
            if (reports) {
                l.token = box.next_token();
                what = "adacode_pack_jobs_report";
                rc = adacode_pack_jobs_report(jobs + l.first, l.n, (int)l.B, (int)l.H, (int)T, (int)l.D, l.nbits, ws.mutable_data_ptr(),
                                              ws.nbytes(), status, m, (uint8_t *)box.host + 2 * l.at, report, l.token, stream);
            } else {
                C10_CUDA_CHECK(cudaMemsetAsync(m, 0, report, stream));
                rc = adacode_pack_jobs(jobs + l.first, l.n, (int)l.B, (int)l.H, (int)T, (int)l.D, l.nbits, ws.mutable_data_ptr(), ws.nbytes(),
                                       status, stream);
                C10_CUDA_CHECK(cudaMemcpyAsync(host + l.at, m, report, cudaMemcpyDeviceToHost, stream));
            }
        }
        // (what is under way still reports, or writes, into this thread's bytes)
        if (rc != ADACODE_OK) (void)cudaStreamSynchronize(stream);
        if (rc == ADACODE_OK && !reports) C10_CUDA_CHECK(cudaStreamSynchronize(stream));
        for (int i = 0; i < n_launches && rc == ADACODE_OK && reports; ++i) {
            what = "adacode_wait_report";
            rc = adacode_wait_report((uint8_t *)box.host + 2 * launch[i].at, (size_t)launch[i].words * 8, launch[i].token, host + launch[i].at, stream);
        }
    }
    check(rc, what);

    Owned parts(PyTuple_New(n)), hists(need_hist ? PyBytes_FromStringAndSize(nullptr, 1024 * n) : Py_NewRef(Py_None));
    if (!parts.p || !hists.p) fail();
    for (int i = 0; i < n_launches; ++i) {
        const Launch &l = launch[i];
        const int64_t *const got = (const int64_t *)(host + l.at);
        const Owned status(PyLong_FromUnsignedLong(*(const uint32_t *)(got + l.n * l.offs)));
        const Tensor counts = need_hist ? l.mail.slice(0, l.n * l.offs + 1).view(at::kInt) : Tensor();
        for (int k = 0; k < l.n; ++k) {
            const int j = l.first + k;
            const Owned offsets(PyList_New(l.offs));
            if (!offsets.p) fail();
            for (int64_t o = 0; o < l.offs; ++o) PyList_SET_ITEM(offsets.p, o, PyLong_FromLongLong(got[k * l.offs + o]));
            const Owned hist(need_hist              ? THPVariable_Wrap(counts.slice(0, 256 * k, 256 * (k + 1)))
                             : given_hist.defined() ? Py_NewRef(args[5])
                                                    : Py_NewRef(Py_None));
            if (need_hist) memcpy(PyBytes_AS_STRING(hists.p) + 1024 * j, (const uint8_t *)(got + l.n * l.offs + 1) + 1024 * k, 1024);
            const Owned o_sm(THPVariable_Wrap(sm[j])), o_cd(THPVariable_Wrap(cd[j])), o_esc(THPVariable_Wrap(esc[j])),
                o_base(THPVariable_Wrap(base[j])), o_seg(THPVariable_Wrap(l.mail.slice(0, k * l.offs, (k + 1) * l.offs)));
            PyObject *part = PyTuple_Pack(8, o_sm.p, o_cd.p, o_esc.p, o_base.p, o_seg.p, hist.p, offsets.p, status.p);
            if (!part) fail();
            PyTuple_SET_ITEM(parts.p, j, part);
        }
    }
    return PyTuple_Pack(2, parts.p, hists.p);
    END_HANDLE_TH_ERRORS
}

// pack_flat(x, right, nbits, block, capacity, histogram or None, workspace)
//   -> (sign_mant, codes, escapes, block_base, total, status)
// A contiguous bf16 tensor on a GPU, a multiple of 8 and fewer than 2**31 elements on a 16-byte boundary.  As with pack,
// trimming and packing again are the caller's.
PyObject *pack_flat(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n_args == 7, "pack_flat: arguments");
    const Tensor &x = tensor(args[0]), &ws = tensor(args[6]);
    const int right = (int)integer(args[1]), nbits = (int)integer(args[2]);
    const int64_t block = integer(args[3]), cap = integer(args[4]), n = x.numel();
    const Tensor hist = args[5] == Py_None ? Tensor() : tensor(args[5]);
    TORCH_CHECK(x.scalar_type() == at::kBFloat16 && x.is_cuda() && x.is_contiguous() && n > 0 && block > 0 && cap >= 0 && nbits >= 1 && nbits <= 4,
                "pack_flat: a contiguous bf16 tensor on a GPU");
    TORCH_CHECK(!hist.defined() || (hist.scalar_type() == at::kInt && hist.numel() == 256 && hist.is_contiguous() && hist.device() == x.device()),
                "pack_flat: a histogram is 256 contiguous int32 on the GPU");
    const c10::cuda::CUDAGuard on(x.device());
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    const auto bytes = at::TensorOptions().device(x.device()).dtype(at::kByte);
    const Tensor sm = at::empty({n}, bytes), cd = at::empty({n * nbits / 8}, bytes), esc = at::empty({cap}, bytes);
    const Tensor base = at::empty({(n + block - 1) / block}, bytes.dtype(at::kInt)), mail = at::empty({ADACODE_FLAT_REPORT_BYTES / 8}, bytes.dtype(at::kLong));
    int64_t got[ADACODE_FLAT_REPORT_BYTES / 8];
    ReportBox &box = report_box();
    box.reserve(2 * sizeof(got));
    const uint32_t token = box.next_token();
    const char *what = "adacode_pack_flat";
    int rc;
    {
        pybind11::gil_scoped_release waits;
        rc = adacode_pack_flat(x.const_data_ptr(), n, right, nbits, (uint8_t *)sm.mutable_data_ptr(), (uint8_t *)cd.mutable_data_ptr(),
                               (uint8_t *)esc.mutable_data_ptr(), cap, (int32_t *)base.mutable_data_ptr(),
                               hist.defined() ? (int32_t *)hist.mutable_data_ptr() : nullptr, ws.mutable_data_ptr(), ws.nbytes(),
                               mail.mutable_data_ptr(), box.host, token, stream);
        if (rc == ADACODE_OK) {
            what = "adacode_wait_report";
            rc = adacode_wait_report(box.host, sizeof(got), token, got, stream);
        }
    }
    check(rc, what);
    const Owned o_sm(THPVariable_Wrap(sm)), o_cd(THPVariable_Wrap(cd)), o_esc(THPVariable_Wrap(esc)), o_base(THPVariable_Wrap(base)),
        total(PyLong_FromLongLong(got[1])), status(PyLong_FromUnsignedLong((uint32_t)got[2]));
    return PyTuple_Pack(6, o_sm.p, o_cd.p, o_esc.p, o_base.p, total.p, status.p);
    END_HANDLE_TH_ERRORS
}

// Whether torch functions are plain calls here: no __torch_function__ of a subclass or of a mode is to see them.
bool plain(PyObject *o) { return THPVariable_CheckExact(o) && !at::impl::torch_function_mode_enabled(); }

// append(buffer, at, states) -> whether `buffer[:, :, at: at + states.shape[2]].copy_(states)` was done here
PyObject *append(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n_args == 3, "append: arguments");
    if (!plain(args[0]) || !plain(args[2])) Py_RETURN_FALSE;
    const Tensor &buf = THPVariable_Unpack(args[0]), &states = THPVariable_Unpack(args[2]);
    const int64_t at = integer(args[1]);
    if (buf.dim() != 4 || states.dim() != 4 || at < 0 || at + states.size(2) > buf.size(2)) Py_RETURN_FALSE;
    {
        pybind11::gil_scoped_release no_gil;
        buf.slice(2, at, at + states.size(2)).copy_(states);
    }
    Py_RETURN_TRUE;
    END_HANDLE_TH_ERRORS
}

// Whether `src`'s rows can be copied behind the segments of `dst` by the unpack launch, i.e. copy_ would do no more than
// move bytes (the conditions of rows.row_record; both are plain bf16 [B, H, T, D] here).
bool plain_rows(const Tensor &src, const Tensor &dst) {
    if (src.scalar_type() != at::kBFloat16 || !src.is_cuda() || src.device() != dst.device()) return false;
    constexpr auto wrappers = c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                   c10::DispatchKey::Functionalize, c10::DispatchKey::Python,
                                                   c10::DispatchKey::Conjugate, c10::DispatchKey::Negative});
    if (src.key_set().has_any(wrappers) || dst.key_set().has_any(wrappers)) return false;
    if (torch::autograd::ForwardADLevel::try_get_by_idx(0)) return false;
    if (c10::GradMode::is_enabled() && (src.requires_grad() || dst.requires_grad())) return false;
    if (dst.is_inference() && !c10::InferenceMode::is_enabled()) return false;
    return true;
}

// dense_view(parts, prefix, rows) -> (dense, ...) or None
// parts: (workspace, table, n_segments, B, H, seq_tile, D, tail) per tensor.  The segments of `table` are unpacked into the
// front of a [B, H, prefix + rows, D] view of the flat `workspace` and the first `rows` tokens of `tail` copied behind
// them, in one launch for parts of one shape.  None, and nothing done, where that is not all that the calls from
// Python would do, or where they would refuse.
PyObject *dense_view(PyObject *, PyObject *const *args, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    TORCH_CHECK_TYPE(n_args == 4 && PyTuple_Check(args[0]), "dense_view: arguments");
    const int n = (int)PyTuple_GET_SIZE(args[0]);
    const int64_t prefix = integer(args[1]), rows = integer(args[2]);
    const Tensor &status = tensor(args[3]);
    if (n < 1 || n > 4 || prefix <= 0 || rows < 0) Py_RETURN_NONE;
    adacode_unpack_job jobs[4];
    adacode_row_copy copies[4];
    int64_t shape[4][4];
    Tensor dense[4];
    const Tensor *spaces[4], *tails[4];
    // everything is looked at before anything is written
    for (int j = 0; j < n; ++j) {
        PyObject *part = PyTuple_GET_ITEM(args[0], j);
        TORCH_CHECK_TYPE(PyTuple_Check(part) && PyTuple_GET_SIZE(part) == 8, "dense_view: a part");
        PyObject *space = PyTuple_GET_ITEM(part, 0), *tail = PyTuple_GET_ITEM(part, 7);
        if (!plain(space)) Py_RETURN_NONE;
        spaces[j] = &THPVariable_Unpack(space);
        const Tensor &table = tensor(PyTuple_GET_ITEM(part, 1));
        const int64_t n_seg = integer(PyTuple_GET_ITEM(part, 2));
        for (int i = 0; i < 4; ++i) shape[j][i] = integer(PyTuple_GET_ITEM(part, 3 + i));
        const int64_t B = shape[j][0], H = shape[j][1], T = shape[j][2], D = shape[j][3], total = prefix + rows;
        const Tensor &s = *spaces[j];
        if (s.scalar_type() != at::kBFloat16 || s.dim() != 1 || s.stride(0) != 1 || !s.is_cuda() || s.device() != spaces[0]->device() ||
            table.device() != s.device() || status.device() != s.device() || B <= 0 || H <= 0 || T <= 0 || D <= 0 || D % 8 != 0 || n_seg <= 0 ||
            n_seg * T > prefix || B * H * total * D > s.numel() ||
            table.nbytes() < n_seg * sizeof(adacode_segment) || B * H * total * D >= (1ll << 31))
            Py_RETURN_NONE;
        jobs[j].segments_dev = (const adacode_segment *)table.const_data_ptr();
        jobs[j].n_segments = (int)n_seg, jobs[j].reserved = 0;
        jobs[j].dst_bf16 = const_cast<void *>(s.const_data_ptr());
        jobs[j].dstride_b = H * total * D, jobs[j].dstride_h = total * D, jobs[j].dstride_s = D;
        if (((uintptr_t)jobs[j].dst_bf16 & 15) != 0) Py_RETURN_NONE;
        if (rows == 0) continue;
        if (!plain(tail)) Py_RETURN_NONE;
        const Tensor &t = THPVariable_Unpack(tail);
        tails[j] = &t;
        if (t.dim() != 4 || !plain_rows(t, s) || t.size(0) != B || t.size(1) != H || t.size(2) < rows || t.size(3) != D || t.stride(3) != 1 ||
            ((t.stride(0) | t.stride(1) | t.stride(2)) & 7) != 0)
            Py_RETURN_NONE;
        adacode_row_copy &c = copies[j];
        c.src_bf16 = t.const_data_ptr(), c.dst_bf16 = (uint16_t *)jobs[j].dst_bf16 + prefix * D;
        c.src_b = t.stride(0), c.src_h = t.stride(1), c.src_s = t.stride(2);
        c.dst_b = jobs[j].dstride_b, c.dst_h = jobs[j].dstride_h, c.dst_s = D;
        c.B = (int)B, c.H = (int)H, c.rows = (int)rows, c.D = (int)D;
        if ((((uintptr_t)c.src_bf16 | (uintptr_t)c.dst_bf16) & 15) != 0) Py_RETURN_NONE;
    }
    const c10::Device device = spaces[0]->device();
    const c10::cuda::CUDAGuard on(device);
    void *const stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    for (int j = 0; j < n; ++j) {
        const int64_t *d = shape[j], total = prefix + rows;
        dense[j] = spaces[j]->as_strided({d[0], d[1], total, d[3]}, {d[1] * total * d[3], total * d[3], d[3], 1});
    }
    for (int j = 0; j < n;) {
        int k = j + 1;
        while (k < n && std::equal(shape[k], shape[k] + 4, shape[j])) ++k;
        check(adacode_unpack_jobs_with_rows(jobs + j, k - j, (int)shape[j][0], (int)shape[j][1], (int)shape[j][2], (int)shape[j][3],
                                            rows ? copies + j : nullptr, rows ? k - j : 0, (int32_t *)status.mutable_data_ptr(), stream),
              "adacode_unpack_jobs_with_rows");
        j = k;
    }
    Owned out(PyTuple_New(n));
    if (!out.p) fail();
    for (int j = 0; j < n; ++j) {
        // (autograd has to know that memory that it may have saved was overwritten)
        if (rows) torch::autograd::impl::bump_version(dense[j]);
        PyTuple_SET_ITEM(out.p, j, THPVariable_Wrap(dense[j]));
    }
    return out.release();
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"pack", (PyCFunction)(void (*)(void))pack, METH_FASTCALL, nullptr},
    {"pack_flat", (PyCFunction)(void (*)(void))pack_flat, METH_FASTCALL, nullptr},
    {"append", (PyCFunction)(void (*)(void))append, METH_FASTCALL, nullptr},
    {"dense_view", (PyCFunction)(void (*)(void))dense_view, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "built_for", ADACODE_BUILT_FOR) != 0) Py_CLEAR(m);
    return m;
}
