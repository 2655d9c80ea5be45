// The short way from a torch tensor to a launch: what ops.py does for a call in its plain form, in one C function.
//
// Each function looks at its arguments, allocates the outputs, fills the parameter block of the C ABI and launches. It returns
// what the operator returns (True where that is None), or None for "not taken": arguments in any other form than the plain
// one, anything ops.py would refuse. ops.py then goes its own way, which raises the errors. A launch that failed is not tried
// again: its error is raised here.
// No state is kept here: scratch comes from the calling thread's pool in ops.py.
//
// Why: decode_attention at B=1 took 14.6 us a call on the host (ctypes fields one by one, shape tuples, dictionary look-ups)
// for 5.7 us of GPU work; a paged decode step of two calls 21.9 us for 10.7.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "sca_b200.h"

namespace {

constexpr int64_t kMaxSplits = 64;         // as MAX_SPLITS, DECODE_STEP_TOKENS in ops.py
constexpr int64_t kDecodeStepTokens = 64;

PyObject* g_scratch = nullptr;          // ops._scratch: threading.local with the dict `pool`
PyObject* g_acquire_scratch = nullptr;  // ops.acquire_scratch_fp32
PyObject* g_check = nullptr;            // _lib.check: raises the error of a status code

// ---- arguments ---------------------------------------------------------------------------------------------------------
// A plain CUDA tensor with memory of its own kind; null for anything else (subclasses, transforms' wrappers, sparse, ...).
const at::Tensor* Plain(PyObject* obj) {
    if (!THPVariable_CheckExact(obj)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(obj);
    if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage()) return nullptr;
    const c10::DispatchKeySet wrappers({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                        c10::DispatchKey::Functionalize, c10::DispatchKey::ZeroTensor});
    return t.key_set().has_any(wrappers) ? nullptr : &t;
}
bool DtypeId(const at::Tensor& t, int32_t* id) {
    switch (t.scalar_type()) {
        case at::kFloat: *id = SCA_DTYPE_F32; return true;
        case at::kHalf: *id = SCA_DTYPE_F16; return true;
        case at::kBFloat16: *id = SCA_DTYPE_BF16; return true;
        default: return false;
    }
}
bool Flag(PyObject* obj, bool* value) {
    *value = obj == Py_True;
    return obj == Py_True || obj == Py_False;
}
// cfg.scale > 0 wins, otherwise float(1 / sqrt(double(D)))
bool Scale(PyObject* obj, int64_t head_dim, float* scale) {
    if (obj != Py_None) {
        if (!PyFloat_CheckExact(obj)) return false;
        const double v = PyFloat_AS_DOUBLE(obj);
        if (v > 0) {
            *scale = static_cast<float>(v);
            return true;
        }
    }
    *scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(head_dim)));
    return true;
}
bool Int(PyObject* obj, int64_t* value) {
    if (!PyLong_CheckExact(obj)) return false;
    int overflow = 0;
    *value = PyLong_AsLongLongAndOverflow(obj, &overflow);
    return overflow == 0;
}
// A device list of at least `count` int32 entries.
bool Ints(const at::Tensor& t, int64_t count) { return t.scalar_type() == at::kInt && t.is_contiguous() && t.numel() >= count; }
// A page table of at least `rows` rows.
bool Table(const at::Tensor& t, int64_t rows) { return t.scalar_type() == at::kInt && t.dim() == 2 && t.size(0) >= rows && t.is_contiguous(); }
bool SameType(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
    return q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type();
}
// An int32 array on the host (numpy), one-dimensional and contiguous.
class HostInts {
public:
    ~HostInts() {
        if (held_) PyBuffer_Release(&view_);
    }
    bool Take(PyObject* obj) {
        if (THPVariable_Check(obj) || !PyObject_CheckBuffer(obj)) return false;
        if (PyObject_GetBuffer(obj, &view_, PyBUF_FORMAT | PyBUF_C_CONTIGUOUS) != 0) {
            PyErr_Clear();
            return false;
        }
        held_ = true;
        return view_.ndim == 1 && view_.itemsize == 4 && view_.format != nullptr && view_.format[0] == 'i' && view_.format[1] == '\0';
    }
    const int32_t* data() const { return static_cast<const int32_t*>(view_.buf); }
    int64_t size() const { return view_.shape[0]; }

private:
    Py_buffer view_{};
    bool held_ = false;
};

// ---- launches ------------------------------------------------------------------------------------------------------------
void* CurrentStream() { return c10::cuda::getCurrentCUDAStream().stream(); }
PyObject* NotTaken() { Py_RETURN_NONE; }
PyObject* Done() { Py_RETURN_TRUE; }
at::Tensor Empty(at::IntArrayRef shape, const at::Tensor& like, at::ScalarType type) {
    return at::empty(shape, at::TensorOptions().dtype(type).device(like.device()));
}
// Other threads run while a launch waits for room in the stream's queue.
class OtherThreadsRun {
public:
    OtherThreadsRun() : state_(PyEval_SaveThread()) {}
    ~OtherThreadsRun() { PyEval_RestoreThread(state_); }  // also when the launch throws
    OtherThreadsRun(const OtherThreadsRun&) = delete;
    OtherThreadsRun& operator=(const OtherThreadsRun&) = delete;

private:
    PyThreadState* state_;
};
template <typename F>
int Launch(const F& f) {
    OtherThreadsRun here;
    return f();
}
// What a launch that did not return SCA_OK comes to. A refusal leaves nothing behind, so the general path may meet it again and
// say what it is. Anything else has been told once: the last error and the word of a prefill that gave up have been read, and
// a second launch that succeeds would hide them.
PyObject* NotLaunched(int rc) {
    if (rc == SCA_INVALID_ARGUMENT || rc == SCA_NOT_IMPLEMENTED) return NotTaken();
    PyObject* none = PyObject_CallFunction(g_check, "i", rc);
    if (none != nullptr) {
        Py_DECREF(none);
        PyErr_Format(PyExc_RuntimeError, "a launch failed with status %d", rc);
    }
    return nullptr;
}
// Nothing else that goes wrong here is an error of its own: the general path meets it again.
template <typename F>
PyObject* Guarded(const F& f) {
    try {
        return f();
    } catch (const std::exception&) {
        PyErr_Clear();
        return NotTaken();
    }
}

// fp32 scratch of this thread on the current stream, as ops.acquire_scratch_fp32 keeps it; null with no error set: not taken.
float* Scratch(int64_t elements, const at::Tensor& like, void* stream, PyObject* device) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const bool plain = cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    if (!plain) return nullptr;
    PyObject* pool = PyObject_GetAttrString(g_scratch, "pool");
    if (pool == nullptr) throw std::runtime_error("scratch pool");
    PyObject* key = Py_BuildValue("(iiK)", static_cast<int>(like.device().index()), 1, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)));
    PyObject* found = key != nullptr ? PyDict_GetItemWithError(pool, key) : nullptr;  // borrowed
    float* data = nullptr;
    if (found != nullptr && THPVariable_CheckExact(found) && THPVariable_Unpack(found).numel() >= elements) {
        data = static_cast<float*>(THPVariable_Unpack(found).data_ptr());
    }
    Py_XDECREF(key);
    Py_DECREF(pool);
    if (data != nullptr) return data;
    PyErr_Clear();
    PyObject* made = PyObject_CallFunction(g_acquire_scratch, "LO", static_cast<long long>(elements), device);
    if (made == nullptr) throw std::runtime_error("scratch");
    data = static_cast<float*>(THPVariable_Unpack(made).data_ptr());  // the pool keeps it
    Py_DECREF(made);
    return data;
}

// flash(q, k, v, causal, scale, return_lse, layout, simt)
PyObject* Flash(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 8) return NotTaken();
        const at::Tensor *q = Plain(a[0]), *k = Plain(a[1]), *v = Plain(a[2]);
        bool causal, want_lse, simt, bshd;
        ScaFlashFwdParams p{};
        if (!q || !k || !v || !Flag(a[3], &causal) || !Flag(a[5], &want_lse) || !Flag(a[7], &simt) || !PyUnicode_Check(a[6])) return NotTaken();
        bshd = PyUnicode_CompareWithASCIIString(a[6], "bshd") == 0;
        if (!bshd && PyUnicode_CompareWithASCIIString(a[6], "bhsd") != 0) return NotTaken();
        if (q->dim() != 4 || k->dim() != 4 || !q->is_contiguous() || !k->is_contiguous() || !v->is_contiguous() ||
            k->sizes() != v->sizes() || !SameType(*q, *k, *v) || !DtypeId(*q, &p.dtype_id) ||
            (!simt && p.dtype_id == SCA_DTYPE_F32)) {
            return NotTaken();
        }
        const int head = bshd ? 2 : 1, seq = bshd ? 1 : 2;
        p.batch = q->size(0), p.num_heads = q->size(head), p.seq_q = q->size(seq), p.head_dim = q->size(3);
        p.num_kv_heads = k->size(head), p.seq_kv = k->size(seq);
        if (k->size(0) != p.batch || k->size(3) != p.head_dim || (causal && p.seq_kv < p.seq_q) || !Scale(a[4], p.head_dim, &p.scale)) return NotTaken();
        const int64_t d = p.head_dim;
        p.q_sb = p.num_heads * p.seq_q * d, p.q_sh = bshd ? d : p.seq_q * d, p.q_ss = bshd ? p.num_heads * d : d;
        p.k_sb = p.num_kv_heads * p.seq_kv * d, p.k_sh = bshd ? d : p.seq_kv * d, p.k_ss = bshd ? p.num_kv_heads * d : d;
        p.v_sb = p.k_sb, p.v_sh = p.k_sh, p.v_ss = p.k_ss;
        p.o_sb = p.num_heads * p.seq_q * d, p.o_sh = p.seq_q * d, p.o_ss = d;
        p.causal = causal, p.return_lse = want_lse, p.diagonal = causal ? p.seq_kv - p.seq_q : 0;
        at::Tensor out = Empty({p.batch, p.num_heads, p.seq_q, d}, *q, q->scalar_type()), lse;
        if (want_lse) lse = Empty({p.batch, p.num_heads, p.seq_q}, *q, at::kFloat);
        p.q = q->data_ptr(), p.k = k->data_ptr(), p.v = v->data_ptr(), p.out = out.data_ptr();
        p.lse = want_lse ? static_cast<float*>(lse.data_ptr()) : nullptr;
        void* stream = CurrentStream();
        if (const int rc = Launch([&] { return simt ? sca_launch_simt_forward(&p, stream) : sca_launch_flash_fwd(&p, stream); })) return NotLaunched(rc);
        if (!want_lse) return THPVariable_Wrap(std::move(out));
        return Py_BuildValue("(NN)", THPVariable_Wrap(std::move(out)), THPVariable_Wrap(std::move(lse)));
    });
}

// Partial slots per row, as slots_for_schedule in ops.py.
int64_t SlotsForSchedule(int64_t column_steps, int64_t longest_steps, int64_t columns, int64_t sms) {
    if (column_steps <= 0 || longest_steps <= 1) return 1;
    const int64_t sharers = std::max<int64_t>(1, 2 * sms / std::max<int64_t>(1, columns));
    const int64_t per_cta = std::max<int64_t>(1, (column_steps + sharers - 1) / sharers);
    return std::max<int64_t>(2, std::min((longest_steps + per_cta - 1) / per_cta + 1, kMaxSplits));
}
int64_t Steps(int64_t tokens) { return (tokens + kDecodeStepTokens - 1) / kDecodeStepTokens; }

// The rest of a decode call whose inputs and strides are in `p`: scratch, output, launch.
PyObject* FinishDecode(ScaDecodeFwdParams& p, const at::Tensor& q, PyObject* q_obj) {
    void* stream = CurrentStream();
    const int64_t base = p.batch * p.num_heads * p.num_splits, d = p.head_dim;
    PyObject* device = PyObject_GetAttrString(q_obj, "device");
    if (device == nullptr) throw std::runtime_error("device");
    float* scratch = nullptr;
    try {
        scratch = Scratch(base * (2 + d), q, stream, device);
    } catch (...) {
        Py_DECREF(device);
        throw;
    }
    Py_DECREF(device);
    if (scratch == nullptr) return NotTaken();
    at::Tensor out = Empty({p.batch, p.num_heads, 1, d}, q, q.scalar_type());
    p.out = out.data_ptr();
    p.partial_m = scratch, p.partial_l = scratch + base, p.partial_o = scratch + 2 * base;
    if (const int rc = Launch([&] { return sca_launch_decode_auto(&p, nullptr, stream); })) return NotLaunched(rc);
    return THPVariable_Wrap(std::move(out));
}

// decode(q, k, v, scale, layout, seq_lens)
PyObject* Decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 6) return NotTaken();
        const at::Tensor *q = Plain(a[0]), *k = Plain(a[1]), *v = Plain(a[2]), *lens = nullptr;
        if (!q || !k || !v || !PyUnicode_Check(a[4])) return NotTaken();
        if (a[5] != Py_None && (lens = Plain(a[5])) == nullptr) return NotTaken();
        const bool bshd = PyUnicode_CompareWithASCIIString(a[4], "bshd") == 0;
        if (!bshd && PyUnicode_CompareWithASCIIString(a[4], "bhsd") != 0) return NotTaken();
        ScaDecodeFwdParams p{};
        if (q->dim() != 4 || k->dim() != 4 || !q->is_contiguous() || !k->is_contiguous() || !v->is_contiguous() ||
            k->sizes() != v->sizes() || !SameType(*q, *k, *v) || !DtypeId(*q, &p.dtype)) {
            return NotTaken();
        }
        const int head = bshd ? 2 : 1, seq = bshd ? 1 : 2;
        p.batch = q->size(0), p.num_heads = q->size(head), p.head_dim = q->size(3), p.num_kv_heads = k->size(head), p.seq_kv = k->size(seq);
        const int64_t d = p.head_dim;
        if (q->size(seq) != 1 || k->size(0) != p.batch || k->size(3) != d || p.num_kv_heads < 1 || p.num_heads % p.num_kv_heads != 0 ||
            (lens != nullptr && !Ints(*lens, p.batch)) || !Scale(a[3], d, &p.scale)) {
            return NotTaken();
        }
        const int64_t group = p.num_heads / p.num_kv_heads, steps = Steps(p.seq_kv);
        const int64_t sms = at::cuda::getDeviceProperties(q->device().index())->multiProcessorCount;
        p.num_splits = p.seq_kv <= 0 ? 1 : SlotsForSchedule(std::max<int64_t>(1, p.batch) * steps, steps, p.num_kv_heads * ((group + 15) / 16), sms);
        p.q = q->data_ptr(), p.k = k->data_ptr(), p.v = v->data_ptr();
        p.q_stride = bshd ? ScaDecodeStrides{p.num_heads * d, d, p.num_heads * d} : ScaDecodeStrides{p.num_heads * d, d, d};
        p.k_stride = bshd ? ScaDecodeStrides{p.seq_kv * p.num_kv_heads * d, d, p.num_kv_heads * d}
                          : ScaDecodeStrides{p.num_kv_heads * p.seq_kv * d, p.seq_kv * d, d};
        p.v_stride = p.k_stride;
        p.o_stride = ScaDecodeStrides{p.num_heads * d, d, d};
        p.seq_lens = lens != nullptr ? static_cast<const int32_t*>(lens->data_ptr()) : nullptr;
        return FinishDecode(p, *q, a[0]);
    });
}

// paged(q, k_pool, v_pool, page_table, seq_lens, block_size, scale, typical_len, longest_len)
PyObject* Paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 9) return NotTaken();
        const at::Tensor *q = Plain(a[0]), *k = Plain(a[1]), *v = Plain(a[2]), *table = Plain(a[3]), *lens = nullptr;
        int64_t block_size, typical, longest;
        ScaDecodeFwdParams p{};
        if (!q || !k || !v || !table || !Int(a[5], &block_size) || !Int(a[7], &typical) || !Int(a[8], &longest)) return NotTaken();
        if (a[4] != Py_None && (lens = Plain(a[4])) == nullptr) return NotTaken();
        if (q->dim() != 4 || q->size(2) != 1 || k->dim() != 4 || k->size(1) != block_size || k->size(3) != q->size(3) || k->sizes() != v->sizes() ||
            !q->is_contiguous() || !k->is_contiguous() || !v->is_contiguous() || !SameType(*q, *k, *v) || !Table(*table, q->size(0)) ||
            (lens != nullptr && !Ints(*lens, q->size(0))) || !DtypeId(*q, &p.dtype)) {
            return NotTaken();
        }
        p.batch = q->size(0), p.num_heads = q->size(1), p.head_dim = q->size(3), p.num_kv_heads = k->size(2);
        const int64_t d = p.head_dim, blocks = k->size(0);
        if (p.num_kv_heads < 1 || !Scale(a[6], d, &p.scale)) return NotTaken();
        p.seq_kv = blocks * block_size;
        const int64_t mean = typical > 0 ? typical : std::min(p.seq_kv, table->size(1) * block_size), steps = Steps(mean);
        const int64_t most = longest > 0 ? Steps(longest) : 2 * steps, group = p.num_heads / p.num_kv_heads;
        const int64_t sms = at::cuda::getDeviceProperties(q->device().index())->multiProcessorCount;
        p.num_splits = mean <= 0 ? 1 : SlotsForSchedule(std::max<int64_t>(1, p.batch) * steps, most, p.num_kv_heads * ((group + 15) / 16), sms);
        p.q = q->data_ptr(), p.k = k->data_ptr(), p.v = v->data_ptr();
        p.q_stride = ScaDecodeStrides{p.num_heads * d, d, d};
        p.o_stride = p.q_stride;
        p.k_stride = ScaDecodeStrides{0, d, p.num_kv_heads * d};  // row = one token of the pool
        p.v_stride = p.k_stride;
        p.seq_lens = lens != nullptr ? static_cast<const int32_t*>(lens->data_ptr()) : nullptr;
        p.page_table = static_cast<const int32_t*>(table->data_ptr());
        if (p.page_table == nullptr) return NotTaken();
        p.block_size = block_size, p.max_blocks_per_seq = table->size(1), p.num_kv_blocks = blocks;
        return FinishDecode(p, *q, a[0]);
    });
}

// ---- packed prefill ------------------------------------------------------------------------------------------------------
at::Tensor VarlenWorkspace(int64_t seqs, int64_t tokens, const at::Tensor& like) {
    return Empty({std::max<int64_t>(sca_flash_varlen_workspace_bytes(seqs, tokens), 16)}, like, at::kByte);
}

// varlen(q, k, v, cu_q, cu_kv, causal, scale)
PyObject* Varlen(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 7) return NotTaken();
        const at::Tensor *q = Plain(a[0]), *k = Plain(a[1]), *v = Plain(a[2]);
        HostInts cu_q, cu_kv;
        bool causal;
        ScaFlashVarlenParams p{};
        if (!q || !k || !v || !cu_q.Take(a[3]) || !cu_kv.Take(a[4]) || !Flag(a[5], &causal) || !DtypeId(*q, &p.dtype_id)) return NotTaken();
        if (q->dim() != 3 || k->dim() != 3 || k->size(2) != q->size(2) || k->sizes() != v->sizes() || !SameType(*q, *k, *v) || !q->is_contiguous() || !k->is_contiguous() || !v->is_contiguous() ||
            cu_q.size() != cu_kv.size() || cu_q.size() < 2 || !Scale(a[6], q->size(2), &p.scale)) {
            return NotTaken();
        }
        p.total_q = q->size(0), p.num_heads = q->size(1), p.head_dim = q->size(2), p.total_kv = k->size(0), p.num_kv_heads = k->size(1);
        p.num_seqs = cu_q.size() - 1;
        at::Tensor out = Empty(q->sizes(), *q, q->scalar_type()), ws = VarlenWorkspace(p.num_seqs, p.total_q, *q);
        p.q = q->data_ptr(), p.k = k->data_ptr(), p.v = v->data_ptr(), p.out = out.data_ptr();
        p.cu_seqlens_q = cu_q.data(), p.cu_seqlens_kv = cu_kv.data(), p.causal = causal;
        p.workspace = ws.data_ptr(), p.workspace_bytes = ws.numel();
        void* stream = CurrentStream();
        if (const int rc = Launch([&] { return sca_launch_flash_varlen(&p, stream); })) return NotLaunched(rc);
        return THPVariable_Wrap(std::move(out));
    });
}

// chunk(q, k_pool, v_pool, page_table, cu_q, seq_lens, causal, scale)
PyObject* Chunk(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 8) return NotTaken();
        const at::Tensor *q = Plain(a[0]), *k = Plain(a[1]), *v = Plain(a[2]), *table = Plain(a[3]);
        HostInts cu_q, lens;
        bool causal;
        ScaFlashPagedParams p{};
        if (!q || !k || !v || !table || !cu_q.Take(a[4]) || !lens.Take(a[5]) || !Flag(a[6], &causal) || !DtypeId(*q, &p.dtype_id)) return NotTaken();
        if (q->dim() != 3 || k->dim() != 4 || k->sizes() != v->sizes() || !SameType(*q, *k, *v) || !q->is_contiguous() || !k->is_contiguous() ||
            !v->is_contiguous() || !Table(*table, lens.size()) || cu_q.size() != lens.size() + 1 || k->size(3) != q->size(2) || !Scale(a[7], q->size(2), &p.scale)) {
            return NotTaken();
        }
        p.total_q = q->size(0), p.num_heads = q->size(1), p.head_dim = q->size(2), p.num_seqs = lens.size();
        p.num_blocks = k->size(0), p.block_size = k->size(1), p.num_kv_heads = k->size(2), p.max_blocks_per_seq = table->size(1);
        at::Tensor out = Empty(q->sizes(), *q, q->scalar_type()), ws = VarlenWorkspace(p.num_seqs, p.total_q, *q);
        p.q = q->data_ptr(), p.out = out.data_ptr(), p.k_pool = k->data_ptr(), p.v_pool = v->data_ptr();
        p.page_table = static_cast<const int32_t*>(table->data_ptr());
        p.cu_seqlens_q = cu_q.data(), p.seq_lens_kv = lens.data(), p.causal = causal;
        p.workspace = ws.data_ptr(), p.workspace_bytes = ws.numel();
        void* stream = CurrentStream();
        if (const int rc = Launch([&] { return sca_launch_flash_paged(&p, stream); })) return NotLaunched(rc);
        return THPVariable_Wrap(std::move(out));
    });
}

// ---- KV cache ------------------------------------------------------------------------------------------------------------
bool PoolShape(const at::Tensor& pool, ScaKvCacheShape* s) {
    if (pool.dim() != 4 || !pool.is_contiguous()) return false;
    *s = ScaKvCacheShape{pool.size(0), pool.size(1), pool.size(2), pool.size(3)};
    return true;
}
// As _same_kind, _require_pools and _require_rows in ops.py.
bool SameKind(const at::Tensor& a, const at::Tensor& b) {
    return a.scalar_type() == b.scalar_type() || (a.element_size() == b.element_size() && !(a.is_floating_point() && b.is_floating_point()));
}
bool Pools(const at::Tensor& k, const at::Tensor& v, ScaKvCacheShape* s) {
    return PoolShape(k, s) && v.dim() == 4 && v.is_contiguous() && v.sizes().slice(1) == k.sizes().slice(1) && v.size(0) >= k.size(0) && SameKind(v, k);
}
bool Rows(const at::Tensor& t, int64_t rows, const at::Tensor& pool) {
    return t.is_contiguous() && t.size(0) >= rows && t.numel() == t.size(0) * pool.size(2) * pool.size(3) && SameKind(t, pool);
}
// New K / V of `kn`'s rows for the pools.
bool NewRows(const at::Tensor& k, const at::Tensor& v, const at::Tensor& kn, const at::Tensor& vn, ScaKvCacheShape* s) {
    return Pools(k, v, s) && kn.dim() >= 1 && vn.dim() >= 1 && Rows(kn, kn.size(0), k) && Rows(vn, kn.size(0), k);
}

// append(k_pool, v_pool, k_new, v_new, slots)
PyObject* Append(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 5) return NotTaken();
        const at::Tensor *k = Plain(a[0]), *v = Plain(a[1]), *kn = Plain(a[2]), *vn = Plain(a[3]), *slots = Plain(a[4]);
        ScaKvCacheShape shape;
        if (!k || !v || !kn || !vn || !slots || !NewRows(*k, *v, *kn, *vn, &shape) || !Ints(*slots, kn->size(0))) return NotTaken();
        void* stream = CurrentStream();
        const int rc = Launch([&] {
            return sca_launch_kv_append(k->data_ptr(), v->data_ptr(), kn->data_ptr(), vn->data_ptr(), static_cast<const int32_t*>(slots->data_ptr()),
                                        kn->size(0), &shape, k->element_size(), stream);
        });
        return rc == SCA_OK ? Done() : NotLaunched(rc);
    });
}

// append_batched(k_pool, v_pool, k_new, v_new, page_table, seq_lens)
PyObject* AppendBatched(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 6) return NotTaken();
        const at::Tensor *k = Plain(a[0]), *v = Plain(a[1]), *kn = Plain(a[2]), *vn = Plain(a[3]), *table = Plain(a[4]), *lens = Plain(a[5]);
        ScaKvCacheShape shape;
        if (!k || !v || !kn || !vn || !table || !lens || !NewRows(*k, *v, *kn, *vn, &shape) || !Table(*table, kn->size(0)) ||
            !Ints(*lens, kn->size(0))) {
            return NotTaken();
        }
        void* stream = CurrentStream();
        const int rc = Launch([&] {
            return sca_launch_kv_append_batched(k->data_ptr(), v->data_ptr(), kn->data_ptr(), vn->data_ptr(), static_cast<const int32_t*>(table->data_ptr()),
                                                static_cast<const int32_t*>(lens->data_ptr()), kn->size(0), table->size(1), &shape,
                                                k->element_size(), stream);
        });
        return rc == SCA_OK ? Done() : NotLaunched(rc);
    });
}

// reset(k_pool, v_pool, block_ids)
PyObject* Reset(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 3) return NotTaken();
        const at::Tensor *k = Plain(a[0]), *v = Plain(a[1]), *ids = Plain(a[2]);
        ScaKvCacheShape shape;
        if (!k || !v || !ids || !Pools(*k, *v, &shape) || !Ints(*ids, 0)) return NotTaken();
        void* stream = CurrentStream();
        const int rc = Launch([&] {
            return sca_launch_kv_reset_block(k->data_ptr(), v->data_ptr(), static_cast<const int32_t*>(ids->data_ptr()), ids->numel(), &shape,
                                             k->element_size(), stream);
        });
        return rc == SCA_OK ? Done() : NotLaunched(rc);
    });
}

// gather(pool, block_ids)
PyObject* Gather(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return Guarded([&]() -> PyObject* {
        if (n != 2) return NotTaken();
        const at::Tensor *pool = Plain(a[0]), *ids = Plain(a[1]);
        ScaKvCacheShape shape;
        if (!pool || !ids || !PoolShape(*pool, &shape) || !Ints(*ids, 0)) return NotTaken();
        at::Tensor out = Empty({ids->numel(), pool->size(1), pool->size(2), pool->size(3)}, *pool, pool->scalar_type());
        void* stream = CurrentStream();
        const int rc = Launch([&] {
            return sca_launch_kv_gather(pool->data_ptr(), static_cast<const int32_t*>(ids->data_ptr()), ids->numel(), out.data_ptr(), &shape,
                                        pool->element_size(), stream);
        });
        return rc == SCA_OK ? THPVariable_Wrap(std::move(out)) : NotLaunched(rc);
    });
}

// init(scratch_local, acquire_scratch, check)
PyObject* Init(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 3) {
        PyErr_SetString(PyExc_TypeError, "init(scratch_local, acquire_scratch, check)");
        return nullptr;
    }
    Py_XSETREF(g_scratch, Py_NewRef(a[0]));
    Py_XSETREF(g_acquire_scratch, Py_NewRef(a[1]));
    Py_XSETREF(g_check, Py_NewRef(a[2]));
    Py_RETURN_NONE;
}

// slots(column_steps, longest_steps, columns, sms): the slot rule, so that a test can hold it against ops.py's
PyObject* Slots(PyObject*, PyObject* const* a, Py_ssize_t n) {
    int64_t v[4];
    for (Py_ssize_t i = 0; i < 4; ++i) {
        if (n != 4 || !Int(a[i], &v[i])) {
            PyErr_SetString(PyExc_TypeError, "slots(column_steps, longest_steps, columns, sms)");
            return nullptr;
        }
    }
    return PyLong_FromLongLong(SlotsForSchedule(v[0], v[1], v[2], v[3]));
}

#define SCA_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {SCA_METHOD("init", Init), SCA_METHOD("flash", Flash), SCA_METHOD("decode", Decode), SCA_METHOD("paged", Paged),
                           SCA_METHOD("varlen", Varlen), SCA_METHOD("chunk", Chunk), SCA_METHOD("append", Append),
                           SCA_METHOD("append_batched", AppendBatched), SCA_METHOD("reset", Reset), SCA_METHOD("gather", Gather),
                           SCA_METHOD("slots", Slots), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Plain operator calls without the Python in between.", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    PyObject* module = PyModule_Create(&g_module);
    if (module != nullptr && PyModule_AddStringConstant(module, "built_with", SCA_BUILT_WITH) != 0) Py_CLEAR(module);
    return module;
}
