// The host side of a chunk's decode and encode calls, on torch's tensors: what stands between a Python call and the launches.
//
// A 37-token chunk keeps the GPU busy for 14 us; reading its tensors' shapes and addresses, making the result and filling in
// the job descriptors took 33 us of Python.  Here it takes 10 with the launches.  The decode looks at its chunks and does the
// usual case (plain contiguous tensors on the current GPU, everything of the right shape and type); whatever is different
// in any way, malformed chunks included, it leaves to the caller, whose general path decodes it or says what is wrong.
// An encode's buffers are made, its job is filled in and its kernels are launched in one call, and in another its sizes are waited
// for, its payload is made and gathered, with nothing in between that the GPU would have to wait for.
//
// The library's entries come as addresses from the binding (bind), so that one copy of the library is in use.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <vector>

#include "../../include/cachegen_b200.h"

namespace {

decltype(&cg_decode_kv) decode_kv;
decltype(&cg_encode_kv) encode_kv;
decltype(&cg_encode_kv_workspace) encode_kv_workspace;
decltype(&cg_encode_kv_wait) encode_kv_wait;
decltype(&cg_encode_kv_gather) encode_kv_gather;

// attribute names
PyObject *s_cdf, *s_max_tensors_key, *s_max_tensors_value, *s_data_chunks, *s_num_heads, *s_head_size, *s_bytestream,
    *s_bytestream_lengths, *s_ntokens, *s_blob, *s_header, *s_sub_off, *s_group_off, *s_captured;
const char *const kHeaderNames[] = {"L", "H", "D", "T", "lp", "nsub", "scale_code", "table_kind", "length_kind", "bins_checksum",
                                    "off_scales", "off_tables", "off_lengths", "off_payload"};
enum HeaderField {
    kL, kH, kD, kT, kLp, kNsub, kScaleCode, kTableKind, kLengthKind, kChecksum, kOffScales, kOffTables, kOffLengths, kOffPayload, kHeaderFields
};
PyObject *s_header_fields[kHeaderFields];

// A new reference that is given back.
struct Ref {
    PyObject *p;
    explicit Ref(PyObject *o) : p(o) {}
    ~Ref() { Py_XDECREF(p); }
    Ref(const Ref &) = delete;
    Ref &operator=(const Ref &) = delete;
};

// Released while the library works, as ctypes does, and while torch's allocator may wait, as torch does.
struct WithoutGil {
    PyThreadState *s = PyEval_SaveThread();
    ~WithoutGil() { PyEval_RestoreThread(s); }
};

at::Tensor make(at::IntArrayRef shape, at::TensorOptions options) {
    const WithoutGil released;
    return at::empty(shape, options);
}

bool plain(PyObject *o) { return o && THPVariable_CheckExact(o); }

// A plain contiguous tensor of this type on this GPU: the only kind that is taken as it is.
bool usable(const at::Tensor &t, at::ScalarType type, at::Device dev) {
    return t.defined() && t.unsafeGetTensorImpl()->has_storage() && t.layout() == at::kStrided && t.scalar_type() == type &&
           t.device() == dev && t.is_contiguous() && !t.is_conj() && !t.is_neg();
}

bool small_int(PyObject *o, int64_t *v) {
    if (!o || !PyLong_CheckExact(o)) return false;
    *v = PyLong_AsLongLong(o);
    if (*v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

bool attribute_int(PyObject *o, PyObject *name, int64_t *v) {
    const Ref a(PyObject_GetAttr(o, name));
    if (!a.p) PyErr_Clear();
    return small_int(a.p, v);
}

// The tensor under a name, alive as long as the object that has it: nobody else can run between here and the launch but
// while the library works, and then `held` keeps it.
bool attribute_tensor(PyObject *o, PyObject *name, std::vector<at::Tensor> *held) {
    const Ref a(PyObject_GetAttr(o, name));
    if (!a.p) PyErr_Clear();
    if (!plain(a.p)) return false;
    held->push_back(THPVariable_Unpack(a.p));
    return true;
}

struct Shape {
    int64_t L = 0, H = 0, D = 0, lp = 0, T = 0;
    at::ScalarType scale = at::kHalf;
};

bool is_16bit(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }
int code(at::ScalarType t) { return t == at::kBFloat16 ? CG_BF16 : CG_F16; }

// Whether this chunk is of the shape of those before it; adds its tokens to theirs.
bool merge(const Shape &s, Shape *all, bool first) {
    if (!first && (s.L != all->L || s.H != all->H || s.D != all->D || s.lp != all->lp || s.scale != all->scale)) return false;
    const int64_t before = first ? 0 : all->T;
    *all = s;
    all->T = before + s.T;
    return true;
}

// One chunk's jobs, without what depends on the output.  false: not the usual case.
bool add_chunk(PyObject *eo, PyTypeObject *piece_type, at::Device dev, Shape *all, bool first, std::vector<cg_decode_job> *jobs,
               std::vector<at::Tensor> *held) {
    Shape s;
    if (!attribute_int(eo, s_num_heads, &s.H) || !attribute_int(eo, s_head_size, &s.D)) return false;
    if (s.H <= 0 || s.D <= 0 || s.H > 0xFFFFFF || s.D > 0xFFFFFF) return false;
    const size_t at = held->size();
    if (!attribute_tensor(eo, s_cdf, held) || !attribute_tensor(eo, s_max_tensors_key, held) || !attribute_tensor(eo, s_max_tensors_value, held))
        return false;
    // (by value: the vector grows)
    const at::Tensor cdf = (*held)[at], mk = (*held)[at + 1], mv = (*held)[at + 2];
    if (!usable(cdf, at::kShort, dev) || cdf.dim() != 3 || cdf.size(0) % 2 || cdf.size(1) != s.H * s.D) return false;
    s.L = cdf.size(0) / 2;
    s.lp = cdf.size(2);
    s.scale = mk.scalar_type();
    if (!is_16bit(s.scale) || !usable(mk, s.scale, dev) || !usable(mv, s.scale, dev) || mk.dim() < 2 || mv.dim() < 2) return false;
    s.T = mk.size(1);
    if (s.L <= 0 || s.T <= 0 || s.T > 0x7FFFFFFF || mk.size(0) != s.L || mv.size(0) != s.L || mv.size(1) != s.T || mk.numel() != s.L * s.T ||
        mv.numel() != s.L * s.T)
        return false;
    if (!merge(s, all, first)) return false;
    const Ref pieces(PyObject_GetAttr(eo, s_data_chunks));
    if (!pieces.p) PyErr_Clear();
    if (!pieces.p || !PyList_CheckExact(pieces.p)) return false;
    const int64_t streams = 2 * s.L * s.H * s.D;
    int64_t tokens = 0;
    for (Py_ssize_t k = 0; k < PyList_GET_SIZE(pieces.p); ++k) {
        PyObject *piece = PyList_GET_ITEM(pieces.p, k);
        int64_t n;
        if (Py_TYPE(piece) != piece_type || !attribute_int(piece, s_ntokens, &n) || n <= 0 || n > CG_MAX_TOKENS_PER_STREAM) return false;
        if (!attribute_tensor(piece, s_bytestream, held) || !attribute_tensor(piece, s_bytestream_lengths, held)) return false;
        const at::Tensor &bytes = (*held)[held->size() - 2], &lengths = held->back();
        if (!usable(bytes, at::kByte, dev) || bytes.dim() != 1 || !usable(lengths, at::kInt, dev) || lengths.numel() != streams) return false;
        cg_decode_job j{};
        j.tables = cdf.data_ptr();
        j.bytes = static_cast<const uint8_t *>(bytes.data_ptr());
        j.lengths = lengths.data_ptr();
        j.scales_k = static_cast<const uint16_t *>(mk.data_ptr()) + tokens;
        j.scales_v = static_cast<const uint16_t *>(mv.data_ptr()) + tokens;
        j.nbytes = bytes.numel();
        j.tables_nbytes = 2 * cdf.numel();
        j.ntokens = static_cast<int32_t>(n);
        j.scale_stride = static_cast<int32_t>(s.T);
        j.table_kind = CG_TABLES_CDF;
        j.length_kind = CG_LENGTHS_I32;
        jobs->push_back(j);
        tokens += n;
    }
    return tokens == s.T;
}

// Containers' kind of tables, what the bins of the decode say about them (see _HostBins), and the row offsets of their byte counts
// or masks.
struct FlatBins {
    int64_t kind = 0, checksum = 0, counts_bytes = 0, sparse_bytes = 0;
    at::Tensor row_off;
};

// The same for a container (flat_format.FlatChunk).
bool add_container(PyObject *chunk, at::Device dev, const FlatBins &bins, Shape *all, bool first, std::vector<cg_decode_job> *jobs,
                   std::vector<at::Tensor> *held) {
    if (!attribute_tensor(chunk, s_blob, held)) return false;
    const at::Tensor blob = held->back();
    if (!usable(blob, at::kByte, dev) || blob.dim() != 1) return false;
    const Ref header(PyObject_GetAttr(chunk, s_header));
    if (!header.p) PyErr_Clear();
    if (!header.p) return false;
    int64_t f[kHeaderFields];
    for (int k = 0; k < kHeaderFields; ++k)
        if (!attribute_int(header.p, s_header_fields[k], f + k) || f[k] < 0 || f[k] >= int64_t{1} << 48) return false;
    if (f[kL] < 1 || f[kL] > 0x7FFF || f[kH] < 1 || f[kD] < 1 || f[kH] > 0xFFFFFF || f[kD] > 0xFFFFFF || f[kH] * f[kD] > 0xFFFFFF || f[kT] < 1 ||
        f[kT] > 0x7FFFFFFF || f[kNsub] != (f[kT] + CG_MAX_TOKENS_PER_STREAM - 1) / CG_MAX_TOKENS_PER_STREAM || f[kScaleCode] > 1 || f[kLengthKind] > 1)
        return false;
    Shape s;
    s.L = f[kL];
    s.H = f[kH];
    s.D = f[kD];
    s.lp = f[kLp];
    s.T = f[kT];
    s.scale = f[kScaleCode] ? at::kBFloat16 : at::kHalf;
    if (!merge(s, all, first)) return false;
    if (f[kChecksum] && f[kChecksum] != bins.checksum) return false;
    const int64_t table_bytes = f[kOffLengths] - f[kOffTables];
    if (f[kTableKind] != bins.kind) return false;
    const int64_t least = bins.kind == CG_TABLES_COUNTS   ? bins.counts_bytes
                          : bins.kind == CG_TABLES_SPARSE ? bins.sparse_bytes
                                                          : 4 * s.L * s.H * s.D * s.lp;
    if (bins.kind > CG_TABLES_SPARSE || table_bytes < least) return false;
    if (bins.kind != CG_TABLES_CDF) {
        if (!usable(bins.row_off, at::kLong, dev) || bins.row_off.numel() != 2 * s.L + 1) return false;
        held->push_back(bins.row_off);
    }
    const Ref sub_off(PyObject_GetAttr(header.p, s_sub_off));
    if (!sub_off.p) PyErr_Clear();
    if (!sub_off.p || !PyList_CheckExact(sub_off.p) || PyList_GET_SIZE(sub_off.p) != f[kNsub] + 1) return false;
    uint8_t *const at = static_cast<uint8_t *>(blob.data_ptr());
    const int64_t size = blob.numel(), wide = f[kLengthKind] == CG_LENGTHS_U16 ? 2 : 4, row = 2 * s.L * s.H * s.D * wide;
    const uintptr_t a = reinterpret_cast<uintptr_t>(at);
    if (size < f[kOffLengths] + f[kNsub] * row || size < f[kOffScales] + 4 * s.L * s.T || (a + f[kOffScales]) % 2 || (a + f[kOffLengths]) % wide ||
        (bins.kind == CG_TABLES_CDF && (a + f[kOffTables]) % 2))
        return false;
    for (int64_t k = 0; k < f[kNsub]; ++k) {
        int64_t from, to;
        if (!small_int(PyList_GET_ITEM(sub_off.p, k), &from) || !small_int(PyList_GET_ITEM(sub_off.p, k + 1), &to) || from < 0 || from > to ||
            to > int64_t{1} << 48)
            return false;
        from = std::min(f[kOffPayload] + from, size);
        to = std::min(f[kOffPayload] + to, size);
        const int64_t t0 = k * CG_MAX_TOKENS_PER_STREAM;
        cg_decode_job j{};
        j.tables = at + f[kOffTables];
        j.bytes = at + from;
        j.lengths = at + f[kOffLengths] + k * row;
        j.scales_k = at + f[kOffScales] + 2 * t0;
        j.scales_v = at + f[kOffScales] + 2 * s.L * s.T + 2 * t0;
        j.table_row_off = bins.row_off.defined() ? static_cast<const int64_t *>(bins.row_off.data_ptr()) : nullptr;
        j.nbytes = to - from;
        j.tables_nbytes = table_bytes;
        j.ntokens = static_cast<int32_t>(std::min<int64_t>(CG_MAX_TOKENS_PER_STREAM, s.T - t0));
        j.scale_stride = static_cast<int32_t>(s.T);
        j.table_kind = static_cast<int32_t>(bins.kind);
        j.length_kind = static_cast<int32_t>(f[kLengthKind]);
        jobs->push_back(j);
    }
    return true;
}

// Adds a tensor to the set that a workspace holds for graphs (see _keep_for_graph in cachegen_decoder.py).
bool keep_for_graph(PyObject *workspace, PyObject *tensor) {
    if (tensor == Py_None) return true;
    PyObject *held = PyDict_GetItem(workspace, s_captured);
    if (!held) {
        const Ref made(PySet_New(nullptr));
        if (!made.p || PyDict_SetItem(workspace, s_captured, made.p)) return false;
        held = made.p;
    }
    return PySet_Add(held, tensor) == 0;
}

// decode(chunks, chunk type, piece type or None, bins, vllm, bf16 out, out or None, workspace, status word, of containers
//        (kind of tables, checksum, counts_bytes, sparse_bytes, row offsets or None))
// -> the KV blob, or the library's error code, or None: not the usual case, nothing has been done.
PyObject *decode(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10 || !PyList_CheckExact(a[0]) || !PyType_Check(a[1]) || !PyList_GET_SIZE(a[0])) Py_RETURN_NONE;
    const bool containers = a[2] == Py_None;
    FlatBins flat;
    if (containers) {
        if (!PyTuple_CheckExact(a[9]) || PyTuple_GET_SIZE(a[9]) != 5) Py_RETURN_NONE;
        int64_t *const to[4] = {&flat.kind, &flat.checksum, &flat.counts_bytes, &flat.sparse_bytes};
        for (int k = 0; k < 4; ++k)
            if (!small_int(PyTuple_GET_ITEM(a[9], k), to[k])) Py_RETURN_NONE;
        if (plain(PyTuple_GET_ITEM(a[9], 4))) flat.row_off = THPVariable_Unpack(PyTuple_GET_ITEM(a[9], 4));
    } else if (!PyType_Check(a[2])) {
        Py_RETURN_NONE;
    }
    if (!plain(a[3]) || !PyDict_CheckExact(a[7]) || !plain(a[8]) || !(a[6] == Py_None || plain(a[6]))) Py_RETURN_NONE;
    const at::Tensor bins = THPVariable_Unpack(a[3]), status = THPVariable_Unpack(a[8]);
    const at::Device dev = bins.device();
    if (dev.type() != at::kCUDA || dev.index() != c10::cuda::current_device()) Py_RETURN_NONE;
    const bool vllm = a[4] == Py_True;
    const at::ScalarType type = a[5] == Py_True ? at::kBFloat16 : at::kHalf;
    Shape s;
    std::vector<cg_decode_job> jobs;
    std::vector<at::Tensor> held;
    const Py_ssize_t chunks = PyList_GET_SIZE(a[0]);
    jobs.reserve(static_cast<size_t>(chunks));
    held.reserve(static_cast<size_t>(5 * chunks));
    for (Py_ssize_t k = 0; k < chunks; ++k) {
        PyObject *eo = PyList_GET_ITEM(a[0], k);
        if (Py_TYPE(eo) != reinterpret_cast<PyTypeObject *>(a[1])) Py_RETURN_NONE;
        if (!(containers ? add_container(eo, dev, flat, &s, k == 0, &jobs, &held)
                         : add_chunk(eo, reinterpret_cast<PyTypeObject *>(a[2]), dev, &s, k == 0, &jobs, &held)))
            Py_RETURN_NONE;
    }
    const int64_t C = s.H * s.D, groups = 2 * s.L * ((C + CG_GROUP_CHANNELS - 1) / CG_GROUP_CHANNELS);
    const int64_t njobs = static_cast<int64_t>(jobs.size());
    if (!usable(bins, at::kFloat, dev) || bins.numel() != 2 * s.L || !usable(status, at::kInt, dev) || status.numel() != 1 || !njobs)
        Py_RETURN_NONE;
    const int64_t shape[5] = {s.L, 2, vllm ? s.T : s.H, vllm ? s.H : s.T, s.D};
    at::Tensor out;
    if (a[6] == Py_None) {
        out = make(shape, at::TensorOptions().dtype(type).device(dev));
    } else {
        out = THPVariable_Unpack(a[6]);
        if (!out.unsafeGetTensorImpl()->has_storage() || out.layout() != at::kStrided || out.scalar_type() != type || out.device() != dev ||
            out.sizes() != at::IntArrayRef(shape) || out.stride(4) != 1 || out.is_conj() || out.is_neg())
            Py_RETURN_NONE;
    }
    // The group offsets' buffer is kept in the workspace between calls.  A graph writes to its buffer at every replay: it gets one of
    // its own memory, and what else it uses of the workspace's stays there when other calls replace it.
    at::Tensor goff;
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
        goff = make({njobs * groups}, at::TensorOptions().dtype(at::kLong).device(dev));
        for (PyObject *used : {a[3], a[8], containers ? PyTuple_GET_ITEM(a[9], 4) : Py_None})
            if (!keep_for_graph(a[7], used)) throw python_error();
    } else {
        PyObject *const kept = PyDict_GetItem(a[7], s_group_off);
        if (plain(kept)) goff = THPVariable_Unpack(kept);
        if (!usable(goff, at::kLong, dev) || goff.numel() < njobs * groups) {
            goff = make({njobs * groups}, at::TensorOptions().dtype(at::kLong).device(dev));
            const Ref made(THPVariable_Wrap(goff));
            if (PyDict_SetItem(a[7], s_group_off, made.p)) throw python_error();
        }
    }
    const int64_t o_token = out.stride(vllm ? 2 : 3), o_head = out.stride(vllm ? 3 : 2);
    uint8_t *at_out = static_cast<uint8_t *>(out.data_ptr());
    int64_t *at_goff = static_cast<int64_t *>(goff.data_ptr());
    for (cg_decode_job &j : jobs) {
        j.out = at_out;
        j.group_off = at_goff;
        at_out += 2 * o_token * j.ntokens;
        at_goff += groups;
    }
    const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(dev.index());
    int rc;
    {
        const WithoutGil released;
        rc = decode_kv(jobs.data(), static_cast<int>(njobs), static_cast<int>(s.L), static_cast<int>(s.H), static_cast<int>(s.D),
                       static_cast<int>(s.lp), static_cast<const float *>(bins.data_ptr()), 0,
                       nullptr, code(s.scale), code(type), out.stride(0), out.stride(1), o_token,
                       o_head, static_cast<int32_t *>(status.data_ptr()), stream.stream());
    }
    if (rc) return PyLong_FromLong(rc);
    {
        const WithoutGil released;
        for (const at::Tensor &t : held) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), stream);
    }
    return THPVariable_Wrap(out);
    END_HANDLE_TH_ERRORS
}

int64_t integer(PyObject *o) {
    const int64_t v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}

// encode_start(address of a cg_encode_kv_job with delta_group and res_bins set, kv, bins, max_bins, address of the tail,
//              workspace or None, row offsets of byte counts or None, their size, stream or None: the current one, launch)
// -> (error code, stream, scales [2, L, T, 1], scales_k, scales_v, cdf, workspace, counts or None).  kv: [L, 2, T, H, D] on a GPU, 16-bit,
// unit innermost stride.  With counts the two scales are parts of one tensor, else tensors of their own and the first is None.
PyObject *encode_start(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10 || !THPVariable_Check(a[1]) || !THPVariable_Check(a[2])) {
        PyErr_SetString(PyExc_TypeError, "encode_start: wrong arguments");
        return nullptr;
    }
    cg_encode_kv_job &job = *reinterpret_cast<cg_encode_kv_job *>(integer(a[0]));
    const at::Tensor kv = THPVariable_Unpack(a[1]), bins = THPVariable_Unpack(a[2]);
    const int64_t max_bins = integer(a[3]), L = kv.size(0), T = kv.size(2), H = kv.size(3), D = kv.size(4);
    const bool with_counts = a[6] != Py_None;
    const c10::cuda::CUDAGuard device(kv.device());
    const at::TensorOptions on = at::TensorOptions().device(kv.device()), bytes = on.dtype(at::kByte);
    at::Tensor scales, scales_k, scales_v, counts, workspace;
    if (with_counts) {
        scales = make({2, L, T, 1}, on.dtype(kv.scalar_type()));
        scales_k = scales.select(0, 0);
        scales_v = scales.select(0, 1);
    } else {
        scales_k = make({L, T, 1}, on.dtype(kv.scalar_type()));
        scales_v = make({L, T, 1}, on.dtype(kv.scalar_type()));
    }
    const at::Tensor cdf = make({2 * L, H * D, max_bins + 1}, on.dtype(at::kShort));
    const int64_t need = encode_kv_workspace(static_cast<int>(L), static_cast<int>(T), static_cast<int>(H), static_cast<int>(D));
    if (need < 0) return Py_BuildValue("(LOOOOOOO)", static_cast<long long>(need), Py_None, Py_None, Py_None, Py_None, Py_None, Py_None, Py_None);
    if (a[5] != Py_None) workspace = THPVariable_Unpack(a[5]);
    if (!workspace.defined() || workspace.numel() < need) workspace = make({need}, bytes);
    job.kv = kv.data_ptr();
    job.bins = static_cast<const float *>(bins.data_ptr());
    job.scales_k = scales_k.data_ptr();
    job.scales_v = scales_v.data_ptr();
    job.cdf = static_cast<int16_t *>(cdf.data_ptr());
    if (with_counts) {
        counts = make({integer(a[7])}, bytes);
        job.counts = static_cast<uint8_t *>(counts.data_ptr());
        job.table_row_off = static_cast<const int64_t *>(THPVariable_Unpack(a[6]).data_ptr());
    }
    job.workspace = workspace.data_ptr();
    job.workspace_bytes = workspace.numel();
    job.tail = reinterpret_cast<int64_t *>(integer(a[4]));
    job.s_layer = kv.stride(0);
    job.s_kv = kv.stride(1);
    job.s_token = kv.stride(2);
    job.s_head = kv.stride(3);
    job.dtype = code(kv.scalar_type());
    job.nlayers = static_cast<int32_t>(L);
    job.ntokens = static_cast<int32_t>(T);
    job.nheads = static_cast<int32_t>(H);
    job.head_size = static_cast<int32_t>(D);
    job.max_bins = static_cast<int32_t>(max_bins);
    void *const stream = a[8] == Py_None ? c10::cuda::getCurrentCUDAStream(kv.device().index()).stream() : reinterpret_cast<void *>(integer(a[8]));
    int rc = CG_OK;
    if (a[9] == Py_True) {
        const WithoutGil released;
        rc = encode_kv(&job, stream);
    }
    const auto wrap = [](const at::Tensor &t) { return t.defined() ? THPVariable_Wrap(t) : Py_NewRef(Py_None); };
    return Py_BuildValue("(iKNNNNNN)", rc, static_cast<unsigned long long>(reinterpret_cast<uintptr_t>(stream)), wrap(scales),
                         wrap(scales_k), wrap(scales_v), wrap(cdf), wrap(workspace), wrap(counts));
    END_HANDLE_TH_ERRORS
}

// encode_finish(address of a job that has been launched, number of its GPU, stream, its tensors of lengths or None)
// -> (error code, tail, pieces or None): waits for the sizes; with lengths, and if no stream is bad, makes a tensor for
// every sub-chunk's streams (a view would pickle the whole buffer) and launches the gather.
// tail: the nsub + 1 payload offsets, the status bits and the number of non-zero byte counts.
PyObject *encode_finish(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4 || !(a[3] == Py_None || PyList_CheckExact(a[3]))) {
        PyErr_SetString(PyExc_TypeError, "encode_finish: wrong arguments");
        return nullptr;
    }
    cg_encode_kv_job &job = *reinterpret_cast<cg_encode_kv_job *>(integer(a[0]));
    const c10::cuda::CUDAGuard device(static_cast<c10::DeviceIndex>(integer(a[1])));
    void *stream = reinterpret_cast<void *>(integer(a[2]));
    const int nsub = (job.ntokens + CG_MAX_TOKENS_PER_STREAM - 1) / CG_MAX_TOKENS_PER_STREAM;
    int rc;
    {
        const WithoutGil released;
        rc = encode_kv_wait(&job, stream);
    }
    if (rc) return Py_BuildValue("(iOO)", rc, Py_None, Py_None);
    // the tail goes back to its pool before anything can fail
    const std::vector<int64_t> sizes(job.tail, job.tail + nsub + 3);
    PyObject *pieces = nullptr;
    if (a[3] != Py_None && !(sizes[nsub + 1] & ~CG_S_COUNT_OVERFLOW)) {
        if (PyList_GET_SIZE(a[3]) != nsub) {
            PyErr_SetString(PyExc_TypeError, "encode_finish: wrong arguments");
            return nullptr;
        }
        std::vector<uint8_t *> to(static_cast<size_t>(nsub));
        std::vector<int32_t *> lengths(static_cast<size_t>(nsub));
        std::vector<at::Tensor> made(static_cast<size_t>(nsub));
        for (int k = 0; k < nsub; ++k) {
            const at::Tensor t = THPVariable_Unpack(PyList_GET_ITEM(a[3], k));
            lengths[k] = static_cast<int32_t *>(t.data_ptr());
            made[k] = make({sizes[k + 1] - sizes[k]}, at::TensorOptions().dtype(at::kByte).device(t.device()));
            to[k] = static_cast<uint8_t *>(made[k].data_ptr());
        }
        {
            const WithoutGil released;
            rc = encode_kv_gather(&job, to.data(), lengths.data(), stream);
        }
        pieces = PyList_New(nsub);
        for (int k = 0; k < nsub; ++k) PyList_SET_ITEM(pieces, k, THPVariable_Wrap(made[k]));
    }
    PyObject *tail = PyList_New(nsub + 3);
    for (int k = 0; k < nsub + 3; ++k) PyList_SET_ITEM(tail, k, PyLong_FromLongLong(sizes[k]));
    return Py_BuildValue("(iNN)", rc, tail, pieces ? pieces : Py_NewRef(Py_None));
    END_HANDLE_TH_ERRORS
}

// bind({name: address})
PyObject *bind(PyObject *, PyObject *addresses) {
    HANDLE_TH_ERRORS
    const auto address = [&](const char *name) {
        PyObject *v = PyDict_GetItemString(addresses, name);
        if (!v) throw std::runtime_error(std::string("bind: no ") + name);
        return reinterpret_cast<void *>(integer(v));
    };
    decode_kv = reinterpret_cast<decltype(decode_kv)>(address("cg_decode_kv"));
    encode_kv = reinterpret_cast<decltype(encode_kv)>(address("cg_encode_kv"));
    encode_kv_workspace = reinterpret_cast<decltype(encode_kv_workspace)>(address("cg_encode_kv_workspace"));
    encode_kv_wait = reinterpret_cast<decltype(encode_kv_wait)>(address("cg_encode_kv_wait"));
    encode_kv_gather = reinterpret_cast<decltype(encode_kv_gather)>(address("cg_encode_kv_gather"));
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr},
                         {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(decode)), METH_FASTCALL, nullptr},
                         {"encode_start", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(encode_start)), METH_FASTCALL, nullptr},
                         {"encode_finish", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(encode_finish)), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
    s_cdf = PyUnicode_InternFromString("cdf");
    s_max_tensors_key = PyUnicode_InternFromString("max_tensors_key");
    s_max_tensors_value = PyUnicode_InternFromString("max_tensors_value");
    s_data_chunks = PyUnicode_InternFromString("data_chunks");
    s_num_heads = PyUnicode_InternFromString("num_heads");
    s_head_size = PyUnicode_InternFromString("head_size");
    s_bytestream = PyUnicode_InternFromString("bytestream");
    s_bytestream_lengths = PyUnicode_InternFromString("bytestream_lengths");
    s_ntokens = PyUnicode_InternFromString("ntokens");
    s_group_off = PyUnicode_InternFromString("group_off");
    s_captured = PyUnicode_InternFromString("captured");
    s_blob = PyUnicode_InternFromString("blob");
    s_header = PyUnicode_InternFromString("header");
    s_sub_off = PyUnicode_InternFromString("sub_off");
    for (int k = 0; k < kHeaderFields; ++k) s_header_fields[k] = PyUnicode_InternFromString(kHeaderNames[k]);
    PyObject *const m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "built_for", CG_BUILT_FOR)) {  // see build.py
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}
