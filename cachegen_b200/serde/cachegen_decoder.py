"""CacheGenDeserializer (reference: LMCache/lmcache/storage_backend/serde/cachegen_decoder.py:114-173).

`from_bytes` keeps the reference's contract -- pickled CacheGenGPUEncoderOutput in, KV blob tensor on
the GPU out, bf16 [L,2,T,H,D] for "vllm" and fp16 [L,2,H,T,D] for "huggingface" -- with the cumsum of
dec.py:70, the per-sub-chunk launches and the fp32 dequantise / stack / permute / cast chain replaced by one
C-ABI call, cg_decode_kv (two launches per 40 sub-chunks).  Its two halves, cg_decode_offsets and
cg_decode_dequant, are what a plan's run_offsets and run_decode call.
(dec.py = cachegen_decoder.py of the reference.)

One deserializer's calls share its offset buffer and status word: they belong on one stream, from one thread at a
time.  Serializers share nothing between calls.
"""
import _thread
import ctypes
import functools
import queue
from typing import List

import torch

from .. import _lib
from .. import torchac_cuda
from ..config import LMCacheEngineConfig, LMCacheEngineMetadata
from ..utils import _lmcache_nvtx_annotate
from . import cachegen_basics as CGBasics
from . import flat_format
from .cachegen_basics import CacheGenConfig, CacheGenGPUBytestream, CacheGenGPUEncoderOutput, on_device
from .serde import Deserializer

_DTYPES = {torch.float16: _lib.CG_F16, torch.bfloat16: _lib.CG_BF16}


def _stream(device):
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def do_dequantize(t: torch.Tensor, bins: torch.Tensor, maxtensors: torch.Tensor) -> torch.Tensor:
    """The reference's dequantisation formula on torch tensors (dec.py:24-34); the product path
    computes the same values inside cg_decode_dequant.  t [L,T,C] float, bins [L], maxtensors [L,T,1]."""
    C = (bins // 2 - 1)[:, None, None]
    t = t - C
    t = t / C
    t = t * maxtensors
    return t


@_lmcache_nvtx_annotate
def bytes_to_tensor(bs: bytes, device="cuda") -> torch.Tensor:
    """A byte string as a uint8 tensor on `device` (dec.py:37-41); to a GPU through pinned staging."""
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # a read-only buffer, and it is only read
        view = torch.frombuffer(bs, dtype=torch.uint8)
    device = torch.device(device)
    if device.type == "cuda":
        device = torch.device("cuda", torch.cuda.current_device() if device.index is None else device.index)
        return CGBasics.staging().whole_to_device(view, device)
    return view.clone()


@_lmcache_nvtx_annotate
def recombine_bytes(bytes_tensor: torch.Tensor, output_lengths: torch.Tensor) -> torch.Tensor:
    """Back-to-back streams as padded rows [nlayers, nchannels, 256] for decode_fast_new
    (dec.py:43-49): row (r, c) holds the 256 bytes that start where stream (r, c) starts, reading
    no further than the last byte of `bytes_tensor`.  The legacy layout; from_bytes does not use it."""
    width = CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK
    lengths = output_lengths.reshape(-1).to(torch.int64)
    starts = lengths.cumsum(0) - lengths
    index = starts[:, None] + torch.arange(width, device=starts.device)
    index.clamp_(max=bytes_tensor.numel() - 1)
    return bytes_tensor[index].reshape(*output_lengths.shape, width)


@_lmcache_nvtx_annotate
def decode_chunk(cdf: torch.Tensor, data_chunk: CacheGenGPUBytestream, target_buffer: torch.Tensor) -> None:
    """Symbols of one sub-chunk into target_buffer [2L, ntokens, C] uint8, strided ok (dec.py:53-75)."""
    torchac_cuda.decode_by_lengths(cdf, data_chunk.bytestream, data_chunk.bytestream_lengths, target_buffer)


@_lmcache_nvtx_annotate
def decode_function_gpu(cdf: torch.Tensor, data_chunks: List[CacheGenGPUBytestream], layers_in_key: int,
                        chunk_size: int, output: torch.Tensor):
    """Symbol-level decode with the reference's signature (dec.py:78-112): fills `output`
    (uint8 [chunk_size, 2L*C]) and returns (key, value) symbols as float32 [L, chunk_size, C]."""
    nlayers, nchannels, _ = cdf.shape
    output = output.reshape((nlayers, chunk_size, nchannels))
    start = 0
    for data_chunk in data_chunks:
        end = start + data_chunk.ntokens
        decode_chunk(cdf, data_chunk, output[:, start:end, :])
        start = end
    out = output.reshape((2, layers_in_key, chunk_size, nchannels))
    key, value = out.float()
    return key, value


def _check_chunk(eo: CacheGenGPUEncoderOutput):
    """Shape checks of an unpickled reference blob -> (L, C, lp, T)."""
    cdf = eo.cdf
    if cdf.dim() != 3 or cdf.dtype != torch.int16:
        raise RuntimeError("CDF must be an int16 tensor [2L, C, Lp]")
    NL, C, lp = cdf.shape
    L = NL // 2
    mk, mv = eo.max_tensors_key, eo.max_tensors_value
    T = mk.shape[1]
    if eo.num_heads * eo.head_size != C or mk.shape[0] != L or mv.shape[0] != L or mv.shape[1] != T or not (
            mk.numel() == mv.numel() == L * T):  # one scale per (layer, token): they are read by address
        raise RuntimeError("inconsistent shapes in the encoded chunk")
    if mk.dtype not in _DTYPES or mk.dtype != mv.dtype:
        raise TypeError(f"scales must be float16 or bfloat16, got {mk.dtype} / {mv.dtype}")
    if sum(dc.ntokens for dc in eo.data_chunks) != T:
        raise RuntimeError("sub-chunk token counts do not add up to the chunk's tokens")
    return L, C, lp, T


def _staged(t: torch.Tensor, dev) -> torch.Tensor:
    """Encoded chunks may arrive with their tensors in (pinned) host memory: stage them on `dev`, contiguous."""
    if t.device != dev:
        t = t.to(dev, non_blocking=True)
    return t if t.is_contiguous() else t.contiguous()


class _HostBins:
    """What the bins of a decode say about the containers it reads and about delta coding.  The values of a tensor
    on a GPU are read back when they are first asked for, which plain pickled chunks never do."""

    def __init__(self, bins: torch.Tensor):
        self._bins = bins
        self._checksums, self._counts, self._sparse = {}, {}, {}

    @functools.cached_property
    def cpu(self) -> torch.Tensor:
        return self._bins.cpu()

    @functools.cached_property
    def values(self) -> tuple:
        return tuple(self.cpu.tolist())

    @functools.cached_property
    def sparse(self) -> bool:
        return flat_format.sparse_representable(self.cpu)

    def checksum(self, delta) -> int:
        key = None if delta is None else (delta.group, delta.divisor, delta.rows)
        if key not in self._checksums:
            self._checksums[key] = flat_format.bins_checksum(self.cpu, delta)
        return self._checksums[key]

    def counts_bytes(self, nchannels: int) -> int:
        if nchannels not in self._counts:
            self._counts[nchannels] = flat_format.table_row_offsets(self.cpu, nchannels)[-1]
        return self._counts[nchannels]

    def sparse_bytes(self, nchannels: int) -> int:
        """Of the masks and what stands in front of them."""
        if nchannels not in self._sparse:
            masks = flat_format.mask_row_offsets(self.cpu, nchannels)[-1]
            self._sparse[nchannels] = flat_format.sparse_parts(self.cpu.numel(), nchannels, masks)[1]
        return self._sparse[nchannels]


class _ChunkView:
    """What a decode needs from one encoded chunk, whichever container it came in, on the GPU."""

    def __init__(self, eo, dev, bins, delta=None):
        """`bins`: a _HostBins.  tables, mk, mv and the first and third part of each of `subs` are addresses."""
        self.keep = []
        if isinstance(eo, flat_format.FlatChunk):
            fc = eo if eo.blob.device == dev else eo.to(dev, non_blocking=True)
            h = fc.header
            self.L, self.H, self.D, self.T, self.lp = h.L, h.H, h.D, h.T, h.lp
            self.C = h.H * h.D
            self.scale_dtype = fc.scale_dtype
            self.table_kind, self.length_kind = h.table_kind, h.length_kind
            # int16 tables decode with any bins, but a chunk written with delta coding does not
            if h.bins_checksum and h.bins_checksum != bins.checksum(delta):
                raise RuntimeError("the container was written with other bin or delta settings")
            if h.table_kind == flat_format.TABLES_COUNTS:
                if h.off_lengths - h.off_tables < bins.counts_bytes(self.C):
                    raise RuntimeError("the container's byte-count tables are smaller than the configured bins need")
            elif h.table_kind == flat_format.TABLES_SPARSE:
                if not bins.sparse:
                    raise RuntimeError("sparse tables cannot describe the configured bins")
                if h.off_lengths - h.off_tables < bins.sparse_bytes(self.C):
                    raise RuntimeError("the container's sparse tables are smaller than the configured bins need")
            # addresses inside the container: a view for each takes longer to make than a short chunk to decode
            at, size, wide = fc.blob.data_ptr(), fc.blob.numel(), 2 if h.length_kind == flat_format.LENGTHS_U16 else 4
            row = 2 * h.L * self.C * wide
            if size < h.off_lengths + h.nsub * row or (at + h.off_scales) % 2 or (at + h.off_lengths) % wide or (
                    h.table_kind == flat_format.TABLES_CDF and (at + h.off_tables) % 2):
                raise RuntimeError("the container's sections are cut short or misaligned")
            self.mk = at + h.off_scales
            self.mv = self.mk + 2 * h.L * h.T
            self.tables = at + h.off_tables
            self.subs = []
            for j in range(h.nsub):
                start, end = (min(h.off_payload + o, size) for o in h.sub_off[j:j + 2])
                self.subs.append((at + start, end - start, at + h.off_lengths + j * row, fc.sub_tokens(j)))
            self.table_bytes = h.off_lengths - h.off_tables
            self.length_bytes = h.off_payload - h.off_lengths
            self.keep.append(fc.blob)
        else:
            L, C, lp, T = _check_chunk(eo)
            self.L, self.C, self.lp, self.T = L, C, lp, T
            self.H, self.D = eo.num_heads, eo.head_size
            self.scale_dtype = eo.max_tensors_key.dtype
            mk, mv, tables = (_staged(t, dev) for t in (eo.max_tensors_key, eo.max_tensors_value, eo.cdf))
            self.mk, self.mv, self.tables = mk.data_ptr(), mv.data_ptr(), tables.data_ptr()
            self.keep += (mk, mv, tables)
            self.table_kind = _lib.CG_TABLES_CDF
            self.length_kind = _lib.CG_LENGTHS_I32
            self.subs = []
            for dc in eo.data_chunks:
                bs, ln = dc.bytestream, dc.bytestream_lengths
                if bs.dtype != torch.uint8 or bs.dim() != 1:
                    raise RuntimeError("bytestream must be a 1-D uint8 tensor")
                if ln.dtype != torch.int32 or ln.numel() != 2 * L * C:
                    raise RuntimeError("bytestream_lengths must be int32 [2L, C]")
                bs, ln = _staged(bs, dev), _staged(ln, dev)
                self.subs.append((bs.data_ptr(), bs.numel(), ln.data_ptr(), dc.ntokens))
                self.keep += (bs, ln)
            self.table_bytes = tables.numel() * 2
            self.length_bytes = len(self.subs) * 2 * L * C * 4
        if sum(s[3] for s in self.subs) != self.T:
            raise RuntimeError("sub-chunk token counts do not add up to the chunk's tokens")
        for s in self.subs:
            if not 0 < s[3] <= CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK:
                raise RuntimeError("a sub-chunk holds 1..256 tokens")


def _on_gpu(eo) -> bool:
    return eo.blob.is_cuda if isinstance(eo, flat_format.FlatChunk) else eo.cdf.is_cuda


def _device_of(eo):
    return eo.blob.device if isinstance(eo, flat_format.FlatChunk) else eo.cdf.device


def _keep_for_graph(ws: dict, *tensors) -> bool:
    """Whether the current stream is being captured.  If so the launches of this call run again at every replay, whatever other calls do
    to the workspace: what they use of it is held there for good."""
    if not torch.cuda.is_current_stream_capturing():
        return False
    ws.setdefault("captured", set()).update(tensors)
    return True


def _status_word(ws: dict, dev) -> torch.Tensor:
    status = ws.get("status")
    if status is None or status.device != dev:
        with torch.inference_mode(False):  # kept, and written to by later calls in whatever mode those run
            status = torch.zeros(1, dtype=torch.int32, device=dev)
        if not _keep_for_graph(ws, status):  # (one that a graph makes is zero only once that has run)
            ws["status"] = status
    return status


_ROW_OFFSETS = {_lib.CG_TABLES_COUNTS: ("table_row_off", flat_format.table_row_offsets),
                _lib.CG_TABLES_SPARSE: ("mask_row_off", flat_format.mask_row_offsets)}


def _row_offsets(ws: dict, kind: int, host_bins: _HostBins, nchannels: int, dev) -> torch.Tensor:
    """Where the rows' byte counts, or masks, start in tables of this kind: a tensor that the workspace keeps."""
    name, fn = _ROW_OFFSETS[kind]
    t, key = ws.get(name), (nchannels, host_bins.values)
    if t is None or t.device != dev or ws.get(name + "_of") != key:
        t = torch.tensor(fn(host_bins.cpu, nchannels), dtype=torch.int64, device=dev)
        ws[name], ws[name + "_of"] = t, key
    return t


class DecodePlan:
    """Everything cg_decode_kv needs for a list of encoded chunks, built once:
    device-resident inputs, the job descriptors, the output blob and the launch arguments.  Chunks are
    CacheGenGPUEncoderOutput objects (the reference's blob, unpickled) or flat_format.FlatChunk
    containers, on the GPU or in (pinned) host memory."""

    def __init__(self, encoder_outputs: list, bins: torch.Tensor, fmt: str,
                 out_dtype: torch.dtype, out: torch.Tensor = None, workspace: dict = None, device=None,
                 peer_out: bool = False, delta=None, host_bins: _HostBins = None):
        if not encoder_outputs:
            raise RuntimeError("nothing to decode")
        if fmt not in ("vllm", "huggingface"):
            raise ValueError(f"unknown KV format {fmt!r}")
        first = encoder_outputs[0]
        dev = torch.device(device) if device is not None else (
            _device_of(first) if _on_gpu(first) else torch.device("cuda", torch.cuda.current_device()))
        ws = workspace if workspace is not None else {}
        if host_bins is None:  # a workspace may serve calls with other bins
            host_bins = _HostBins(bins)
        with on_device(dev):
            views = [_ChunkView(eo, dev, host_bins, delta) for eo in encoder_outputs]
        v0 = views[0]
        L, C, lp, H, D, scale_dtype = v0.L, v0.C, v0.lp, v0.H, v0.D, v0.scale_dtype
        NL = 2 * L
        for v in views:
            if (v.L, v.C, v.lp, v.H, v.scale_dtype) != (L, C, lp, H, scale_dtype):
                raise RuntimeError("chunks of one decode call must share layers, channels, table length and dtype")
        if scale_dtype not in _DTYPES:
            raise TypeError(f"scales must be float16 or bfloat16, got {scale_dtype}")
        total_T = sum(v.T for v in views)
        if bins.numel() != NL:
            raise RuntimeError(f"bins describe {bins.numel() // 2} layers, the blob has {L}")
        shape = (L, 2, total_T, H, D) if fmt == "vllm" else (L, 2, H, total_T, D)
        if out is None:
            out = torch.empty(shape, dtype=out_dtype, device=dev)
        elif (tuple(out.shape) != shape or out.dtype != out_dtype or out.stride(4) != 1 or
              (out.device != dev and not peer_out)):
            # peer_out: `out` is memory of another GPU of the box that this GPU can address
            # (cachegen_b200.parallel.buffer_on_root); the kernel stores into it over NVLink
            raise RuntimeError("output tensor has the wrong shape, dtype, device or innermost stride")
        if fmt == "vllm":
            o_layer, o_kv, o_token, o_head = out.stride(0), out.stride(1), out.stride(2), out.stride(3)
        else:
            o_layer, o_kv, o_head, o_token = out.stride(0), out.stride(1), out.stride(2), out.stride(3)
        nslab = (C + _lib.CG_GROUP_CHANNELS - 1) // _lib.CG_GROUP_CHANNELS
        ngroups = NL * nslab
        njobs_total = sum(len(v.subs) for v in views)
        status = ws.get("status")
        if status is None or status.device != dev:
            status = _status_word(ws, dev)
        row_offs = {kind: _row_offsets(ws, kind, host_bins, C, dev) for kind in {v.table_kind for v in views} if kind in _ROW_OFFSETS}
        goff = ws.get("group_off")
        if torch.cuda.is_current_stream_capturing():
            _keep_for_graph(ws, bins, status, *row_offs.values())
            goff = torch.empty(njobs_total * ngroups, dtype=torch.int64, device=dev)  # of the graph's own memory
        elif goff is None or goff.numel() < njobs_total * ngroups or goff.device != dev:
            goff = torch.empty(njobs_total * ngroups, dtype=torch.int64, device=dev)
            ws["group_off"] = goff

        esz = out.element_size()
        self.keep = list(row_offs.values())  # tensors that must outlive the launches
        jobs = self.jobs = (_lib.DecodeJob * njobs_total)()
        self.payload_bytes = self.table_bytes = self.length_bytes = 0
        at_out, at_off = out.data_ptr(), goff.data_ptr()
        k = 0
        for v in views:
            self.keep += v.keep
            self.table_bytes += v.table_bytes
            self.length_bytes += v.length_bytes
            mk, mv = v.mk, v.mv
            row_off = row_offs[v.table_kind].data_ptr() if v.table_kind in row_offs else None
            for at_bytes, nbytes, at_lengths, ntok in v.subs:
                self.payload_bytes += nbytes
                job = jobs[k]
                job.tables, job.bytes, job.lengths, job.group_off = v.tables, at_bytes, at_lengths, at_off
                job.scales_k, job.scales_v, job.out, job.table_row_off = mk, mv, at_out, row_off
                job.nbytes, job.tables_nbytes, job.ntokens, job.scale_stride = nbytes, v.table_bytes, ntok, v.T
                job.table_kind, job.length_kind = v.table_kind, v.length_kind
                mk += 2 * ntok
                mv += 2 * ntok
                at_out += esz * o_token * ntok
                at_off += 8 * ngroups
                k += 1
        self.njobs = njobs_total
        self.delta_group, self.res_bins = 0, None
        if delta is not None:
            self.delta_group = delta.group
            self.res_bins = delta.residual_bins(host_bins.cpu[:L], host_bins.cpu[L:], dev)
            self.keep.append(self.res_bins)
        self.out, self.dev, self.bins, self.status, self.goff = out, dev, bins, status, goff
        self.dims = (L, H, D, C, lp, NL, total_T)
        self.strides = (o_layer, o_kv, o_token, o_head)
        self.dtypes = (_DTYPES[scale_dtype], _DTYPES[out_dtype])
        # bytes one decode pass must move: 16-bit KV out, payload, tables, lengths, scales in
        self.scale_bytes = NL * total_T * 2
        self.output_bytes = NL * total_T * C * esz

    @functools.cached_property
    def batches(self):
        """(jobs, how many, their group offsets) of every cg_decode_offsets / cg_decode_dequant call."""
        ngroups = self.dims[5] * ((self.dims[3] + _lib.CG_GROUP_CHANNELS - 1) // _lib.CG_GROUP_CHANNELS)
        most, size = _lib.CG_MAX_DECODE_JOBS, ctypes.sizeof(_lib.DecodeJob)
        return [((_lib.DecodeJob * min(most, self.njobs - b)).from_buffer(self.jobs, b * size), min(most, self.njobs - b),
                 ctypes.c_void_p(self.goff.data_ptr() + 8 * b * ngroups)) for b in range(0, self.njobs, most)]

    # launches per call: 2 per batch
    def run_offsets(self) -> None:
        lib = _lib.lib()
        NL, C = self.dims[5], self.dims[3]
        with on_device(self.dev):
            st = _stream(self.dev)
            for arr, n, goff in self.batches:
                rc = lib.cg_decode_offsets(arr, n, NL, C, goff, self.status.data_ptr(), st)
                _lib.check(rc, "cg_decode_offsets")

    # launches per call: 1 per batch
    def run_decode(self) -> None:
        lib = _lib.lib()
        L, H, D, C, lp, NL, _ = self.dims
        with on_device(self.dev):
            st = _stream(self.dev)
            for arr, n, _ in self.batches:
                if self.delta_group:
                    rc = lib.cg_decode_dequant_delta(arr, n, L, H, D, lp, self.bins.data_ptr(), self.delta_group,
                                                     self.res_bins.data_ptr(), *self.dtypes, *self.strides,
                                                     self.status.data_ptr(), st)
                else:
                    rc = lib.cg_decode_dequant(arr, n, L, H, D, lp, self.bins.data_ptr(), *self.dtypes, *self.strides,
                                               self.status.data_ptr(), st)
                _lib.check(rc, "cg_decode_dequant")

    # launches per call: 2 per batch
    def run(self) -> torch.Tensor:
        L, H, D, _, lp, _, _ = self.dims
        cur = torch.cuda.current_stream(self.dev)
        with on_device(self.dev):
            rc = _lib.lib().cg_decode_kv(self.jobs, self.njobs, L, H, D, lp, self.bins.data_ptr(), self.delta_group,
                                         self.res_bins.data_ptr() if self.delta_group else None, *self.dtypes, *self.strides,
                                         self.status.data_ptr(), cur.cuda_stream)
        _lib.check(rc, "cg_decode_kv")
        for t in self.keep:
            t.record_stream(cur)
        return self.out

    @property
    def launches(self) -> int:
        return 2 * ((self.njobs + _lib.CG_MAX_DECODE_JOBS - 1) // _lib.CG_MAX_DECODE_JOBS)


def decode_many(encoder_outputs: List[CacheGenGPUEncoderOutput], bins: torch.Tensor, fmt: str,
                out_dtype: torch.dtype, out: torch.Tensor = None, workspace: dict = None, delta=None,
                host_bins: _HostBins = None) -> torch.Tensor:
    """Fused decode of consecutive encoded chunks of one KV cache into one blob.

    The chunks' tokens are laid one after the other along the token axis of the result, which has
    shape [L,2,T,H,D] ("vllm") or [L,2,H,T,D] ("huggingface"), T the total token count -- what
    LMCacheEngine.retrive builds with torch.cat from per-chunk from_bytes calls
    (LMCache/lmcache/cache_engine.py:282-320 in the reference).  All sub-chunks of all chunks go
    through one cg_decode_kv, in batches of up to 40 per launch.

    The chunks' tensors may live on the GPU or in (pinned) host memory; host tensors are copied to the
    GPU on the current stream first.  bins: float32 [2L] on the GPU (key bins then value bins).
    `out`, when given, must have the result's shape and dtype with a unit innermost stride (any other
    strides).  `workspace` caches the small offset / status buffers between calls; a graph that captures a decode needs it, or
    the deserializer that has it, for as long as it is replayed.  `host_bins`: the values of `bins`,
    when the caller knows them; read from the tensor otherwise, if the chunks ask for them.
    """
    if delta is None and workspace is not None:
        decoded = _decode_usual(encoder_outputs, bins, fmt, out_dtype, out, workspace, host_bins)
        if decoded is not None:
            return decoded
    return DecodePlan(encoder_outputs, bins, fmt, out_dtype, out=out, workspace=workspace, delta=delta,
                      host_bins=host_bins).run()


def _decode_usual(encoder_outputs, bins, fmt, out_dtype, out, workspace, host_bins):
    """What DecodePlan(...).run() does for chunks, all of one kind, of plain contiguous tensors on the current GPU, in native code.
    None, and nothing has been done but for buffers that the workspace keeps, for any other chunks."""
    if not encoder_outputs or not _on_gpu(encoder_outputs[0]):  # asked first: the rest takes a tenth of a short chunk's call
        return None
    if type(encoder_outputs) is not list or fmt not in ("vllm", "huggingface") or out_dtype not in _DTYPES or not bins.is_cuda:
        return None
    kind, piece, flat = CacheGenGPUEncoderOutput, CacheGenGPUBytestream, None
    if type(encoder_outputs[0]) is flat_format.FlatChunk:
        header = encoder_outputs[0].header
        if host_bins is None or header.table_kind == _lib.CG_TABLES_SPARSE and not host_bins.sparse:
            return None
        kind, piece, C = flat_format.FlatChunk, None, header.H * header.D
        flat = (header.table_kind, host_bins.checksum(None), host_bins.counts_bytes(C), host_bins.sparse_bytes(C),
                _row_offsets(workspace, header.table_kind, host_bins, C, bins.device) if header.table_kind in _ROW_OFFSETS else None)
    decoded = _lib.calls().decode(encoder_outputs, kind, piece, bins, fmt == "vllm", out_dtype == torch.bfloat16, out, workspace,
                                  _status_word(workspace, bins.device), flat)
    if type(decoded) is int:
        _lib.check(decoded, "cg_decode_kv")
    return decoded


_copy_streams = {}


def _copy_stream(dev) -> torch.cuda.Stream:
    stream = _copy_streams.get(dev)
    if stream is None:
        stream = _copy_streams[dev] = torch.cuda.Stream(device=dev)
    return stream


def _chunk_tokens(eo) -> int:
    return eo.num_tokens if isinstance(eo, flat_format.FlatChunk) else eo.max_tensors_key.shape[1]


def decode_many_pipelined(encoder_outputs: List[CacheGenGPUEncoderOutput], bins: torch.Tensor, fmt: str,
                          out_dtype: torch.dtype, out: torch.Tensor = None, groups: int = 4,
                          workspaces: list = None, delta=None, host_bins: _HostBins = None) -> torch.Tensor:
    """decode_many for encoded chunks held in pinned host memory, with the host-to-device copies of
    one group of chunks overlapped with the decode of the previous group (a copy stream per device;
    the decode launches stay on the caller's current stream).  `workspaces`: one dict per group; `host_bins`: as for
    decode_many."""
    host_bins = host_bins or _HostBins(bins)
    n = len(encoder_outputs)
    groups = max(1, min(groups, n))
    first = encoder_outputs[0]
    if groups == 1 or _on_gpu(first):
        return decode_many(encoder_outputs, bins, fmt, out_dtype, out=out,
                           workspace=workspaces[0] if workspaces else None, delta=delta, host_bins=host_bins)
    dev = torch.device("cuda", torch.cuda.current_device())
    L, H, D = bins.numel() // 2, first.num_heads, first.head_size
    total_T = sum(_chunk_tokens(eo) for eo in encoder_outputs)
    shape = (L, 2, total_T, H, D) if fmt == "vllm" else (L, 2, H, total_T, D)
    if out is None:
        out = torch.empty(shape, dtype=out_dtype, device=dev)
    elif tuple(out.shape) != shape:
        raise RuntimeError("output tensor has the wrong shape")
    copy_stream = _copy_stream(dev)
    cur = torch.cuda.current_stream(dev)
    captured = torch.cuda.is_current_stream_capturing()  # and so is the copy stream, which waits for it
    copy_stream.wait_stream(cur)
    if workspaces is None:
        workspaces = [dict() for _ in range(groups)]
    per = (n + groups - 1) // groups
    t0 = 0
    for g in range(groups):
        part = encoder_outputs[g * per:(g + 1) * per]
        if not part:
            break
        tg = sum(_chunk_tokens(eo) for eo in part)
        view = out[:, :, t0:t0 + tg] if fmt == "vllm" else out[:, :, :, t0:t0 + tg]
        with torch.cuda.stream(copy_stream):
            part = _stage_flat(part, workspaces[g], dev, captured)
            plan = DecodePlan(part, bins, fmt, out_dtype, out=view, workspace=workspaces[g], device=dev, delta=delta,
                              host_bins=host_bins)
            ready = torch.cuda.Event()
            ready.record(copy_stream)
        cur.wait_event(ready)
        plan.run()
        # the workspace's tensors come from the copy stream's pool; run sees to the plan's other inputs
        for t in (plan.goff, plan.status):
            t.record_stream(cur)
        t0 += tg
    return out


def _stage_flat(part: list, ws: dict, dev, captured: bool) -> list:
    """Copies a group's CGB2 containers from host memory into one device buffer that the workspace
    keeps between calls (no allocation per call, nothing for the caching allocator to hold back while
    the previous call's kernels still run).  Chunks of other kinds are returned as they are."""
    if not all(isinstance(eo, flat_format.FlatChunk) and not eo.blob.is_cuda for eo in part):
        return part
    starts, need = [], 0
    for eo in part:
        starts.append(need)
        need += (eo.blob.numel() + flat_format.ALIGN - 1) // flat_format.ALIGN * flat_format.ALIGN
    arena = ws.get("arena")
    if arena is None or arena.device != dev or arena.numel() < need:
        with torch.inference_mode(False):
            arena = torch.empty(need, dtype=torch.uint8, device=dev)
        ws["arena"] = arena
    if captured:
        _keep_for_graph(ws, arena)
    staged = []
    for eo, a in zip(part, starts):
        dst = arena[a:a + eo.blob.numel()]
        dst.copy_(eo.blob, non_blocking=True)
        staged.append(flat_format.FlatChunk(dst, eo.header))
    return staged


def decode_to_kv(encoder_output: CacheGenGPUEncoderOutput, bins: torch.Tensor, fmt: str, out_dtype: torch.dtype,
                 out: torch.Tensor = None, workspace: dict = None, delta=None, host_bins: _HostBins = None) -> torch.Tensor:
    """Fused decode of one encoded chunk into its KV blob (see decode_many)."""
    return decode_many([encoder_output], bins, fmt, out_dtype, out=out, workspace=workspace, delta=delta, host_bins=host_bins)


class CacheGenDeserializer(Deserializer):
    """Reference: dec.py:114-173.  `out_dtype` overrides the reference's fixed choice (bf16 for "vllm",
    fp16 for "huggingface"); `cachegen_config` replaces the lookup by model name."""

    def __init__(self, config: LMCacheEngineConfig, metadata: LMCacheEngineMetadata,
                 cachegen_config: CacheGenConfig = None, out_dtype: torch.dtype = None,
                 delta: "CGBasics.DeltaCoding" = None):
        _lib.lib()  # fail at construction if the CUDA library is missing
        self.delta = delta  # anchor-token delta coding: must be what the serializer was given
        self.cachegen_config = cachegen_config or CacheGenConfig.from_model_name(metadata.model_name)
        self.chunk_size = config.chunk_size
        self.fmt = metadata.fmt
        if self.fmt not in ("vllm", "huggingface"):
            raise ValueError(f"unknown KV format {self.fmt!r}")
        self.out_dtype = out_dtype or (torch.bfloat16 if self.fmt == "vllm" else torch.float16)
        self.key_bins = self.make_key_bins(self.cachegen_config)
        self.value_bins = self.make_value_bins(self.cachegen_config)
        self._bins = torch.cat((self.key_bins, self.value_bins)).contiguous()
        # their values: from the configuration, unless somebody else's methods made the tensors
        if (type(self).make_key_bins, type(self).make_value_bins) == _BINS_MAKERS:
            self._host_bins = _HostBins(torch.cat((CGBasics.make_key_bins(self.cachegen_config, "cpu"),
                                                   CGBasics.make_value_bins(self.cachegen_config, "cpu"))))
        else:
            self._host_bins = _HostBins(self._bins)
        self._workspace = {}

    def make_key_bins(self, config: CacheGenConfig) -> torch.Tensor:
        return CGBasics.make_key_bins(config, "cuda")

    def make_value_bins(self, config: CacheGenConfig) -> torch.Tensor:
        return CGBasics.make_value_bins(config, "cuda")

    def decode(self, encoder_output: CacheGenGPUEncoderOutput, out: torch.Tensor = None) -> torch.Tensor:
        """`from_bytes` without the unpickling."""
        ntokens = _chunk_tokens(encoder_output)
        if ntokens > self.chunk_size:
            # the reference slices a chunk_size-row buffer and fails in its reshape (dec.py:138-141,101)
            raise RuntimeError(f"blob holds {ntokens} tokens, more than chunk_size = {self.chunk_size}")
        return decode_to_kv(encoder_output, self._bins_on(_device_of(encoder_output)), self.fmt, self.out_dtype,
                            out=out, workspace=self._workspace, delta=self.delta, host_bins=self._host_bins)

    def decode_many(self, encoder_outputs: List[CacheGenGPUEncoderOutput], out: torch.Tensor = None) -> torch.Tensor:
        """Consecutive chunks of one KV cache into one blob, in as few launches as possible."""
        for eo in encoder_outputs:
            if _chunk_tokens(eo) > self.chunk_size:
                raise RuntimeError(f"a blob holds more tokens than chunk_size = {self.chunk_size}")
        return decode_many(encoder_outputs, self._bins_on(_device_of(encoder_outputs[0])), self.fmt, self.out_dtype,
                           out=out, workspace=self._workspace, delta=self.delta, host_bins=self._host_bins)

    def decode_many_host(self, encoder_outputs: List[CacheGenGPUEncoderOutput], out: torch.Tensor = None,
                         groups: int = None) -> torch.Tensor:
        """decode_many for chunks whose tensors sit in pinned host memory: copies and decodes overlap.
        groups: how many parts the chunks are split into (default: up to 32); the decode of a part
        runs while the next one is copied, so the last part's decode is all that is not hidden."""
        if groups is None:
            groups = min(32, len(encoder_outputs))
        ws = self._workspace.setdefault("groups", [dict() for _ in range(groups)])
        if len(ws) < groups:
            ws += [dict() for _ in range(groups - len(ws))]
        return decode_many_pipelined(encoder_outputs, self._bins_on(_device_of(encoder_outputs[0])), self.fmt,
                                     self.out_dtype, out=out, groups=groups, workspaces=ws, delta=self.delta,
                                     host_bins=self._host_bins)

    def group_status_words(self):
        """Status words of the pipelined path's per-group workspaces."""
        return [w["status"] for w in self._workspace.get("groups", []) if "status" in w]

    def plan(self, encoder_outputs: List[CacheGenGPUEncoderOutput], out: torch.Tensor = None,
             peer_out: bool = False, workspace: dict = None) -> DecodePlan:
        """The launch plan decode_many would run, for callers that decode the same chunks repeatedly.
        peer_out: `out` lives on another GPU of the box (see DecodePlan).  Plans built on one workspace
        (default: this object's) share its offset buffer: `run` recomputes the offsets every time, but
        `run_decode` alone is only valid while no other plan of the workspace has run in between."""
        return DecodePlan(encoder_outputs, self._bins_on(_device_of(encoder_outputs[0])), self.fmt, self.out_dtype,
                          out=out, workspace=self._workspace if workspace is None else workspace, peer_out=peer_out,
                          delta=self.delta, host_bins=self._host_bins)

    def _bins_on(self, dev) -> torch.Tensor:
        if not dev.type == "cuda":
            dev = torch.device("cuda", torch.cuda.current_device())
        if self._bins.device != dev:
            self._bins = self._bins.to(dev)
        return self._bins

    def check_status(self) -> None:
        """Synchronises and raises if a decode since the last check met malformed stream lengths."""
        words = ([self._workspace["status"]] if "status" in self._workspace else []) + self.group_status_words()
        for status in words:
            bits = int(status.item())
            if bits:
                status.zero_()
                raise RuntimeError("cachegen decode: " + _lib.status_text(bits))

    def from_bytes_many(self, blobs: List[bytes], out: torch.Tensor = None) -> torch.Tensor:
        """from_bytes for the blobs of consecutive chunks of one KV cache: one result tensor, as
        decode_many builds it.  Three things run side by side: the blobs' bytes on their way to the GPU (on a
        copy stream), the parsing of the blobs after the first (on a thread; the copies leave the interpreter to
        it), and the decode of each chunk that has arrived.  A pickled chunk's tensors come back on the GPU they were
        saved from; all are decoded on the first chunk's."""
        if not blobs:
            raise RuntimeError("nothing to decode")
        total = len(blobs)
        parsed = queue.SimpleQueue()
        cur = copies = None

        def parse(blob, dev, ahead=False):
            load = CGBasics.BlobLoad()
            with load:
                if ahead and isinstance(blob, bytes) and not flat_format.is_flat(blob):
                    CGBasics.staging().start(blob)
                chunk = (load.flat(blob, dev) if flat_format.is_flat(blob) else load.unpickle(blob))
            ntokens = _chunk_tokens(chunk)
            if ntokens > self.chunk_size:
                raise RuntimeError(f"a blob holds more tokens than chunk_size = {self.chunk_size}")
            return load, chunk, ntokens

        def parse_rest():
            try:
                with torch.cuda.device(dev), torch.cuda.stream(cur):
                    for blob in blobs[1:]:
                        parsed.put(parse(blob, dev))
            except BaseException as e:  # handed to the caller's thread
                parsed.put(e)

        chunks, tokens, done, at = [], 0, 0, 0
        waiting = []
        try:
            here = torch.device("cuda", torch.cuda.current_device())
            first = parse(blobs[0], here, ahead=True)  # the others are parsed while their predecessors travel
            dev = _device_of(first[1]) if _on_gpu(first[1]) else here
            cur, copies = torch.cuda.current_stream(dev), _copy_stream(dev)
            copies.wait_stream(cur)  # the tensors come from the current stream's pool
            if total > 1:
                # (a threading.Thread's start waits until the thread runs: 140 us before the first bytes left)
                _thread.start_new_thread(parse_rest, ())
            while done < total:
                item = first if done == 0 else (waiting.pop(0) if waiting else parsed.get())
                if isinstance(item, BaseException):
                    raise item
                load, chunk, ntokens = item
                # tensors of another GPU, made on a stream there that is not known here
                others = {p[2].device for p in load.pairs if p[2].device != dev}
                for d in others:
                    torch.cuda.synchronize(d)
                load.send(copies)
                for d in others:
                    torch.cuda.synchronize(d)
                arrived = torch.cuda.Event()
                arrived.record(copies)
                chunks.append((chunk, ntokens, arrived))
                tokens += ntokens
                done += 1
                while not parsed.empty():
                    waiting.append(parsed.get())
                if done + len(waiting) < total or any(isinstance(w, BaseException) for w in waiting):
                    continue  # the result's size is not known yet
                if at == 0:
                    out = self._blob_for(chunks[0][0], tokens + sum(w[2] for w in waiting), dev, out)
                    start = 0
                for chunk, n, arrived in chunks[at:]:
                    cur.wait_event(arrived)
                    part = out[:, :, start:start + n] if self.fmt == "vllm" else out[:, :, :, start:start + n]
                    DecodePlan([chunk], self._bins_on(dev), self.fmt, self.out_dtype, out=part, workspace=self._workspace,
                               device=dev, delta=self.delta, host_bins=self._host_bins).run()
                    start += n
                at = len(chunks)
        finally:
            CGBasics.staging().finish()
            if copies is not None:
                cur.wait_stream(copies)
        return out

    def _blob_for(self, chunk, ntokens, dev, out):
        """The result of a decode of ntokens tokens: `out`, checked, or a new tensor."""
        L, H, D = self._bins.numel() // 2, chunk.num_heads, chunk.head_size
        shape = (L, 2, ntokens, H, D) if self.fmt == "vllm" else (L, 2, H, ntokens, D)
        if out is None:
            return torch.empty(shape, dtype=self.out_dtype, device=dev)
        if tuple(out.shape) != shape:
            raise RuntimeError("output tensor has the wrong shape, dtype, device or innermost stride")
        return out

    @_lmcache_nvtx_annotate
    def from_bytes(self, bs: bytes) -> torch.Tensor:
        if flat_format.is_flat(bs):
            # a CGB2 container: one copy to the GPU, decoded in place
            return self.decode(flat_format.from_bytes(bs, device=torch.device("cuda", torch.cuda.current_device())))
        # tensors pickled on a GPU come back on that GPU; anything else is staged by the decode plan
        return self.decode(CacheGenGPUEncoderOutput.from_bytes(bs))


_BINS_MAKERS = (CacheGenDeserializer.make_key_bins, CacheGenDeserializer.make_value_bins)
