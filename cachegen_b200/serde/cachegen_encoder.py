"""CacheGenSerializer (reference: LMCache/lmcache/storage_backend/serde/cachegen_encoder.py:247-348).

`to_bytes` keeps the reference's contract -- KV blob tensor in, pickled CacheGenGPUEncoderOutput out,
byte-identical to what the reference produces from the same input -- with the reference's chain of
torch ops and per-sub-chunk launches replaced by three C-ABI calls:

    cg_encode_kv         split K/V + quantise + tables + every sub-chunk's streams + offsets  (enc.py:257-292, 225-236)
    cg_encode_kv_wait    waits for the payload sizes, all that the host needs to know
    cg_encode_kv_gather  gather of the streams                                                (enc.py:210-222)

Beside it: encode_many (a whole cache, chunks in flight on several streams and no wait in between), encode_levels
(one chunk at several bin settings) and encode_flat (the CGB2 container of flat_format.py, filled by
cg_encode_kv_flat).  quantize_and_tables and encode_streams are the same steps one by one.

(enc.py = cachegen_encoder.py of the reference.)
"""
import collections
import ctypes
import dataclasses
import operator
import threading
from typing import Tuple

import torch

from .. import _lib
from ..config import LMCacheEngineConfig, LMCacheEngineMetadata
from ..utils import _lmcache_nvtx_annotate
from . import cachegen_basics as CGBasics
from . import flat_format
from .cachegen_basics import CacheGenConfig, CacheGenGPUBytestream, CacheGenGPUEncoderOutput, on_device
from .serde import Serializer

_DTYPES = {torch.float16: _lib.CG_F16, torch.bfloat16: _lib.CG_BF16}


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream(device):
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def _split_kv(tensor: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """[L, 2, T, H, D] -> K and V as [L, T, H*D] (enc.py:72-83)."""
    num_layers, _, num_tokens, num_heads, head_size = tensor.shape
    return torch.unbind(tensor.reshape(num_layers, 2, num_tokens, num_heads * head_size), dim=1)


@_lmcache_nvtx_annotate
def torch_quant_vectorized(bins: torch.Tensor, input_groups: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """The reference's quantiser with its own signature (enc.py:42-59), on the quantise kernel: bins
    [R] (any numeric type), input_groups [R, T, C] float16 / bfloat16 on the GPU -> (symbols int8
    [R, T, C], max|x| per (row, token) [R, T, 1] in the input's dtype).  The serializer does not go
    through here (it quantises K and V of the blob in place, tables in the same pass)."""
    if input_groups.dim() != 3 or input_groups.dtype not in _DTYPES or not input_groups.is_cuda:
        raise TypeError("expected a CUDA float16 / bfloat16 tensor [nlayers, ntokens, nchannels]")
    x = input_groups.contiguous()
    R, T, C = x.shape
    if bins.numel() != R:
        raise RuntimeError(f"bins describe {bins.numel()} rows, the input has {R}")
    b = bins.to(device=x.device, dtype=torch.float32).contiguous()
    if R % 2:  # the kernel takes rows in two halves: give an odd count one more row to chew on
        x = torch.cat((x, x[-1:]))
        b = torch.cat((b, b[-1:]))
    half = x.shape[0] // 2
    max_bins = max(int(b.max()), 1)
    sym = torch.empty(x.shape, dtype=torch.int8, device=x.device)
    scales = torch.empty(x.shape[:2], dtype=x.dtype, device=x.device)
    cdf = torch.empty((x.shape[0], C, max_bins + 1), dtype=torch.int16, device=x.device)
    null = ctypes.c_void_p(None)
    with torch.cuda.device(x.device):
        rc = _lib.lib().cg_quantize_cdf(_ptr(x), _DTYPES[x.dtype], T * C, half * T * C, C, C, half, T, 1, C, _ptr(b),
                                        max_bins, _ptr(sym), _ptr(scales), _ptr(cdf), null, null, null,
                                        _stream(x.device))
    _lib.check(rc, "cg_quantize_cdf")
    return sym[:R], scales[:R].unsqueeze(-1)


@_lmcache_nvtx_annotate
def concat_max(max1) -> torch.Tensor:
    """A sequence of per-layer max tensors as one tensor with a leading layer axis (enc.py:62-70)."""
    return torch.stack([max1[i] for i in range(len(max1))])


@_lmcache_nvtx_annotate
def collect_bytes(output_buffer: torch.Tensor, output_lengths: torch.Tensor) -> torch.Tensor:
    """The first output_lengths[r, c] bytes of every row output_buffer[r, c, :], back to back in
    (r, c) order, as one uint8 tensor (enc.py:210-222), on the offset and compaction kernels."""
    return _collect(output_buffer, output_lengths)[0]


def _collect(output_buffer: torch.Tensor, output_lengths: torch.Tensor, status: torch.Tensor = None):
    """collect_bytes with one wait, for the total size; also returns the status word as it then is."""
    if output_buffer.dim() != 3 or output_buffer.dtype != torch.uint8 or not output_buffer.is_cuda:
        raise TypeError("expected a CUDA uint8 buffer [nlayers, nchannels, row]")
    buf, lengths = output_buffer.contiguous(), output_lengths.to(torch.int32).contiguous()
    NL, C, stride = buf.shape
    dev = buf.device
    if tuple(lengths.shape) != (NL, C) or lengths.device != dev:
        raise RuntimeError("output_lengths must have shape [nlayers, nchannels], on the buffer's GPU")
    nslab = (C + _lib.CG_GROUP_CHANNELS - 1) // _lib.CG_GROUP_CHANNELS
    offsets = torch.empty(NL * nslab, dtype=torch.int64, device=dev)
    lib, stream = _lib.lib(), _stream(dev)
    with on_device(dev):
        if NL * nslab <= _lib.CG_MAX_OFFSET_GROUPS:
            tail = _take_tail(4)
            try:
                rc = lib.cg_stream_sizes(_ptr(lengths), NL, C, min(stride, 1 << 20),
                                         None if status is None else status.data_ptr(), offsets.data_ptr(), tail.data_ptr(), stream)
                if rc == 0:
                    rc = lib.cg_wait_word(tail.data_ptr() + 24, stream)
                total, outside, bits, _ = tail[:4].tolist()
            except BaseException:
                torch.cuda.current_stream(dev).synchronize()  # the GPU may still be about to write to it
                raise
            finally:
                _give_tail(tail)
        else:
            total, outside, bits = torch.stack((lengths.sum(dtype=torch.int64),
                                                ((lengths < 0) | (lengths > stride)).sum(dtype=torch.int64),
                                                lengths.new_zeros((), dtype=torch.int64) if status is None else status[0].to(torch.int64))).tolist()
            job = _lib.DecodeJob()
            job.lengths, job.nbytes, job.length_kind = lengths.data_ptr(), total, _lib.CG_LENGTHS_I32
            rc = lib.cg_decode_offsets((_lib.DecodeJob * 1)(job), 1, NL, C, _ptr(offsets), None, stream)
        _lib.check(rc, "cg_stream_sizes")
        if outside:
            raise RuntimeError("collect_bytes: a length is negative or exceeds the buffer's row size")
        out = torch.empty(total, dtype=torch.uint8, device=dev)
        # the only sub-chunk starts where its first group does, at 0
        rc = lib.cg_compact_streams(_ptr(buf), stride, _ptr(lengths), _ptr(offsets), _ptr(offsets), 1, NL, C, _ptr(out), stream)
    _lib.check(rc, "cg_compact_streams")
    return out, bits


@_lmcache_nvtx_annotate
def encode_ntokens(cdf_int: torch.Tensor, encode_input: torch.Tensor, output_buffer: torch.Tensor,
                   output_lengths: torch.Tensor) -> torch.Tensor:
    """encode_fast_new into the caller's buffers, then collect_bytes (enc.py:225-242)."""
    from .. import torchac_cuda
    torchac_cuda.encode_fast_new(cdf_int, encode_input, output_buffer, output_lengths)
    status = torchac_cuda._status_word(cdf_int.device)
    # a stream that outgrew its row has a length that collect_bytes would refuse: the status comes first
    try:
        out, bits = _collect(output_buffer, output_lengths, status)
    except RuntimeError:
        torchac_cuda.check_status(cdf_int.device)
        raise
    if bits:
        torchac_cuda.check_status(cdf_int.device)
    return out


def quantize_and_tables(kv: torch.Tensor, key_bins: torch.Tensor, value_bins: torch.Tensor, max_bins: int,
                        with_counts: bool = False, delta: "CGBasics.DeltaCoding" = None):
    """Fused torch_quant_vectorized (K and V) + calculate_cdf (K and V) + the two torch.cat of
    encode_function (enc.py:42-59, 257-267).

    kv: CUDA fp16/bf16 blob addressed as [L, 2, T, H, D] (any strides with a unit innermost stride, so
        the permuted view of a "huggingface" blob is read in place).
    Returns (symbols int8 [2L, T, C], scales [2L, T] in kv.dtype, tables int16 [2L, C, max_bins + 1]);
    with_counts adds (byte counts uint8 of the compact table form, int32 status word whose
    CG_S_COUNT_OVERFLOW bit says they are unusable for this chunk).
    """
    if kv.dim() != 5 or kv.shape[1] != 2:
        raise RuntimeError(f"expected a KV blob of shape [L, 2, T, H, D], got {tuple(kv.shape)}")
    if kv.dtype not in _DTYPES:
        raise TypeError(f"the codec takes float16 or bfloat16 KV, got {kv.dtype}")
    if not kv.is_cuda:
        raise RuntimeError("KV must be a CUDA tensor")
    if kv.stride(4) != 1:
        kv = kv.contiguous()
    L, _, T, H, D = kv.shape
    C = H * D
    dev = kv.device
    bins = torch.cat((key_bins, value_bins)).to(device=dev, dtype=torch.float32).contiguous()
    if bins.numel() != 2 * L:
        raise RuntimeError(f"bins describe {bins.numel() // 2} layers, the KV blob has {L}")
    sym = torch.empty((2 * L, T, C), dtype=torch.int8, device=dev)
    scales = torch.empty((2 * L, T), dtype=kv.dtype, device=dev)
    cdf = torch.empty((2 * L, C, max_bins + 1), dtype=torch.int16, device=dev)
    counts = row_off = status = None
    if with_counts:
        offs = flat_format.table_row_offsets(bins.cpu(), C)
        row_off = torch.tensor(offs, dtype=torch.int64, device=dev)
        counts = torch.empty(offs[-1], dtype=torch.uint8, device=dev)
        status = torch.zeros(1, dtype=torch.int32, device=dev)
    null = ctypes.c_void_p(None)
    tail = (_ptr(cdf), _ptr(counts) if with_counts else null, _ptr(row_off) if with_counts else null,
            _ptr(status) if with_counts else null, _stream(dev))
    head = (_ptr(kv), _DTYPES[kv.dtype], kv.stride(0), kv.stride(1), kv.stride(2), kv.stride(3), L, T, H, D,
            _ptr(bins), int(max_bins))
    with torch.cuda.device(dev):
        if delta is not None:
            res_bins = delta.residual_bins(key_bins, value_bins, dev)
            rc = _lib.lib().cg_quantize_cdf_delta(*head, delta.group, _ptr(res_bins), _ptr(sym), _ptr(scales), *tail)
        else:
            rc = _lib.lib().cg_quantize_cdf(*head, _ptr(sym), _ptr(scales), *tail)
    _lib.check(rc, "cg_quantize_cdf")
    if with_counts:
        return sym, scales, cdf, counts, status
    return sym, scales, cdf


def encode_streams(cdf: torch.Tensor, sym: torch.Tensor, scratch_stride: int = None):
    """The sub-chunk loop of encode_function in one pass (enc.py:269-292).

    cdf int16 [2L, C, Lp], sym int8 [2L, T, C] contiguous.  Returns (bytes uint8 [total], lengths int32
    [nsub, 2L, C], sub_off: python list of nsub+1 byte offsets of the sub-chunks inside `bytes`).
    Synchronises once, to size the output.
    """
    NL, T, C = sym.shape
    lp = cdf.shape[2]
    dev = sym.device
    nsub = (T + CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK - 1) // CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK
    stride = scratch_stride or _lib.stream_capacity(min(T, CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK))
    stride = (stride + 3) // 4 * 4
    nslab = (C + _lib.CG_GROUP_CHANNELS - 1) // _lib.CG_GROUP_CHANNELS
    scratch = torch.empty((nsub, NL * C, stride), dtype=torch.uint8, device=dev)
    lengths = torch.empty((nsub, NL, C), dtype=torch.int32, device=dev)
    group_off = torch.empty((nsub, NL * nslab), dtype=torch.int64, device=dev)
    sub_off = torch.empty(nsub + 1, dtype=torch.int64, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    L = _lib.lib()
    with torch.cuda.device(dev):
        rc = L.cg_encode_chunk(_ptr(cdf), _ptr(sym), NL, T, C, lp, _ptr(scratch), stride, _ptr(lengths),
                               _ptr(group_off), _ptr(sub_off), _ptr(status), _stream(dev))
        _lib.check(rc, "cg_encode_chunk")
        host = torch.cat((sub_off, status.to(torch.int64))).cpu()  # the one synchronisation
        bits = int(host[nsub + 1])
        if bits:
            raise RuntimeError("cachegen encode: " + _lib.status_text(bits))
        offs = [int(v) for v in host[:nsub + 1]]
        out = torch.empty(offs[-1], dtype=torch.uint8, device=dev)
        rc = L.cg_compact_streams(_ptr(scratch), stride, _ptr(lengths), _ptr(group_off), _ptr(sub_off), nsub, NL,
                                  C, _ptr(out), _stream(dev))
        _lib.check(rc, "cg_compact_streams")
    return out, lengths, offs


class _BinsInfo:
    """What the values of a pair of bins tensors mean to an encode.  Tensors on a GPU are read back here, which waits
    for it, and what is kept belongs to these values: whoever keeps an info must know that the tensors it came from
    have not been written to since (see CacheGenSerializer._bins)."""

    def __init__(self, key_bins, value_bins):
        keys, values = (t.detach().cpu().to(torch.float32) for t in (key_bins, value_bins))
        self.cpu = torch.cat((keys, values))
        self.kmax, self.vmax = int(keys.max()), int(values.max())
        self.on_device = {}   # device -> float32 [2L]
        self.sparse = flat_format.sparse_representable(self.cpu)
        self.checksums = {}   # delta settings -> bins_checksum
        self.row_offsets = {}  # (device, channels) -> (int64 offsets of the byte counts, size, of the masks, size)

    def on(self, dev):
        t = self.on_device.get(dev)
        if t is None:
            t = self.on_device[dev] = self.cpu.to(dev)
        return t

    def checksum(self, delta):
        key = None if delta is None else (delta.group, delta.divisor, delta.rows)
        if key not in self.checksums:
            self.checksums[key] = flat_format.bins_checksum(self.cpu, delta)
        return self.checksums[key]

    def offsets(self, dev, nchannels):
        o = self.row_offsets.get((dev, nchannels))
        if o is None:
            counts = flat_format.table_row_offsets(self.cpu, nchannels)
            masks = flat_format.mask_row_offsets(self.cpu, nchannels)
            o = (torch.tensor(counts, dtype=torch.int64, device=dev), counts[-1],
                 torch.tensor(masks, dtype=torch.int64, device=dev), masks[-1])
            self.row_offsets[dev, nchannels] = o
        return o

    def table_bins(self, max_bins=None):
        """max_bins of the chunk's tables.  The reference builds key and value tables with their own
        maximum and concatenates them, which needs the two to be equal (enc.py:265-267).  `max_bins`
        overrides that: a layer shard of a model must use the whole model's value so that its tables and
        streams are the ones an unsharded encode produces."""
        if max_bins is not None:
            if max_bins < max(self.kmax, self.vmax):
                raise RuntimeError(f"max_bins {max_bins} is below the largest bin count {max(self.kmax, self.vmax)}")
            return int(max_bins)
        if self.kmax != self.vmax:
            raise RuntimeError(f"Sizes of tensors must match: key tables have {self.kmax + 1} entries, value tables {self.vmax + 1}")
        return self.kmax


_local = threading.local()
_KEPT_TAILS = 32


def _take_tail(n: int) -> torch.Tensor:
    """Pinned int64 memory for an encode's sizes, from this thread's pool (at most _KEPT_TAILS buffers)."""
    pool = _local.__dict__.setdefault("tails", [])
    for i in range(len(pool) - 1, -1, -1):
        if pool[i].numel() >= n:
            return pool.pop(i)
    return torch.empty(max(n, 64), dtype=torch.int64, pin_memory=True)


def _give_tail(t: torch.Tensor) -> None:
    pool = _local.__dict__.setdefault("tails", [])
    if len(pool) < _KEPT_TAILS:
        pool.append(t)


class _PendingChunk:
    """One chunk whose kernels up to the streams and their offsets are enqueued on `stream` (default: the
    current one), but whose payload size is not yet known on the host.  finish() waits for that and
    enqueues the gather.  Buffers come from the current stream's pool whatever `stream` is.  enqueue=False leaves the
    launches to _encode_infos."""

    def __init__(self, kv, info, max_bins, delta=None, stream=None, workspace=None, with_counts=False, enqueue=True):
        if kv.dim() != 5 or kv.shape[1] != 2:
            raise RuntimeError(f"expected a KV blob of shape [L, 2, T, H, D], got {tuple(kv.shape)}")
        if kv.dtype not in _DTYPES:
            raise TypeError(f"the codec takes float16 or bfloat16 KV, got {kv.dtype}")
        if not kv.is_cuda:
            raise RuntimeError("KV must be a CUDA tensor")
        if kv.stride(4) != 1:
            kv = kv.contiguous()
        L, _, T, H, D = kv.shape
        if info.cpu.numel() != 2 * L:  # the kernels read 2L of them
            raise RuntimeError(f"bins describe {info.cpu.numel() // 2} layers, the KV blob has {L}")
        dev = kv.device
        self.kv, self.info, self.dev = kv, info, dev
        self.L, self.T, self.H, self.D, self.max_bins = L, T, H, D, max_bins
        step = CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK
        self.nsub = (T + step - 1) // step
        self.lib = _lib.lib()
        self.on = None if stream is None else stream.cuda_stream  # the stream's address; None: the current one
        self.bins = info.on(dev)
        self.tail = _take_tail(self.nsub + 4)
        job = self.job = _lib.EncodeKvJob()
        self.res_bins = None
        try:
            if delta is not None:
                self.res_bins = delta.residual_bins(info.cpu[:L], info.cpu[L:], dev)
                job.delta_group, job.res_bins = delta.group, self.res_bins.data_ptr()
            row_off = size = None
            if with_counts:
                row_off, size, self.mask_off, self.mask_bytes = info.offsets(dev, H * D)
            self.start(workspace, row_off, size, enqueue)
            self.lengths = []
            if enqueue and not with_counts:
                self.make_lengths()
        except BaseException:
            self.abandon()
            raise

    def start(self, workspace, row_off, counts_bytes, enqueue):
        """Makes the buffers (`workspace`, if it is large enough, is taken), fills the job in and launches its kernels."""
        rc, self.on, self.scales, self.scales_k, self.scales_v, self.cdf, self.workspace, self.counts = _lib.calls().encode_start(
            ctypes.addressof(self.job), self.kv, self.bins, self.max_bins, self.tail.data_ptr(), workspace, row_off, counts_bytes,
            self.on, enqueue)
        _lib.check(rc, "cg_encode_kv_workspace" if self.cdf is None else "cg_encode_kv")

    def make_lengths(self):
        """Made while the GPU works: what is done after its sizes have arrived is time in which it has nothing to do."""
        self.lengths = [torch.empty((2 * self.L, self.H * self.D), dtype=torch.int32, device=self.dev) for _ in range(self.nsub)]

    @property
    def stream_ptr(self):
        return ctypes.c_void_p(self.on)

    @property
    def pointers(self):
        return ctypes.c_void_p * self.nsub

    @property
    def length_pointers(self):
        return self.pointers(*[t.data_ptr() for t in self.lengths])

    def another(self, info, max_bins):
        """The same KV at other bins, prepared like this chunk (one without delta coding or counts) and not enqueued."""
        if info.cpu.numel() != 2 * self.L:
            raise RuntimeError(f"bins describe {info.cpu.numel() // 2} layers, the KV blob has {self.L}")
        p = object.__new__(_PendingChunk)
        p.__dict__.update(self.__dict__)
        p.info, p.max_bins, p.bins = info, max_bins, info.on(self.dev)
        p.tail = _take_tail(self.nsub + 4)
        p.job = _lib.EncodeKvJob()
        p.start(None, None, None, False)
        return p

    def sizes(self, lengths=None):
        """Waits for (payload offsets [nsub + 1], status bits, number of non-zero byte counts, pieces): with `lengths`, the tensors
        for them, the streams are gathered into pieces of their own as soon as their sizes are known."""
        rc, host, pieces = _lib.calls().encode_finish(ctypes.addressof(self.job), self.dev.index, self.on, lengths)
        if host is not None:
            _give_tail(self.tail)
            self.tail = None
        _lib.check(rc, "cg_encode_kv_wait" if host is None else "cg_encode_kv_gather")
        bits = host[self.nsub + 1]
        if bits & ~_lib.CG_S_COUNT_OVERFLOW:
            raise RuntimeError("cachegen encode: " + _lib.status_text(bits & ~_lib.CG_S_COUNT_OVERFLOW))
        return host[:self.nsub + 1], bits, host[self.nsub + 2], pieces

    def pieces(self):
        """Waits for the sizes; a tensor for every sub-chunk's streams (a view would pickle the whole buffer)."""
        offs = self.sizes()[0]
        return [torch.empty(offs[j + 1] - offs[j], dtype=torch.uint8, device=self.dev) for j in range(self.nsub)]

    def finish(self) -> CacheGenGPUEncoderOutput:
        return self.output(self.sizes(self.lengths)[3])

    def output(self, pieces) -> CacheGenGPUEncoderOutput:
        step = CGBasics.CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK
        return CacheGenGPUEncoderOutput([CacheGenGPUBytestream(piece, lengths, min(step, self.T - j * step))
                                         for j, (piece, lengths) in enumerate(zip(pieces, self.lengths))],
                                        self.cdf, self.scales_k, self.scales_v, self.H, self.D)

    def abandon(self) -> None:
        """Gives the buffers up after an error: the GPU may still be writing to them, the pinned one among them, which
        would go to whoever asks torch for pinned memory next.  Nothing to do once the sizes have been read."""
        if self.tail is not None:
            (torch.cuda.current_stream(self.dev) if self.on is None else
             torch.cuda.ExternalStream(self.on, device=self.dev)).synchronize()
            _give_tail(self.tail)
            self.tail = None


def encode_many(kv: torch.Tensor, key_bins: torch.Tensor, value_bins: torch.Tensor, chunk_tokens: int,
                batch: int = 16, max_bins: int = None, delta=None, streams: int = 3, info: _BinsInfo = None) -> list:
    """Encodes a whole KV cache [L, 2, T, H, D] (GPU, unit innermost stride) chunk by chunk, as
    LMCacheEngine.store does with one to_bytes call per chunk (LMCache/lmcache/cache_engine.py:205-255
    in the reference), but without waiting for a chunk's payload size before the next chunk's kernels
    are enqueued: up to `batch` chunks, but no more than two a stream (six by default), are in flight; a chunk's
    streams are gathered when its turn to be replaced comes, so the host waits for sizes that arrived long ago.  Every chunk in
    flight keeps its own workspace (200 MB for a 7B-shape chunk).  Consecutive chunks run on `streams` side
    streams in turn (see _side_streams); the caller's stream waits for them before the call returns.
    Returns the chunks' CacheGenGPUEncoderOutput objects, identical to per-chunk encode_function calls.
    `info`: what the bins are, when the caller knows (see CacheGenSerializer._bins); read from the tensors otherwise."""
    info = info or _BinsInfo(key_bins, value_bins)
    kmax = info.table_bins(max_bins)
    if kv.stride(4) != 1:
        kv = kv.contiguous()  # on the caller's stream, before the others wait for it
    T = kv.shape[2]
    info.on(kv.device)
    caller = torch.cuda.current_stream(kv.device)
    lanes = _side_streams(kv.device, streams)
    for side in lanes:
        side.wait_stream(caller)  # the cache is ready on the caller's stream
    spare = [[] for _ in lanes]   # workspaces whose chunk has been gathered on that stream
    result, in_flight = [], collections.deque()

    def finish_oldest():
        p, lane = in_flight.popleft()
        try:
            result.append(p.finish())
        finally:
            p.abandon()
        spare[lane].append(p.workspace)

    try:
        for i, s in enumerate(range(0, T, chunk_tokens)):
            lane = i % len(lanes)
            if len(in_flight) >= max(1, min(batch, 2 * len(lanes))):
                finish_oldest()
            ws = spare[lane].pop() if spare[lane] else None
            # tensors come from the caller's stream's pool, and go back to it after the waits below
            in_flight.append((_PendingChunk(kv[:, :, s:s + chunk_tokens], info, kmax, delta=delta, stream=lanes[lane],
                                            workspace=ws), lane))
        while in_flight:
            finish_oldest()
    finally:
        for p, _ in in_flight:
            p.abandon()
        for side in lanes:
            caller.wait_stream(side)
    return result


_SIDE_STREAMS = {}


def _side_streams(device, n):
    """n streams of `device`, made once and kept: consecutive chunks of encode_many go to different
    streams, so that one chunk's quantisation, which is bound by memory, runs beside another's coder, which
    is bound by instruction issue, and fills what its last wave leaves idle."""
    key = (torch.device(device).index if torch.device(device).index is not None else torch.cuda.current_device())
    have = _SIDE_STREAMS.setdefault(key, [])
    while len(have) < n:
        have.append(torch.cuda.Stream(device=device))
    return have[:n]


def encode_levels(kv: torch.Tensor, levels: list) -> list:
    """One chunk of KV, [L, 2, T, H, D] on the GPU, encoded at several bin settings: `levels` is a list
    of (key_bins, value_bins) pairs, the result one CacheGenGPUEncoderOutput per pair, each identical
    to what encode_function gives with those bins.  This is what the reference's adaptation scripts
    store per chunk (one blob per QUANT_LEVEL, run_adaptation.py:61-72) so that config_selection can
    pick a level per chunk (src/utils.py:294-314).  Up to four levels share one read of the KV and one launch
    for each step."""
    return _encode_infos(kv, [_BinsInfo(kb, vb) for kb, vb in levels])


def _encode_infos(kv, infos) -> list:
    if kv.stride(4) != 1:
        kv = kv.contiguous()
    groups, step = [], _lib.CG_MAX_ENCODE_LEVELS
    # Groups share a read and their launches; what is left over goes first, so that the GPU works on it while the host prepares four
    # others.  Three settings of a 256-token chunk of 32 layers x 8 heads take 193.5 us together, 199 with the first of them alone
    # in front (of 30 tokens 118 and 129); five 272 us as one and four, 295 as four and one.
    left = (len(infos) - 1) % step + 1
    slices = [infos[:left]] + [infos[s:s + step] for s in range(left, len(infos), step)] if infos else []
    try:
        first = None
        for part in slices:
            groups.append([])
            for info in part:
                groups[-1].append(first.another(info, info.table_bins()) if first else
                                  _PendingChunk(kv, info, info.table_bins(), enqueue=False))
                first = first or groups[-1][0]
            jobs = (_lib.EncodeKvJob * len(groups[-1]))(*[p.job for p in groups[-1]])
            with on_device(first.dev):
                _lib.check(first.lib.cg_encode_kv_levels(jobs, len(jobs), first.stream_ptr), "cg_encode_kv_levels")
            for p in groups[-1]:
                p.make_lengths()
        result = []
        for group in groups:
            first = group[0]
            jobs = (_lib.EncodeKvJob * len(group))(*[p.job for p in group])
            pieces = [p.pieces() for p in group]
            pointers = ctypes.c_void_p * (len(group) * first.nsub)
            with on_device(first.dev):
                rc = first.lib.cg_encode_kv_levels_gather(jobs, len(group), pointers(*[t.data_ptr() for one in pieces for t in one]),
                                                          pointers(*[t.data_ptr() for p in group for t in p.lengths]),
                                                          first.stream_ptr)
            _lib.check(rc, "cg_encode_kv_levels_gather")
            result += [p.output(one) for p, one in zip(group, pieces)]
        return result
    finally:
        for group in groups:
            for p in group:
                p.abandon()


@_lmcache_nvtx_annotate
def encode_function(kv: torch.Tensor, config: CacheGenConfig, key_bins: torch.Tensor, value_bins: torch.Tensor,
                    chunk_size: int, max_bins: int = None, delta=None, info: _BinsInfo = None) -> CacheGenGPUEncoderOutput:
    """Encodes one chunk of KV, [L, 2, T, H, D] on the GPU, T == chunk_size (enc.py:247-301).  `info`: as for encode_many."""
    if kv.shape[2] != chunk_size:
        raise RuntimeError(f"chunk_size {chunk_size} does not match the {kv.shape[2]} tokens of the blob")
    info = info or _BinsInfo(key_bins, value_bins)
    p = _PendingChunk(kv, info, info.table_bins(max_bins), delta=delta)
    try:
        return p.finish()
    finally:
        p.abandon()


def encode_flat(kv: torch.Tensor, key_bins: torch.Tensor, value_bins: torch.Tensor,
                compact_tables=True, max_bins: int = None, delta=None, info: _BinsInfo = None) -> flat_format.FlatChunk:
    """Encodes one chunk of KV, [L, 2, T, H, D] on the GPU, into a CGB2 container on the GPU
    (flat_format.py): the same tables, lengths and streams as encode_function, with uint16 lengths and
    the tables in the smallest form that can hold them.  compact_tables: True (sparse byte counts when
    every non-centre histogram count fits a byte and no row has more than 32 of them, else dense byte
    counts when the counts fit, else the int16 tables), "counts" (never sparse) or False (always int16)."""
    info = info or _BinsInfo(key_bins, value_bins)
    kmax = info.table_bins(max_bins)
    p = _PendingChunk(kv, info, kmax, delta=delta, with_counts=True)
    try:
        # while the GPU works
        f, checksum = _lib.FlatLayout(), info.checksum(delta)
        off_masks, off_counts = flat_format.sparse_parts(2 * p.L, p.H * p.D, p.mask_bytes)
        f.mask_row_off, f.off_masks, f.off_counts = p.mask_off.data_ptr(), off_masks, off_counts
        offs, bits, nonzero, _ = p.sizes()
    finally:
        p.abandon()
    fits = bool(compact_tables) and not (bits & _lib.CG_S_COUNT_OVERFLOW)
    if fits and compact_tables is True and info.sparse:
        kind, size = flat_format.TABLES_SPARSE, off_counts + nonzero
    elif fits:
        kind, size = flat_format.TABLES_COUNTS, p.counts.numel()
    else:
        kind, size = flat_format.TABLES_CDF, 2 * p.cdf.numel()
    header = flat_format.layout(p.L, p.H, p.D, p.T, kmax + 1, p.kv.dtype, kind, size, flat_format.LENGTHS_U16, offs,
                                bins_checksum=checksum)
    head = header.pack()
    blob = torch.empty(header.total, dtype=torch.uint8, device=p.dev)
    sub_off = (ctypes.c_int64 * p.nsub)(*offs[:p.nsub])
    f.blob, f.table_kind = blob.data_ptr(), kind
    f.header_host, f.header_bytes = ctypes.cast(head, ctypes.c_void_p), len(head)
    f.sub_off_host = ctypes.addressof(sub_off)
    f.off_scales, f.off_tables, f.tables_bytes = header.off_scales, header.off_tables, size
    f.off_lengths, f.off_payload = header.off_lengths, header.off_payload
    with on_device(p.dev):
        _lib.check(p.lib.cg_encode_kv_flat(ctypes.byref(p.job), ctypes.byref(f), p.stream_ptr), "cg_encode_kv_flat")
    return flat_format.FlatChunk(blob, header)


_settings_of = operator.attrgetter(*[f.name for f in dataclasses.fields(CacheGenConfig)])


class CacheGenSerializer(Serializer):
    """Reference: enc.py:303-348.  `cachegen_config` may be given instead of looking it up from
    metadata.model_name (quality levels other than the built-in ones).  wire_format: "pickle" (the
    reference's blob, default) or "flat" (the CGB2 container of flat_format.py, which the reference
    cannot read)."""

    def __init__(self, config: LMCacheEngineConfig, metadata: LMCacheEngineMetadata,
                 cachegen_config: CacheGenConfig = None, wire_format: str = "pickle", table_max_bins: int = None,
                 delta: "CGBasics.DeltaCoding" = None):
        if wire_format not in ("pickle", "flat"):
            raise ValueError(f"unknown wire format {wire_format!r}")
        self.wire_format = wire_format
        self.delta = delta  # anchor-token delta coding: off (None) is the reference's behaviour
        self.table_max_bins = table_max_bins  # see _table_bins: set for a layer shard of a model
        _lib.lib()  # fail at construction if the CUDA library is missing
        self.cachegen_config = cachegen_config or CacheGenConfig.from_model_name(metadata.model_name)
        self.chunk_size = config.chunk_size
        self.fmt = metadata.fmt
        self._key_bins = self.make_key_bins(self.cachegen_config)
        self._value_bins = self.make_value_bins(self.cachegen_config)
        # the values are known from the configuration, unless somebody else's methods made the tensors
        self._bins_shared = (type(self).make_key_bins, type(self).make_value_bins) != _BINS_MAKERS
        self._info = (_BinsInfo(self._key_bins, self._value_bins) if self._bins_shared else
                      self._config_info(self.cachegen_config))
        self._levels = {}  # settings -> _BinsInfo

    # The bins tensors are the caller's to read, write and replace.  Once one has been handed out, or was handed in, nothing
    # says whether it has been written to (a tensor made in inference mode has no version counter, and writes
    # through .data do not count in one): from then on every call reads them back.
    @property
    def key_bins(self) -> torch.Tensor:
        self._bins_shared = True
        return self._key_bins

    @key_bins.setter
    def key_bins(self, bins: torch.Tensor) -> None:
        self._key_bins, self._bins_shared = bins, True

    @property
    def value_bins(self) -> torch.Tensor:
        self._bins_shared = True
        return self._value_bins

    @value_bins.setter
    def value_bins(self, bins: torch.Tensor) -> None:
        self._value_bins, self._bins_shared = bins, True

    def _bins(self) -> _BinsInfo:
        info = self._info
        if self._bins_shared:
            now = _BinsInfo(self._key_bins, self._value_bins)
            if (now.kmax, now.vmax) != (info.kmax, info.vmax) or not torch.equal(now.cpu, info.cpu):
                info = self._info = now
        return info

    @staticmethod
    def _config_info(config: CacheGenConfig) -> _BinsInfo:
        return _BinsInfo(CGBasics.make_key_bins(config, "cpu"), CGBasics.make_value_bins(config, "cpu"))

    def make_key_bins(self, config: CacheGenConfig) -> torch.Tensor:
        return CGBasics.make_key_bins(config, "cuda")

    def make_value_bins(self, config: CacheGenConfig) -> torch.Tensor:
        return CGBasics.make_value_bins(config, "cuda")

    def encode(self, tensor: torch.Tensor) -> CacheGenGPUEncoderOutput:
        """`to_bytes` without the final pickle: the encoded chunk with its tensors on the GPU."""
        if self.fmt == "huggingface":
            tensor = tensor.permute(0, 1, 3, 2, 4)  # a view; the kernels read it through its strides
        ntokens = tensor.shape[2]
        return encode_function(tensor.cuda(), self.cachegen_config, self._key_bins, self._value_bins, ntokens,
                               max_bins=self.table_max_bins, delta=self.delta, info=self._bins())

    def encode_many(self, tensor: torch.Tensor, chunk_tokens: int = None, batch: int = 16, streams: int = 3) -> list:
        """A whole KV cache, one encoded chunk per `chunk_tokens` (default: the configured chunk size)
        tokens, with up to `batch` chunks, but no more than two a stream, in flight on the GPU, on `streams` streams
        in turn."""
        if self.fmt == "huggingface":
            tensor = tensor.permute(0, 1, 3, 2, 4)
        tensor = tensor.cuda()
        if tensor.stride(4) != 1:
            tensor = tensor.contiguous()
        return encode_many(tensor, self._key_bins, self._value_bins, chunk_tokens or self.chunk_size, batch,
                           max_bins=self.table_max_bins, delta=self.delta, streams=streams, info=self._bins())

    def encode_levels(self, tensor: torch.Tensor, cachegen_configs: list) -> list:
        """The chunk encoded with each of `cachegen_configs` (CacheGenConfig objects, e.g. the three
        QUANT_LEVEL settings) in one go: one CacheGenGPUEncoderOutput per configuration, equal to what
        a serializer built with that configuration returns from `encode`."""
        if self.fmt == "huggingface":
            tensor = tensor.permute(0, 1, 3, 2, 4)
        return _encode_infos(tensor.cuda(), [self._level_info(c) for c in cachegen_configs])

    def _level_info(self, config: CacheGenConfig) -> _BinsInfo:
        """The bins of a quality level, made once per setting."""
        key = _settings_of(config) if type(config) is CacheGenConfig else dataclasses.astuple(config)
        info = self._levels.get(key)
        if info is None:
            info = self._levels[key] = self._config_info(config)
        return info

    def encode_flat(self, tensor: torch.Tensor, compact_tables=True) -> flat_format.FlatChunk:
        """The chunk as a CGB2 container on the GPU."""
        if self.fmt == "huggingface":
            tensor = tensor.permute(0, 1, 3, 2, 4)
        tensor = tensor.cuda()
        if tensor.stride(4) != 1:
            tensor = tensor.contiguous()
        return encode_flat(tensor, self._key_bins, self._value_bins, compact_tables, max_bins=self.table_max_bins,
                           delta=self.delta, info=self._bins())

    @_lmcache_nvtx_annotate
    def to_bytes(self, tensor: torch.Tensor) -> bytes:
        """KV blob ([L,2,T,H,D] for "vllm", [L,2,H,T,D] for "huggingface") -> bytes (enc.py:324-348):
        the reference's pickle, or a CGB2 container when wire_format == "flat"."""
        if self.wire_format == "flat":
            return self.encode_flat(tensor).tobytes()
        return self.encode(tensor).to_bytes()


_BINS_MAKERS = (CacheGenSerializer.make_key_bins, CacheGenSerializer.make_value_bins)
