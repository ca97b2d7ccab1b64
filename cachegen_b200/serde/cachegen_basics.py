"""CacheGenConfig and the wire dataclasses
(reference: LMCache/lmcache/storage_backend/serde/cachegen_basics.py:8-156).

The blob format is the reference's: `pickle` of a CacheGenGPUEncoderOutput whose tensors are CUDA
tensors.  So that blobs travel both ways between this package and the reference, the two wire
classes pickle under the reference's module path `lmcache.storage_backend.serde.cachegen_basics`;
when no `lmcache` package is importable, alias modules of that name are registered at import time
(see cachegen_b200.compat).
"""
import contextlib
import ctypes
import functools
import io
import os
import pickle
import sys
import threading
from collections import OrderedDict
from dataclasses import dataclass, replace
from typing import List

import torch

from .. import _lib

CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK = 256

REFERENCE_MODULE = "lmcache.storage_backend.serde.cachegen_basics"


@dataclass
class CacheGenConfig:
    """Per-layer-group bin counts: keys in three groups, values in two (cachegen_basics.py:10-21)."""
    key_first_layers: int
    key_second_layers: int
    key_third_layers: int
    key_first_bins: int
    key_second_bins: int
    key_third_bins: int
    value_first_layers: int
    value_first_bins: int
    value_second_bins: int

    def __getitem__(self, key: str) -> int:
        return getattr(self, key)

    @property
    def num_layers(self) -> int:
        return self.key_third_layers

    @property
    def max_bins(self) -> int:
        return max(self.key_first_bins, self.key_second_bins, self.key_third_bins,
                   self.value_first_bins, self.value_second_bins)

    def with_bins_divided(self, divisor: int, minimum: int = 4) -> "CacheGenConfig":
        """A lower quality level: every bin count divided by `divisor`, not below `minimum`."""
        d = lambda b: max(minimum, b // divisor)
        return replace(self, key_first_bins=d(self.key_first_bins), key_second_bins=d(self.key_second_bins),
                       key_third_bins=d(self.key_third_bins), value_first_bins=d(self.value_first_bins),
                       value_second_bins=d(self.value_second_bins))

    def layer_slice(self, start: int, stop: int) -> "CacheGenConfig":
        """The settings of layers [start, stop) as a configuration of their own (layer-sharded runs)."""
        n = stop - start
        if not 0 <= start < stop <= self.key_third_layers:
            raise ValueError(f"bad layer range [{start}, {stop}) of {self.key_third_layers}")
        clip = lambda b: min(max(b - start, 0), n)
        return replace(self, key_first_layers=clip(self.key_first_layers), key_second_layers=clip(self.key_second_layers),
                       key_third_layers=n, value_first_layers=clip(self.value_first_layers))

    @staticmethod
    def from_model_name(model_name: str) -> "CacheGenConfig":
        """Same lookup as cachegen_basics.py:23-96: any name containing "Mistral-7B" reads the
        QUANT_LEVEL environment variable ("1", "2" or "3"; KeyError when unset), the 7B and 70B
        families have fixed settings, anything else raises ValueError."""
        family_7b = ["mistralai/Mistral-7B-Instruct-v0.2", "mistral-community/Mistral-7B-v0.2",
                     "lmsys/longchat-7b-16k"]
        family_70b = ["Yukang/LongAlpaca-70B-16k"]
        if "Mistral-7B" in model_name:
            level = os.environ["QUANT_LEVEL"]
            if level == "1":
                return CacheGenConfig(10, 20, 32, 16, 16, 12, 2, 16, 12)
            if level == "2":
                return CacheGenConfig(10, 20, 32, 32, 16, 16, 2, 32, 16)
            if level == "3":
                return CacheGenConfig(10, 20, 32, 32, 32, 32, 2, 32, 32)
            raise ValueError(f"QUANT_LEVEL must be 1, 2 or 3, got {level!r}")
        elif model_name in family_7b:
            return CacheGenConfig(10, 20, 32, 32, 16, 16, 2, 32, 16)
        elif model_name in family_70b:
            return CacheGenConfig(20, 40, 80, 32, 32, 16, 20, 32, 16)
        else:
            raise ValueError(f"Model {model_name} is not supported")


class DeltaCoding:
    """Settings of anchor-token delta coding (cg_quantize_cdf_delta / cg_decode_dequant_delta; the
    reference has no such step, so chunks written with it are only readable by this package and only by a
    deserializer given the same settings).

    group:    tokens per group, a power of two in 2..256; the first token of a group is the anchor
    divisor:  residual tokens use max(4, bins // divisor) bins
    rows:     "keys" (key rows only: keys are the smooth ones) or "all"
    """

    def __init__(self, group: int, divisor: int = 2, rows: str = "keys"):
        if group < 2 or group > CACHEGEN_GPU_MAX_TOKENS_PER_CHUNK or group & (group - 1):
            raise ValueError(f"delta group must be a power of two in 2..256, got {group}")
        if divisor < 1:
            raise ValueError("delta divisor must be at least 1")
        if rows not in ("keys", "all"):
            raise ValueError(f"delta rows must be 'keys' or 'all', got {rows!r}")
        self.group, self.divisor, self.rows = int(group), int(divisor), rows
        self._res_bins = {}

    def residual_bins(self, key_bins: torch.Tensor, value_bins: torch.Tensor, device) -> torch.Tensor:
        """float32 [2L] on `device`: residual bin counts of the key rows then the value rows, 0 = no delta.  The
        result is kept by the bins' values, so tensors on a GPU are read back on every call."""
        kb, vb = key_bins.detach().cpu().float(), value_bins.detach().cpu().float()
        key = (str(device), tuple(kb.tolist()), tuple(vb.tolist()))
        t = self._res_bins.get(key)
        if t is None:
            res_k = torch.clamp(torch.div(kb, self.divisor, rounding_mode="floor"), min=4.0)
            res_v = torch.clamp(torch.div(vb, self.divisor, rounding_mode="floor"), min=4.0)
            if self.rows == "keys":
                res_v = torch.zeros_like(res_v)
            t = torch.cat((res_k, res_v)).to(device=device, dtype=torch.float32).contiguous()
            self._res_bins[key] = t
        return t

    def __repr__(self):
        return f"DeltaCoding(group={self.group}, divisor={self.divisor}, rows={self.rows!r})"


def make_key_bins(config: CacheGenConfig, device="cuda") -> torch.Tensor:
    """float32 [L] (cachegen_encoder.py:311-316 / cachegen_decoder.py:122-127)."""
    ret = torch.zeros(config.key_third_layers)
    ret.fill_(config.key_third_bins)
    ret[:config.key_second_layers] = config.key_second_bins
    ret[:config.key_first_layers] = config.key_first_bins
    return ret.to(device)


def make_value_bins(config: CacheGenConfig, device="cuda") -> torch.Tensor:
    """float32 [L] (cachegen_encoder.py:318-322 / cachegen_decoder.py:129-135)."""
    ret = torch.zeros(config.key_third_layers)
    ret.fill_(config.value_second_bins)
    ret[:config.value_first_layers] = config.value_first_bins
    return ret.to(device)


@dataclass
class CacheGenGPUBytestream:
    """One sub-chunk (<= 256 tokens) of encoded streams (cachegen_basics.py:124-131)."""
    bytestream: torch.Tensor          # uint8 [sum of lengths]: streams in (row, channel) order
    bytestream_lengths: torch.Tensor  # int32 [2L, C]
    ntokens: int

    def __getitem__(self, key: str):
        return getattr(self, key)


@dataclass
class CacheGenGPUEncoderOutput:
    """One encoded chunk (cachegen_basics.py:133-156)."""
    data_chunks: List[CacheGenGPUBytestream]
    cdf: torch.Tensor                # int16 [2L, C, Lp]
    max_tensors_key: torch.Tensor    # [L, T, 1], input dtype
    max_tensors_value: torch.Tensor  # [L, T, 1], input dtype
    num_heads: int
    head_size: int

    def __getitem__(self, key: str):
        return getattr(self, key)

    def to_bytes(self) -> bytes:
        try:
            return dump_blob(self)
        except Exception:
            # dump_blob follows torch's legacy storage stream by hand; should a torch release change
            # that format, the plain pickle is still the reference's blob (slower: torch copies every
            # CUDA tensor through pageable memory)
            f = io.BytesIO()
            pickle.dump(self, f)
            return f.getvalue()

    @staticmethod
    def from_bytes(bs: bytes) -> "CacheGenGPUEncoderOutput":
        return load_blob(bs)


# ---- writing a blob ---------------------------------------------------------------------------------------
# pickle.dump of the object gives the reference's blob, but torch pickles a CUDA tensor by copying
# its storage to pageable host memory, writing a legacy `torch.save` stream of it into one buffer,
# copying that into the pickle and the pickle into the result: 34 ms for a 30 MB chunk.  dump_blob
# writes the same bytes -- the same outer pickle, and for each storage the same legacy stream, built
# by _legacy_stream_head.  The outer pickle is made with placeholders of the storages' sizes while the tensors
# are on their way into pinned memory, and every tensor's bytes are copied once, from there to their place in
# the result, by several threads as they arrive (cg_host_download).

class _PersistentId:
    def __init__(self, pid):
        self.pid = pid


class _LegacyPickler(pickle.Pickler):
    def persistent_id(self, obj):
        return obj.pid if isinstance(obj, _PersistentId) else None


def _legacy_preamble() -> bytes:
    """Magic number, protocol version and system info of a legacy stream, as three pickles."""
    ser = torch.serialization
    info = {"protocol_version": ser.PROTOCOL_VERSION, "little_endian": sys.byteorder == "little",
            "type_sizes": {"short": ser.SHORT_SIZE, "int": ser.INT_SIZE, "long": ser.LONG_SIZE}}
    return b"".join(pickle.dumps(part, protocol=ser.DEFAULT_PROTOCOL)
                    for part in (ser.MAGIC_NUMBER, ser.PROTOCOL_VERSION, info))


def _pickle_stream_head(dtype: torch.dtype, key: str, location: str, numel: int) -> bytes:
    """What torch.save(storage, f, _use_new_zipfile_serialization=False) writes before the storage's
    raw data (torch/serialization.py, _legacy_save): the preamble, the storage as a persistent id, the list
    of storage keys, the element count."""
    f = io.BytesIO()
    f.write(_legacy_preamble())
    storage_type = getattr(torch, torch.storage._dtype_to_storage_type_map()[dtype])
    _LegacyPickler(f, protocol=torch.serialization.DEFAULT_PROTOCOL).dump(
        _PersistentId(("storage", storage_type, key, location, numel, None)))
    pickle.dump([key], f, protocol=torch.serialization.DEFAULT_PROTOCOL)
    f.write(int(numel).to_bytes(8, sys.byteorder))
    return f.getvalue()


_HEAD_PARTS = {}  # (dtype, location) -> the constant pieces of a head around its key, element count and key
_KEY, _COUNT = "<a storage's key>", 0x01234567


def _pickled_str(v: str) -> bytes:
    raw = v.encode("utf-8", "surrogatepass")
    return b"X" + len(raw).to_bytes(4, "little") + raw


def _pickled_int(v: int) -> bytes:
    return pickle.dumps(v, protocol=torch.serialization.DEFAULT_PROTOCOL)[2:-1]


def _legacy_stream_head(dtype: torch.dtype, key: str, location: str, numel: int) -> bytes:
    """_pickle_stream_head's bytes, put together from the pieces of one made before."""
    parts = _HEAD_PARTS.get((dtype, location))
    if parts is None:
        sample = _pickle_stream_head(dtype, _KEY, location, _COUNT)[:-8]
        before, between, after = sample.split(_pickled_str(_KEY))
        first, second = between.split(_pickled_int(_COUNT))
        parts = _HEAD_PARTS[dtype, location] = (before, first, second, after)
    k = _pickled_str(key)
    return b"".join((parts[0], k, parts[1], _pickled_int(numel), parts[2], k, parts[3], int(numel).to_bytes(8, sys.byteorder)))


class _StreamedStorage:
    """Stands in for a tensor's TypedStorage while pickling: reduces to what the storage itself
    reduces to, (torch.storage._load_from_bytes, (legacy stream,))."""

    def __init__(self, stream: bytes):
        self.stream = stream

    def __reduce__(self):
        return (torch.storage._load_from_bytes, (self.stream,))


def _owns_its_storage(t: torch.Tensor) -> bool:
    return (t.layout == torch.strided and t.is_contiguous() and t.storage_offset() == 0 and not t.requires_grad and
            type(t) is torch.Tensor and t.untyped_storage().nbytes() == t.numel() * t.element_size() and
            t.dtype in torch.storage._dtype_to_storage_type_map())


_PLACEHOLDER_LEN = 1 << 16  # pickle writes byte strings of at least this size outside its frames


class _BlobPickler(pickle.Pickler):
    """Pickles the tensors in `sizes` (id -> bytes of raw data) with a placeholder for their storage stream;
    everything else as pickle.dump does.  A placeholder of _PLACEHOLDER_LEN bytes stands for a stream of at
    least that size (pickle frames both the same way: outside the frames) and reaches the file as the object
    it is; a smaller one is as long as its stream and is found again by the marker it starts with.
    `streams` lists (placeholder, head, tensor, stream length) in the order written."""

    def __init__(self, file, sizes: dict):
        super().__init__(file)
        self.sizes = sizes
        self.streams = []

    def reducer_override(self, obj):
        if isinstance(obj, torch.Tensor) and id(obj) in self.sizes:
            head = _legacy_stream_head(obj.dtype, str(obj.untyped_storage()._cdata),
                                       torch.serialization.location_tag(obj.untyped_storage()), obj.numel())
            n = len(head) + self.sizes[id(obj)]
            if n >= 1 << 32:
                return NotImplemented  # another opcode: left to torch
            marker = _MARKER + len(self.streams).to_bytes(4, "little")
            stream = bytes(_PLACEHOLDER_LEN) if n >= _PLACEHOLDER_LEN else marker + bytes(n - len(marker))
            self.streams.append((stream, head, obj, n))
            return (torch._utils._rebuild_tensor_v2,
                    (_StreamedStorage(stream), 0, tuple(obj.size()), obj.stride(), False, OrderedDict()))
        return NotImplemented


_MARKER = bytes.fromhex("e1f7c36a905d4b2887d21e5cb0394fa6")


class _PartsWriter:
    """File object that keeps what is written as a list of byte strings: the pickler hands a large
    byte string over as the object it was given, so nothing is copied until the blob is put together."""

    def __init__(self):
        self.parts = []

    def write(self, b):
        self.parts.append(b if isinstance(b, bytes) else bytes(b))
        return len(b)


def _place_streams(parts: list, streams: list):
    """Where everything goes: ([(offset, bytes)] of the pickle itself and the streams' heads, [(offset, tensor)]
    of the streams' raw data, total size), every placeholder replaced by its stream and the 4-byte
    length before a large one corrected."""
    large = {id(s[0]): s for s in streams if len(s[0]) == _PLACEHOLDER_LEN}
    small = [(i, s) for i, s in enumerate(streams) if len(s[0]) < _PLACEHOLDER_LEN]
    fixed, raw, pos, last = [], [], 0, -1  # last: the pickle's own piece before
    for part in parts:
        d = large.get(id(part))
        if d is not None:
            _, head, t, n = d
            at, before = fixed[last] if last >= 0 else (0, b"")
            # BINBYTES + length, the last thing written before the payload
            if at + len(before) != pos or not before.endswith(b"B" + _PLACEHOLDER_LEN.to_bytes(4, "little")):
                raise RuntimeError("unexpected pickle layout around a storage stream")
            fixed[last] = (at, before[:-4] + n.to_bytes(4, "little"))
            fixed.append((pos, head))
            raw.append((pos + len(head), t))
            pos += n
            continue
        last = len(fixed)
        fixed.append((pos, part))
        k = 0
        while small:
            i, (stream, head, t, n) = small[0]
            k = part.find(_MARKER + i.to_bytes(4, "little"), k)
            if k < 0:
                break
            fixed.append((pos + k, head))
            raw.append((pos + k + len(head), t))
            small.pop(0)
            k += n
        pos += len(part)
    if small or len(raw) != len(streams):
        raise RuntimeError("a storage stream's placeholder is missing from the pickle")
    return fixed, raw, pos


_bytes_new = ctypes.pythonapi.PyBytes_FromStringAndSize
_bytes_new.restype, _bytes_new.argtypes = ctypes.py_object, [ctypes.c_char_p, ctypes.c_ssize_t]
_bytes_at = ctypes.pythonapi.PyBytes_AsString
_bytes_at.restype, _bytes_at.argtypes = ctypes.c_void_p, [ctypes.py_object]


class BytesView:
    """A byte string where a uint8 tensor over its bytes is expected for its address and size."""

    def __init__(self, bs: bytes):
        self.bs = bs

    def data_ptr(self) -> int:
        return _bytes_at(self.bs)

    def numel(self) -> int:
        return len(self.bs)

    def to(self, device) -> torch.Tensor:
        return torch.frombuffer(bytearray(self.bs), dtype=torch.uint8).to(device)


def dump_blob(eo: "CacheGenGPUEncoderOutput") -> bytes:
    """The pickle of an encoded chunk, byte for byte what pickle.dump writes (cachegen_basics.py:146-151).
    Tensors that own their storage have their legacy streams built here; the others are left to torch."""
    tensors = [eo.cdf, eo.max_tensors_key, eo.max_tensors_value]
    for dc in eo.data_chunks:
        tensors += [dc.bytestream, dc.bytestream_lengths]
    sizes = {id(t): t.numel() * t.element_size() for t in tensors if isinstance(t, torch.Tensor) and _owns_its_storage(t)}
    devices = {t.device for t in tensors if id(t) in sizes and t.is_cuda}
    if len(devices) > 1:  # one stream carries the transfers: the tensors of another GPU are left to torch
        sizes = {id(t): sizes[id(t)] for t in tensors if id(t) in sizes and (not t.is_cuda or t.device == tensors[0].device)}
    on_gpu = [t for t in tensors if id(t) in sizes and t.is_cuda and t.numel()]
    st = staging()
    try:
        if on_gpu:
            st.fetch(on_gpu)
        out = _PartsWriter()
        pickler = _BlobPickler(out, sizes)
        pickler.dump(eo)
        fixed, raw, total = _place_streams(out.parts, pickler.streams)
        blob = _bytes_new(None, total)  # uninitialised, ours alone until it is returned
        base = _bytes_at(blob)
        for at, piece in fixed:
            ctypes.memmove(base + at, piece, len(piece))
        where = {id(t): base + at for at, t in raw}
        for at, t in raw:
            if not t.is_cuda and t.numel():
                ctypes.memmove(base + at, t.data_ptr(), sizes[id(t)])
    except BaseException:
        st.cancel()
        raise
    if on_gpu:
        st.collect([where[id(t)] for t in on_gpu])
    return blob


# `CacheGenEncoderOutput.from_bytes` is what the reference's tests call on a blob
# (LMCache/tests/test_serde.py:43); with pickle it is the same loader.
CacheGenEncoderOutput = CacheGenGPUEncoderOutput


class _StorageRecord(pickle.Unpickler):
    """Reads the one persistent id of a torch legacy storage stream without building the storage."""

    def __init__(self, f):
        super().__init__(f)
        self.seen = []

    def persistent_load(self, saved_id):
        self.seen.append(saved_id)
        return None


def _load_storage_from_bytes(b: bytes):
    """Replacement for torch.storage._load_from_bytes while unpickling a blob.

    Pickling a tensor stores its storage as the bytes of a legacy `torch.save` stream: three small
    pickles (magic, protocol, system info), the pickled storage whose persistent id names type,
    location and size, the list of storage keys, then an int64 element count and the raw data.
    torch's loader copies that data into a CPU storage and then to the GPU; here the data is viewed
    in place inside `b` and copied once, straight to its device.  Anything unexpected falls back to
    torch's own loader."""
    import warnings
    try:
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")  # TypedStorage deprecation notes; read-only buffer note
            return _load_storage_fast(b)
    except Exception:
        return torch.storage._load_from_bytes(bytes(b))


_HEAD_START = _legacy_preamble() + b"\x80\x02(X\x07\x00\x00\x00storageq\x00ctorch\n"
_INT_SIZES = {75: 1, 77: 2, 74: 4}  # BININT1, BININT2, BININT


def _read_stream_head(b):
    """(storage class name, location, element count, offset of the raw data) of a legacy stream as
    _pickle_stream_head writes it, or None."""
    head = bytes(b[:1024])
    at = len(_HEAD_START)
    end = head.find(b"\n", at)
    if head[:at] != _HEAD_START or end < 0 or head[end + 1:end + 4] != b"q\x01X":
        return None
    name = head[at:end]
    at = end + 8 + int.from_bytes(head[end + 4:end + 8], "little")
    key = head[end + 3:at]
    n = int.from_bytes(head[at + 3:at + 7], "little")
    location = head[at + 7:at + 7 + n]
    if head[at:at + 3] != b"q\x02X" or head[at + 7 + n:at + 9 + n] != b"q\x03":
        return None
    at += 9 + n
    size = _INT_SIZES.get(head[at]) if at < len(head) else None
    if size is None:
        return None
    numel = int.from_bytes(head[at + 1:at + 1 + size], "little")
    tail = b"Ntq\x04Q.\x80\x02]q\x00" + key + b"q\x01a." + numel.to_bytes(8, "little")
    at += 1 + size
    if head[at:at + len(tail)] != tail:
        return None
    return name.decode(), location.decode(), numel, at + len(tail)


def _parse_stream_head(b):
    """The same from any legacy stream, by unpickling its parts; raises what it cannot read."""
    f = io.BytesIO(bytes(b[:1 << 16]))  # the stream's head: small pickles, then the raw data (b may be a view)
    if pickle.load(f) != torch.serialization.MAGIC_NUMBER or pickle.load(f) != torch.serialization.PROTOCOL_VERSION:
        raise ValueError("not a legacy stream")
    info = pickle.load(f)
    if not info.get("little_endian", True):
        raise ValueError("big-endian stream")
    rec = _StorageRecord(f)
    rec.load()
    keys = pickle.load(f)
    if len(rec.seen) != 1 or len(keys) != 1:
        raise ValueError("more than one storage")
    typename, storage_type, key, location, numel, view = rec.seen[0]
    if typename != "storage" or view is not None or keys[0] != key:
        raise ValueError("storage view")
    off = f.tell()
    if off + 8 > min(len(b), 1 << 16):
        raise ValueError("header too long")
    if int.from_bytes(b[off:off + 8], "little") != numel:
        raise ValueError("size mismatch")
    return storage_type.__name__, location, numel, off + 8


def _load_storage_fast(b):
    name, location, numel, off = _read_stream_head(b) or _parse_stream_head(b)
    storage_type = getattr(torch, name)
    dtype = torch.uint8 if storage_type is torch.UntypedStorage else storage_type.dtype
    nbytes = numel * torch._utils._element_size(dtype)
    if off + nbytes != len(b):
        raise ValueError("size mismatch")
    device = torch.device(location)
    if device.type == "cuda" and not (torch.cuda.is_available() and (device.index or 0) < torch.cuda.device_count()):
        raise ValueError("device not present")
    if nbytes == 0:
        raw = torch.empty(0, dtype=torch.uint8, device=device)
    else:
        view_cpu = torch.frombuffer(b, dtype=torch.uint8, count=nbytes, offset=off)  # read-only, only read
        if device.type == "cpu":
            raw = view_cpu.clone()
        else:
            raw = staging().to_device(view_cpu, device)
    return torch.storage.TypedStorage(wrap_storage=raw.untyped_storage(), dtype=dtype, _internal=True)


_NOTHING = contextlib.nullcontext()
_EARLY_SPARE = 256 << 10  # room behind the byte string for tensors that are not part of it
_AHEAD_SPARE = 64  # room behind a byte string that is sent as it is
_EARLY_FROM = 2 << 20  # below, parsing and copying take less time than the threads take to wake


def on_device(dev):
    """Context in which `dev` is the current device; nothing to do in the usual case."""
    return _NOTHING if torch.cuda.current_device() == dev.index else torch.cuda.device(dev)


class _Staging:
    """Pinned host memory that a thread's blob loads and dumps pass through: bytes are copied into it
    by several threads and leave it by asynchronous copies on the current stream (or arrive in it from
    the GPU), several times faster than a copy to or from pageable memory (cg_host_upload,
    cg_host_download).  Two buffers per thread, used in turn and grown on demand, so that filling one overlaps
    the copies still leaving the other; `begin` waits until the chosen buffer's last copies are done."""

    def __init__(self):
        self.bufs = [None, None]
        self.events = [None, None]     # (device, event) of each buffer's last copies, recorded again and again
        self.leaving = [False, False]  # whether that event may still be outstanding
        self.turn = 0
        self.buf = None
        self.waiting = None  # (host view, device tensor) pairs of the load in progress
        self.early = None    # (handle, address, size, _Ahead or None) of a byte string whose copy runs ahead of its parsing
        self.fetched = None  # the tensors whose transfers into the chosen buffer are on their way, and their stream
        self.fetching = None

    def begin(self, nbytes: int) -> None:
        self.turn ^= 1
        i = self.turn
        if self.leaving[i]:
            self.events[i][1].synchronize()
            self.leaving[i] = False
        if self.bufs[i] is None or self.bufs[i].numel() < nbytes:
            self.bufs[i] = None
            # an eighth to spare: payloads differ from chunk to chunk, and pinning 30 MB takes 28 ms
            self.bufs[i] = torch.empty(max(nbytes + nbytes // 8, 1 << 20), dtype=torch.uint8,
                                       pin_memory=torch.cuda.is_available())
        self.buf = self.bufs[i]

    def end(self) -> None:
        self.buf = None

    def __del__(self):
        # the thread has ended: torch would give its buffers to others while copies may still leave them
        for i in range(2):
            if self.leaving[i]:
                try:
                    self.events[i][1].synchronize()
                except Exception:
                    pass  # the process is ending, or the GPU has failed: nobody gets the memory

    # -- to the GPU: a load collects the tensors it makes, and sends them together
    def open(self) -> None:
        self.waiting = []

    def to_device(self, view_cpu: torch.Tensor, device) -> torch.Tensor:
        if self.waiting is None:
            return view_cpu.to(device)  # no load in progress
        out = torch.empty(view_cpu.numel(), dtype=torch.uint8, device=device)
        self.waiting.append((view_cpu.data_ptr(), view_cpu.numel(), out, view_cpu))
        return out

    def start(self, bs: bytes, ahead: bool = False) -> None:
        """Has the helper threads copy a byte string that is about to be parsed, from _EARLY_FROM bytes on: parsing a
        blob takes 130 to 200 us, as long as a third of its 30 MB take over the bus, and waking the threads 50.
        ahead: one of them sends it to the current GPU as well, on the current stream, and the tensors are cut out of it
        there (a 256-token chunk to pickled bytes and back 2,070 -> 1,940 us; several blobs after each other keep the bus
        busy as it is).  Until they are, the GPU holds the blob's size (30 MB) beside them.  Only for a blob whose first
        tensor belongs there: what is to stay on the host, or goes to another GPU, would be sent for nothing."""
        if len(bs) < _EARLY_FROM or not torch.cuda.is_available():
            return
        where = _blob_location(bs)
        if where == "cpu":
            return
        device = torch.device("cuda", torch.cuda.current_device())
        on, raw = torch.cuda.current_stream(device), None
        if ahead and where == str(device) and not torch.cuda.is_current_stream_capturing():
            try:
                raw = torch.empty(len(bs) + _AHEAD_SPARE, dtype=torch.uint8, device=device)
            except torch.cuda.OutOfMemoryError:
                pass  # the tensors alone may fit
        self.begin(len(bs) + _EARLY_SPARE)
        handle, at = ctypes.c_void_p(), _bytes_at(bs)
        lib, args = _lib.lib(), (at, len(bs), self.buf.data_ptr(), self.buf.numel())
        if raw is None:
            _lib.check(lib.cg_host_stage(*args, ctypes.byref(handle)), "cg_host_stage")
        else:
            _lib.check(lib.cg_host_stage_ahead(*args, raw.data_ptr(), on.cuda_stream, ctypes.byref(handle)), "cg_host_stage_ahead")
        self.early = (handle, at, len(bs), None if raw is None else (raw, device, on))

    def _send_early(self, pairs: list, stream) -> list:
        """Sends the tensors that lie in the byte string of `start`, and small ones beside it (a blob's scales: the
        unpickler copies short streams), if they are on one GPU; returns the others."""
        handle, at, size, ahead = self.early
        mine, others, spare = [], [], _EARLY_SPARE - 256
        for p in pairs:
            if not at <= p[0] < at + size:
                spare -= (p[1] + 255) // 256 * 256
                if spare < 0:
                    others.append(p)
                    continue
            mine.append(p)
        try:
            if not mine or any(p[2].device != mine[0][2].device for p in mine):
                return pairs
            if ahead is not None and (mine[0][2].device != ahead[1] or self._stream_for(ahead[1], stream) != ahead[2]):
                return pairs  # it went elsewhere
            segs = (_lib.HostSegment * len(mine))(*[(a, o.data_ptr(), n) for a, n, o, _ in mine])
            self._send(lambda on: _lib.lib().cg_host_stage_send(handle, segs, len(mine), on), mine[0][2].device, stream)
        finally:
            self.finish()
        return others

    def finish(self) -> None:
        """Ends a `start` whose bytes are not wanted (any more)."""
        if self.early is not None:
            (handle, _, _, ahead), self.early = self.early, None
            _lib.lib().cg_host_stage_end(handle)
            if ahead is not None:  # transfers that were begun still read the buffer, wanted or not
                self._mark(ahead[1], ahead[2])
            self.end()

    @staticmethod
    def _stream_for(device, stream):
        return torch.cuda.current_stream(device) if stream is None or stream.device != device else stream

    def _mark(self, device, on) -> None:
        """Notes that copies from the chosen buffer may be on this stream."""
        if self.events[self.turn] is None or self.events[self.turn][0] != device:
            self.events[self.turn] = (device, torch.cuda.Event())
        with on_device(device):
            self.events[self.turn][1].record(on)
        self.leaving[self.turn] = True

    def _send(self, upload, device, stream) -> None:
        """Runs an upload from the chosen buffer on `stream`, if it is one of the device's, or its current one."""
        with on_device(device):
            on = self._stream_for(device, stream)
            try:
                rc = upload(on.cuda_stream)
            finally:
                self._mark(device, on)
        _lib.check(rc, "cg_host_upload")

    def send(self, pairs: list = None, stream=None) -> None:
        """The collected tensors' bytes (or another load's) on their way, in the order they were made; on `stream`,
        or each device's current one."""
        if pairs is None:
            pairs, self.waiting = self.waiting, None
        if self.early is not None:
            pairs = self._send_early(pairs, stream)
        while pairs:
            device = pairs[0][2].device
            mine = [p for p in pairs if p[2].device == device]
            pairs = [p for p in pairs if p[2].device != device]
            segs = (_lib.HostSegment * len(mine))(*[(at, o.data_ptr(), n) for at, n, o, _ in mine])
            self.begin(sum((n + 255) // 256 * 256 for _, n, _, _ in mine))
            try:
                self._send(lambda on: _lib.lib().cg_host_upload(segs, len(mine), self.buf.data_ptr(), self.buf.numel(), on),
                           device, stream)
            finally:
                self.end()

    def drop(self) -> None:
        """Forgets a load that failed, or that another send takes over."""
        self.waiting = None

    def whole_to_device(self, view_cpu: torch.Tensor, device) -> torch.Tensor:
        """One host buffer (any memory) to the GPU through the staging memory."""
        n = view_cpu.numel()
        out = torch.empty(n, dtype=torch.uint8, device=device)
        if n:
            seg = _lib.HostSegment(view_cpu.data_ptr(), out.data_ptr(), n)
            self.begin((n + 255) // 256 * 256)
            try:
                self._send(lambda on: _lib.lib().cg_host_upload(ctypes.byref(seg), 1, self.buf.data_ptr(), self.buf.numel(), on),
                           out.device, None)
            finally:
                self.end()
        return out

    # -- from the GPU
    def fetch(self, tensors: list) -> None:
        """Enqueues the transfers of contiguous tensors of one GPU; `collect` does the rest."""
        sizes = [t.numel() * t.element_size() for t in tensors]
        self.segs = (_lib.HostSegment * len(tensors))(*[(None, t.data_ptr(), n) for t, n in zip(tensors, sizes)])
        self.begin(sum((n + 255) // 256 * 256 for n in sizes))
        self.fetched, self.fetching = tensors, torch.cuda.current_stream(tensors[0].device)
        try:
            self._download(1)
        except BaseException:
            self.cancel()
            raise

    def collect(self, pointers: list) -> None:
        """The bytes of the fetched tensors to these addresses."""
        try:
            for seg, at in zip(self.segs, pointers):
                seg.host = at
            self._download(2)
        except BaseException:
            self.cancel()
            raise
        self.fetched = self.fetching = None
        self.end()

    def cancel(self) -> None:
        """Ends a fetch whose bytes are not wanted (any more): waits for the transfers that still write to the buffer."""
        if self.fetched is not None:
            self.fetching.synchronize()
            self.fetched = self.fetching = None
        self.end()

    def _download(self, phase: int) -> None:
        with on_device(self.fetched[0].device):
            rc = _lib.lib().cg_host_download(self.segs, len(self.segs), self.buf.data_ptr(), self.buf.numel(), phase,
                                             self.fetching.cuda_stream)
        _lib.check(rc, "cg_host_download")

    def whole_from_device(self, t: torch.Tensor) -> bytes:
        """The bytes of a contiguous GPU tensor."""
        n = t.numel() * t.element_size()
        out = _bytes_new(None, n)
        seg = _lib.HostSegment(_bytes_at(out), t.data_ptr(), n)
        self.begin((n + 255) // 256 * 256)
        try:
            with on_device(t.device):
                on = torch.cuda.current_stream(t.device)
                try:
                    rc = _lib.lib().cg_host_download(ctypes.byref(seg), 1, self.buf.data_ptr(), self.buf.numel(), 0, on.cuda_stream)
                    _lib.check(rc, "cg_host_download")
                except BaseException:
                    on.synchronize()  # transfers may still write to the buffer
                    raise
        finally:
            self.end()
        return out


_staging_local = threading.local()


def staging() -> _Staging:
    st = getattr(_staging_local, "staging", None)
    if st is None:
        st = _staging_local.staging = _Staging()
    return st


class _ViewReader:
    """File-like reader over a bytes-like object that hands large reads out as memoryview slices
    (no copy) and small ones as bytes."""

    def __init__(self, data):
        self.mv = memoryview(data)
        self.pos = 0

    def read(self, n: int = -1):
        if n is None or n < 0:
            n = len(self.mv) - self.pos
        piece = self.mv[self.pos:self.pos + n]
        self.pos += len(piece)
        return piece if len(piece) >= (1 << 16) else bytes(piece)

    def readline(self):
        end = self.pos
        while end < len(self.mv) and self.mv[end] != 10:
            end += 1
        end = min(end + 1, len(self.mv))
        piece = bytes(self.mv[self.pos:end])
        self.pos = end
        return piece


def _find_wire_class(module, name):
    if name in ("CacheGenGPUEncoderOutput", "CacheGenGPUBytestream") and module in (REFERENCE_MODULE, __name__):
        return globals()[name]
    if module == "torch.storage" and name == "_load_from_bytes":
        return _load_storage_from_bytes
    return None


class _Unpickler(pickle.Unpickler):
    """pickle loader that resolves the two wire classes to this module, whichever module path the
    blob was written under, and reads tensor storages with one copy (see _load_storage_from_bytes)."""

    def find_class(self, module, name):
        return _find_wire_class(module, name) or super().find_class(module, name)


class _ViewUnpickler(pickle._Unpickler):
    """The same loader on the standard library's Python unpickler reading through a _ViewReader: the
    blob's large byte strings (the pickled tensor storages) reach _load_storage_from_bytes as views
    of the blob instead of copies.  A blob has a few hundred opcodes, so the interpreter's speed
    does not matter; copying its 30 MB once more does."""

    def __init__(self, data):
        super().__init__(_ViewReader(data))

    def find_class(self, module, name):
        return _find_wire_class(module, name) or super().find_class(module, name)


_MAGIC_PICKLE = pickle.dumps(torch.serialization.MAGIC_NUMBER, protocol=torch.serialization.DEFAULT_PROTOCOL)
_TOKEN = b"cachegen storage"


def _cut_streams(bs: bytes):
    """The pickle with its large storage streams cut out, and those streams: ([bytes of the pickle, a token in
    place of each stream], {token: (offset, view) of the stream}).  A legacy stream starts with torch's magic number, and
    the four bytes before it, behind the BINBYTES opcode, are its length; the search goes on behind it, so
    that the tensors' own bytes are never looked at."""
    view, pieces, streams, start, at = memoryview(bs), [], {}, 0, 0
    while True:
        p = bs.find(_MAGIC_PICKLE, at)
        if p < 0:
            break
        at = p + 1
        if p < 5 or bs[p - 5] != 66:  # BINBYTES; another opcode stays as it is
            continue
        n = int.from_bytes(bs[p - 4:p], "little")
        if p + n > len(bs):
            raise ValueError("truncated storage stream")
        at = p + n
        if n < _PLACEHOLDER_LEN:
            continue  # inside a frame of the pickle, whose length counts it
        token = _TOKEN + len(streams).to_bytes(4, "little")
        streams[token] = (p, view[p:p + n])
        pieces += [bs[start:p - 4], len(token).to_bytes(4, "little"), token]
        start = p + n
    pieces.append(bs[start:])
    return b"".join(pieces), streams


_STORAGE_DTYPES = {name: dtype for dtype, name in torch.storage._dtype_to_storage_type_map().items()}
_dtype_of = _STORAGE_DTYPES.get


def _blob_location(bs: bytes):
    """The device that a blob's first storage names ("cpu", "cuda:0"); None if the blob does not start as one does."""
    at = bs.find(_MAGIC_PICKLE, 0, _FIRST_STREAM_WITHIN)
    head = _read_stream_head(memoryview(bs)[at:at + 1024]) if at >= 0 else None
    return head[1] if head else None


_FIRST_STREAM_WITHIN = 4096  # the names of a blob's classes and fields come first, a few hundred bytes


class _CudaStream:
    """A storage on a GPU whose bytes are still in the blob."""

    def __init__(self, at, dtype, numel, device, view):
        self.at, self.dtype, self.numel, self.device, self.view = at, dtype, numel, device, view


def _stream_storage(streams, base, b):
    """What a pickled storage is: its bytes b, or a token in place of a stream that was cut out."""
    at, stream = streams.get(b, (0, b))
    head = _read_stream_head(stream) if at and torch.cuda.is_available() else None
    if head is not None and head[1].startswith("cuda"):
        name, location, numel, off = head
        dtype = _dtype_of(name)
        device = torch.device(location)
        if (dtype is not None and off + numel * dtype.itemsize == len(stream) and numel and
                (device.index or 0) < torch.cuda.device_count()):
            return _CudaStream(base + at + off, dtype, numel, device, stream)
    return _load_storage_from_bytes(stream)


def _stream_tensor(storage, offset, size, stride, requires_grad, hooks, metadata=None):
    """torch._utils._rebuild_tensor_v2 on what _stream_storage gives."""
    if isinstance(storage, _CudaStream):
        if offset == 0 and not requires_grad and metadata is None:
            t = torch.empty(size, dtype=storage.dtype, device=storage.device)
            if t.numel() == storage.numel and t.stride() == stride:
                staging().waiting.append((storage.at, storage.numel * t.element_size(), t, storage.view))
                return t
        storage = _load_storage_from_bytes(storage.view)
    return torch._utils._rebuild_tensor_v2(storage, offset, size, stride, requires_grad, hooks, metadata)


class _CutUnpickler(pickle.Unpickler):
    """The loader for a pickle whose large streams were cut out: on the C unpickler, which would copy them.
    What it puts in its memo must not refer back to it: the cycle would keep the blob until a collection."""

    def __init__(self, bs: bytes):
        skeleton, streams = _cut_streams(bs)
        self.storage = functools.partial(_stream_storage, streams, _bytes_at(bs))
        super().__init__(io.BytesIO(skeleton))

    def find_class(self, module, name):
        if module == "torch.storage" and name == "_load_from_bytes":
            return self.storage
        if module == "torch._utils" and name == "_rebuild_tensor_v2":
            return _stream_tensor
        return _find_wire_class(module, name) or super().find_class(module, name)


def _unpickle(bs):
    """The object in a blob, its tensors collected in the open staging load."""
    if isinstance(bs, bytes):
        try:
            return _CutUnpickler(bs).load()
        except Exception:
            staging().open()
    try:
        return _ViewUnpickler(bs).load()
    except Exception:
        staging().open()
    with io.BytesIO(bs) as f:
        return _Unpickler(f).load()


class BlobLoad:
    """One blob parsed, its tensors made, but their bytes not yet sent: parsing and sending may be done by two
    threads.  unpickle / flat inside the `with`, send after it."""

    def __enter__(self):
        staging().open()
        return self

    def __exit__(self, *exc):
        self.pairs = staging().waiting
        staging().drop()

    def unpickle(self, bs):
        return _unpickle(bs)

    def flat(self, buf, device):
        from . import flat_format
        return flat_format.wrap(buf, lambda view: staging().to_device(view, device))

    def send(self, stream) -> None:
        staging().send(self.pairs, stream)


def load_blob(bs):
    """Unpickles a CacheGenGPUEncoderOutput written by this package or by the reference."""
    st = staging()
    st.open()
    try:
        if isinstance(bs, bytes):
            st.start(bs, ahead=True)
        eo = _unpickle(bs)
        st.send()
    finally:
        st.drop()
        st.finish()
    return eo


def _adopt_reference_module_path():
    from .. import compat
    if compat.install_wire_aliases(__name__):
        CacheGenGPUBytestream.__module__ = REFERENCE_MODULE
        CacheGenGPUEncoderOutput.__module__ = REFERENCE_MODULE


_adopt_reference_module_path()
