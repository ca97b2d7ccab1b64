"""What csrc/cg_calls.cpp does, in Python, for where that module could not be built: the same entries with the same arguments and results,
through the same library.  A call takes 10 to 30 us longer on the host."""
import ctypes

import torch

from . import _lib

_DTYPES = {torch.float16: _lib.CG_F16, torch.bfloat16: _lib.CG_BF16}


def decode(*_):
    """No call is taken: DecodePlan decodes them all."""
    return None


def encode_start(job_at, kv, bins, max_bins, tail_at, workspace, row_off, counts_bytes, on, launch):
    L, _, T, H, D = kv.shape
    dev, lib, job = kv.device, _lib.lib(), _lib.EncodeKvJob.from_address(job_at)
    scales = counts = None
    if row_off is None:
        scales_k, scales_v = (torch.empty((L, T, 1), dtype=kv.dtype, device=dev) for _ in range(2))
    else:
        scales = torch.empty((2, L, T, 1), dtype=kv.dtype, device=dev)
        scales_k, scales_v = scales[0], scales[1]
    cdf = torch.empty((2 * L, H * D, max_bins + 1), dtype=torch.int16, device=dev)
    need = lib.cg_encode_kv_workspace(L, T, H, D)
    if need < 0:
        return (need,) + (None,) * 7
    if workspace is None or workspace.numel() < need:
        workspace = torch.empty(need, dtype=torch.uint8, device=dev)
    job.kv, job.bins, job.cdf = kv.data_ptr(), bins.data_ptr(), cdf.data_ptr()
    job.scales_k, job.scales_v = scales_k.data_ptr(), scales_v.data_ptr()
    if row_off is not None:
        counts = torch.empty(counts_bytes, dtype=torch.uint8, device=dev)
        job.counts, job.table_row_off = counts.data_ptr(), row_off.data_ptr()
    job.workspace, job.workspace_bytes, job.tail = workspace.data_ptr(), workspace.numel(), tail_at
    job.s_layer, job.s_kv, job.s_token, job.s_head, _ = kv.stride()
    job.dtype, job.nlayers, job.ntokens, job.nheads, job.head_size, job.max_bins = _DTYPES[kv.dtype], L, T, H, D, max_bins
    rc = 0
    with torch.cuda.device(dev):
        if on is None:
            on = torch.cuda.current_stream(dev).cuda_stream
        if launch:
            rc = lib.cg_encode_kv(ctypes.byref(job), on)
    return rc, on, scales, scales_k, scales_v, cdf, workspace, counts


def encode_finish(job_at, device_index, on, lengths):
    lib, job = _lib.lib(), _lib.EncodeKvJob.from_address(job_at)
    step = _lib.CG_MAX_TOKENS_PER_STREAM
    nsub = (job.ntokens + step - 1) // step
    with torch.cuda.device(device_index):
        rc = lib.cg_encode_kv_wait(ctypes.byref(job), on)
        if rc:
            return rc, None, None
        sizes, pieces = list((ctypes.c_int64 * (nsub + 3)).from_address(job.tail)), None
        if lengths is not None and not sizes[nsub + 1] & ~_lib.CG_S_COUNT_OVERFLOW:
            pieces = [torch.empty(sizes[k + 1] - sizes[k], dtype=torch.uint8, device=lengths[k].device) for k in range(nsub)]
            pointers = ctypes.c_void_p * nsub
            rc = lib.cg_encode_kv_gather(ctypes.byref(job), pointers(*[t.data_ptr() for t in pieces]),
                                         pointers(*[t.data_ptr() for t in lengths]), on)
    return rc, sizes, pieces
