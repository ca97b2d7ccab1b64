"""Argument checks of the calls for several bin settings; nothing is launched."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from cachegen_b200 import _lib
    return _lib.lib()


def jobs_of(lib, n):
    from cachegen_b200 import _lib
    jobs = (_lib.EncodeKvJob * n)()
    need = lib.cg_encode_kv_workspace(1, 4, 1, 8)
    for j in jobs:
        j.kv = j.bins = j.scales_k = j.scales_v = j.cdf = j.workspace = j.tail = 256
        j.workspace_bytes = need
        j.nlayers, j.ntokens, j.nheads, j.head_size, j.max_bins = 1, 4, 1, 8, 32
    return jobs


def test_levels_arguments(lib):
    from cachegen_b200 import _lib
    most = _lib.CG_MAX_ENCODE_LEVELS
    for call in (lib.cg_encode_kv_levels, lambda j, n, s: lib.cg_encode_kv_levels_gather(j, n, None, None, s)):
        assert call(None, 1, None) == -1
        assert call(jobs_of(lib, 1), 0, None) == -2
        assert call(jobs_of(lib, most + 1), most + 1, None) == -6
        for field, value in (("kv", 512), ("dtype", 1), ("ntokens", 3), ("s_token", 8), ("s_head", 8)):
            jobs = jobs_of(lib, 2)
            setattr(jobs[1], field, value)
            assert call(jobs, 2, None) == -2, field
        jobs = jobs_of(lib, 2)
        jobs[1].max_bins = 64
        assert call(jobs, 2, None) == -4
        jobs[1].max_bins, jobs[1].cdf = 32, None
        assert call(jobs, 2, None) == -1
    assert lib.cg_encode_kv_levels_gather(jobs_of(lib, 2), 2, None, None, None) == -1
