"""Encode with given tables: groups of symbols with and without the table's last one, at the groups' edges, and symbols
above it, which are reported and coded as the last."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lp", [2, 3, 17, 33, 40])
@pytest.mark.parametrize("C,T", [(1, 16), (130, 15), (130, 17), (128, 32), (200, 100), (96, 256)])
def test_last_symbols_in_some_groups(oracle, lp, C, T):
    from cachegen_b200 import torchac_cuda
    rng = np.random.default_rng(lp * 1000 + C + T)
    top = lp - 2
    cdf, sym = np.zeros((2, C, lp), np.uint16), rng.integers(0, max(top, 1), size=(2, T, C)).astype(np.int8)
    for r in range(2):
        for c in range(C):
            cdf[r, c] = np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), size=lp - 2, replace=False)), [65535]))
    # the lanes of one warp differ in where their last symbols are; row 1 has one group with a single one
    for c in range(0, C, 3):
        sym[0, rng.random(T) < 0.1, c] = top
    sym[1, T - 1 - T // 3, C // 2] = top
    want, want_len = oracle.encode_chunk(cdf.view(np.int16), sym)
    out = torch.zeros((2, C, 4 * T + 16), dtype=torch.uint8, device="cuda")
    lengths = torch.zeros((2, C), dtype=torch.int32, device="cuda")
    torchac_cuda.encode_fast_new(torch.from_numpy(cdf.view(np.int16)).cuda(), torch.from_numpy(sym).cuda(), out, lengths)
    n, rows = lengths.cpu().numpy(), out.cpu().numpy()
    assert (n == want_len).all()
    assert b"".join(rows[r, c, :n[r, c]].tobytes() for r in range(2) for c in range(C)) == want.tobytes()


@pytest.mark.parametrize("above", [1, 100])
def test_symbols_above_the_last(oracle, above):
    from cachegen_b200 import _lib
    rng = np.random.default_rng(above)
    lp, C, T = 17, 64, 40
    cdf, sym = np.zeros((1, C, lp), np.uint16), rng.integers(0, lp - 2, size=(1, T, C)).astype(np.int8)
    for c in range(C):
        cdf[0, c] = np.concatenate(([0], np.sort(rng.choice(np.arange(1, 65535), size=lp - 2, replace=False)), [65535]))
    wrong = sym.copy()
    wrong[0, 20, 5], sym[0, 20, 5] = lp - 2 + above, lp - 2
    want, want_len = oracle.encode_chunk(cdf.view(np.int16), sym)
    out = torch.zeros((1, C, 128), dtype=torch.uint8, device="cuda")
    lengths, status = torch.zeros((1, C), dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    dev, x = torch.from_numpy(cdf.view(np.int16)).cuda(), torch.from_numpy(wrong).cuda()
    strides = (ctypes.c_int64 * 3)(*x.stride())
    rc = _lib.lib().cg_encode_padded(dev.data_ptr(), x.data_ptr(), strides, 1, T, C, lp, out.data_ptr(), 128, lengths.data_ptr(),
                                     status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "cg_encode_padded")
    n, rows = lengths.cpu().numpy(), out.cpu().numpy()
    assert status.item() == _lib.CG_S_BAD_SYMBOL
    assert (n == want_len).all()
    assert b"".join(rows[0, c, :n[0, c]].tobytes() for c in range(C)) == want.tobytes()
