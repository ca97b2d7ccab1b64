"""Encoded chunks whose parts do not fit together are refused before anything is read by address."""
import dataclasses

import pytest
import torch


def chunk(L=2, T=5, H=1, D=4, lp=9):
    from cachegen_b200.serde.cachegen_basics import CacheGenGPUBytestream, CacheGenGPUEncoderOutput
    return CacheGenGPUEncoderOutput([CacheGenGPUBytestream(torch.zeros(7, dtype=torch.uint8), torch.ones(2 * L, H * D, dtype=torch.int32), T)],
                                    torch.zeros(2 * L, H * D, lp, dtype=torch.int16), torch.ones(L, T, 1).half(),
                                    torch.ones(L, T, 1).half(), H, D)


def test_a_chunk_that_fits():
    from cachegen_b200.serde.cachegen_decoder import _check_chunk
    eo = chunk()
    assert _check_chunk(eo) == (2, 4, 9, 5)
    flat = dataclasses.replace(eo, max_tensors_key=eo.max_tensors_key[..., 0], max_tensors_value=eo.max_tensors_value[..., 0])
    assert _check_chunk(flat) == (2, 4, 9, 5)


@pytest.mark.parametrize("field", ["max_tensors_key", "max_tensors_value"])
@pytest.mark.parametrize("shape", [(2, 5, 2), (2, 5, 0), (2, 5, 1, 3), (2, 4, 1), (3, 5, 1)])
def test_scales_of_another_shape(field, shape):
    from cachegen_b200.serde.cachegen_decoder import _check_chunk
    with pytest.raises(RuntimeError):
        _check_chunk(dataclasses.replace(chunk(), **{field: torch.ones(shape).half()}))
