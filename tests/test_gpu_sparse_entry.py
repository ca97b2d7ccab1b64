"""cg_pack_sparse_tables through the C ABI: the parts it makes of byte counts are those of an encoded container."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,T,H,D", [(2, 40, 2, 64), (1, 256, 3, 80), (3, 255, 1, 8)])
def test_sparse_parts_of_byte_counts(L, T, H, D):
    from cachegen_b200 import _lib
    from cachegen_b200.serde import cachegen_encoder as E, flat_format as ff
    C = H * D
    kv = torch.randn((L, 2, T, H, D), generator=torch.Generator().manual_seed(C)).half().cuda()
    kb, vb = torch.full((L,), 32.0).cuda(), torch.full((L,), 16.0).cuda()
    counts = E.quantize_and_tables(kv, kb, vb, 32, with_counts=True)[3]
    flat = E.encode_flat(kv, kb, vb, max_bins=32)
    assert flat.header.table_kind == ff.TABLES_SPARSE
    bins = torch.cat((kb, vb))
    offs, moffs = ff.table_row_offsets(bins.cpu(), C), ff.mask_row_offsets(bins.cpu(), C)
    off_masks, off_counts = ff.sparse_parts(2 * L, C, moffs[-1])
    tables = torch.zeros(off_counts + counts.numel(), dtype=torch.uint8, device="cuda")
    dev = [torch.tensor(o, dtype=torch.int64, device="cuda") for o in (offs, moffs)]
    rc = _lib.lib().cg_pack_sparse_tables(counts.data_ptr(), dev[0].data_ptr(), bins.data_ptr(), 2 * L, C, tables.data_ptr(),
                                          tables.data_ptr() + off_masks, dev[1].data_ptr(), tables.data_ptr() + off_counts,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    ngroups = 2 * L * ((C + 127) // 128)
    used = off_counts + int(tables[4 * ngroups:4 * ngroups + 4].view(torch.int32))
    assert torch.equal(tables[:used], flat.tables()[:used])
