"""The encoder's parse with two warps per chunk (few chunks) and with one (many):
the same bytes for the same chunks, at every effort, for LZ4 and for the parse
of the DEFLATE encoder, with records and without, one and several per chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(nblocks):
    import torch
    g = torch.Generator().manual_seed(8)
    f = torch.randn((nblocks, 32, 32, 32), generator=g).cuda()
    f[1::5] = 0.0                                    # one long match
    f[2::5] = torch.round(f[2::5] * 2) / 2           # short matches
    f[3::5, :, :, 8:] = 1.0
    return f.view(32 * nblocks, 32, 32)


@pytest.fixture(scope="module")
def field(gpu_lib):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return _field(2 * (16 * sms + 1))


@pytest.mark.parametrize("bpc", [1, 2])
@pytest.mark.parametrize("encoder,shuffle", [("lz4", True), ("lz4", False), ("zlib", True)])
@pytest.mark.parametrize("effort", [0, 1, 2])
def test_same_bytes(field, encoder, shuffle, effort, bpc):
    import torch
    import cubismz_gb300 as cz
    nblocks = field.shape[0] // 32 * bpc // 2
    few = 11 * bpc - (bpc > 1)  # the last chunk short where it can be
    ctx = cz.context(0)
    ctx.set_lz4_effort(effort)
    try:
        big = cz.compress_field(field[:32 * nblocks], 0.3, 1, 4, shuffle, encoder=encoder, blocks_per_chunk=bpc)
        d, o = (t.cpu().numpy() for t in big.to_device())
        small = cz.compress_field(field[:32 * few], 0.3, 1, 4, shuffle, encoder=encoder, blocks_per_chunk=bpc)
        ds, os_ = small.to_device()
        back = cz.decompress_field(ds, os_, (32 * few, 32, 32), 1, shuffle, encoder=encoder, blocks_per_chunk=bpc)
    finally:
        ctx.set_lz4_effort(1)
    ds, os_ = ds.cpu().numpy(), os_.cpu().numpy()
    n = few // bpc  # whole chunks
    assert np.array_equal(os_[:n + 1], o[:n + 1])
    assert np.array_equal(ds[:o[n]], d[:o[n]])
    plain = cz.compress_field(field[:32 * few], 0.3, 1, 4, shuffle, encoder="none")
    dp, op = plain.to_device()
    want = cz.decompress_field(dp, op, (32 * few, 32, 32), 1, shuffle, encoder="none")
    assert torch.equal(back.view(torch.int32), want.view(torch.int32))
