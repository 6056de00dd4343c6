"""Error norms with the decoded field written over the reference: the field is
the decoded one and the statistics are its own against itself, every time."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype,encoder,bpc", [(1, "lz4", 1), (3, "none", 15), (2, "zlib", 1)])
def test_out_is_the_reference(gpu_lib, wtype, encoder, bpc):
    import torch
    import cubismz_gb300 as cz
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    f = torch.randn((160, 128, 192), generator=g, device="cuda")
    kw = dict(shuffle=True, encoder=encoder, blocks_per_chunk=bpc)
    data, off = cz.compress_field(f, 0.5, wtype, 4, **kw).to_device()
    dec = cz.decompress_field(data, off, f.shape, wtype, **kw)
    want = cz.diff_field(data, off, f.shape, dec, wtype, **kw)
    assert want["e_inf"] == 0.0 and want["n_inf"] > 0.0
    for _ in range(3):
        ref = f.clone()
        got = cz.diff_field(data, off, f.shape, ref, wtype, out=ref, **kw)
        assert got == want and torch.equal(ref, dec)
