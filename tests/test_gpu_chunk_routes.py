"""One record per chunk: chunk offsets summed by the gather's own CTAs or by a
scan (the line lies at 1024 chunks), and records found from the offset table
and the decoded lengths alone, malformed ones included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _noise(nblocks, seed):
    import torch
    g = torch.Generator().manual_seed(seed)
    f = torch.randn((32 * nblocks, 32, 32), generator=g)
    f[::3] = 0.0
    return f.cuda()


@pytest.mark.parametrize("nblocks", [1, 256, 257, 1024, 1025])
@pytest.mark.parametrize("encoder", ["none", "lz4", "zlib"])
def test_offsets_on_both_routes(gpu_lib, nblocks, encoder):
    """A block's bytes do not depend on its neighbours: the first nblocks of
    1100 blocks give the first nblocks chunks of their stream, which the
    scan places."""
    import torch
    import cubismz_gb300 as cz
    f = _noise(1100, 5)
    data, off = (t.cpu().numpy() for t in cz.compress_field(f, 0.5, 1, 0, True, encoder=encoder).to_device())
    cf = cz.compress_field(f[:32 * nblocks], 0.5, 1, 0, True, encoder=encoder)
    d, o = (t.cpu().numpy() for t in cf.to_device())
    assert np.array_equal(o, off[:nblocks + 1]) and cf.nbytes == o[-1]
    assert np.array_equal(d[:o[-1]], data[:o[-1]])
    back = cz.decompress_field(torch.from_numpy(d).cuda(), torch.from_numpy(o).cuda(), (32 * nblocks, 32, 32), 1, True,
                               encoder=encoder)
    full = cz.decompress_field(torch.from_numpy(data).cuda(), torch.from_numpy(off).cuda(), tuple(f.shape), 1, True,
                               encoder=encoder)
    assert torch.equal(back.view(torch.int32), full[:32 * nblocks].view(torch.int32))


@pytest.mark.parametrize("encoder", ["none", "lz4", "zlib"])
@pytest.mark.parametrize("fault", ["size", "short", "empty", "backwards"])
def test_malformed_chunk(gpu_lib, encoder, fault):
    import torch
    import cubismz_gb300 as cz
    n, hit = 6, 3
    f = _noise(n, 6)
    data, off = cz.compress_field(f, 0.5, 1, 0, True, encoder=encoder).to_device()
    want = cz.decompress_field(data, off, tuple(f.shape), 1, True, encoder=encoder)
    d, o = data.cpu().numpy().copy(), off.cpu().numpy().copy()
    chunks = [d[o[i]:o[i + 1]] for i in range(n)]
    if fault == "size":  # a record that claims more bytes than its chunk has
        raw = chunks[hit] if encoder == "none" else np.frombuffer(
            (cz.lz4_decompress if encoder == "lz4" else cz.zlib_decompress)(chunks[hit].tobytes(), 200000), np.uint8)
        raw = raw.copy()
        raw[:4] = np.frombuffer(np.int32(raw.size).tobytes(), np.uint8)
        chunks[hit] = raw if encoder == "none" else np.frombuffer(
            (cz.lz4_compress if encoder == "lz4" else cz.zlib_compress)(raw.tobytes()), np.uint8)
    elif fault == "short":
        chunks[hit] = chunks[hit][:chunks[hit].size // 8 * 4]
    elif fault == "empty":
        chunks[hit] = chunks[hit][:0]
    o2 = np.concatenate([[0], np.cumsum([c.size for c in chunks])]).astype(np.int64)
    if fault == "backwards":  # the last chunk's end before its start
        o2[n] = o2[n - 1] - 4
        hit = n - 1
    d2 = np.concatenate(chunks + [np.zeros(64, np.uint8)])
    out = torch.full(tuple(f.shape), 7.0, device="cuda")
    with pytest.raises(cz.CzError):
        cz.decompress_field(torch.from_numpy(d2).cuda(), torch.from_numpy(o2).cuda(), tuple(f.shape), 1, True,
                            encoder=encoder, out=out)
    keep = torch.ones(n, dtype=torch.bool)
    keep[hit] = False
    a, b = out.view(n, -1)[keep], want.view(n, -1)[keep]
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert torch.equal(cz.decompress_field(data, off, tuple(f.shape), 1, True, encoder=encoder), want)
