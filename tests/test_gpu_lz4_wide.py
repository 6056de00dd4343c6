"""The two LZ4 decoders (a CTA per chunk for few chunks, a warp per chunk for
many) on both sides of the rule that picks one, and the CTA decoder where its
steps can go wrong: sequence counts around a step's, outputs around the ring's
and the stage's size, long length fields, deep chains of copies, sources at
every distance. Streams are the restated reference encoder's; the output is
the input."""
import numpy as np
import pytest

from oracle import czoracle as O

pytestmark = pytest.mark.gpu


def _cases():
    rng = np.random.default_rng(5)
    yield b"abcd" * 3
    yield bytes(20)
    for n in (4095, 4096, 4097, 32767, 32768, 40000):  # one run: off 1, chains as deep as the step
        yield bytes([7]) * n
    for n in (255, 270, 2070, 2080, 4200, 70000):  # long literal runs between matches
        lit = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
        yield b"headerhead" * 4 + lit + b"headerhead" * 40 + lit[:64] * 3 + b"tail!"
    small = rng.integers(0, 4, 60000, dtype=np.uint8).tobytes()  # short matches, many sequences a step
    yield small
    yield small[:1021]
    base = rng.integers(0, 256, 65000, dtype=np.uint8).tobytes()
    yield base + base[300:900] + base[20000:20600] + base[40000:64000]  # sources behind the ring
    words = [rng.integers(0, 256, k, dtype=np.uint8).tobytes() for k in (4, 5, 6, 7, 9, 17, 33)]
    yield b"".join(words[i] for i in rng.integers(0, len(words), 20000))


def test_cta_decoder(gpu_lib):
    import cubismz_gb300 as cz
    for data in _cases():
        assert cz.lz4_decompress(O.lz4_compress(data), len(data)) == data


@pytest.mark.parametrize("nblocks", [1216, 1220])
def test_both_sides_of_the_rule(gpu_lib, nblocks):
    """8 chunks per SM and just above, one record per chunk."""
    import torch
    import cubismz_gb300 as cz
    from cubismz_gb300 import synth
    f = synth.generate((32, 64, 16 * nblocks), seed=nblocks, blobs=40, interfaces=2)
    d = torch.from_numpy(f).cuda()
    cf = cz.compress_field(d, 2e-3, 1, 4, True, encoder="lz4")
    data, off = cf.to_device()
    assert off.numel() == nblocks + 1
    got = cz.decompress_field(data, off, f.shape, 1, True, encoder="lz4")
    raw = cz.compress_field(d, 2e-3, 1, 4, True, encoder="none")
    rdata, roff = raw.to_device()
    want = cz.decompress_field(rdata, roff, f.shape, 1, True, encoder="none")
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
