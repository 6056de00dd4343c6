"""The CTA-per-chunk zlib encoder where its blocks and lanes can go wrong:
blocks that share output words, a last block of a few bits, literal runs and
matches on both sides of what a lane takes alone (32 bytes, 4 pieces), stored
blocks at every bit offset, more blocks than warps. zlib inflates every stream
to its input."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data():
    rng = np.random.default_rng(21)
    noise = rng.integers(0, 256, 200000, dtype=np.uint8).tobytes()
    out = [b"", b"x", b"xyz" * 9, bytes(100), bytes(65535), bytes(65536), bytes(1 << 20)]
    for n in (31, 32, 33, 127, 128, 129):  # literal runs between matches
        out.append(b"".join(noise[n * i:n * i + n] + b"matchmatch" for i in range(200)))
    for m in (257, 258, 259, 1032, 1033, 1100, 5000):  # matches of 1 to 20 pieces
        out.append(noise[:40] + b"".join(bytes([i]) * m + noise[i:i + 3] for i in range(60)))
    out.append(rng.geometric(0.05, 150000).clip(0, 255).astype(np.uint8).tobytes())
    for n in (65534, 65535, 65536, 131071):  # stored blocks and their neighbours
        out.append(noise[:n] + b"tail" * 50)
    return out


def test_streams_inflate_to_their_input(gpu_lib):
    import cubismz_gb300 as cz
    for data in _data():
        assert zlib.decompress(cz.zlib_compress(data)) == data


@pytest.mark.parametrize("bpc", [1, 4, 15])
def test_record_chunks(gpu_lib, bpc):
    """5, 20 and 75 blocks per chunk."""
    import torch
    import cubismz_gb300 as cz
    from cubismz_gb300 import synth
    f = torch.from_numpy(synth.generate((96, 160, 64), seed=bpc, blobs=8, interfaces=2)).cuda()
    data, off = cz.compress_field(f, 1e-3, 1, 4, True, encoder="zlib", blocks_per_chunk=bpc).to_device()
    raw, roff = cz.compress_field(f, 1e-3, 1, 4, True, encoder="none", blocks_per_chunk=bpc).to_device()
    d, o, r, ro = (t.cpu().numpy() for t in (data, off, raw, roff))
    for k in range(o.size - 1):
        assert zlib.decompress(d[o[k]:o[k + 1]].tobytes()) == r[ro[k]:ro[k + 1]].tobytes()
