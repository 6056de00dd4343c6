"""The two-warp zlib decoder where its ring, its queue of records and its
tables can go wrong: sources at every distance up to 32 KiB (inside and behind
the ring), matches of 3 to 258 bytes and long runs, codes longer than the
lookup tables', stored blocks between others, sizes around a batch, capacities
one byte short. Streams are zlib's; the output is the input."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data():
    rng = np.random.default_rng(9)
    noise = rng.integers(0, 256, 40000, dtype=np.uint8).tobytes()
    out = [b"", b"a", b"ab" * 3, bytes([5]) * 258, bytes([5]) * 259, bytes([5]) * 40000]
    for dist in (1, 2, 3, 31, 32, 7000, 8191, 16380, 16384, 24000, 32506):  # zlib's own window ends at 32 506
        out.append(noise[:dist] + noise[:min(dist, 300)] * 2 + b"end")
    skew = rng.geometric(0.02, 60000).clip(0, 255).astype(np.uint8).tobytes()  # code lengths up to 15
    out.append(skew)
    out.append(skew[:20000] + noise + skew[:20000])
    text = b"".join(bytes([i % 7]) * (i % 300) for i in range(600))
    out.append(text)
    out += [noise[:n] for n in (383, 384, 385, 768, 769)]
    return out


@pytest.mark.parametrize("level,strategy", [(1, zlib.Z_DEFAULT_STRATEGY), (9, zlib.Z_DEFAULT_STRATEGY),
                                            (6, zlib.Z_FIXED), (6, zlib.Z_HUFFMAN_ONLY), (6, zlib.Z_RLE),
                                            (0, zlib.Z_DEFAULT_STRATEGY)])
def test_inflate_streams(gpu_lib, level, strategy):
    import cubismz_gb300 as cz
    for data in _data():
        c = zlib.compressobj(level, zlib.DEFLATED, 15, 9, strategy)
        z = c.compress(data[:len(data) // 3]) + c.flush(zlib.Z_FULL_FLUSH) + c.compress(data[len(data) // 3:]) + c.flush()
        assert cz.zlib_decompress(z, len(data)) == data
        if data:
            with pytest.raises(cz.CzError):
                cz.zlib_decompress(z, len(data) - 1)
