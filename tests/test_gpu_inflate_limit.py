"""Inflating past a capacity near 2^31 bytes ends with the error and writes
nothing behind the output."""
import zlib

import pytest

pytestmark = pytest.mark.gpu


def _zeros(pieces, size):
    """A zlib stream of pieces * size zeros up to its last block (no trailer:
    the capacity ends first)."""
    z = zlib.compressobj(9, zlib.DEFLATED, -15)
    piece = z.compress(bytes(size)) + z.flush(zlib.Z_FULL_FLUSH)
    return b"\x78\x9c" + piece * pieces


def test_output_past_the_largest_capacity(gpu_lib):
    import cubismz_gb300 as cz
    with pytest.raises(cz.CzError):
        cz.zlib_decompress(_zeros(33, 1 << 26), 2 ** 31 - 1)  # 2.2e9 bytes
    assert cz.zlib_decompress(zlib.compress(b"abc" * 1000), 3000) == b"abc" * 1000
