"""The codec kernels where their block bookkeeping can go wrong, against the
oracle bit for bit: nothing and everything kept (empty and full quarters),
signed zeros, wide exponent spreads (the out-of-line stencils), infinities,
several blocks per CTA (the plane ring wraps) and a single one."""
import numpy as np
import pytest

from oracle import czoracle as O

pytestmark = pytest.mark.gpu


def _field(nblocks, seed):
    """nblocks blocks along z, of seven kinds in turn."""
    rng = np.random.default_rng(seed)
    b = np.zeros((nblocks, 32, 32, 32), np.float32)
    for i in range(nblocks):
        kind, n = i % 7, (32, 32, 32)
        if kind == 0:
            b[i] = rng.standard_normal(n)
        elif kind == 1:
            b[i] = np.where(rng.random(n) < 0.5, -0.0, 0.0)
        elif kind == 2:
            b[i] = rng.standard_normal(n) * 10.0 ** rng.uniform(-9, 9, n)
        elif kind == 3:
            b[i] = np.where(rng.random(n) < 0.02, rng.standard_normal(n), -0.0)
        elif kind == 4:
            b[i] = 1.0 + 1e-3 * rng.standard_normal(n)
        elif kind == 5:
            b[i, :, :, 16:] = 3.0
            b[i, 7:20] *= 1e-30
        else:
            b[i] = rng.standard_normal(n) * 1e-39  # subnormal
    return b.reshape(32 * nblocks, 32, 32)


@pytest.mark.parametrize("nblocks", [1, 560])
@pytest.mark.parametrize("wtype,eps,shuffle", [(1, -1.0, True), (1, 1e-3, False), (2, 0.0, True), (3, 1e-4, True),
                                               (1, 1e38, True), (3, -1.0, False)])
def test_blocks_bit_exact(gpu_lib, nblocks, wtype, eps, shuffle):
    import torch
    import cubismz_gb300 as cz
    f = _field(nblocks, 3 + wtype)
    cf = cz.compress_field(torch.from_numpy(f).cuda(), eps, wtype, 0, shuffle, encoder="none")
    data, off = cf.to_device()
    raw, ooff = O.field_compress(f, eps, wtype, 0, int(shuffle), 0, 1)
    assert np.array_equal(off.cpu().numpy(), ooff)
    assert np.array_equal(data.cpu().numpy(), raw)
    dec = cz.decompress_field(data, off, f.shape, wtype, shuffle, encoder="none").cpu().numpy()
    want = O.field_decompress(raw, ooff, f.shape, wtype, int(shuffle))
    assert np.array_equal(dec.view(np.uint32), want.view(np.uint32))


def test_infinities_and_nan(gpu_lib):
    """Lines with an infinity or a NaN take the binary64 path: same mask and
    sizes as the oracle, same survivors wherever they are numbers."""
    import torch
    import cubismz_gb300 as cz
    f = _field(3, 1)
    f[3, 4, 5], f[40, 2, 30], f[70, 31, 31] = np.inf, -np.inf, np.nan
    cf = cz.compress_field(torch.from_numpy(f).cuda(), 1e-3, 1, 0, False, encoder="none")
    data, off = cf.to_device()
    raw, ooff = O.field_compress(f, 1e-3, 1, 0, 0, 0, 1)
    assert np.array_equal(off.cpu().numpy(), ooff)
    a, b = data.cpu().numpy().view(np.uint32), raw.view(np.uint32)
    nan = lambda u: (u & 0x7fffffff) > 0x7f800000
    assert np.array_equal(np.where(nan(a), 0, a), np.where(nan(b), 0, b))
