"""The lines that the kernels' main path has to carry or leave, on the CPU: a -0
among a line's sources does not take it off the main path, and lines whose
exponents spread too far are bit-exact to the oracle off it."""
import ctypes as C

import numpy as np
import pytest

from oracle import czoracle as O
from tests.test_emu import emu, fp, u8p  # noqa: F401 (fixture)

N = (32, 32, 32)


def _stats(emu, block, wtype):  # noqa: F811
    """Lines, lines off the main path, stencils of those on no grid."""
    st = np.zeros(3, np.int64)
    b = np.ascontiguousarray(block, np.float32).copy()
    emu.emu_fwt(b.ctypes.data_as(fp), wtype, st.ctypes.data_as(C.c_void_p))
    return st


@pytest.mark.parametrize("wtype", [1, 2, 3])
def test_a_negative_zero_stays_on_the_main_path(emu, wtype):  # noqa: F811
    rng = np.random.default_rng(4)
    f = 1.0 + 0.1 * rng.random(N)
    scattered = np.where(rng.random(N) < 0.02, -0.0, f)
    background = np.where((np.indices(N) ** 2).sum(0) < 400, f, -0.0)
    for b in (np.full(N, -0.0), scattered, background):
        zero = np.where(b == 0.0, 0.0, b)  # the same field with +0
        assert _stats(emu, b, wtype)[1] == _stats(emu, zero, wtype)[1]


def _wide(seed):
    rng = np.random.default_rng(seed)
    with np.errstate(over="ignore"):
        yield rng.standard_normal(N) * np.exp(8 * rng.standard_normal(N))
        yield rng.standard_normal(N) * 2.0 ** rng.integers(-16, 1, N)  # just past one grid
        yield rng.standard_normal(N) * 2.0 ** rng.integers(-12, 1, N)  # past the last predictions' grid
        yield np.where(rng.random(N) < 0.5, -0.0, rng.standard_normal(N) * 2.0 ** rng.integers(-30, 1, N))
        yield rng.integers(-3, 4, N) * 2.0 ** rng.integers(-140, -120, N)
        yield rng.integers(-3, 4, N) * 2.0 ** rng.integers(100, 126, N)
        r = np.sqrt((np.indices(N) ** 2).sum(0))
        yield 6e-8 + (1 - 6e-8) * 0.5 * (1 - np.tanh((r - 24) / 2))  # a volume fraction's interface


@pytest.mark.parametrize("wtype", [1, 2, 3])
def test_wide_lines_bit_exact(emu, wtype):  # noqa: F811
    for b in _wide(9):
        b = np.ascontiguousarray(b.astype(np.float32))
        with np.errstate(all="ignore"):
            phys, pos = b.copy(), np.zeros(N, np.float32)
            emu.emu_fwt(phys.ctypes.data_as(fp), wtype, None)
            emu.emu_to_positional(phys.ctypes.data_as(fp), pos.ctypes.data_as(fp))
            want = O.fwt(b, wtype)
            assert _same(pos, want)
            rec = O.block_compress(b, -1.0, wtype, 0, 0)
            dec = np.zeros(N, np.float32)
            assert emu.emu_block_decompress(rec.ctypes.data_as(u8p), rec.size, wtype, 0, dec.ctypes.data_as(fp)) == 0
            assert _same(dec, O.block_decompress(rec, wtype, 0))


def _same(a, b):
    both = np.isnan(a) & np.isnan(b)
    return np.array_equal(np.where(both, 0, a.view(np.uint32)), np.where(both, 0, b.view(np.uint32)))


def signed_zero_fields():
    """Zeros of both signs beside values that cancel exactly in a stencil."""
    rng = np.random.default_rng(12)
    yield rng.choice(np.array([0.0, -0.0, -0.0, 1.0, -1.0, 0.5, -0.5], np.float32), size=N)
    yield rng.choice(np.array([0.0, -0.0, -0.0, 7.0, -1.0, 1.0, -7.0], np.float32), size=N)  # -5 v0 = 35 v2
    yield np.where(rng.random(N) < 0.7, rng.choice(np.array([0.0, -0.0], np.float32), size=N),
                   rng.integers(-2, 3, N)).astype(np.float32)


@pytest.mark.parametrize("wtype", [1, 2, 3])
def test_signs_of_zeros(emu, wtype):  # noqa: F811
    for b in signed_zero_fields():
        phys, pos = b.copy(), np.zeros(N, np.float32)
        emu.emu_fwt(phys.ctypes.data_as(fp), wtype, None)
        emu.emu_to_positional(phys.ctypes.data_as(fp), pos.ctypes.data_as(fp))
        assert np.array_equal(pos.view(np.uint32), O.fwt(b, wtype).view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("wtype", [1, 2, 3])
def test_signs_of_zeros_on_the_gpu(gpu_lib, wtype):
    """The same fields through the kernels, everything kept, bit for bit."""
    import torch
    import cubismz_gb300 as cz
    f = np.concatenate(list(signed_zero_fields()) * 60)  # several blocks per CTA
    cf = cz.compress_field(torch.from_numpy(f).cuda(), -1.0, wtype, 0, False, encoder="none")
    data, off = cf.to_device()
    raw, ooff = O.field_compress(f, -1.0, wtype, 0, 0, 0, 1)
    assert np.array_equal(off.cpu().numpy(), ooff) and np.array_equal(data.cpu().numpy(), raw)
    dec = cz.decompress_field(data, off, f.shape, wtype, False, encoder="none").cpu().numpy()
    assert np.array_equal(dec.view(np.uint32), O.field_decompress(raw, ooff, f.shape, wtype, 0).view(np.uint32))
