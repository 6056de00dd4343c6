"""The refit's two routes for its sums (integers where binary64 holds the sum
exactly, binary64 else: thread sums more than 2^20 apart) and its step count,
against the same steps in FP64 with the oracle's operators; the dense operators
where a CTA takes one, several or a last odd block."""
import numpy as np
import pytest

from oracle import czoracle as O

pytestmark = pytest.mark.gpu


def _blocks(kind):
    rng = np.random.default_rng(21)
    b = rng.standard_normal((2, 32, 32, 32))
    if kind == "wide":  # planes from 1e-15 to 1e5
        b *= 10.0 ** np.linspace(-15, 5, 32)[None, :, None, None]
    elif kind == "empty":  # a block without anything
        b[1] = 0.0
    return b.astype(np.float32)


@pytest.mark.parametrize("wtype", [1, 2, 3])
@pytest.mark.parametrize("kind", ["even", "wide", "empty"])
@pytest.mark.parametrize("iters", [1, 2])
def test_steps_match_fp64(gpu_lib, kind, wtype, iters):
    import torch
    import cubismz_gb300 as cz
    x = _blocks(kind)
    eps = 0.5
    f = torch.from_numpy(x.reshape(64, 32, 32)).cuda()
    cf = cz.refit_field(f, eps, iters=iters, wtype=wtype, zerobits=0, shuffle=False, encoder="none")
    data, off = cf.to_device()
    dec = cz.decompress_field(data, off, (64, 32, 32), wtype, False, encoder="none").cpu().numpy().reshape(x.shape)
    d, o = data.cpu().numpy(), off.cpu().numpy()
    for g in range(2):
        mask = np.unpackbits(d[o[g] + 4:o[g] + 4 + 4096], bitorder="little").reshape(32, 32, 32).astype(bool)
        c = np.where(mask, O.fwt(x[g], wtype), 0).astype(np.float64)
        W = lambda v: O.iwt_f64(v.astype(np.float64), wtype)
        r = x[g].astype(np.float64) - W(c)
        p = s = np.where(mask, O.iwt_adj_f64(r, wtype), 0)
        gamma = np.vdot(s, s)
        for _ in range(iters):
            q = W(p)
            delta = np.vdot(q, q)
            if not (gamma > 0 and delta > 0):
                break
            c = c + gamma / delta * p
            r = r - gamma / delta * q
            s = np.where(mask, O.iwt_adj_f64(r, wtype), 0)
            gamma, old = np.vdot(s, s), gamma
            p = s + gamma / old * p
        want = W(c)
        # an operator is within 2e-5 of the largest entry; 2 per step, 2 to start, 1 to decode
        assert np.abs(dec[g] - want).max() <= 2e-5 * (2 * iters + 3) * max(np.abs(x[g]).max(), 1e-30)


@pytest.mark.parametrize("nblocks", [1, 152, 153, 307])
def test_operators_over_several_blocks(gpu_lib, nblocks):
    """Each block's result is that of the block alone."""
    import torch
    import cubismz_gb300 as cz
    c = torch.randn((nblocks, 32, 32, 32), generator=torch.Generator().manual_seed(nblocks)).cuda()
    for f in (cz.iwt_linear, cz.iwt_adjoint):
        all_ = f(c, 1)
        for g in {0, nblocks // 2, nblocks - 1}:
            assert torch.equal(all_[g], f(c[g:g + 1].contiguous(), 1)[0])
