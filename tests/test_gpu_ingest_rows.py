"""The tiled layout transforms with 32, 64 and 128 rows per tile, odd plane counts
and extents just off a tile, against torch's permute."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("nx,ny,nz", [(32, 1, 32), (96, 5, 160), (64, 3, 64), (192, 7, 320), (128, 1, 128),
                                      (256, 3, 384), (640, 2, 96), (96, 9, 128), (160, 3, 48)])
def test_rows(gpu_lib, nx, ny, nz, dtype):
    import torch
    import cubismz_gb300 as cz
    g = torch.Generator().manual_seed(nx + nz)
    a = torch.randn((nx, ny, nz), generator=g, dtype=torch.float64).to(getattr(torch, dtype)).cuda()
    f = cz.field_from_zfastest(a)
    assert torch.equal(f, a.float().permute(2, 1, 0).contiguous())
    assert torch.equal(cz.field_to_zfastest(f), a.float())
