"""The plan's tuner times a kernel once: with few chunks the LZ4 widths 2, 4 and
8 are the same kernel, so they have one time and are not chosen among."""
import pytest

pytestmark = pytest.mark.gpu


def test_one_kernel_one_time(gpu_lib):
    import torch
    import cubismz_gb300 as cz
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    fields = [torch.randn((96, 64, 32 * (1 + k)), generator=g, device="cuda") for k in range(4)]
    plan = cz.Plan(fields, [1e-2] * 4, 1, 4, True, "lz4", tune=True)
    info = plan.info()
    lz = info["lz4_stage_ms"]
    assert lz[2] == lz[4] == lz[8] > 0 and lz[16] > 0
    assert info["shape"]["lz4_chunks_per_cta"] == (4 if lz[4] <= lz[16] else 16)
    plan.close()


def test_many_chunks_are_timed_by_width(gpu_lib):
    import torch
    import cubismz_gb300 as cz
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    f = torch.randn((32 * (9 * sms + 1), 32, 32), device="cuda")
    plan = cz.Plan([f], [1e-2], 1, 4, True, "lz4", tune=True)
    lz = plan.info()["lz4_stage_ms"]
    assert len(set(lz.values())) > 1 and min(lz.values()) > 0
    plan.close()
