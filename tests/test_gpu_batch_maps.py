"""Launches over several fields read their tensor maps from device memory, at
an address that the next batch of the same context uses again: every batch must
see its own fields, whatever the batch before had at the same place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the same number of fields in every batch, so that the maps lie at the same
# addresses: equal shapes with other pointers, the fields in another order,
# other shapes (other strides), fields freed in between
SHAPES = [(64, 96, 32), (32, 32, 160), (96, 64, 64)]
BATCHES = [SHAPES, SHAPES, SHAPES[::-1], [(32, 64, 128), (160, 32, 32), (64, 64, 96)], SHAPES]


@pytest.mark.parametrize("encoder", ["none", "lz4"])
def test_batches_on_one_context(gpu_lib, encoder):
    import torch
    import cubismz_gb300 as cz
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    for k, shapes in enumerate(BATCHES):
        fields = [torch.randn(s, generator=g, device="cuda") + 10.0 * (k + i) for i, s in enumerate(shapes)]
        eps = [1e-3 * (i + 1) for i in range(len(fields))]
        got = [cf.to_device() for cf in cz.batch_compress(fields, eps, 1, 4, True, encoder=encoder)]
        for f, e, (d, o) in zip(fields, eps, got):
            sd, so = cz.compress_field(f, e, 1, 4, True, encoder=encoder).to_device()
            assert torch.equal(o, so) and torch.equal(d, sd)
        del fields, got
        torch.cuda.empty_cache()


def test_plans_one_after_the_other(gpu_lib):
    """A plan can get the address of a destroyed one's list."""
    import torch
    import cubismz_gb300 as cz
    for k, shapes in enumerate(BATCHES):
        fields = [torch.from_numpy(np.random.default_rng(10 * k + i).standard_normal(s).astype(np.float32)).cuda()
                  for i, s in enumerate(shapes)]
        eps = [1e-3 * (i + 1) for i in range(len(fields))]
        plan = cz.Plan(fields, eps, 1, 4, True, "none", tune=True)
        plan.launch()
        data, off = plan.result().to_device()
        for i, (f, e) in enumerate(zip(fields, eps)):
            d, o = plan.field_chunks(data, off, i)
            sd, so = cz.compress_field(f, e, 1, 4, True, encoder="none").to_device()
            assert torch.equal(o, so) and torch.equal(d, sd)
        plan.close()


def test_plan_list_is_there_before_its_first_launch(gpu_lib):
    """cz_plan_create copies the fields' list on a stream of its own; a launch
    on another stream right after it, with the copy engine still busy with
    something else, reads the whole list."""
    import torch
    import cubismz_gb300 as cz
    shapes = SHAPES * 3
    fields = [torch.from_numpy(np.random.default_rng(50 + i).standard_normal(s).astype(np.float32)).cuda()
              for i, s in enumerate(shapes)]
    eps = [1e-3 * (i + 1) for i in range(len(fields))]
    host = torch.empty(1 << 28, pin_memory=True).fill_(1.0)
    dev = torch.empty(1 << 28, device="cuda")
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        dev.copy_(host, non_blocking=True)
    plan = cz.Plan(fields, eps, 1, 4, True, "none", tune=False)
    plan.launch()
    data, off = plan.result().to_device()
    torch.cuda.synchronize()
    for i, (f, e) in enumerate(zip(fields, eps)):
        d, o = plan.field_chunks(data, off, i)
        sd, so = cz.compress_field(f, e, 1, 4, True, encoder="none").to_device()
        assert torch.equal(o, so) and torch.equal(d, sd)
    plan.close()
