"""The launch shape of level-ordered IC(0) by the rows of a level: one block of
256 threads per SM on narrow levels, two on wider ones in mixed precision, four
on the widest; whatever the shape, the same apply."""
import numpy as np
import pytest

from conftest import tflows
from test_gpu_numbered_boxes import _dev, _permuted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,wide", [((30, 25, 20), False), ((92, 90, 88), True)])
def test_blocks_per_sm(dims, wide):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, ptr, col, diag, val = _permuted(dims, "random")
    topo, v = tflows.Topology(n, ptr, col, diag), _dev(val)
    b = _dev(np.random.default_rng(1).uniform(-1, 1, n))
    want = min(4 if wide else 1, -(-n // 256) / sms) * sms
    for precision in (tflows.FP64, tflows.FP64_FMA, tflows.MIXED):
        x = torch.zeros_like(b)
        r = topo.solve(v, b, x, "cg", 2, 4, 0.0, opts=tflows.options(precision=precision))
        assert (r["block_size"], r["grid_blocks"]) == (256, round(want))
    z = []
    for kw in ({}, {"block_size": 256, "grid_blocks": 7}):
        z.append(torch.empty_like(b))
        assert topo.ic_apply(v, b, z[-1], opts=tflows.options(**kw))["status"] == tflows.OK
    assert torch.equal(z[0].view(torch.int64), z[1].view(torch.int64))
    topo.close()
