"""Which IC(0) calls run the tiled sweeps: the box that a topology reports, and
the block size of the launch (512 threads for tiled sweeps, 256 for
level-ordered ones of this size)."""
import numpy as np
import pytest

from conftest import tflows
from test_gpu_numbered_boxes import _dev, _permuted

pytestmark = pytest.mark.gpu
DIMS = (17, 8, 9)


def _apply(topo, n, val, **kw):
    import torch
    z = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    r = _dev(np.random.default_rng(n).uniform(-1, 1, n))
    res = topo.ic_apply(val, r, z, opts=tflows.options(**kw))
    assert res["status"] == tflows.OK
    return res["block_size"], z.cpu().numpy().view(np.uint64)


def test_other_numberings_are_looked_for_on_first_use():
    import torch
    n, ptr, col, diag, val = _permuted(DIMS, "blocks")
    topo, v = tflows.Topology(n, ptr, col, diag), _dev(val)
    assert topo.box is None
    x, b = torch.zeros(n, dtype=torch.float64, device="cuda"), _dev(np.ones(n))
    assert topo.solve(v, b, x, "cg", 1, 200, 1e-6)["status"] == tflows.OK
    _apply(topo, n, v, ic_tiled=0)
    assert topo.box is None
    _apply(topo, n, v, ic_tiled=1)
    assert topo.box == DIMS
    topo.close()


@pytest.mark.parametrize("kind,box", [("box", True), ("blocks", True), ("x-blocks", True), ("z-fastest", True),
                                      ("wavefronts", True), ("reversed-block", False), ("random", False)])
def test_route_of_a_numbering(kind, box):
    if kind == "box":
        s = tflows.mesh.pressure_system(*DIMS, perturb=0.2, seed=sum(DIMS), variable_density=True)
        n, val, topo = s.N, s.A[:-1].copy(), tflows.Topology.from_system(s)
    else:
        n, ptr, col, diag, val = _permuted(DIMS, kind)
        topo = tflows.Topology(n, ptr, col, diag)
    v = _dev(val)
    block, z = _apply(topo, n, v)
    assert (topo.box is not None) == box
    assert not box or sorted(topo.box) == sorted(DIMS)
    assert block == (512 if box else 256)
    level_block, level = _apply(topo, n, v, ic_tiled=0)
    assert level_block == 256
    assert np.array_equal(z, level)
    for threads in (64, 128, 160, 288):  # (64: too few for a patch's four warps)
        assert np.array_equal(_apply(topo, n, v, ic_tiled=1, block_size=threads)[1], level)
    topo.close()
