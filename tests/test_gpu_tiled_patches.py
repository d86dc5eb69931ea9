"""The tiled IC(0) sweeps at the edges of their patches (8 x 4 columns),
tiles (up to four patches) and chunks (4 steps), with more tiles than blocks
and with one block: the apply must equal the level-ordered one bit for bit in
reference arithmetic, and mixed solves (FP32 and BF16 entries) must reach
their FP64 tolerance."""
import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("dims", [(2, 2, 2), (8, 4, 6), (9, 5, 2), (16, 8, 7), (17, 8, 9),
                                  (16, 9, 22), (31, 3, 23), (3, 33, 24), (40, 25, 5)])
@pytest.mark.parametrize("block,grid", [(64, 0), (128, 0), (128, 3), (256, 2), (480, 5), (512, 1),
                                        (0, 0)])
def test_patch_edges_equal_level_apply(dims, block, grid):
    import torch
    s = mesh.pressure_system(*dims, perturb=0.2, seed=sum(dims), variable_density=True)
    topo = tflows.Topology.from_system(s)
    val = _dev(s.A[:-1])
    r = _dev(np.random.default_rng(block + grid).uniform(-1, 1, s.N))
    out = {}
    for tiled in (0, 1):
        z = torch.full((s.N,), float("nan"), dtype=torch.float64, device="cuda")
        opts = tflows.options(ic_tiled=tiled, block_size=block, grid_blocks=grid)
        for _ in range(2):  # the second apply starts from the first one's buffers
            res = topo.ic_apply(val, r, z, opts=opts)
            assert res["status"] == tflows.OK
        out[tiled] = z.cpu().numpy()
    topo.close()
    assert np.array_equal(out[0].view(np.uint64), out[1].view(np.uint64))


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("dims,grid", [((17, 9, 30), 2), ((33, 20, 11), 1), ((26, 41, 13), 0)])
def test_mixed_solves_on_ragged_tiles(bf16, dims, grid):
    s = mesh.pressure_system(*dims, perturb=0.2, seed=1, variable_density=True)
    tol = 1e-10 * float(np.linalg.norm(s.b))
    x, r = s.x.copy(), s.b.copy()
    opts = tflows.options(precision=tflows.MIXED, ic_bf16=bf16, ic_tiled=1, grid_blocks=grid)
    out = tflows.solve_ex("cg", s.N, s.NB, s.NONZ, s.A, s.Acol, s.Arow, s.Adia, s.Ab, x, r, 2,
                          20000, tol, opts=opts)
    assert out.status == tflows.OK
    assert np.linalg.norm(s.b - s.scipy() @ x[s.NB + 1:]) < tol
