"""IC(0) on boxes in other numberings.  Where every cell comes after its three
neighbours before it the tiled sweeps run, and must equal the level-ordered
ones bit for bit in reference arithmetic, whatever the order of a row's
entries; other numberings keep the level-ordered sweeps."""
import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


def _numbering(kind, nx, ny, nz):
    """The new number of each cell x + nx (y + ny z)."""
    c = np.arange(nx * ny * nz)
    x, y, z = c % nx, c // nx % ny, c // (nx * ny)
    if kind == "blocks":
        key = (x >= nx * 2 // 5) + 2 * (y >= ny // 2) + 4 * (z >= nz // 3)
    elif kind == "x-blocks":          # x outermost: the x neighbours come first in a row
        key = x // 3 * 1000 + z // 2
    elif kind == "z-fastest":
        key = (x * ny + y) * nz + z
    elif kind == "wavefronts":
        key = x + y + z
    elif kind == "reversed-block":    # breaks the order across one face
        key = -(x >= nx // 2).astype(int)
    else:
        key = np.random.default_rng(0).permutation(c.size)
    order = np.lexsort((c, key))
    new = np.empty_like(c)
    new[order] = c
    return new


def _permuted(dims, kind):
    s = mesh.pressure_system(*dims, perturb=0.2, seed=sum(dims), variable_density=True)
    a = s.scipy().tocoo()
    new = _numbering(kind, *dims)
    row, col = new[a.row], new[a.col]
    key = np.lexsort((col, row))
    row, col, val = row[key], col[key], a.data[key]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=s.N))])
    return s.N, ptr, col, np.flatnonzero(row == col), val


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("kind", ["blocks", "x-blocks", "z-fastest", "wavefronts", "reversed-block", "random"])
@pytest.mark.parametrize("dims", [(2, 2, 2), (9, 5, 2), (17, 8, 9), (16, 9, 22), (31, 3, 23), (40, 25, 12)])
@pytest.mark.parametrize("block,grid", [(0, 0), (128, 3)])
def test_other_numberings_equal_level_apply(dims, kind, block, grid):
    import torch
    n, ptr, col, diag, val = _permuted(dims, kind)
    topo = tflows.Topology(n, ptr, col, diag)
    v, r = _dev(val), _dev(np.random.default_rng(n).uniform(-1, 1, n))
    out = {}
    for tiled in (0, 1):
        z = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        opts = tflows.options(ic_tiled=tiled, block_size=block, grid_blocks=grid)
        for _ in range(2):
            assert topo.ic_apply(v, r, z, opts=opts)["status"] == tflows.OK
        out[tiled] = z.cpu().numpy()
    topo.close()
    assert np.array_equal(out[0].view(np.uint64), out[1].view(np.uint64))


@pytest.mark.parametrize("kind", ["blocks", "wavefronts"])
@pytest.mark.parametrize("precision", ["FP64_FMA", "MIXED"])
@pytest.mark.parametrize("bf16", [0, 1])
def test_other_numberings_solve(kind, precision, bf16):
    import torch
    import scipy.sparse as sp
    n, ptr, col, diag, val = _permuted((26, 21, 13), kind)
    b = np.random.default_rng(5).uniform(-1, 1, n)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    topo = tflows.Topology(n, ptr, col, diag)
    tol = 1e-10 * float(np.linalg.norm(b))
    res = topo.solve(_dev(val), _dev(b), x, "cg", 2, 5000, tol,
                     opts=tflows.options(precision=getattr(tflows, precision), ic_bf16=bf16, ic_tiled=1))
    topo.close()
    assert res["status"] == tflows.OK
    # the recurrence's residual is below tol; the true one differs by rounding
    # (eps ||A|| ||x|| is 1e-13 ||b|| here)
    rest = np.linalg.norm(b - sp.csr_matrix((val, col, ptr)) @ x.cpu().numpy())
    assert rest < tol + 1e-12 * np.linalg.norm(b)
