"""Every solver on the four kinds of systems that have kernels of their own (a
box, a box in another numbering, a mesh that is no box, long rows), alone and
together in one batch: each reaches its tolerance."""
import numpy as np
import pytest

from conftest import tflows
from test_gpu_numbered_boxes import _permuted
from test_gpu_product_rows import _system

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def systems():
    import scipy.sparse as sp
    out = {}
    s = tflows.mesh.pressure_system(13, 12, 11, perturb=0.2, seed=1, variable_density=True)
    out["box"] = s.scipy().tocsr()
    out["box"].sort_indices()
    for kind, dims in (("blocks", (17, 9, 10)), ("random", (14, 11, 9))):
        n, ptr, col, diag, val = _permuted(dims, kind)
        out[kind] = sp.csr_matrix((val, col, ptr))
    out["long"] = _system(1500, 30, 5, [])[0]
    made = {}
    for k, a in out.items():
        n = a.shape[0]
        diag = np.flatnonzero(np.repeat(np.arange(n), np.diff(a.indptr)) == a.indices)
        made[k] = (a, tflows.Topology(n, a.indptr, a.indices, diag), np.random.default_rng(n).uniform(-1, 1, n))
    yield made
    for _, topo, _ in made.values():
        topo.close()


SOLVES = [("cg", 0, {}), ("cg", 1, {}), ("cg", 2, {}), ("cgs", 1, {}), ("cgs", 2, {}), ("bicg", 1, {})]
SOLVES_MIXED = SOLVES + [("cg", 0, {"refine_restart": 1}), ("cg", 1, {"refine_restart": 1}),
                         ("cg", 2, {"refine_restart": 1}), ("cg", 2, {"ic_bf16": 1}), ("cg", 2, {"ic_sweeps": 2}),
                         ("cg", 2, {"ic_sweeps": 1, "refine_restart": 1})]
CASES = [(p, *c) for p, cs in (("FP64", SOLVES), ("FP64_FMA", SOLVES + [("cg", 2, {"ic_sweeps": 2})]),
                               ("MIXED", SOLVES_MIXED)) for c in cs]


@pytest.mark.parametrize("precision,method,prec,kw", CASES)
def test_alone_and_in_a_batch(systems, precision, method, prec, kw):
    import torch
    opts = tflows.options(precision=getattr(tflows, precision), **kw)
    rtol = 1e-8
    dev = {k: (torch.from_numpy(a.data).cuda(), torch.from_numpy(b).cuda()) for k, (a, _, b) in systems.items()}
    tol = [rtol * float(np.linalg.norm(b)) for _, _, b in systems.values()]

    def check(k, res, x, what):
        a, _, b = systems[k]
        assert res["status"] == tflows.OK, (k, what, res)
        # the true residual differs from the recurrence's by the rounding of
        # the iterates (CGS: its residual may first rise a thousandfold)
        rest = np.linalg.norm(b - a @ x.cpu().numpy())
        assert rest <= (rtol + (1e-9 if method == "cgs" else 1e-11)) * np.linalg.norm(b), (k, what, rest)

    for (k, (_, topo, _)), t in zip(systems.items(), tol):
        x = torch.zeros_like(dev[k][1])
        check(k, topo.solve(*dev[k], x, method, prec, 5000, t, opts=opts), x, "alone")
    xs = [torch.zeros_like(d[1]) for d in dev.values()]
    n = len(xs)
    res = tflows.solve_batched([s[1] for s in systems.values()], [d[0] for d in dev.values()],
                               [d[1] for d in dev.values()], xs, [method] * n, [prec] * n, [5000] * n, tol, opts=opts)
    for k, r, x in zip(systems, res, xs):
        check(k, r, x, "batch")
