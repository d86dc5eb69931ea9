"""How many systems a batch takes: four per SM, whatever the preconditioner, in
the default shape and with 256 threads (the register budget's limit), two per
SM with 512; one more is refused."""
import numpy as np
import pytest

from conftest import tflows

mesh = tflows.mesh
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "FP64_FMA", "MIXED"])
@pytest.mark.parametrize("block,per_sm", [(0, 2.1), (0, 3), (0, 4), (256, 4), (512, 2)])
def test_batches_of_small_boxes(precision, block, per_sm):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count = int(per_sm * sms)
    systems = [mesh.pressure_system(*d, perturb=0.2, seed=1, variable_density=True)
               for d in ((5, 4, 3), (9, 5, 4), (17, 3, 2))]
    topos = [tflows.Topology.from_system(s) for s in systems]
    vals = [torch.from_numpy(s.A[:-1].copy()).cuda() for s in systems]
    rhs = [torch.from_numpy(s.b).cuda() for s in systems]
    opts = tflows.options(precision=getattr(tflows, precision), tol_mode=tflows.TOL_RELATIVE,
                          block_size=block)

    def run(n):
        k = np.arange(n) % 3
        xs = [torch.zeros_like(rhs[i]) for i in k]
        res = tflows.solve_batched([topos[i] for i in k], [vals[i] for i in k], [rhs[i] for i in k],
                                   xs, ["cg"] * n, [2] * n, [500] * n, [1e-10] * n, opts=opts)
        return k, xs, res

    k, xs, res = run(count)
    for i, x, r in zip(k, xs, res):
        s = systems[i]
        assert r["status"] == tflows.OK
        # the recurrence's residual is below 1e-10 ||b||, the true one differs by rounding
        assert np.linalg.norm(s.b - s.scipy() @ x.cpu().numpy()) <= 2e-10 * np.linalg.norm(s.b)
    if per_sm == 4:
        with pytest.raises(tflows.SolverError) as e:
            run(8 * sms + 1)
        assert e.value.status == tflows.BAD_INPUT
    for t in topos:
        t.close()
