"""Planes that a cluster of CTAs shares in the yz pass, with variable mobility:
its three modes (import, main with the flux of the c planes, C2) and the side
branch of the graph, from the smallest number of fields on.  The fields are held
to the FP64 GPU path at the FP32 path's stated 1e-5, and two runs in one batch
to the same runs alone, bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import TOL32, _check_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,var", [(128, 1), (160, 1), (200, 1), (200, 2), (256, 1)])
def test_variable_mobility(pkg, oracle, n, var):
    p = oracle.Params(n, n, n, var, t_step=0.01, mobility="c1mc")
    start = pkg.ic_voronoi(p, 3, 12, 0.02, 0.45, 0.02)
    out = []
    for precision in (pkg.PF_FP64_PLAIN, pkg.PF_FP32_FUSED):
        run = pkg.Run(p, precision=precision)
        run.set_fields(*start)
        run.step(2)
        out.append(run.get_fields())
        run.close()
    _check_fields(*out[1], *out[0], TOL32)


def test_batch_equals_alone(pkg, oracle):
    ps = [oracle.Params(160, 160, 160, 1, t_step=dt, mobility="c1mc") for dt in (0.01, 0.02)]
    starts = [pkg.ic_voronoi(p, s, 8, 0.02, 0.45, 0.02) for s, p in enumerate(ps, 1)]
    batch = pkg.Batch(ps)
    for r, st in enumerate(starts):
        batch.set_fields(r, *st)
    batch.step(3)
    both = [batch.get_fields(r) for r in range(2)]
    batch.close()
    for p, st, (phi, con) in zip(ps, starts, both):
        run = pkg.Run(p)
        run.set_fields(*st)
        run.step(3)
        a, b = run.get_fields()
        run.close()
        assert np.array_equal(a, phi) and np.array_equal(b, con)
