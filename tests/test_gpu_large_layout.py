"""Runs above 512 MB of mixed-space state keep a z row of all kx together.  Under
variable mobility all modes of both passes read and write that layout: import,
the flux of the c planes into J, the mobility's x pass, the C2 pass, export and
the float fields of the analysis; planes in one CTA (128^2, the first variant)
and in clusters.  The fields are held to the FP64 GPU path at the FP32 path's
stated 1e-5; what an export or an analysis hands out twice is equal bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import TOL32, _check_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,var,variant", [(128, 64, 0), (128, 64, 1), (160, 33, 0), (256, 8, 0)])
def test_variable_mobility(pkg, oracle, monkeypatch, n, var, variant):
    import torch

    assert (var + 1) * (n // 2 + 1) * n * n * 8 > 512 << 20
    monkeypatch.setenv("PFGPU_YZ_VARIANT", str(variant))
    p = oracle.Params(n, n, n, var, t_step=0.01, mobility="c1mc")
    start = pkg.ic_voronoi(p, 3, 40, 0.02, 0.45, 0.02)
    run = pkg.Run(p, precision=pkg.PF_FP64_PLAIN)
    run.set_fields(*start)
    run.step(2)
    want = run.get_fields()
    run.close()
    run = pkg.Run(p)
    try:
        run.set_fields(*start)
        run.step(2)
        phi, con = run.get_fields()
        _check_fields(phi, con, *want, TOL32)
        pinned = torch.empty(n ** 3 * (var + 1), dtype=torch.float64, pin_memory=True).numpy()
        run.get_fields_aos(pinned[: n ** 3 * var], pinned[n ** 3 * var:])
        assert np.array_equal(pinned[: n ** 3 * var].reshape(n, n, n, var), np.moveaxis(phi, 0, -1))
        assert np.array_equal(pinned[n ** 3 * var:].reshape(n, n, n), con)
        seen = pkg.analyze_run(run, 0.3, want=("phi_3", "con"))
        assert np.array_equal(seen["phi_3"], phi[2]) and np.array_equal(seen["con"], con)
    finally:
        run.close()
