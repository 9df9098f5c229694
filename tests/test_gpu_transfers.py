"""Fields in and out of a run, from every kind of host memory the entry points
take: pageable and pinned memory that the kernels read and write themselves,
and memory that does not start on a double, which goes through copies.  All
hold the same values, so the results are equal bit for bit.  Also the FP64
path's batched transforms (a last chunk of fewer fields) and the voxel
analysis at the edges of its 32-cell groups."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import TOL64, _check_diag, _check_fields, _run_lib

pytestmark = pytest.mark.gpu


def _buffer(n, kind):
    if kind == "pinned":
        import torch

        return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
    if kind == "odd":  # four bytes off a double
        return np.empty(8 * n + 4, dtype=np.uint8)[4:].view(np.float64)
    return np.empty(n)


@pytest.mark.parametrize("shape,var", [((32, 16, 32), 1), ((64, 64, 32), 5), ((102, 102, 102), 2), ((96, 96, 96), 17)])
def test_fields_from_and_to_any_host_memory(pkg, oracle, shape, var):
    nx, ny, nz = shape
    p = oracle.Params(nx, ny, nz, var, t_step=0.01, mobility="c1mc")
    rng = np.random.default_rng(var)
    n = nx * ny * nz
    phi, con = rng.random(n * var) - 0.5, rng.random(n)
    lib, dp = pkg.load_library(), ctypes.POINTER(ctypes.c_double)
    run = pkg.Run(p)
    try:
        want = None
        for kind_in in ("pageable", "pinned", "odd"):
            a, c = _buffer(n * var, kind_in), _buffer(n, kind_in)
            a[:], c[:] = phi, con
            for kind_out in ("pageable", "pinned", "odd"):
                assert lib.pf_set_fields(run.h, a.ctypes.data_as(dp), c.ctypes.data_as(dp)) == 0
                run.step(2)
                b, d = _buffer(n * var, kind_out), _buffer(n, kind_out)
                assert lib.pf_get_fields(run.h, b.ctypes.data_as(dp), d.ctypes.data_as(dp)) == 0
                assert np.array_equal(a, phi) and np.array_equal(c, con)  # the caller's fields are only read
                if want is None:
                    want = b.copy(), d.copy()
                assert np.array_equal(b, want[0]) and np.array_equal(d, want[1]), (kind_in, kind_out)
    finally:
        run.close()


def test_batch_records_when_runs_stand_apart(pkg, oracle):
    """Records come back for all runs at once while the runs stand at the same
    step, and run by run after one of them has started afresh."""
    p = oracle.Params(32, 32, 32, 3, t_step=0.02)
    phi, con = oracle.ic_noise(p, 5, 0.01, 0.5, 0.01)
    b = pkg.Batch([p, p, p])
    try:
        for r in range(3):
            b.set_fields(r, phi, con)
        first = b.step(7)
        b.set_fields(1, phi, con)
        second = b.step(1030)  # longer than the ring of 1024 records
    finally:
        b.close()
    assert first[0] == first[1] == first[2]
    assert [d["step"] for d in second[0]] == list(range(8, 1038))
    assert [d["step"] for d in second[1]] == list(range(1, 1031))
    assert second[1][:7] == first[0]
    assert second[1][7:] == second[0][:1023] and second[2] == second[0]


def test_fp64_path_with_a_short_last_chunk(pkg, oracle):
    """9 fields of 100 x 96 x 90: transformed five at a time, then one by one."""
    p = oracle.Params(100, 96, 90, 9, t_step=0.002, D_gb=0.5, am=0.5, ap=2.0, con_0_mat=0.3, con_0_ppt=0.7)
    phi, con = pkg.ic_voronoi(p, 3, 12, 0.05, 0.5, 0.02)
    gp, gc, gd = _run_lib(pkg, p, phi, con, 2, precision=64)
    op, oc, od = oracle.run(p, phi, con, 2, faithful=True, workers=8)
    _check_fields(gp, gc, op, oc, TOL64)
    _check_diag(gd, od, 1e-9, oracle.stats(phi, con))


@pytest.mark.parametrize("shape,var", [((1, 1, 3), 3), ((3, 3, 7), 31), ((4, 4, 4), 32), ((3, 5, 9), 33), ((2, 3, 11), 255),
                                       ((3, 3, 5), 700)])
def test_analysis_at_group_edges(pkg, oracle, shape, var):
    import pf_paraview

    nz, ny, nx = shape
    p = oracle.Params(Nx=nx, Ny=ny, Nz=nz, var=var)
    rng = np.random.default_rng(var)
    phi, con = rng.random((var,) + shape) ** 3, rng.random(shape)
    got = pkg.analyze_fields(p, phi, con, 0.2)
    want = pf_paraview.analyze(phi, con, 0.2)
    for k in ("phi_sq", "var_num", "phi_3", "grad_phi_3", "boundary"):
        assert np.array_equal(got[k], want[k]), k
    for k in ("precipitate_voxels", "boundary_voxels", "precipitate_fraction"):
        assert got[k] == want[k], k
