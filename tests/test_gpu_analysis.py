"""The voxel analysis where its route changes with var -- the widest cells that
one warp's shared memory holds (799) and the general kernel beyond -- and from
several threads whose cells need different amounts of it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARRAYS = ("phi_sq", "var_num", "phi_3", "grad_phi_3", "boundary")
COUNTS = ("precipitate_voxels", "boundary_voxels", "precipitate_fraction")


def _case(oracle, shape, var):
    nz, ny, nx = shape
    rng = np.random.default_rng(var)
    return oracle.Params(Nx=nx, Ny=ny, Nz=nz, var=var), rng.random((var,) + shape) ** 3, rng.random(shape)


def _same(got, want):
    return all(np.array_equal(got[k], want[k]) for k in ARRAYS) and all(got[k] == want[k] for k in COUNTS)


@pytest.mark.parametrize("var", [799, 800, 1001])
def test_around_the_widest_cells(pkg, oracle, var):
    import pf_paraview

    p, phi, con = _case(oracle, (3, 3, 5), var)
    assert _same(pkg.analyze_fields(p, phi, con, 0.2), pf_paraview.analyze(phi, con, 0.2))


def test_threads_of_different_var(pkg, oracle):
    import pf_paraview

    errors = []

    def work(var):
        try:
            p, phi, con = _case(oracle, (4, 4, 4), var)
            want = pf_paraview.analyze(phi, con, 0.2)
            for _ in range(100):
                assert _same(pkg.analyze_fields(p, phi, con, 0.2), want)
        except BaseException as e:  # noqa: BLE001 - reported by the test's own thread
            errors.append((var, repr(e)))

    threads = [threading.Thread(target=work, args=(var,)) for var in (200, 255, 320)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
