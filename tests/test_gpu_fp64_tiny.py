"""The FP64 path's bulk terms where sum phi^4 is tiny.  Uniform fields have no
gradient, so that one step is phi - L dt dF/dphi of a single cell and leaves c
alone; the fourth term's ratios phi^3 phi_P^4 / (sum phi^4)^2 and phi_P^3 N4 /
(sum phi^4)^2 go as 1/phi and hold as long as sum phi^4 is a normal number.
Tolerance: some 30 roundings of the bulk terms and a transform there and back,
with a margin of 10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [0.5, 1e-10, 1e-30, 1e-38, 3e-39, 1e-39, 1e-45, 1e-70])
def test_uniform_cells(pkg, oracle, size):
    p = oracle.Params(8, 4, 6, 3, t_step=0.01, am=0.5, ap=5.0, con_0_mat=0.1, con_0_ppt=0.9)
    phi, c = size * np.array([1.0, 2.0, 1.5]), 0.4
    r = phi / size  # the ratios do not depend on the size
    n4, s4 = (r[:2] ** 4).sum(), (r ** 4).sum()
    d = p.am * (c - p.con_0_mat) ** 2 - p.ap * (c - p.con_0_ppt) ** 2
    term4 = np.array([*(4.0 * r[:2] ** 3 * r[2] ** 4), -4.0 * r[2] ** 3 * n4]) / s4 ** 2 * d / size
    others = (phi ** 2).sum() - phi ** 2
    want = phi - p.mob_phi * p.t_step * (phi ** 3 - phi + 2.0 * p.sigma_1 * phi * others + term4)
    assert p.sigma_1 == p.sigma_2
    run = pkg.Run(p, precision=pkg.PF_FP64_PLAIN)
    try:
        run.set_fields(np.broadcast_to(phi[:, None, None, None], (3, 6, 4, 8)).copy(), np.full((6, 4, 8), c))
        run.step(1)
        got, con = run.get_fields()
    finally:
        run.close()
    scale = np.abs(want).max() + np.abs(p.mob_phi * p.t_step * term4).max()
    assert np.abs(got - want[:, None, None, None]).max() <= 10 * 60 * 2.3e-16 * scale
    assert np.abs(con - c).max() <= 10 * 30 * 2.3e-16
