"""What the autotuner times: steps of runs that hold fields, every run of the
batch, so that the bulk terms take the branch they take in earnest.  The
tuner's report ends with the least sum of phi^2 that its last step found in
each run."""
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/oracle"]
import __graft_entry__ as ge, pf_ref
pkg = ge.load_package()
n, var, mobility = {n}, {var}, {mobility!r}
bulk = dict(am=0.5, ap=5.0, con_0_mat=0.1) if mobility == "reference" else {{}}  # with M(c) no start holds under these
ps = [pf_ref.Params(n, n, n, var, mob_phi=m, mobility=mobility, **bulk) for m in {mob_phi}]
pkg.Batch(ps).close()
"""


@pytest.mark.parametrize("n,var,mobility,mob_phi", [(64, 1, "reference", (1.0,)), (64, 8, "reference", (1.0, 0.0, 5.0)),
                                                    (80, 12, "c1mc", (1.0, 0.1)), (96, 55, "reference", (1.0,))])
def test_every_run_holds_fields(n, var, mobility, mob_phi):
    root = str(Path(__file__).resolve().parents[1])
    env = {k: v for k, v in os.environ.items() if not k.startswith("PFGPU_")}
    r = subprocess.run([sys.executable, "-c", CODE.format(root=root, n=n, var=var, mobility=mobility, mob_phi=mob_phi)],
                       env=dict(env, PFGPU_AUTOTUNE_REPORT="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    state = re.findall(r"run (\d+): phi_min (\S+), (\d+) non-finite", r.stderr)
    assert [int(s[0]) for s in state] == list(range(len(mob_phi))), r.stderr
    for _, phi_min, bad in state:
        assert float(phi_min) > 0.1 and bad == "0", r.stderr
