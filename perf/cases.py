"""Measured cases of the framework: what its users have it compute, through its
public entry points (the C ABI of include/pfgpu.h by the ctypes binding).

Kinds of work (``kind``):

* ``run``      a resident run between two outputs: pf_step(n) with every step's
               record, then pf_get_fields -- the loop of pf_var_diff and of
               every host that links the library;
* ``batch``    the same for several runs stepped together (pf_batch_*), as the
               sweep driver and the server do;
* ``job``      a whole short run from host arrays: pf_set_fields, pf_step(n),
               pf_get_fields, in pageable memory as a Fortran host has it;
* ``fp64``     ``run`` on the FP64 path, which serves every grid that the FP32
               path does not (any even Nx) and the precision reports;
* ``analysis`` the post-processor's voxel analysis of one output step;
* ``shim``     f_trans_ and inv_trans_ as the Fortran driver calls them.

The FP32 path keeps its fields in FP32 and hands them out as REAL*8, so its
fields and records come back here in FP32 (converted on the device); the FP64
paths' results stay FP64.
"""
import ctypes
import importlib.util
import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
DEVICE = "cuda"


def _package():
    """The package directory's name is not a Python identifier."""
    name = "pfgb300"
    if name not in sys.modules:
        root = ROOT / "phase-field-microstructure-evolution_gb300"
        spec = importlib.util.spec_from_file_location(name, root / "__init__.py", submodule_search_locations=[str(root)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _case(kind, nx, ny, nz, var, steps=0, mobility="const", start="voronoi", runs=1, **more):
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, var=var, steps=steps, mobility=mobility, start=start, runs=runs, **more)


def listed():
    return [
        # a host that looks at every step of a small run: latency and launches
        _case("run", 32, 32, 32, 4, 1, "c1mc", name="run_32_each_step"),
        # the small single run (64^3, 4 order parameters, noise start)
        _case("run", 64, 64, 64, 4, 100, "const", "noise", name="run_64_noise"),
        # the reference's own grid and coefficients (inputs/config.yaml): 96^3, 55 variants, grain-boundary mobility
        _case("run", 96, 96, 96, 55, 50, "boundary", name="run_96_config"),
        # its weak-scaling grids, ragged for an FFT: 102 = 6 x 17 ...
        _case("run", 102, 102, 102, 12, 60, "boundary", name="run_102_ragged"),
        # ... and 200, whose planes no single block holds
        _case("run", 200, 200, 200, 6, 40, "c1mc", name="run_200_scaling"),
        # the polycrystal run: 128^3, 16 order parameters, M(c)
        _case("run", 128, 128, 128, 16, 100, "c1mc", name="run_128_polycrystal"),
        # the large single run: 256^3, 32 order parameters
        _case("run", 256, 256, 256, 32, 40, "const", name="run_256_large"),
        # a parametric ensemble with coefficients of its own for every run
        _case("batch", 64, 64, 64, 8, 40, "const", "noise", 64, name="batch_64_ensemble"),
        # a short request: start up, a few steps, result down
        _case("job", 128, 128, 128, 8, 10, "const", name="job_128_short"),
        # a grid outside the FP32 path's list
        _case("fp64", 100, 100, 90, 6, 3, "boundary", name="fp64_100x100x90"),
        # one output step of the reference's own grid through the post-processor
        _case("analysis", 96, 96, 96, 55, name="analysis_96_config"),
        # one forward and one inverse transform of a Fortran host
        _case("shim", 128, 128, 128, 1, name="shim_128"),
    ]


CUBES = (16, 32, 64, 80, 96, 102, 128, 160, 200, 256)
# planes that go with every nx (rows of 102 and 200 do not divide into every x tile)
PLANES = [(n, n) for n in CUBES if n not in (102, 200)] + [(16, 32), (32, 16), (32, 64), (64, 32)]
# no drawn case has more than a sixth of the largest run's cell-steps
MAX_CELL_STEPS = 256 ** 3 * 33 * 40 // 6
MAX_FIELD_CELLS = 256 ** 3 * 17


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "run", "batch", "job", "fp64", "analysis", "shim"))
    mobility = rng.choice(("const", "boundary", "c1mc"))
    start = "noise" if mobility == "const" and rng.random() < 0.5 else "voronoi"
    if kind in ("run", "batch", "job"):
        # per-run coefficients go with small grids, as in an ensemble
        sizes = [n for n in CUBES if n <= 80] if kind == "batch" else CUBES
        nx = rng.choice(sizes)
        ny, nz = (nx, nx) if rng.random() < 0.6 else rng.choice([p for p in PLANES if p[0] <= max(sizes)])
        cells = nx * ny * nz
        runs = _log_int(rng, 2, 64) if kind == "batch" else 1
        var = _log_int(rng, 1, max(1, min(60, MAX_FIELD_CELLS // (cells * runs) - 1)))
        steps = _log_int(rng, 1, max(1, min(100 if kind != "job" else 10, MAX_CELL_STEPS // (cells * runs * (var + 1)))))
        return _case(kind, nx, ny, nz, var, steps, mobility, start, runs)
    if kind == "fp64":
        nx, ny, nz = 2 * _log_int(rng, 6, 50), _log_int(rng, 12, 100), _log_int(rng, 12, 100)
        return _case(kind, nx, ny, nz, _log_int(rng, 1, 6), rng.randint(1, 3), mobility, start)
    nx, ny, nz = (_log_int(rng, 16, 128) for _ in range(3))
    if kind == "analysis":
        return _case(kind, nx, ny, nz, _log_int(rng, 3, 24))
    return _case(kind, nx - nx % 2, ny, nz, 1)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _params(case, gen):
    """The run's coefficients: the polycrystal set, the reference's baseline
    set (grain-boundary mobility, chemical free energy), or an ensemble member's."""
    p = SimpleNamespace(Nx=case["nx"], Ny=case["ny"], Nz=case["nz"], var=case["var"], t_step=0.05, grad_coeff_phi=1.0,
                        grad_coeff_c=1.0, D_S=1.0, D_L=1.0, D_gb=0.0, mob_phi=1.0, sigma_1=1.5, sigma_2=1.5, am=0.0,
                        ap=0.0, con_0_mat=0.0, con_0_ppt=1.0, mobility="reference")
    if case["mobility"] == "boundary":
        p.t_step, p.D_gb, p.am, p.ap, p.con_0_mat = 1e-4, 1.0, 0.5, 5.0, 0.1
    elif case["mobility"] == "c1mc":
        p.t_step, p.mobility = 0.1, "c1mc"
    if case["kind"] == "batch":
        a, b, c = torch.rand(3, generator=gen, device=DEVICE, dtype=torch.float64).tolist()
        p.mob_phi = 0.1 * 100.0 ** a if case["mobility"] == "const" else 0.5 + a
        p.grad_coeff_phi = p.grad_coeff_c = 0.5 + 3.5 * b
        p.sigma_1 = p.sigma_2 = 1.0 + c
    return p


def _uniform(shape, amp, gen):
    return torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float64).mul_(2.0).sub_(1.0).mul_(amp)


def _grains(case, gen):
    """Variant of every cell: nearest of some seed points, periodic."""
    n = (case["nz"], case["ny"], case["nx"])
    count = max(2, min(256, n[0] * n[1] * n[2] // 16384))
    at = torch.rand((count, 3), generator=gen, device=DEVICE).tolist()
    axes = [torch.arange(k, device=DEVICE, dtype=torch.float32) for k in n]
    best = torch.full(n, float("inf"), device=DEVICE)
    label = torch.zeros(n, dtype=torch.int64, device=DEVICE)
    for g, point in enumerate(at):
        d = []
        for k in range(3):
            x = (axes[k] - point[k] * n[k]).abs()
            d.append(torch.minimum(x, n[k] - x).square())
        dist = d[0][:, None, None] + d[1][None, :, None] + d[2][None, None, :]
        near = dist < best
        best = torch.where(near, dist, best)
        label.masked_fill_(near, g % case["var"])
    return label


def _start(case, gen):
    """phi[z, y, x, var] and con[z, y, x] in FP64 on the GPU."""
    n = (case["nz"], case["ny"], case["nx"])
    if case["start"] == "noise":
        return _uniform(n + (case["var"],), 0.001, gen), _uniform(n, 0.01, gen).add_(0.5)
    label = _grains(case, gen)
    phi = _uniform(n + (case["var"],), 0.01, gen)
    one = torch.ones((), device=DEVICE, dtype=torch.float64)
    phi.scatter_add_(3, label.unsqueeze(3), one.expand(n + (1,)))
    if case["kind"] == "analysis":  # interfaces a few cells wide, as a run has them
        phi.add_(torch.roll(phi, (1, 1, 2), (0, 1, 2))).mul_(0.5)
    return phi, _uniform(n, 0.02, gen).add_(0.5)


def _members(case, seed):
    """(coefficients, phi, con) of every run of the case, one at a time."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    for _ in range(case["runs"]):
        p = _params(case, gen)
        yield (p,) + _start(case, gen)


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    pkg = _package()
    lib = pkg.load_library()
    cells, var, runs = case["nx"] * case["ny"] * case["nz"], case["var"], case["runs"]
    s = SimpleNamespace(case=case, lib=lib, pkg=pkg, cells=cells, split=cells * var)
    if case["kind"] == "shim":
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed)
        s.field = _uniform((cells,), 1.0, gen).cpu()
        s.spec = torch.empty(2 * (case["nx"] // 2 + 1) * case["ny"] * case["nz"], dtype=torch.float64)
        s.back = torch.empty(cells, dtype=torch.float64)
        ints = ctypes.c_int * 3
        s.n = [ctypes.c_int(case[k]) for k in ("nx", "ny", "nz")]
        s.first = ints(1, 1, 1)
        s.ien = ints(case["nx"], case["ny"], case["nz"])
        s.fen = ints(case["nz"], case["ny"], case["nx"] // 2 + 1)
        return s
    if case["kind"] == "analysis":
        p, phi, con = next(_members(case, seed))
        s.cfg = pkg.make_config(p)
        s.phi, s.con = phi.cpu(), con.cpu()
        n = (case["nz"], case["ny"], case["nx"])
        s.out = {k: torch.empty(n, dtype=torch.int32 if k == "var_num" else torch.float64)
                 for k in ("phi_sq", "var_num", "phi_3", "grad_phi_3", "boundary")}
        s.ptrs, s.counts = pkg.AnalysisOut(), pkg.VoxelCounts()
        for k, t in s.out.items():
            setattr(s.ptrs, k, ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_int if k == "var_num" else ctypes.c_double)))
        return s
    # the fields of every run: phi(var, x, y, z), then con(x, y, z)
    s.fields = torch.empty((runs, cells * (var + 1)), dtype=torch.float64, pin_memory=case["kind"] != "job")
    s.diag = (pkg.Diag * (runs * case["steps"]))()
    ps = []
    for r, (p, phi, con) in enumerate(_members(case, seed)):
        s.fields[r, :s.split].copy_(phi.reshape(-1))
        s.fields[r, s.split:].copy_(con.reshape(-1))
        ps.append(p)
        del phi, con
    if case["kind"] == "batch":
        s.owner = pkg.Batch(ps)
        for r in range(runs):
            _ok(s, lib.pf_batch_set_fields(s.owner.h, r, _ptr(s.fields[r]), _ptr(s.fields[r, s.split:])))
        return s
    s.owner = pkg.Run(ps[0], precision=pkg.PF_FP64_PLAIN if case["kind"] == "fp64" else pkg.PF_FP32_FUSED)
    if case["kind"] == "job":
        s.start, s.fields = s.fields, torch.empty_like(s.fields)
    else:
        _ok(s, lib.pf_set_fields(s.owner.h, _ptr(s.fields), _ptr(s.fields[0, s.split:])))
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
ENERGIES = ("f_int", "f_eta", "f_ch", "e_tot")
EXTREMES = ("c_max", "c_min", "phi_min", "phi_P_max")
RECORD = np.dtype([("step", "i4"), ("nonfinite", "i4")] + [(k, "f8") for k in ENERGIES + EXTREMES + ("mass",)])


def _ok(s, rc):
    if rc:
        raise s.pkg.PFError(rc, s.lib.pf_last_error().decode())


def _results(s):
    """Fields and records of a pass: on the FP32 path in FP32, on the device."""
    real = np.float64 if s.case["kind"] == "fp64" else np.float32
    fields = s.fields if real is np.float64 else s.fields.to(DEVICE).to(torch.float32)
    rec = np.frombuffer(s.diag, dtype=RECORD)
    return {
        "phi": fields[:, :s.split],
        "con": fields[:, s.split:],
        "energies": np.stack([rec[k] for k in ENERGIES], 1).astype(real),
        "extremes": np.stack([rec[k] for k in EXTREMES], 1).astype(real),
        "mass": rec["mass"].astype(real),
        "counts": np.stack([rec["step"], rec["nonfinite"]], 1),
    }


def run(s):
    lib, case = s.lib, s.case
    if case["kind"] == "shim":
        nx, ny, nz = (ctypes.byref(v) for v in s.n)
        lib.f_trans_(_ptr(s.field), _ptr(s.spec), nx, ny, nz, s.first, s.ien, s.first, s.fen)
        lib.inv_trans_(_ptr(s.spec), _ptr(s.back), s.first, s.ien, s.first, s.fen)
        return {"spec": s.spec, "back": s.back}
    if case["kind"] == "analysis":
        _ok(s, lib.pf_analyze_fields(ctypes.byref(s.cfg), _ptr(s.phi), _ptr(s.con), 0.3, ctypes.byref(s.ptrs),
                                     ctypes.byref(s.counts)))
        return dict(s.out, voxels=[s.counts.precipitate_voxels, s.counts.boundary_voxels],
                    fraction=np.float64(s.counts.precipitate_fraction))
    h = s.owner.h
    if case["kind"] == "batch":
        _ok(s, lib.pf_batch_step(h, case["steps"], s.diag))
        for r in range(case["runs"]):
            _ok(s, lib.pf_batch_get_fields(h, r, _ptr(s.fields[r]), _ptr(s.fields[r, s.split:])))
        return _results(s)
    if case["kind"] == "job":
        _ok(s, lib.pf_set_fields(h, _ptr(s.start), _ptr(s.start[0, s.split:])))
    _ok(s, lib.pf_step(h, case["steps"], s.diag))
    _ok(s, lib.pf_get_fields(h, _ptr(s.fields), _ptr(s.fields[0, s.split:])))
    return _results(s)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    cells, nf = case["nx"] * case["ny"] * case["nz"], case["var"] + 1
    fft = 2.5 * cells * math.log2(cells)  # one real 3-D transform
    if case["kind"] == "shim":
        return {"bytes": 2 * (8 * cells + 16 * (case["nx"] // 2 + 1) * case["ny"] * case["nz"]), "flops": 2 * fft}
    if case["kind"] == "analysis":
        return {"bytes": cells * (8 * nf + 4 * 8 + 4), "flops": cells * (4 * case["var"] + 12)}
    real = 8 if case["kind"] == "fp64" else 4
    # a step reads and writes every field once; it transforms the driving force of every field forward and the new
    # field back, and with variable mobility the flux both ways
    transforms = 2 * nf + (0 if case["mobility"] == "const" else 2)
    steps = case["steps"] * case["runs"]
    move = 8 * cells * nf * case["runs"] * (2 if case["kind"] == "job" else 1)
    return {"bytes": steps * 2 * real * cells * nf + move, "flops": steps * (transforms * fft + 30.0 * cells * nf)}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _wavenumbers(n, count, axis):
    m = torch.arange(count, device=DEVICE, dtype=torch.float64)
    q = torch.where(m <= n // 2, m, m - n) * (2.0 * math.pi / n)
    shape = [1, 1, 1]
    shape[axis] = count
    return q.reshape(shape), torch.where(2 * m == n, torch.zeros_like(q), q).reshape(shape)


def _exact_run(p, phi, con, steps):
    """The semi-implicit steps of one run: Allen-Cahn for phi, Cahn-Hilliard for con."""
    n, cells, dt, last = con.shape, con.numel(), p.t_step, p.var - 1
    qx, gx = _wavenumbers(p.Nx, p.Nx // 2 + 1, 2)
    qy, gy = _wavenumbers(p.Ny, p.Ny, 1)
    qz, gz = _wavenumbers(p.Nz, p.Nz, 0)
    q2, q4 = qx ** 2 + qy ** 2 + qz ** 2, qx ** 4 + qy ** 4 + qz ** 4
    g, g2 = gx + gy + gz, gx ** 2 + gy ** 2 + gz ** 2
    k3 = -(gx * qx ** 2 + gy * qy ** 2 + gz * qz ** 2)
    weight = torch.full((1, 1, p.Nx // 2 + 1), 2.0, device=DEVICE, dtype=torch.float64)
    weight[..., 0] = 1.0
    if p.Nx % 2 == 0:
        weight[..., -1] = 1.0
    g2 = g2 * weight

    def forward(a):
        return torch.fft.rfftn(a, norm="forward")

    def back(a):
        return torch.fft.irfftn(a, s=n, norm="forward")

    def gradient(spectrum):
        return float((g2 * (spectrum.real ** 2 + spectrum.imag ** 2)).sum())

    phi = [phi[..., f].contiguous() for f in range(p.var)]
    spec = [forward(f) for f in phi]
    con_spec = forward(con)
    records = []
    for _ in range(steps):
        fint = 0.5 * cells * (p.grad_coeff_phi * sum(gradient(a) for a in spec) + p.grad_coeff_c * gradient(con_spec))
        pre, quart, pairs = torch.zeros_like(con), torch.zeros_like(con), torch.zeros_like(con)
        for f in range(last):
            a = phi[f] ** 2
            pairs += a * pre
            pre += a
            quart += a * a
        ppt = phi[last]
        pp2 = ppt ** 2
        s2, s4 = pre + pp2, quart + pp2 ** 2
        feta = float((-0.5 * s2 + 0.25 * s4 + p.sigma_1 * pairs + p.sigma_2 * pp2 * pre).sum())
        h = quart / s4
        dm, dp = con - p.con_0_mat, con - p.con_0_ppt
        fm, fp = p.am * dm ** 2, p.ap * dp ** 2
        fch = float((h * fm + (1.0 - h) * fp).sum())
        mu = 2.0 * h * p.am * dm + 2.0 * (1.0 - h) * p.ap * dp
        records.append((fint, feta, fch, fint + feta + fch, max(0.0, float(con.max())), min(1.0, float(con.min())),
                        min(1.0, float(s2.min())), max(0.0, float(ppt.max())), float(con.sum())))
        if p.mobility == "c1mc":
            extra = p.D_L * con * (1.0 - con)
        else:
            extra = 2.0 * (1.0 - s2) * p.D_gb
        t4 = 4.0 * (pp2 / s4) * (pp2 / s4) * (fm - fp)
        t4p = -4.0 * (ppt ** 3 / s4) * h * (fm - fp)
        den = 1.0 + p.mob_phi * p.grad_coeff_phi * dt * q2
        for f in range(p.var):
            a = phi[f]
            if f < last:
                force = a ** 3 - a + 2.0 * a * (p.sigma_1 * (pre - a * a) + p.sigma_2 * pp2) + t4 * a ** 3
            else:
                force = a ** 3 - a + 2.0 * a * p.sigma_2 * pre + t4p
            spec[f] = (spec[f] - p.mob_phi * dt * forward(force)) / den
            phi[f] = back(spec[f])
        mu_spec = forward(mu)
        new = con_spec - p.D_L * dt * q2 * mu_spec
        if p.mobility == "c1mc" or p.D_gb != 0.0:
            flux = back(1j * (g * mu_spec - p.grad_coeff_c * k3 * con_spec)) * extra
            new = new + 1j * g * dt * forward(flux)
        con_spec = new / (1.0 + p.D_L * dt * p.grad_coeff_c * q4)
        con = back(con_spec)
    return torch.stack(phi, -1).reshape(-1), con.reshape(-1), np.array(records)


def _exact_analysis(case, seed):
    _, phi, _ = next(_members(case, seed))
    at3 = phi[..., 2].contiguous()
    grad = torch.zeros_like(at3)
    if min(at3.shape) > 2:
        mid = slice(1, -1)
        d = [(at3[2:, mid, mid] - at3[:-2, mid, mid]) / 2, (at3[mid, 2:, mid] - at3[mid, :-2, mid]) / 2,
             (at3[mid, mid, 2:] - at3[mid, mid, :-2]) / 2]
        grad[mid, mid, mid] = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt()
    above = phi > 0.3
    edge = above.sum(-1) > 1
    count = int(edge.sum())
    fraction = float((edge & above[..., -1]).sum()) / count if count else 0.0
    return {"phi_sq": (phi ** 2).sum(-1), "var_num": None, "phi_3": at3, "grad_phi_3": grad, "boundary": edge.double(),
            "voxels": None, "fraction": np.float64(fraction)}


def exact(case, seed):
    if case["kind"] == "shim":
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed)
        field = _uniform((case["nx"] * case["ny"] * case["nz"],), 1.0, gen)
        spec = torch.fft.rfftn(field.reshape(case["nz"], case["ny"], case["nx"]), norm="forward")
        return {"spec": torch.view_as_real(spec.permute(2, 1, 0).contiguous()).reshape(-1), "back": field}
    if case["kind"] == "analysis":
        return _exact_analysis(case, seed)
    cells = case["nx"] * case["ny"] * case["nz"]
    phi = torch.empty((case["runs"], cells * case["var"]), device=DEVICE, dtype=torch.float64)
    con = torch.empty((case["runs"], cells), device=DEVICE, dtype=torch.float64)
    records = []
    for r, (p, a, c) in enumerate(_members(case, seed)):
        phi[r], con[r], rec = _exact_run(p, a, c, case["steps"])
        records.append(rec)
    rec = np.concatenate(records)
    return {"phi": phi, "con": con, "energies": rec[:, 0:4].copy(), "extremes": rec[:, 4:8].copy(),
            "mass": rec[:, 8].copy(), "counts": None}
