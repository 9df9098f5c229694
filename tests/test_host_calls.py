"""The library's host code against a CUDA runtime of the host (fake_cuda.cpp):
what it allocates and when, and how it leaves a call that fails.  No GPU."""
import ctypes
import importlib.util
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
DP = ctypes.POINTER(ctypes.c_double)
PF_ENOMEM = -3


@pytest.fixture(scope="module")
def fake(pkg, lib, tmp_path_factory):
    out = Path(pkg.__file__).parent / "_build"
    home = importlib.util.spec_from_file_location("recipe", Path(pkg.__file__).parent / "build.py")
    recipe = importlib.util.module_from_spec(home)
    home.loader.exec_module(recipe)
    so = tmp_path_factory.mktemp("fake") / "libpfgpu_fake.so"
    objs = [str(out / (p.stem + ".o")) for p in recipe._sources()]
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(recipe.cuda_home() / "include"),
                    str(ROOT / "tests" / "fake_cuda.cpp"), *objs, "-Wl,-Bsymbolic", "-Wl,-z,defs", "-lpthread",
                    "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so))
    f.fake_order.restype = f.pf_last_error.restype = ctypes.c_char_p
    f.fake_reset()
    return f


@pytest.fixture(autouse=True)
def clean(fake):
    fake.fake_reset()


def _ptr(a):
    return a.ctypes.data_as(DP)


class Run:
    """A run of 16^3 cells, with host fields."""

    def __init__(self, fake, pkg, oracle, precision=32, var=2, **more):
        self.f = fake
        cfg = pkg.make_config(oracle.Params(16, 16, 16, var, **more), precision)
        self.h = ctypes.c_void_p()
        assert fake.pf_create(ctypes.byref(cfg), ctypes.byref(self.h)) == 0, fake.pf_last_error()
        self.phi, self.con = np.zeros(16 ** 3 * var), np.zeros(16 ** 3)

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.f.pf_destroy(self.h)


@pytest.mark.parametrize("coherent", [0, 1])
@pytest.mark.parametrize("precision", [32, 64])
def test_memory_is_allocated_when_the_run_is_made(fake, pkg, oracle, coherent, precision):
    """After pf_create a run needs no more device memory to take fields, step and hand them out."""
    fake.fake_coherent(coherent)
    with Run(fake, pkg, oracle, precision, mobility="c1mc") as r:
        fake.fake_fail(b"cudaMalloc", 1, 2)
        assert fake.pf_set_fields(r.h, _ptr(r.phi), _ptr(r.con)) == 0
        assert fake.pf_step(r.h, 5, None) == 0
        assert fake.pf_get_fields(r.h, _ptr(r.phi), _ptr(r.con)) == 0, fake.pf_last_error()
    fake.fake_reset()
    if precision == 32:  # and where there is none, it is pf_create that says so
        fake.fake_fail(b"cudaMalloc", 3, 2)
        cfg, h = pkg.make_config(oracle.Params(16, 16, 16, 2)), ctypes.c_void_p()
        assert fake.pf_create(ctypes.byref(cfg), ctypes.byref(h)) == PF_ENOMEM


@pytest.mark.parametrize("call,step,nth", [("set", b"cudaLaunchKernelExC", 1), ("set", b"cudaMemsetAsync", 1),
                                           ("get", b"cudaMemcpyAsync", 2), ("set64", b"cudaMemcpyAsync", 2),
                                           ("get64", b"cudaMemcpyAsync", 2), ("f_trans", b"launch", 1),
                                           ("inv_trans", b"cufftExec", 1)])
def test_a_failed_call_leaves_the_callers_memory_alone(fake, pkg, oracle, call, step, nth):
    """Kernels and copies already under way on the caller's arrays have ended when the call reports its error."""
    with Run(fake, pkg, oracle, 64 if call.endswith("64") else 32) as r:
        three = ctypes.c_int * 3
        n, one, ien, fen = ctypes.c_int(16), three(1, 1, 1), three(16, 16, 16), three(16, 16, 9)
        spec = np.zeros(2 * 9 * 256)
        fake.fake_reset()
        fake.fake_fail(step, nth, 700)
        if call == "f_trans":
            fake.f_trans_(_ptr(r.con), _ptr(spec), ctypes.byref(n), ctypes.byref(n), ctypes.byref(n), one, ien, one, fen)
        elif call == "inv_trans":
            fake.inv_trans_(_ptr(spec), _ptr(r.con), one, ien, one, fen)
        else:
            fn = fake.pf_set_fields if call.startswith("set") else fake.pf_get_fields
            assert fn(r.h, _ptr(r.phi), _ptr(r.con)) != 0
        _, failed, after = fake.fake_order().decode().partition("FAILED")
        assert failed and "cudaStreamSynchronize" in after, fake.fake_order()


def test_analysis_never_lowers_a_kernels_shared_memory(fake, pkg, oracle):
    """The limit is the process's: lowered for one call, it would fail another thread's larger one."""
    fields = np.ones((256, 64))
    counts = pkg.VoxelCounts()
    for var in (255, 200, 230, 700, 193):
        cfg = pkg.make_config(oracle.Params(4, 4, 4, var))
        assert fake.pf_analyze_fields(ctypes.byref(cfg), _ptr(np.ones(64 * var)), _ptr(fields[0]), ctypes.c_double(0.3),
                                      None, ctypes.byref(counts)) == 0
    assert fake.fake_count(b"cudaFuncSetAttribute") > 0 and fake.fake_lowered() == 0


class Shim:
    """f_trans_ of a grid no other test uses."""

    def __init__(self, fake, nx, ny, nz):
        three = ctypes.c_int * 3
        self.f, self.n = fake, [ctypes.c_int(v) for v in (nx, ny, nz)]
        self.one, self.ien, self.fen = three(1, 1, 1), three(nx, ny, nz), three(nz, ny, nx // 2 + 1)
        self.real, self.spec = np.zeros(nx * ny * nz), np.zeros(2 * (nx // 2 + 1) * ny * nz)

    def __call__(self):
        self.f.f_trans_(_ptr(self.real), _ptr(self.spec), *map(ctypes.byref, self.n), self.one, self.ien, self.one, self.fen)


def test_shims_use_what_belongs_to_their_device(fake):
    shim = Shim(fake, 6, 4, 2)
    try:
        for device in (0, 1, 0, 1):
            assert fake.pf_shim_device(device) == 0
            shim()
    finally:
        fake.pf_shim_device(0)
    assert fake.fake_strays() == 0
    assert fake.fake_count(b"cufftPlan") == 4  # two a device, kept


@pytest.mark.parametrize("step,nth", [(b"cudaMalloc", 1), (b"cudaMalloc", 3), (b"cufftPlan", 1), (b"cufftPlan", 2)])
def test_shims_give_back_what_they_could_not_finish(fake, capfd, step, nth):
    shim = Shim(fake, 6, 4, 10 + 2 * nth + len(step))
    before = fake.fake_live()
    fake.fake_fail(step, nth, 2)
    shim()
    assert b"FAILED" in fake.fake_order() and fake.fake_live() == before
    assert "f_trans_" in capfd.readouterr().err
    shim()  # and the next call makes them
    assert fake.fake_count(b"cufftExec") == 1 and capfd.readouterr().err == ""


@pytest.mark.parametrize("precision,nth", [(32, 1), (32, 2), (32, 3), (64, 1)])
def test_a_run_that_does_not_fit_is_no_error_of_the_others(fake, pkg, oracle, precision, nth):
    cfg, h = pkg.make_config(oracle.Params(16, 16, 16, 2), precision), ctypes.c_void_p()
    with Run(fake, pkg, oracle) as r:
        before = fake.fake_live()
        fake.fake_fail(b"cudaMalloc", nth, 2)
        assert fake.pf_create(ctypes.byref(cfg), ctypes.byref(h)) < 0
        assert fake.fake_live() == before
        assert fake.pf_set_fields(r.h, _ptr(r.phi), _ptr(r.con)) == 0, fake.pf_last_error()


def test_an_fp64_run_is_one_allocation(fake, pkg, oracle):
    """Short FP64 runs pay for their memory and plans as much as for their steps."""
    with Run(fake, pkg, oracle, 64, mobility="c1mc"):
        assert fake.fake_count(b"cudaMalloc") == 1 and fake.fake_count(b"cufftPlan") == 4
    assert fake.fake_count(b"cudaFree") == 1


@pytest.mark.parametrize("call,step", [("analyze", b"cudaMalloc"), ("analyze_run", b"cudaMalloc"), ("set", b"cudaMemcpyAsync"),
                                       ("get", b"cudaMemcpyAsync"), ("set64", b"cudaMemcpyAsync"), ("f_trans", b"cudaMemcpy")])
def test_a_failed_call_is_no_error_of_the_next_one(fake, pkg, oracle, call, step):
    cfg, counts = pkg.make_config(oracle.Params(16, 16, 16, 3)), pkg.VoxelCounts()
    more = ctypes.c_double(0.3), None, ctypes.byref(counts)
    fake.fake_coherent(0)  # fields go in by copies
    with Run(fake, pkg, oracle) as other, Run(fake, pkg, oracle, 64 if call == "set64" else 32, var=3) as r:
        fake.fake_fail(step, 1, 2)
        if call == "analyze":
            assert fake.pf_analyze_fields(ctypes.byref(cfg), _ptr(r.phi), _ptr(r.con), *more) < 0
        elif call == "analyze_run":
            assert fake.pf_analyze_run(r.h, *more) < 0
        elif call == "f_trans":
            Shim(fake, 6, 4, 8)()
        else:
            assert (fake.pf_get_fields if call == "get" else fake.pf_set_fields)(r.h, _ptr(r.phi), _ptr(r.con)) < 0
        assert b"FAILED" in fake.fake_order()
        assert fake.pf_set_fields(other.h, _ptr(other.phi), _ptr(other.con)) == 0, fake.pf_last_error()
