"""What the library makes of CUDA calls that fail or report an error: in child processes, with the
runtime's calls faked (cuda_fakes.c)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent

CHILD = """
import ctypes as C
import sys

import numpy as np

import yukawacolourednoise_gb300 as yk

fakes = C.CDLL(sys.argv[1])


def params(L, **kw):
    base = dict(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=1.0, cut_fraction=1.0,
                Nt=L, Nx=L, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=20000, fixed_dt=0.01, seed=1234,
                init=yk.YK_INIT_PHILOX, precision=yk.YK_MIXED)
    return yk.Params.default(**(base | kw))


def buffer(a):
    rt, p = C.CDLL("libcudart.so.13"), C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 4) == 0
    return p.value
"""


@pytest.fixture(scope="module")
def child(tmp_path_factory, ylib):
    lib = tmp_path_factory.mktemp("fakes") / "cuda_fakes.so"
    inc = next(p for p in ("/usr/local/cuda/include", os.environ.get("CUDA_HOME", "") + "/include") if Path(p).exists())
    subprocess.run(["gcc", "-shared", "-fPIC", "-I", inc, "-o", str(lib), str(HERE / "cuda_fakes.c"), "-ldl"], check=True)

    def run(body):
        env = dict(os.environ, LD_PRELOAD=str(lib), PYTHONPATH=str(HERE.parent))
        r = subprocess.run([sys.executable, "-c", CHILD + body, str(lib)], env=env, cwd=HERE.parent, capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stderr
    return run


def test_timeout_of_one_group_is_kept(child):
    # a batch whose cluster solves run in groups of one form: an error that is recorded
    # before any of them starts outlasts them all
    child("""
with yk.Context([params(64, n_rhs=40), params(16, wilson_param=0.7), params(128, n_rhs=20)]) as ctx:
    ctx.step(1)
    for launch in (1, 2, 3):
        ctx.profile_begin()   # the step's launches one by one, not as a graph
        fakes.fake_error(launch, yk.YK_ETIMEOUT)
        ctx.step(1)
        try:
            ctx.synchronize()
        except yk.YukawaError as e:
            assert e.status == yk.YK_ETIMEOUT
        else:
            raise AssertionError(launch)
        ctx.step(1)           # the next step's solves start without it
        ctx.synchronize()
        ctx.profile_end()
""")


def test_timeout_of_the_first_plane_solve_is_kept(child):
    child("""
b = np.random.default_rng(1).normal(size=(64 * 64, 8))
with yk.Context(params(64)) as ctx:
    ctx.synchronize()
    fakes.fake_error(2, yk.YK_ETIMEOUT)
    try:
        ctx.cg_solve(buffer(b), buffer(b), tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=5000, precision=yk.YK_MIXED)
    except yk.YukawaError as e:
        assert e.status == yk.YK_ETIMEOUT
    else:
        raise AssertionError
    st = ctx.cg_solve(buffer(b), buffer(b), tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=5000, precision=yk.YK_MIXED)
    assert st.converged == 1
""")


def test_no_memory_for_the_planes(child):
    # a mixed solve that finds no room for the plane solves' workspace runs on the one there
    # is; with room again it takes the planes
    child("""
b, x = (buffer(np.random.default_rng(1).normal(size=(64 * 64, 8))) for _ in range(2))
solve = dict(tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=5000)
with yk.Context(params(64)) as ctx:
    ctx.cg_solve(b, x, precision=yk.YK_FP64, **solve)   # the workspace of every solve
    fakes.fake_no_memory(1)
    st = ctx.cg_solve(b, x, precision=yk.YK_MIXED, **solve)
    assert st.converged == 1
    fakes.fake_no_memory(0)
    assert ctx.cg_solve(b, x, precision=yk.YK_MIXED, **solve).reliable_updates > st.reliable_updates   # two solves' updates
""")


@pytest.mark.parametrize("chains", ["params(32), params(64, wilson_param=0.7)", "params(32, precision=yk.YK_FP64)",
                                    "params(128, precision=yk.YK_FP64)", "params(64, cut_fraction=0.35)", "params(512)",
                                    "params(33), params(20)"])
def test_launches_of_a_profiled_step(child, chains):
    child(f"""
with yk.Context([{chains}]) as ctx:
    ctx.step(1)
    ctx.profile_begin()
    n = fakes.fake_launches()
    ctx.step(2)
    n = fakes.fake_launches() - n
    assert ctx.profile_end().launches == n, n
""")


def test_cluster_kernels_on_another_device(child):
    # kernel attributes hold for one device: a process that makes contexts on two sets them for
    # both (here one device that calls itself another)
    child("""
def attributes():
    n = fakes.fake_cluster_attributes()
    with yk.Context(params(32, precision=yk.YK_FP64)) as ctx:
        ctx.step(1)
        assert ctx.observables().status == 0
    return fakes.fake_cluster_attributes() - n

first = attributes()
assert first > 0 and attributes() == 0
fakes.fake_device(1)
assert attributes() == first
""")
