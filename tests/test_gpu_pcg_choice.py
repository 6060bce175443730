"""Which form of the learned iteration runs: not slower than one launch a phase."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# networks whose tile and halo leave room for two blocks an SM, for one, on lattices with more
# tiles than SMs and fewer
@pytest.mark.parametrize("Nt,Nx,layers", [(512, 512, 5), (512, 512, 8), (256, 512, 7), (256, 256, 8)])
def test_time(ylib, cuda, monkeypatch, Nt, Nx, layers):
    yk = ylib
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.02, cut_fraction=1.0, Nt=Nt,
                          Nx=Nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, fixed_dt=1e-6, seed=1, init=yk.YK_INIT_NONE,
                          precision=yk.YK_MIXED)
    sig = 2.13 + 0.4 * np.random.default_rng(2).normal(size=Nt * Nx)
    best = {}
    for tile in ("", "8x64x1"):
        if tile:
            monkeypatch.setenv("YK_NET_TILE", tile)
        with yk.Context(p) as ctx:
            ctx.set_field(sig)
            ctx.net_setup(layers=layers, seed=1)
            ctx.step_learned(6, True)   # the trials of the first solves
            for _ in range(10):
                t = time.perf_counter()
                ctx.step_learned(2, True)
                ctx.synchronize()
                best[tile] = min(best.get(tile, 1e9), time.perf_counter() - t)
    assert best[""] < 1.15 * best["8x64x1"], best
