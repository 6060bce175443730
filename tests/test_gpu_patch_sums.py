"""The patch kernels' sums of an iteration (the blocks' slot words) against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# one patch (no neighbour, one word a value), counts that neither the words' loads nor
# the polls' strides divide, more blocks than one turn of loads takes (PX = 8: 19 x 16
# patches), four tiles a block; r = 1 and not
@pytest.mark.parametrize("Nt,Nx,patch,r,blocks", [(16, 32, 16, 1.0, 1), (16, 32, 8, 0.7, 2), (32, 64, 32, 1.0, 1),
                                                  (48, 96, 16, 1.3, 9), (96, 192, 32, 1.0, 9), (304, 256, 8, 1.0, 304)])
def test_single_system(ylib, cuda, monkeypatch, Nt, Nx, patch, r, blocks):
    yk = ylib
    monkeypatch.setenv("YK_CG_EO_PATCH", str(patch))
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=r,
                          cut_fraction=1.0, Nt=Nt, Nx=Nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=20000,
                          fixed_dt=0.01, seed=1234, init=yk.YK_INIT_PHILOX, precision=yk.YK_MIXED, reliable_every=50)
    with yk.Context(p) as ctx:
        ctx.profile_begin()
        ctx.step(1)
        pr = ctx.profile_end()
        assert pr.cg_kernel == 3 and pr.cg_grid == blocks, (pr.cg_kernel, pr.cg_grid)
        ctx.step(1)
        got = ctx.get_field()
        assert ctx.observables().status == 0
    a = O.action(m2=-0.5, lam=1.0, g=0.5, m0=0.1, r=r, cut_fraction=1.0)
    phi = O.uniform_field(1234, 0, Nt * Nx)
    for s in range(2):
        phi, _ = O.langevin_step(Nt, Nx, a, phi, 1234, 0, s, tol=1e-10, tol_mode=1, fixed_dt=0.01)
    # the solves stop at 1e-10 |eta|; dt g chi of that is below 1e-8 (the fields of order 1)
    assert np.abs(got - phi).max() < 1e-8
