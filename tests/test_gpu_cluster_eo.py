"""The cluster-resident even-odd solve of the step (cg_eoc_kernel) against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _params(yk, Nt, Nx, m0=0.1, g=0.5, r=1.0, n_rhs=1, **kw):
    base = dict(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=g, fermion_mass=m0, wilson_param=r, cut_fraction=1.0,
                Nt=Nt, Nx=Nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=20000, fixed_dt=0.01, seed=1234,
                init=yk.YK_INIT_PHILOX, n_rhs=n_rhs, precision=yk.YK_MIXED, reliable_every=50)
    return yk.Params.default(**(base | kw))


def _check(yk, ps, ctas, steps=2):
    with yk.Context(ps) as ctx:
        ctx.profile_begin()
        ctx.step(1)
        pr = ctx.profile_end()
        # cg_grid tells the kernels apart: one launch per form, clusters of one to sixteen CTAs a system
        assert pr.cg_grid == ctas, pr.cg_grid
        ctx.step(steps - 1)
        got = [ctx.get_field(c) for c in range(len(ps))]
        obs = [ctx.observables(c) for c in range(len(ps))]
    for c, p in enumerate(ps):
        a = O.action(m2=p.mass, lam=p.g, g=p.yukawa_coupling, m0=p.fermion_mass, r=p.wilson_param,
                     cut_fraction=p.cut_fraction)
        phi = O.uniform_field(1234, c, p.Nt * p.Nx)
        for s in range(steps):
            phi, _ = O.langevin_step(p.Nt, p.Nx, a, phi, 1234, c, s, n_rhs=p.n_rhs, tol=1e-10, tol_mode=1,
                                     fixed_dt=0.01)
        assert obs[c].status == 0
        assert np.abs(got[c] - phi).max() < 1e-8, (c, p.Nt, p.Nx)


# one row a thread to four, alike for all of them and not; one CTA to sixteen; rows
# that clusters do not divide, columns that leave threads of the block idle, the
# smallest and largest lattices
@pytest.mark.parametrize("Nt,Nx,r,ctas", [(2, 4, 1.0, 1), (6, 10, 1.0, 1), (10, 6, 0.7, 1), (54, 44, 1.0, 8),
                                          (70, 96, 1.0, 16), (130, 126, 1.0, 16), (128, 256, 1.0, 16),
                                          (160, 224, 1.0, 16), (192, 224, 1.0, 16), (134, 250, 1.3, 16),
                                          (256, 256, 1.0, 16), (512, 128, 1.0, 16)])
def test_single_chain(ylib, cuda, Nt, Nx, r, ctas):
    _check(ylib, [_params(ylib, Nt, Nx, r=r)], ctas)


# many systems: the fewest CTAs each, in groups of one form (c = 4, 2 and 1; r = 1 and not)
def test_batch(ylib, cuda):
    yk = ylib
    ps = [_params(yk, 64, 64, n_rhs=40), _params(yk, 16, 24, m0=0.2, r=0.7, n_rhs=3),
          _params(yk, 128, 128, m0=0.3, g=0.4, n_rhs=20), _params(yk, 66, 100, m0=0.05, g=0.8, n_rhs=1),
          _params(yk, 36, 56, m0=0.2, r=1.3)]
    _check(yk, ps, 40 + 3 + 80 + 2 + 1, steps=1)


# an absolute stop and a cap that is reached
def test_stops(ylib, cuda):
    yk = ylib
    p = _params(yk, 48, 40, cg_tol=1e-6, cg_tol_mode=yk.YK_TOL_ABS)
    with yk.Context(p) as ctx:
        ctx.step(1)
        got = ctx.get_field()
        assert ctx.observables().status == 0
    a = O.action(m2=-0.5, lam=1.0, g=0.5, m0=0.1, r=1.0, cut_fraction=1.0)
    want, _ = O.langevin_step(48, 40, a, O.uniform_field(1234, 0, 48 * 40), 1234, 0, 0, tol=1e-12, tol_mode=1,
                              fixed_dt=0.01)
    assert np.abs(got - want).max() < 1e-6 * 0.01 * 10   # |dphi| <= dt g |eta| |A_o^-1 ..| |r|
    with yk.Context(_params(yk, 48, 40, cg_max_iter=7)) as ctx:
        ctx.step(1)
        o = ctx.observables()
        assert o.cg_iterations == 7 and o.status == yk.YK_ENOCONV
