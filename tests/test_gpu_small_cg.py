"""The cluster-resident CG of small lattices (cg_small_kernel) against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

KERNEL = 6   # yk_profile.cg_kernel of the cluster-resident solve


def _params(yk, Nt, Nx, **kw):
    base = dict(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=1.0,
                cut_fraction=1.0, Nt=Nt, Nx=Nx, cg_tol=1e-12, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=20000,
                fixed_dt=0.01, seed=1234, init=yk.YK_INIT_PHILOX)
    return yk.Params.default(**(base | kw))


def _action(p):
    return O.action(m2=p.mass, lam=p.g, g=p.yukawa_coupling, m0=p.fermion_mass, r=p.wilson_param,
                    cut_fraction=p.cut_fraction)


# one CTA to sixteen; rows fewer than CTAs, ranges that split rows, one site a
# CTA more than another, one to four units a thread, the largest real lattice
@pytest.mark.parametrize("Nt,Nx,r,n_rhs", [(2, 2, 1.0, 1), (3, 5, 1.0, 2), (9, 8, 0.7, 1), (17, 16, 1.0, 3),
                                           (54, 45, 1.0, 1), (33, 100, 1.3, 1), (128, 96, 1.0, 1)])
def test_fp64_steps(ylib, cuda, Nt, Nx, r, n_rhs):
    yk = ylib
    p = _params(yk, Nt, Nx, wilson_param=r, n_rhs=n_rhs)
    with yk.Context(p) as ctx:
        phi = ctx.get_field()
        ctx.profile_begin()
        ctx.step(2)
        assert ctx.profile_end().cg_kernel == KERNEL
        got, obs = ctx.get_field(), ctx.observables()
    for step in range(2):
        phi, ro = O.langevin_step(Nt, Nx, _action(p), phi, 1234, 0, step, n_rhs=n_rhs, tol=1e-12, tol_mode=1,
                                  fixed_dt=0.01)
    assert np.abs(got - phi).max() < 1e-9
    assert obs.status == 0 and abs(obs.cg_iterations - ro.cg_iters) <= 2 * n_rhs


# caller-given complex sources: FP64 and mixed, D^dag D and D D^dag, up to six
# units a thread (192 x 128)
@pytest.mark.parametrize("mtype", [0, 1])
@pytest.mark.parametrize("Nt,Nx,r", [(2, 3, 1.0), (21, 16, 1.0), (45, 54, 0.7), (192, 128, 1.0)])
def test_complex_solves(ylib, cuda, Nt, Nx, r, mtype):
    yk = ylib
    p = _params(yk, Nt, Nx, wilson_param=r)
    rng = np.random.default_rng(Nt)
    sig = rng.uniform(0.5, 1.5, Nt * Nx)
    b = rng.normal(size=(Nt * Nx, 4)) + 1j * rng.normal(size=(Nt * Nx, 4))
    with yk.Context(p) as ctx:
        ctx.set_field(sig)
        bd = cuda.from_numpy(b).cuda()
        for prec in (yk.YK_FP64, yk.YK_MIXED):
            xd = cuda.zeros_like(bd)
            st = ctx.cg_solve(bd, xd, mtype=mtype, tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=5000, precision=prec)
            x = xd.cpu().numpy()
            a = _action(p)
            ax = O.dirac(Nt, Nx, a, sig, O.dirac(Nt, Nx, a, sig, x, mtype == 0), mtype == 1)
            # the recursive residual of the FP64 solve drifts from the true one by rounding
            assert st.converged == 1 and np.linalg.norm(b - ax) <= 1.05e-10 * np.linalg.norm(b)
