"""Mixed solves of complex sources by their real planes (launch_plane_solve) against the CPU oracle's operator."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# both products, r = 1 and not, one CTA and sixteen a plane, the largest lattice;
# sources with one empty plane, of small norm, of one site; both kinds of target
@pytest.mark.parametrize("mtype", [0, 1])
@pytest.mark.parametrize("Nt,Nx,r,source", [(2, 4, 1.0, "dense"), (64, 48, 0.7, "imag"), (34, 26, 1.0, "point"),
                                            (96, 128, 1.0, "small"), (256, 256, 1.0, "dense")])
def test_residual(ylib, cuda, Nt, Nx, r, source, mtype):
    yk = ylib
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=r,
                          cut_fraction=1.0, Nt=Nt, Nx=Nx, seed=1, init=yk.YK_INIT_NONE, precision=yk.YK_MIXED)
    a = O.action(m2=-0.5, lam=1.0, g=0.5, m0=0.1, r=r, cut_fraction=1.0)
    rng = np.random.default_rng(Nt)
    sig = rng.uniform(0.5, 1.5, Nt * Nx)
    b = rng.normal(size=(Nt * Nx, 4)) + 1j * rng.normal(size=(Nt * Nx, 4))
    if source == "imag":
        b = 1j * b.imag
    elif source == "point":
        b = np.zeros_like(b)
        b[5, 2] = 1 - 2j
    elif source == "small":
        b = b * 1e-9
    with yk.Context(p) as ctx:
        ctx.set_field(sig)
        bd = cuda.from_numpy(b).cuda()
        for mode, tol in ((yk.YK_TOL_REL, 1e-10), (yk.YK_TOL_ABS, 1e-9 * np.linalg.norm(b))):
            xd = cuda.zeros_like(bd)
            st = ctx.cg_solve(bd, xd, mtype=mtype, tol=tol, tol_mode=mode, max_iter=5000, precision=yk.YK_MIXED)
            x = xd.cpu().numpy()
            ax = O.dirac(Nt, Nx, a, sig, O.dirac(Nt, Nx, a, sig, x, mtype == 0), mtype == 1)
            target = tol * (np.linalg.norm(b) if mode == yk.YK_TOL_REL else 1.0)
            # the residual that the solve checked, within FP64 rounding of the two products
            assert st.converged == 1 and np.linalg.norm(b - ax) <= target * (1 + 1e-3)


def test_cap_and_zero(ylib, cuda):
    yk = ylib
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=1.0,
                          cut_fraction=1.0, Nt=32, Nx=48, seed=1, init=yk.YK_INIT_PHILOX, precision=yk.YK_MIXED)
    b = cuda.randn(32 * 48, 4, dtype=cuda.complex128, device="cuda")
    x = cuda.ones_like(b)
    with yk.Context(p) as ctx:
        st = ctx.cg_solve(b, x, tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=4, precision=yk.YK_MIXED, allow_noconv=True)
        assert st.converged == 0 and st.iterations == 4
        st = ctx.cg_solve(cuda.zeros_like(b), x, tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=100, precision=yk.YK_MIXED)
        assert st.converged == 1 and st.iterations == 0 and float(x.abs().max()) == 0.0
