"""Environment switches of the even-odd solves: which solve runs, and that they are read at context creation."""
import pytest

pytestmark = pytest.mark.gpu


def _params(yk, Nt, Nx, m0=0.1, g=0.5, r=1.0, n_rhs=1, **kw):
    return yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=g, fermion_mass=m0, wilson_param=r,
                             cut_fraction=1.0, Nt=Nt, Nx=Nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=20000,
                             fixed_dt=0.01, seed=1234, init=yk.YK_INIT_PHILOX, n_rhs=n_rhs, reliable_every=50,
                             **({"precision": yk.YK_MIXED} | kw))


@pytest.mark.parametrize("switch", ["YK_CG_EO", "YK_CG_EOC"])
def test_complex_sources(ylib, cuda, monkeypatch, switch):
    # two plane solves, or (switched off) the one on the whole complex lattice; a context keeps
    # what it was made with
    yk = ylib
    b = cuda.randn(64 * 48, 4, dtype=cuda.complex128, device="cuda", generator=cuda.Generator("cuda").manual_seed(1))

    def solve(ctx):
        st = ctx.cg_solve(b, cuda.zeros_like(b), tol=1e-10, tol_mode=yk.YK_TOL_REL, max_iter=5000, precision=yk.YK_MIXED)
        return st.iterations, st.reliable_updates

    with yk.Context(_params(yk, 64, 48)) as on:
        planes = solve(on)
        monkeypatch.setenv(switch, "0")
        with yk.Context(_params(yk, 64, 48)) as off:
            whole = solve(off)
            assert solve(on) == planes != whole
            monkeypatch.delenv(switch)
            assert solve(off) == whole


@pytest.mark.parametrize("balance", ["0", "1"])
def test_autotune_of_small_fp64_batches(ylib, cuda, monkeypatch, balance):
    # the clusters of a small FP64 batch have no grid to tune, and none is reported; balanced
    # block ranges are the grid-wide kernel's, whose grid is tuned
    yk = ylib
    monkeypatch.setenv("YK_CG_BALANCE", balance)
    with yk.Context([_params(yk, 32, 32, n_rhs=2, precision=yk.YK_FP64), _params(yk, 32, 32, m0=0.2, precision=yk.YK_FP64)]) as ctx:
        ctx.step(1)
        t = ctx.tune_report()
        ctx.profile_begin()
        ctx.step(1)
        pr = ctx.profile_end()
        if balance == "0":
            assert pr.cg_kernel == 6 and (t.cg_candidates, t.cg_grid, t.cg_grid_max) == (0, 0, 0)
        else:
            assert pr.cg_kernel == 0 and t.cg_candidates > 0 and pr.cg_grid <= t.cg_grid <= t.cg_grid_max
