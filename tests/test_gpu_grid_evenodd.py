"""The even-odd kernels that run on the whole GPU (YK_CG_EOC=0) on lattices that fit clusters, against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (Nt, Nx, m0, g, cut, n_rhs) of each chain
SINGLE = [(64, 64, 0.1, 0.5, 1.0, 1)]
ROWS = [(54, 44, 0.1, 0.5, 1.0, 1)]
BATCH = [(40, 24, 0.1, 0.5, 0.35355339059327373, 2), (8, 8, 0.25, 0.3, 0.2, 1), (64, 64, 0.05, 0.8, 1.0, 3)]
PATCHES = [(32, 64, 0.1, 0.5, 1.0, 2), (32, 32, 0.2, 0.7, 1.0, 1), (128, 128, 0.3, 0.4, 1.0, 4), (256, 256, 0.15, 0.6, 1.0, 1)]


@pytest.mark.parametrize("specs,kernel", [(SINGLE, 3), (ROWS, 3), (BATCH, 4), (PATCHES, 5)],
                         ids=["one_patches", "one_rows", "batch_four_passes", "batch_patches"])
@pytest.mark.parametrize("r", [0.7, 1.0, 1.3])
def test_steps(ylib, cuda, monkeypatch, specs, kernel, r):
    yk = ylib
    monkeypatch.setenv("YK_CG_EOC", "0")
    ps = [yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=g, fermion_mass=m0, wilson_param=r,
                            cut_fraction=s, Nt=nt, Nx=nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=20000,
                            fixed_dt=0.01, seed=1234, init=yk.YK_INIT_PHILOX, n_rhs=nr, precision=yk.YK_MIXED,
                            reliable_every=50) for nt, nx, m0, g, s, nr in specs]

    def profiled(ctx):
        ctx.profile_begin()
        ctx.step(1)
        return ctx.profile_end()
    with yk.Context(ps) as ctx:
        pr = profiled(ctx)
        assert (pr.cg_kernel, pr.cg_cluster_blocks) == (kernel, 0)
        ctx.step(1)
        got = [ctx.get_field(c) for c in range(len(ps))]
        assert all(ctx.observables(c).status == 0 for c in range(len(ps)))
    monkeypatch.delenv("YK_CG_EOC")
    with yk.Context(ps) as ctx:   # on clusters, under the same code (256 x 256 fits one at r = 1)
        pr = profiled(ctx)
        assert pr.cg_kernel == kernel and (1 <= pr.cg_cluster_blocks <= 16) == (r == 1.0 or specs is not PATCHES)
    for c, p in enumerate(ps):
        a = O.action(m2=-0.5, lam=1.0, g=p.yukawa_coupling, m0=p.fermion_mass, r=r, cut_fraction=p.cut_fraction)
        phi = O.uniform_field(1234, c, p.Nt * p.Nx)
        for s in range(2):
            phi, _ = O.langevin_step(p.Nt, p.Nx, a, phi, 1234, c, s, n_rhs=p.n_rhs, tol=1e-10, tol_mode=1, fixed_dt=0.01)
        # the solves stop at 1e-10 |eta|; dt g chi of that is below 1e-8 (the fields of order 1)
        assert np.abs(got[c] - phi).max() < 1e-8, c


def test_small_fp64_clusters_are_reported(ylib, cuda):
    yk = ylib
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, cut_fraction=1.0, Nt=32,
                          Nx=32, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, fixed_dt=0.01, seed=1, init=yk.YK_INIT_PHILOX,
                          n_rhs=2)
    with yk.Context(p) as ctx:
        ctx.profile_begin()
        ctx.step(1)
        pr = ctx.profile_end()
        assert pr.cg_kernel == 6 and pr.cg_cluster_blocks * 2 == pr.cg_grid
