"""The learned solver's two-launch iterations on ragged tiles, against the FP64 CG step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# tiles cut off at both edges, lattices smaller than a tile's halo (staged rows and
# columns wrap more than once), one tile a row and several; with the network and z = r
@pytest.mark.parametrize("use_net", [True, False])
@pytest.mark.parametrize("Nt,Nx,layers", [(41, 25, 2), (9, 7, 4), (4, 130, 3), (67, 96, 2), (256, 72, 4)])
def test_steps_match_the_cg_step(ylib, cuda, Nt, Nx, layers, use_net):
    yk = ylib
    fields = []
    for learned in (False, True):
        p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.05, wilson_param=1.0,
                              cut_fraction=1.0, Nt=Nt, Nx=Nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL,
                              cg_max_iter=20000, seed=1234, init=yk.YK_INIT_PHILOX, fixed_dt=0.01,
                              precision=yk.YK_FP64)
        with yk.Context(p) as ctx:
            if learned:
                ctx.net_setup(layers, 7)
                ctx.net_train(n_sources=2, n_levels=3, base_iter=4, steps=40, batch=2, lr=2e-3, seed=3)
                st = ctx.step_learned(2, use_net=use_net)
                assert st.converged == 1
            else:
                ctx.step(2)
            assert ctx.observables().status == 0
            fields.append(ctx.get_field())
    # both solve to 1e-10 of the source: the fields differ by dt times that and the condition's factor
    assert np.abs(fields[1] - fields[0]).max() < 1e-8 * np.abs(fields[0]).max()
