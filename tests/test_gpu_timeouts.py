"""Bounded device waits that give up: the blocks end in order and the caller hears of it."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_cluster_ends_together(ylib, cuda):
    # one block of a cluster gives up after about 2 s; the others, which pass more
    # barriers and store into its shared memory after that, end with it
    st = C.c_int(-1)
    assert ylib.lib().yk_check_cluster_timeout(None, C.byref(st)) == ylib.YK_ETIMEOUT
    assert st.value == ylib.YK_ETIMEOUT
    p = ylib.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, cut_fraction=1.0, Nt=32,
                            Nx=32, cg_tol=1e-10, cg_tol_mode=ylib.YK_TOL_REL, fixed_dt=0.01, seed=1,
                            init=ylib.YK_INIT_PHILOX)
    with ylib.Context(p) as ctx:   # the device stays usable
        ctx.step(1)
        assert ctx.observables().status == 0
