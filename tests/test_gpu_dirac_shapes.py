"""The Dirac apply where its blocks, bands and warps end, against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# rows shorter than a warp's lanes, at its and the block's ends and past them; one
# row a band, bands that divide the lattice and not
@pytest.mark.parametrize("r", [1.0, 0.7])
@pytest.mark.parametrize("Nt,Nx", [(2, 2), (3, 3), (2, 15), (5, 16), (4, 17), (33, 127), (32, 128), (35, 129), (700, 97),
                                   (1031, 130)])
def test_shapes(ylib, cuda, Nt, Nx, r):
    yk = ylib
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=r,
                          cut_fraction=1.0, Nt=Nt, Nx=Nx, seed=1, init=yk.YK_INIT_NONE)
    a = O.action(m2=-0.5, lam=1.0, g=0.5, m0=0.1, r=r, cut_fraction=1.0)
    rng = np.random.default_rng(Nt * 2000 + Nx)
    sig = rng.uniform(-2.0, 2.0, Nt * Nx)
    v = rng.normal(size=(Nt * Nx, 4)) + 1j * rng.normal(size=(Nt * Nx, 4))
    with yk.Context(p) as ctx:
        ctx.set_field(sig)
        for dagger in (False, True):
            want = O.dirac(Nt, Nx, a, sig, v, dagger)
            for prec, dt, tol in ((yk.YK_FP64, cuda.complex128, 1e-14), (yk.YK_FP32, cuda.complex64, 1e-6)):
                inp = cuda.from_numpy(v).to(dt).cuda()
                out = cuda.empty_like(inp)
                ctx.dirac_apply(inp, out, dagger, prec)
                ctx.synchronize()
                # a site sums nine terms of magnitude up to 4 |v|: a few roundings each
                assert np.abs(out.cpu().numpy() - want).max() < tol * 4 * np.abs(v).max()
