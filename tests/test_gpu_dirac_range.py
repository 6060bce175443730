"""The FP32 Dirac apply on fields and couplings beyond FP32's range, against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# the diagonal 2 r + m0 + g sigma is an FP64 sum rounded to FP32: its factors need not be FP32
# numbers (too large, too small, subnormal), nor all sites' alike
@pytest.mark.parametrize("g,scale", [(0.5, 1.0), (1e-39, 1e39), (1e39, 1e-39), (0.0, 1e39), (1e-10, 1e39), (1e-35, 1e35),
                                     (1e38, 1e-44)])
def test_diagonal(ylib, cuda, g, scale):
    yk, Nt, Nx = ylib, 6, 40
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=g, fermion_mass=0.1, wilson_param=1.0,
                          cut_fraction=1.0, Nt=Nt, Nx=Nx, seed=1, init=yk.YK_INIT_NONE)
    a = O.action(m2=-0.5, lam=1.0, g=g, m0=0.1, r=1.0, cut_fraction=1.0)
    rng = np.random.default_rng(1)
    sig = scale * rng.uniform(-2.0, 2.0, Nt * Nx)
    sig[::7] = 0.0
    v = rng.normal(size=(Nt * Nx, 4)) + 1j * rng.normal(size=(Nt * Nx, 4))
    with yk.Context(p) as ctx:
        ctx.set_field(sig)
        for dagger in (False, True):
            want = O.dirac(Nt, Nx, a, sig, v, dagger)
            inp = cuda.from_numpy(v).to(cuda.complex64).cuda()
            out = cuda.empty_like(inp)
            ctx.dirac_apply(inp, out, dagger, yk.YK_FP32)
            ctx.synchronize()
            # nine terms of magnitude up to (4 + |g sigma|) |v|: a few roundings each
            size = (4 + np.abs(g * sig).reshape(-1, 1)) * np.abs(v).max()
            assert (np.abs(out.cpu().numpy() - want) < 1e-6 * size).all()
