"""The coloured noise's transforms over the lengths they factor differently, against the CPU oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


# powers of four and of two with a two over, powers of odd primes, products of all
# kinds, primes (one stage), the longest length that is no power of two
@pytest.mark.parametrize("Nt,Nx", [(2, 3), (3, 7), (4, 9), (64, 27), (128, 25), (45, 54), (160, 224), (49, 75), (12, 121),
                                   (210, 143), (251, 8), (6, 255), (512, 256), (1024, 2)])
def test_lengths(ylib, cuda, Nt, Nx):
    yk = ylib
    s = 0.35355339059327373
    p = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.0, fermion_mass=0.1, wilson_param=1.0,
                          cut_fraction=s, Nt=Nt, Nx=Nx, seed=1234, init=yk.YK_INIT_NONE)
    w = np.random.default_rng(Nt * 1000 + Nx).normal(size=Nt * Nx)
    with yk.Context(p) as ctx:
        xi = cuda.empty(Nt * Nx, dtype=cuda.float64, device="cuda")
        ctx.coloured_noise(xi, cuda.from_numpy(w).cuda())
        ctx.synchronize()
        # |xi| is of order 1: a transform's rounding error is a few units of 1e-16 times
        # the square root of its depth, the oracle's direct sums' of their length
        assert np.abs(xi.cpu().numpy() - O.coloured_noise(Nt, Nx, s, w)).max() < 1e-13
