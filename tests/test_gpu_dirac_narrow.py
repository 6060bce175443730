"""The Dirac apply on narrow lattices: as many busy lanes as on square ones."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("Nt,Nx,square", [(4096, 2, (128, 64)), (2048, 40, (256, 320)), (4096, 64, (512, 512))])
def test_time(ylib, cuda, Nt, Nx, square, prec):
    # the same number of sites takes at most twice as long on rows of two (a site's neighbours
    # come from memory there), where a block's 256 threads for each band took nine times as long
    yk = ylib
    dt, p = (cuda.complex64, yk.YK_FP32) if prec == "fp32" else (cuda.complex128, yk.YK_FP64)
    assert square[0] * square[1] == Nt * Nx
    a = cuda.randn(Nt * Nx, 4, dtype=dt, device="cuda")
    b = cuda.empty_like(a)
    us = []
    for nt, nx in ((Nt, Nx), square):
        q = yk.Params.default(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, cut_fraction=1.0,
                              Nt=nt, Nx=nx, seed=1, init=yk.YK_INIT_PHILOX)
        stream = cuda.cuda.Stream()
        with yk.Context(q) as ctx:
            ctx.set_stream(stream.cuda_stream)
            best = 1e9
            for _ in range(8):
                e0, e1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
                ctx.dirac_apply(a, b, True, p)
                e0.record(stream)
                for _ in range(20):
                    ctx.dirac_apply(a, b, True, p)
                e1.record(stream)
                e1.synchronize()
                best = min(best, e0.elapsed_time(e1) / 20 * 1e3)
            us.append(best)
    assert us[0] < 2.0 * us[1] + 1.0, us
