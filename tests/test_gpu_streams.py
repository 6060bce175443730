"""Chains that step at the same time on streams of their own: the same fields as one after another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_contexts_side_by_side(ylib, cuda):
    # cluster solves of every kind (even-odd at r = 1 and not, FP64, complex), a batch, and a solve on
    # the whole GPU; the graphs of all are launched before any is waited for, several times
    yk = ylib

    def p(Nt, Nx, **kw):
        base = dict(use_mass=1, mass=-0.5, g=1.0, yukawa_coupling=0.5, fermion_mass=0.1, wilson_param=1.0,
                    cut_fraction=0.35355339059327373, Nt=Nt, Nx=Nx, cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL,
                    cg_max_iter=20000, fixed_dt=0.01, seed=7, init=yk.YK_INIT_PHILOX, precision=yk.YK_MIXED)
        return yk.Params.default(**(base | kw))
    chains = [[p(256, 256)], [p(64, 96, wilson_param=0.7)], [p(32, 32, precision=yk.YK_FP64)], [p(54, 45, precision=yk.YK_FP64)],
              [p(64, 48, pions=1)], [p(128, 128, n_rhs=2), p(32, 64, wilson_param=1.3), p(64, 64)], [p(256, 256)], [p(512, 512)],
              [p(33, 31)]]
    want = []
    for ps in chains:
        with yk.Context(ps) as ctx:
            for _ in range(6):
                ctx.step(1)
            want.append([ctx.get_field(c) for c in range(len(ps))])
    ctxs = [yk.Context(ps) for ps in chains]
    streams = [cuda.cuda.Stream() for _ in chains]
    for ctx, s in zip(ctxs, streams):
        ctx.set_stream(s.cuda_stream)
    for _ in range(6):
        for ctx in ctxs:
            ctx.step(1)
    for ctx, w in zip(ctxs, want):
        assert all(np.array_equal(ctx.get_field(c), w[c]) for c in range(len(w)))
        ctx.close()
