"""The work whose speed matters to a user of this framework, as measurable cases.

A case is a dict of plain values.  Every case goes through the package's public
entry points: Langevin steps of one chain or of a batch (``Context.step``, the
host-exchanging ``step_io``, the learned-preconditioner ``step_learned``), the
Wilson-Dirac apply (``dirac_apply``) and the CG solve on caller-given sources
(``cg_solve``).

Fields come in two kinds.  "thermal" is what a chain meets after burn-in at
m^2 = -0.5, lambda = 1: a mean near 2.13 and Gaussian fluctuations with the free
spectrum 1 / (1.75 + p^2) below the noise cutoff (the statistics of the
thermalised 256 x 256 field that the benchmark starts from).  "young" is a chain
twenty steps of 0.01 after its start from iid Uniform[-1, 1]: the linear Langevin
evolution of that start, with the mean that a 256 x 256 chain has by then.  The mean
is still small, the fermion matrix ill-conditioned, and the solver works hardest.
A thermal chain just keeps stepping.  A young chain is put back to its field before
each step (a copy on the device), so that every pass does the same work, as a
program does that draws several noises on one configuration.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import yukawacolourednoise_gb300 as yk

M2, LAMBDA, G = -0.5, 1.0, 0.5
CUT = 0.35355339059327373      # Lambda = pi / 2
MEAN, GAP = 2.13, 1.75         # the thermal field's mean and its spectrum's constant
AGE, YOUNG_MEAN, RATE = 0.2, 0.175, -0.35   # the young field: its Langevin time, mean and p = 0 rate


# --------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest run configuration (32 x 32, the reference's plain FP64 method): a step is all latency
        dict(name="step_fp64_32x32", kind="step", Nt=32, Nx=32, precision="fp64", m0=0.1, start="thermal",
             adaptive=False),
        # the reference's default method (FP64, adaptive step size) on an odd, ragged lattice
        dict(name="step_fp64_54x45", kind="step", Nt=54, Nx=45, precision="fp64", m0=0.1, start="thermal",
             adaptive=True),
        # the headline: one mixed-precision step at 256 x 256
        dict(name="step_mixed_256x256", kind="step", Nt=256, Nx=256, precision="mixed", m0=0.1, start="thermal",
             adaptive=False),
        # a host program that owns the field and exchanges it every step, on edges that are no powers of two
        dict(name="step_io_160x224", kind="io", Nt=160, Nx=224, precision="mixed", m0=0.1, start="thermal",
             adaptive=True),
        # near the chiral regime of a young chain: hundreds of solver iterations per step
        dict(name="step_mixed_512x512_young", kind="step", Nt=512, Nx=512, precision="mixed", m0=0.02, start="young",
             adaptive=False),
        # many independent chains of uneven sizes, four sources each, in one step
        dict(name="step_batch_64_chains", kind="batch", chains=64, rhs=4, pick=1234, start="thermal"),
        # the largest lattices: several sources per chain, near the chiral regime, of a young chain
        dict(name="step_large_2x1024x1024", kind="large", Nt=1024, Nx=1024, chains=2, rhs=4, m0=0.01, start="young"),
        # four fields (sigma and the pions): the complex operator
        dict(name="step_pions_64x48", kind="pions", Nt=64, Nx=48, precision="mixed", m0=0.1, start="thermal"),
        # the same chiral regime with the trained preconditioner
        dict(name="step_learned_512x512_young", kind="learned", Nt=512, Nx=512, layers=2, m0=0.02, start="young"),
        # the operator alone, FP32, on a lattice beyond L2
        dict(name="dirac_fp32_2048x2048", kind="dirac", Nt=2048, Nx=2048, precision="fp32", dagger=False),
        # the operator alone, FP64 and daggered, rows of an odd length
        dict(name="dirac_fp64_1000x749_dag", kind="dirac", Nt=1000, Nx=749, precision="fp64", dagger=True),
        # a solve on a complex source of the caller, as propagators and correlators need
        dict(name="cg_mixed_192x128_young", kind="cg", Nt=192, Nx=128, precision="mixed", m0=0.1, start="young"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))))))


def _edge(rng, lo, hi):
    """A lattice edge: a power of two, or any length up to 256 (the longest that is no power of two)."""
    if rng.random() < 0.4:
        return 1 << rng.randint(math.ceil(math.log2(lo)), int(math.log2(hi)))
    return _log(rng, lo, min(hi, 256))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "io", "batch", "large", "pions", "learned", "dirac", "dirac", "cg"])
    m0 = round(rng.uniform(0.05, 0.3), 4)
    start = rng.choice(["thermal", "thermal", "young"])
    if kind == "step":
        return dict(kind=kind, Nt=_edge(rng, 32, 512), Nx=_edge(rng, 32, 512),
                    precision=rng.choice(["fp64", "mixed", "mixed"]), m0=m0, start=start, adaptive=rng.random() < 0.5)
    if kind == "io":
        return dict(kind=kind, Nt=_edge(rng, 64, 256), Nx=_edge(rng, 64, 256), precision="mixed", m0=m0,
                    start="thermal", adaptive=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, chains=_log(rng, 4, 64), rhs=rng.randint(1, 4), pick=rng.randint(1, 10 ** 6),
                    start="thermal")
    if kind == "large":
        return dict(kind=kind, Nt=1024, Nx=rng.choice([512, 1024]), chains=rng.randint(1, 2), rhs=rng.randint(1, 4),
                    m0=round(rng.uniform(0.01, 0.1), 4), start="young")
    if kind == "pions":
        return dict(kind=kind, Nt=_edge(rng, 16, 128), Nx=_edge(rng, 16, 128),
                    precision=rng.choice(["fp64", "mixed"]), m0=m0, start="thermal")
    if kind == "learned":
        edges = [128, 144, 192, 256, 512]      # above 256 the noise takes powers of two
        return dict(kind=kind, Nt=rng.choice(edges), Nx=rng.choice(edges), layers=rng.randint(2, 4),
                    m0=round(rng.uniform(0.02, 0.1), 4), start="young")
    if kind == "dirac":
        return dict(kind=kind, Nt=_log(rng, 64, 2048), Nx=rng.choice([_log(rng, 64, 2048), 32 * _log(rng, 2, 64)]),
                    precision=rng.choice(["fp32", "fp64"]), dagger=rng.random() < 0.5)
    return dict(kind=kind, Nt=_edge(rng, 32, 256), Nx=_edge(rng, 32, 256), precision=rng.choice(["fp64", "mixed"]),
                m0=m0, start=start)


def _chains(case):
    """(Nt, Nx, m0, g) of every chain of the case."""
    if case["kind"] == "batch":
        # the batching configuration: seeded sizes, masses and couplings
        r = np.random.default_rng(case["pick"])
        n = case["chains"]
        L = r.choice([32, 64, 128, 256], size=n)
        return [(int(a), int(a), float(m), float(g)) for a, m, g in
                zip(L, r.uniform(0.05, 0.3, size=n), r.uniform(0.3, 0.8, size=n))]
    g = 0.6 if case["kind"] == "large" else G
    return [(case["Nt"], case["Nx"], case.get("m0", 0.1), g)] * case.get("chains", 1)


def _params(case, seed):
    mixed = case.get("precision", "mixed") == "mixed"
    many = case["kind"] in ("batch", "large", "learned")
    return [yk.Params.default(
        use_mass=1, mass=M2, g=LAMBDA, yukawa_coupling=g, fermion_mass=m0, wilson_param=1.0,
        cut_fraction=1.0 if case["kind"] in ("dirac", "cg") else CUT, Nt=Nt, Nx=Nx, fixed_dt=0.0 if case.get("adaptive") else 0.01, precision=yk.YK_MIXED if mixed else yk.YK_FP64,
        cg_tol=1e-10, cg_tol_mode=yk.YK_TOL_REL, cg_max_iter=50000, reliable_every=50,
        reliable_delta=1e-3 if many else 1e-5, n_rhs=case.get("rhs", 1), seed=seed, init=yk.YK_INIT_NONE,
        pions=int(case["kind"] == "pions")) for Nt, Nx, m0, g in _chains(case)]


# -------------------------------------------------------------------- inputs
def _generator(seed, chain=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + chain)


def _p2(Nt, Nx):
    """p^2 of every mode, in the order of operations that decides which modes at the cutoff's edge are kept."""
    def axis(k, L):
        return np.where(k <= L // 2, k, k - L) * 2.0 * math.pi / L
    kt, kx = np.arange(Nt)[:, None], np.arange(Nx)[None, :]
    upper = kx > Nx // 2       # the half spectrum's mirror image
    kt, kx = np.where(upper, (Nt - kt) % Nt, kt), np.where(upper, Nx - kx, kx + 0 * kt)
    return axis(kt, Nt) ** 2 + axis(kx, Nx) ** 2


def _kept(Nt, Nx):
    return torch.from_numpy(_p2(Nt, Nx) <= (math.sqrt(2.0) * math.pi * CUT) ** 2).cuda()


def _lattice_p2(Nt, Nx):
    kt, kx = [4 * torch.sin(math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n) ** 2 for n in (Nt, Nx)]
    return kt[:, None] + kx[None, :]


def _shaped(w, amplitude):
    return torch.fft.ifft2(torch.fft.fft2(w) * amplitude).real.contiguous()


def _white(Nt, Nx, gen):
    return torch.randn(Nt, Nx, generator=gen, device="cuda", dtype=torch.float64)


def _smooth(Nt, Nx, gen):
    """Gaussian fluctuations with the thermal spectrum."""
    return _shaped(_white(Nt, Nx, gen), (_kept(Nt, Nx) / (GAP + _lattice_p2(Nt, Nx))).sqrt())


def _field(Nt, Nx, start, gen):
    if start == "thermal":
        return MEAN + _smooth(Nt, Nx, gen)
    first = 1 - 2 * torch.rand(Nt, Nx, generator=gen, device="cuda", dtype=torch.float64)
    rate = RATE + _lattice_p2(Nt, Nx)
    noise = (_kept(Nt, Nx) * -torch.expm1(-2 * AGE * rate) / rate).sqrt()
    return YOUNG_MEAN + _shaped(first - first.mean(), torch.exp(-AGE * rate)) + _shaped(_white(Nt, Nx, gen), noise)


def _inputs(case, seed):
    """The tensors that a case starts from: every chain's field, and what else the call takes."""
    fields, more = [], {}
    for c, (Nt, Nx, _, _) in enumerate(_chains(case)):
        gen = _generator(seed, c)
        fields.append(_field(Nt, Nx, case.get("start", "thermal"), gen))
        if case["kind"] == "pions":
            more["pions"] = torch.stack([_smooth(Nt, Nx, gen) for _ in range(3)])
        if case["kind"] in ("dirac", "cg"):
            dt = torch.complex64 if case["precision"] == "fp32" else torch.complex128
            more["source"] = torch.randn(Nt * Nx, 4, generator=gen, device="cuda", dtype=dt)
    return fields, more


class _Device:
    """An array in device memory that a context owns."""

    def __init__(self, ctx, ptr, shape):
        self.ctx = ctx     # the memory lives as long as the context
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _view(ctx, ptr, *shape):
    return torch.as_tensor(_Device(ctx, ptr, shape), device="cuda")


def prepare(case, seed):
    fields, more = _inputs(case, seed)
    ctx = yk.Context(_params(case, seed))
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    for c, f in enumerate(fields):
        ctx.set_field(f.cpu().numpy(), chain=c)
    s = dict(kind=case["kind"], ctx=ctx, stream=stream)
    if case["kind"] in ("dirac", "cg"):
        s["source"], s["out"] = more["source"], torch.empty_like(more["source"])
        s["precision"] = dict(fp64=yk.YK_FP64, fp32=yk.YK_FP32, mixed=yk.YK_MIXED)[case["precision"]]
        s["dagger"] = case.get("dagger", False)
        return s
    if case["kind"] == "io":
        s["here"] = fields[0].cpu().reshape(-1).pin_memory()
        s["there"] = torch.empty_like(s["here"]).pin_memory()
        return s
    s["fields"] = [_view(ctx, ctx.field_ptr(c), *f.shape) for c, f in enumerate(fields)]
    s["again"] = fields if case["start"] == "young" else None
    if case["kind"] == "pions":
        ctx.set_pions(more["pions"].cpu().numpy())
        s["fields"].append(_view(ctx, ctx.pions_ptr(), *more["pions"].shape))
    if case["kind"] == "learned":
        # a program trains once, after burn-in, and steps with the trained network from there on
        ctx.net_setup(case["layers"], 7)
        ctx.net_train(n_sources=2, n_levels=5, base_iter=4, steps=150, batch=4, lr=2e-3, seed=3)
    return s


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "dirac":
        ctx.dirac_apply(state["source"], state["out"], state["dagger"], state["precision"])
        return state["out"]
    if state["kind"] == "cg":
        ctx.cg_solve(state["source"], state["out"], yk.YK_DAGGER, 1e-10, yk.YK_TOL_REL, 50000, state["precision"])
        return state["out"]
    if state["kind"] == "io":
        obs = ctx.step_io(state["here"], state["there"])
        state["here"], state["there"] = state["there"], state["here"]
        return [state["here"], obs.sum_phi, obs.sum_phi2, obs.eps, obs.max_drift]
    if state["again"] is not None:
        with torch.cuda.stream(state["stream"]):
            for f, start in zip(state["fields"], state["again"]):
                f.copy_(start)
    if state["kind"] == "learned":
        ctx.step_learned(1)
    else:
        ctx.step(1)
    return state["fields"]


def work(case):
    """One pass's inputs read once and outputs written once, and the operations of the method it asks for.

    A step's operations are its solves': per site, iteration and source two applications of the real operator
    (11 operations for each of four components) and ten for the vectors' updates and products; on an even lattice
    half the sites of the even-odd system.  Iterations: what these fields take, about."""
    sites = sum(Nt * Nx for Nt, Nx, _, _ in _chains(case))
    if case["kind"] == "dirac":
        spinor = 32 if case["precision"] == "fp32" else 64
        return {"bytes": sites * (2 * spinor + 8), "flops": sites * 8 * 11}
    edge = max(max(Nt, Nx) for Nt, Nx, _, _ in _chains(case))
    iterations = 25 if case["start"] == "thermal" else 60 + 6 / (case["m0"] + 6 / edge)
    per_site = (2 * 4 * 11 + 4 * 10) * iterations * case.get("rhs", 1)
    if case["kind"] in ("cg", "pions"):
        per_site *= 2          # complex
    if case["kind"] == "cg":
        return {"bytes": sites * (2 * 64 + 8), "flops": sites * per_site * 2}
    return {"bytes": sites * (64 if case["kind"] == "pions" else 16), "flops": sites * per_site}


# ------------------------------------------------- the same results, in 64 bits
def _philox(seed, chain, step, kind, rhs, n):
    """Philox4x32-10 of counters 0 .. n-1: four 32-bit words each."""
    M = 0xFFFFFFFF
    e = torch.arange(n, device="cuda", dtype=torch.int64)
    c = [e, torch.full_like(e, step & M), torch.full_like(e, step >> 32), torch.full_like(e, kind << 24 | rhs)]
    k = [seed & M, (seed >> 32) ^ chain]
    for i in range(10):
        if i:
            k = [(k[0] + 0x9E3779B9) & M, (k[1] + 0xBB67AE85) & M]
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57      # modulo 2^64: the words are its halves
        c = [(b >> 32) & M ^ c[1] ^ k[0], b & M, (a >> 32) & M ^ c[3] ^ k[1], a & M]
    return c


def _f32(v):
    return v.to(torch.float32).to(torch.float64)


def _fma(a, b, c):
    return _f32(a * b + c)       # the product of two floats is exact in 64 bits


def _log1p_core(f):
    s = _f32(f / _f32(2 + f))
    t, z = 2 * s, _f32(s * s)
    p = torch.full_like(z, float.fromhex("0x1.c71c72p-4"))
    for a in ("0x1.24924ap-3", "0x1.99999ap-3", "0x1.555556p-2"):
        p = _fma(z, p, float.fromhex(a))
    return _fma(_f32(t * z), p, t)


def _normal_pairs(a, b):
    """The framework's Box-Muller, which is defined in 32-bit arithmetic, operation for operation."""
    hi, lo = float.fromhex("0x1.62e4p-1"), float.fromhex("0x1.7f7d1cp-20")
    M = 0xFFFFFFFF
    u = _f32(_f32(((2 * a + 1) & M).double()) * 2.0 ** -33)
    m, ex = torch.frexp(u)
    m, ex = 2 * m, ex.double() - 1
    big = m > float.fromhex("0x1.6a09e6p+0")
    m, ex = torch.where(big, m / 2, m), torch.where(big, ex + 1, ex)
    small = -_fma(ex, torch.full_like(ex, hi), _fma(ex, torch.full_like(ex, lo), _log1p_core(_f32(m - 1))))
    w = _f32(_f32(((2 * (a ^ M) + 1) & M).double()) * 2.0 ** -33)
    near = -_log1p_core(-w)
    far = _f32(_f32(hi - _log1p_core(_f32(1 - 2 * w))) + lo)
    neglog = torch.where(a < 0x80000000, small, torch.where(w <= float.fromhex("0x1.2bec34p-2"), near, far))
    R = _f32(torch.sqrt(_f32(2 * neglog)))
    j = ((b + 0x20000000) & M) >> 30
    d = (b - (j << 30)) & M
    d = torch.where(d >= 1 << 31, d - (1 << 32), d)
    y = _f32(_f32((2 * d + 1).double()) * 2.0 ** -33)
    y2 = _f32(y * y)

    def poly(*c):
        p = torch.full_like(y2, float.fromhex(c[0]))
        for q in c[1:]:
            p = _fma(y2, p, float.fromhex(q))
        return p
    sn = _f32(y * poly("0x1.507834p+5", "-0x1.32d2ccp+6", "0x1.466bc6p+6", "-0x1.4abbcep+5", "0x1.921fb6p+2"))
    cs = poly("-0x1.a6d1f2p+4", "0x1.e1f506p+5", "-0x1.55d3c8p+6", "0x1.03c1f0p+6", "-0x1.3bd3ccp+4", "0x1p+0")
    c = torch.where(j == 0, cs, torch.where(j == 1, -sn, torch.where(j == 2, -cs, sn)))
    s = torch.where(j == 0, sn, torch.where(j == 1, cs, torch.where(j == 2, -sn, -cs)))
    return _f32(R * c), _f32(R * s)


def _normals(seed, chain, kind, rhs, n):
    """Normals 0 .. n-1 of a stream at step 0."""
    w = _philox(seed, chain, 0, kind, rhs, -(-n // 4))
    p, q = _normal_pairs(w[0], w[1]), _normal_pairs(w[2], w[3])
    return torch.stack([*p, *q], dim=1).reshape(-1)[:n]


def _dirac(v, sigma, m0, g, dagger, pions=None):
    """D v or D^dag v, Wilson r = 1; v: (..., Nt, Nx, flavour, spin)."""
    sgn = -1.0 if dagger else 1.0
    edge = torch.ones(v.shape[-4], 1, 1, 1, device=v.device, dtype=torch.float64)
    up, dn = edge.clone(), edge.clone()
    up[-1], dn[0] = -1.0, -1.0       # antiperiodic in time
    tu, td = torch.roll(v, -1, -4) * up, torch.roll(v, 1, -4) * dn
    xu, xd = torch.roll(v, -1, -3), torch.roll(v, 1, -3)
    gt = torch.tensor([1.0, -1.0], device=v.device, dtype=torch.float64)
    hops = tu + td + xu + xd - sgn * (gt * (tu - td) + (xu - xd).flip(-1))
    out = (2.0 + m0 + g * sigma)[..., None, None] * v - 0.5 * hops
    if pions is not None:            # i gamma5 tau.pi, gamma5 = sigma_2 on spin
        w = torch.stack([v[..., 1], -v[..., 0]], dim=-1)
        p = [q[..., None] * (sgn * g) for q in pions]
        out = out + torch.stack([p[2] * w[..., 0, :] + (p[0] - 1j * p[1]) * w[..., 1, :],
                                 (p[0] + 1j * p[1]) * w[..., 0, :] - p[2] * w[..., 1, :]], dim=-2)
    return out


def _solve(b, apply):
    """x with A x = b, A = D^dag D, by CG to what 64 bits hold; b: (sources, ...)."""
    def dot(u, v):
        return (u.conj() * v).real.flatten(1).sum(1).reshape(-1, *([1] * (b.dim() - 1)))
    x, r = torch.zeros_like(b), b.clone()
    for _ in range(2):               # the second round takes the first one's true residual
        p, rr = r.clone(), dot(r, r)
        stop = rr * 1e-24
        for it in range(20000):
            q = apply(p)
            a = torch.where(rr > 0, rr / dot(p, q).clamp_min(1e-300), 0.0)
            x = x + a * p
            r = r - a * q
            new = dot(r, r)
            p = r + torch.where(rr > 0, new / rr.clamp_min(1e-300), 0.0) * p
            rr = new
            if it % 16 == 15 and bool((rr <= stop).all()):
                break
        r = b - apply(x)
    return x


def _laplace(f):
    return torch.roll(f, 1, 0) + torch.roll(f, -1, 0) + torch.roll(f, 1, 1) + torch.roll(f, -1, 1) - 4 * f


def _coloured(w):
    return torch.fft.ifft2(torch.fft.fft2(w) * _kept(*w.shape)).real


def _step(case, seed, c, sigma, pions):
    """The fields after one step of chain c: (sigma, pions or None), eps and the largest drift."""
    Nt, Nx, m0, g = _chains(case)[c]
    V = Nt * Nx
    ops = [lambda v, d=d: _dirac(v, sigma, m0, g, d, pions) for d in (False, True)]
    eta = torch.stack([_normals(seed, c, 2, j, 4 * V) for j in range(case.get("rhs", 1))])
    eta = eta.reshape(-1, Nt, Nx, 2, 2)
    if pions is not None:
        eta = eta.to(torch.complex128)
    chi = ops[0](_solve(eta, lambda v: ops[1](ops[0](v))))
    fields, noise = [sigma], [_normals(seed, c, 1, 0, V)]
    units = [eta]
    if pions is not None:
        zero, one = torch.zeros_like(sigma), torch.ones_like(sigma)
        for a in range(3):
            fields.append(pions[a])
            noise.append(_normals(seed, c, 1, a + 1, V))
            only = [one if q == a else zero for q in range(3)]
            # i gamma5 tau_a eta, as the operator with that pion alone less the one without
            units.append(_dirac(eta, zero, 0.0, 1.0, False, only) - _dirac(eta, zero, 0.0, 1.0, False))
    square = sum(f * f for f in fields)
    drift = [-g * (chi.conj() * u).real.sum((-1, -2)).mean(0) + f * (M2 + LAMBDA / 6 * square) - _laplace(f)
             for f, u in zip(fields, units)]
    top = max(float(d.abs().max()) for d in drift)
    top = min(max(top, 1e-5), 1e5)
    eps = 0.02 * 30 / top if case.get("adaptive") else 0.01
    new = [f - eps * d - math.sqrt(2 * eps) * _coloured(w.reshape(Nt, Nx)) for f, d, w in zip(fields, drift, noise)]
    return new[0], (torch.stack(new[1:]) if pions is not None else None), eps, top


def exact(case, seed):
    fields, more = _inputs(case, seed)
    if case["kind"] in ("dirac", "cg"):
        (Nt, Nx, m0, g), sigma = _chains(case)[0], fields[0]
        v = more["source"].to(torch.complex128).reshape(Nt, Nx, 2, 2)
        if case["kind"] == "dirac":
            return _dirac(v, sigma, m0, g, case["dagger"]).reshape(-1, 4)
        return _solve(v[None], lambda u: _dirac(_dirac(u, sigma, m0, g, False), sigma, m0, g, True)).reshape(-1, 4)
    out = []
    for c, sigma in enumerate(fields):
        new, pions, eps, top = _step(case, seed, c, sigma, more.get("pions"))
        out.append(new)
    if case["kind"] == "io":
        return [new.cpu().reshape(-1), float(new.sum()), float((new * new).sum()), eps, top]
    return out + ([pions] if case["kind"] == "pions" else [])
