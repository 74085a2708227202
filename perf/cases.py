"""The work that a user of this framework has it do, as cases that can be timed and compared.

Each case is one call sequence through the Python entry points, from page-locked host arrays
to page-locked (or, for the links, plain) host arrays, on one lattice or one batch of lattices:

  solve       set_trafo, overrelax to theta < eps, get_trafo
  sweeps      set_trafo, a fixed number of overrelaxation sweeps, the functional, get_trafo
  thermalize  a stretch of a heatbath chain with its plaquettes, get_links
  anneal      set_trafo, a stretch of simulated annealing with microcanonical sweeps, get_trafo
  fix         set_links, set_trafo, functional, apply_trafo, plaquette, Polyakov loop, get_links
  batch       Gribov copies of several configurations from Haar starts, the best copy of each

Links are Gram-Schmidt of 1 + eps * complex Gaussian (a weak-coupling-like configuration, mean
plaquette about 0.6 as at beta = 6), starts are Haar.  Both come from the seed alone.
"""
import math

import numpy as np
import torch

import cudagfx_gb300 as gfx

PREC = {"double": gfx.PREC_DOUBLE, "single": gfx.PREC_SINGLE, "mixed": gfx.PREC_MIXED}
GAUGE = {"landau": gfx.LANDAU, "coulomb": gfx.COULOMB}
LINK_EPS = 0.22


def listed():
    return [
        # the smallest lattice that is fixed in earnest, all in FP64 as by default: launches and
        # latency count (omega 1.7, theta < 1e-12, a check every 10 sweeps)
        dict(name="solve_f64_8x8x8x8", kind="solve", lx=8, ly=8, lz=8, lt=8, precision="double",
             link_reals=12, gauge="landau", eps=1e-12, checkinterval=10, near=0),
        # an ordinary mixed-precision Landau solve with the rebased FP32 polish
        dict(name="solve_mixed_16x16x16x32", kind="solve", lx=16, ly=16, lz=16, lt=32,
             precision="mixed", link_reals=18, gauge="landau", eps=1e-12, checkinterval=50, near=10),
        # the headline problem's lattice: mixed, 32^4
        dict(name="solve_mixed_32x32x32x32", kind="solve", lx=32, ly=32, lz=32, lt=32,
             precision="mixed", link_reals=12, gauge="landau", eps=1e-12, checkinterval=50, near=10),
        # the largest lattice: FP32 bulk sweeps that stream the links from HBM
        dict(name="sweeps_f32_48x48x48x96", kind="sweeps", lx=48, ly=48, lz=48, lt=96,
             precision="mixed", link_reals=12, gauge="landau", sweep_prec=0, n=50),
        # FP32 Coulomb sweeps of a lattice whose fields fit in L2
        dict(name="sweeps_f32_24x24x24x24", kind="sweeps", lx=24, ly=24, lz=24, lt=24,
             precision="single", link_reals=12, gauge="coulomb", sweep_prec=0, n=50),
        # FP64 sweeps as the reference runs them, on the layout the tuner chooses
        dict(name="sweeps_f64_32x32x32x32", kind="sweeps", lx=32, ly=32, lz=32, lt=32,
             precision="double", link_reals=18, gauge="landau", sweep_prec=1, n=10),
        # FP64 Coulomb sweeps on a ragged lattice (slices that are no multiple of a block)
        dict(name="sweeps_f64_12x10x14x18", kind="sweeps", lx=12, ly=10, lz=14, lt=18,
             precision="double", link_reals=12, gauge="coulomb", sweep_prec=1, n=20),
        # heatbath chain in FP64, the default precision of thermalize
        dict(name="therm_f64_16x16x16x32", kind="thermalize", lx=16, ly=16, lz=16, lt=32,
             precision="double", link_reals=12, beta=6.0, n=8, heatbath_prec=0),
        # heatbath chain in FP32 arithmetic, as the larger configurations are made
        dict(name="therm_f32_32x32x32x32", kind="thermalize", lx=32, ly=32, lz=32, lt=32,
             precision="mixed", link_reals=18, beta=6.0, n=40, heatbath_prec=1),
        # annealing before the overrelaxation: heatbath and three microcanonical sweeps a step
        dict(name="anneal_16x16x16x32", kind="anneal", lx=16, ly=16, lz=16, lt=32,
             precision="mixed", link_reals=12, steps=200, nmicro=3),
        # what a program does around the fixing: load, observables, the fixed field back
        dict(name="fix_16x16x16x32", kind="fix", lx=16, ly=16, lz=16, lt=32,
             precision="double", link_reals=12, gauge="landau"),
        # Gribov copies of two lattice sizes in one device loop
        dict(name="batch_16x16x16x16_24x24x24x24", kind="batch", la=16, ca=16, lb=24, cb=8,
             eps=1e-12, checkinterval=25),
    ]


def draw(rng):
    def even(lo, hi):
        return 2 * int(round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2)))))

    def dims(least, most):
        while True:
            d = [even(4, 40) for _ in range(4)]
            if least <= math.prod(d) <= most:
                return dict(lx=d[0], ly=d[1], lz=d[2], lt=d[3])

    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "sweeps", "sweeps", "sweeps", "thermalize", "anneal",
                       "fix", "batch"])
    c = dict(kind=kind)
    if kind == "batch":
        la, lb = rng.sample([8, 10, 12, 14, 16, 20, 24], 2)
        return dict(c, la=la, ca=spread(1, 12), lb=lb, cb=spread(1, 8), eps=1e-12,
                    checkinterval=rng.choice([10, 20, 25]))
    if kind == "solve":
        p = rng.choice(["double", "mixed", "mixed"])
        return dict(c, **dims(2000, 40_000 if p == "double" else 600_000), precision=p,
                    link_reals=rng.choice([12, 18]), gauge="landau", eps=1e-12,
                    checkinterval=rng.choice([10, 25, 50]), near=10 if p == "mixed" else 0)
    if kind == "sweeps":
        p = rng.choice([0, 1, 1])
        return dict(c, **dims(2000, 1_000_000), precision=rng.choice(["single", "mixed"]) if p == 0
                    else "double", link_reals=rng.choice([12, 18]),
                    gauge=rng.choice(["landau", "coulomb"]), sweep_prec=p,
                    n=spread(2, 60) if p == 0 else spread(1, 10))
    if kind == "thermalize":
        p = rng.choice([0, 0, 1])
        return dict(c, **dims(2000, 500_000), precision="mixed" if p else
                    rng.choice(["double", "mixed"]), link_reals=rng.choice([12, 18]),
                    beta=rng.choice([5.7, 6.0, 6.2]), n=spread(2, 40) if p else spread(1, 8),
                    heatbath_prec=p)
    if kind == "anneal":
        return dict(c, **dims(2000, 500_000), precision="mixed", link_reals=12,
                    steps=spread(20, 200), nmicro=rng.choice([0, 1, 3]))
    return dict(c, **dims(2000, 500_000), precision=rng.choice(["double", "mixed"]),
                link_reals=rng.choice([12, 18]), gauge=rng.choice(["landau", "coulomb"]))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _dims(c):
    return (c["lx"], c["ly"], c["lz"], c["lt"])


def _volume(c):
    return math.prod(_dims(c))


def _su3(rows):
    """(n, 2, 3) complex rows -> (n, 3, 3): Gram-Schmidt, row 2 = conj(row 0 x row 1)."""
    r0 = rows[:, 0] / torch.linalg.vector_norm(rows[:, 0], dim=1, keepdim=True)
    r1 = rows[:, 1] - torch.sum(rows[:, 1] * r0.conj(), 1, keepdim=True) * r0
    r1 = r1 / torch.linalg.vector_norm(r1, dim=1, keepdim=True)
    return torch.stack([r0, r1, torch.linalg.cross(r0, r1).conj()], 1)


def _random(n, seed, eps=None):
    """n SU(3) matrices on the GPU: Haar, or near the identity with eps."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out = torch.empty((n, 3, 3), dtype=torch.complex128, device="cuda")
    for a in range(0, n, 1 << 22):
        m = min(n - a, 1 << 22)
        z = torch.randn((m, 2, 3, 2), dtype=torch.float64, device="cuda", generator=gen)
        rows = torch.view_as_complex(z)
        if eps is not None:
            rows = eps * rows
            rows[:, 0, 0] += 1.0
            rows[:, 1, 1] += 1.0
        out[a:a + m] = _su3(rows)
    return out


def _pinned(m):
    """(n, 3, 3) complex on the GPU -> the host's su3 array in page-locked memory."""
    out = gfx.pinned_empty((m.shape[0], 3, 3, 2))
    torch.from_numpy(out).copy_(torch.view_as_real(m))
    return out


def _links(c, seed):
    return _random(4 * _volume(c), 2 * seed, LINK_EPS)


def _start(c, seed):
    return _random(_volume(c), 2 * seed + 1)


def _twister_bank(ctx, seed, n_gauss, n_unif):
    r = np.random.RandomState(seed % (1 << 31))
    p = r.randint(0, 1 << 32, size=(4096, 4), dtype=np.uint64).astype(np.uint32)
    p[:, 0] |= np.uint32(0x80000000)
    ctx.mt_load_params(p)
    ctx.mt_seed(seed % (1 << 31))
    # whole rounds of 19 outputs per twister: a stream that goes on from call to call
    per = 4096 * 38
    ctx.mt_init(-(-n_gauss // per) * per, -(-n_unif // per) * per)


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "batch":
        dims = [(c["la"],) * 4, (c["lb"],) * 4]
        b = gfx.Batch(dims, [c["ca"], c["cb"]])
        for k, d in enumerate(dims):
            b.set_links(k, _pinned(_random(4 * math.prod(d), 4 * seed + k, LINK_EPS)))
        s.update(batch=b, seed=seed, params=gfx.Context.or_params(
            maxit=20000, eps=c["eps"], checkinterval=c["checkinterval"], omega=1.7,
            criterion=gfx.CRIT_THETA, checkinterval_double=2, polish=2))
        return s
    ctx = gfx.Context(_dims(c), precision=PREC[c["precision"]], link_reals=c["link_reals"])
    V = ctx.volume
    u = _pinned(_links(c, seed))
    s["ctx"] = ctx
    if c["kind"] == "fix":
        s["u"] = u
    else:
        ctx.set_links(u)
    if c["kind"] != "thermalize":
        s["g0"] = _pinned(_start(c, seed))
        s["g"] = gfx.pinned_empty((V, 3, 3, 2))
    if c["kind"] == "solve":
        s["params"] = gfx.Context.or_params(
            maxit=20000, eps=c["eps"], checkinterval=c["checkinterval"], omega=1.7,
            criterion=gfx.CRIT_THETA, checkinterval_double=2, checkinterval_near=c["near"],
            polish=2)
    if c["kind"] == "thermalize":
        _twister_bank(ctx, seed, 4 * V, 16 * V)
    if c["kind"] == "anneal":
        _twister_bank(ctx, seed, V, 4 * V)
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "batch":
        b = state["batch"]
        b.random_haar(state["seed"] % (1 << 40))
        res, _ = b.overrelax(state["params"])
        best = [b.best(k)[0] for k in range(2)]
        return {"F": np.array([r["F"] for r in res]),
                "iterations": np.array([r["iterations"] for r in res]),
                "best": np.array(best), "g": [b.get_trafo(k, best[k]) for k in range(2)]}
    ctx = state["ctx"]
    if kind == "thermalize":
        plaq = ctx.thermalize(c["beta"], c["n"], checkint=4, variant=gfx.HB_KENNEDY_PENDLETON,
                              precision=c["heatbath_prec"])
        return {"links": ctx.get_links(), "plaq": plaq}
    if kind == "fix":
        gauge = GAUGE[c["gauge"]]
        ctx.set_links(state["u"])
        ctx.set_trafo(state["g0"])
        before = ctx.functional(gauge)
        ctx.apply_trafo()
        plaq, loop = ctx.plaquette(), ctx.polyakov()
        return {"functional": before.as_dict(), "plaq": plaq, "polyakov": [loop.real, loop.imag],
                "links": ctx.get_links()}
    ctx.set_trafo(state["g0"])
    if kind == "solve":
        r = ctx.overrelax(state["params"])
        # theta itself is left out: of a fixed field it is a square of rounding-sized numbers
        return {"F": r.final_values.F, "iterations": r.iterations, "sweeps": r.sweeps,
                "g": ctx.get_trafo_into(state["g"])}
    if kind == "anneal":
        f = ctx.simanneal(0.01, 1.4, c["steps"], nmicro=c["nmicro"])
    else:
        gauge = GAUGE[c["gauge"]]
        ctx.or_sweeps(c["n"], 1.7, gauge, c["sweep_prec"])
        f = ctx.functional(gauge)
    return {"functional": f.as_dict(), "g": ctx.get_trafo_into(state["g"])}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
UPDATE_FLOPS = 4766.0   # per overrelaxation update, the count of overrelax.cu:897
MEASURE_FLOPS = 1950.0  # nine SU(3) products and the norm, per site
SU3 = 198.0             # flops of one product


def work(case):
    """Bytes and flops of one pass: per half-sweep each link and each g once, the updated g
    written; per call each host array once."""
    c = case
    if c["kind"] == "batch":
        va, vb = c["la"] ** 4, c["lb"] ** 4
        v, n = va * c["ca"] + vb * c["cb"], 300.0
        return {"bytes": n * (240.0 * (va + vb) + 192.0 * v) + 144.0 * (va + vb),
                "flops": n * v * UPDATE_FLOPS}
    v = float(_volume(c))
    r = c["link_reals"]
    host_g, host_u = 144.0 * v, 576.0 * v
    if c["kind"] == "thermalize":
        per = 24.0 * (4 + 4) * 4 * c["n"] * v  # a staple and a link a direction, FP64 rows
        fields = 4 * 2 * c["n"] * 4.0 * 20.0 * v
        return {"bytes": per + fields + host_u, "flops": 4 * c["n"] * v * (18 * SU3 + 700.0)}
    if c["kind"] == "anneal":
        sweeps = c["steps"] * (1 + c["nmicro"])
        return {"bytes": sweeps * 528.0 * v + c["steps"] * 2 * 20.0 * v + 2 * host_g,
                "flops": sweeps * v * UPDATE_FLOPS}
    if c["kind"] == "fix":
        dev_u, dev_g = 32.0 * r * v, 96.0 * v
        return {"bytes": 2 * host_u + host_g + 5 * dev_u + 3 * dev_g,
                "flops": v * (MEASURE_FLOPS + 8 * SU3 + 18 * SU3 + SU3)}
    nd = 3 if c["gauge"] == "coulomb" else 4
    f32 = c["precision"] != "double"
    size = 4.0 if f32 else 8.0
    reals = 2 * nd * (12 if f32 else r) + 24 + 12
    n = c["n"] if c["kind"] == "sweeps" else 200.0
    return {"bytes": n * v * size * reals + 2 * host_g + v * (8.0 * nd * r + 96.0),
            "flops": n * v * UPDATE_FLOPS * nd / 4 + v * MEASURE_FLOPS}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------
class _Lattice:
    """Fields as tensors [t, z, y, x, ...]; direction mu = 0..3 = x, y, z, t."""

    def __init__(self, c):
        self.lx, self.ly, self.lz, self.lt = _dims(c)
        self.shape = (self.lt, self.lz, self.ly, self.lx)
        self.V = math.prod(self.shape)
        t, z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in self.shape],
                                    indexing="ij")
        self.parity = (t + z + y + x) & 1

    def g(self, m):
        return m.reshape(*self.shape, 3, 3)

    def u(self, m):
        return m.reshape(*self.shape, 4, 3, 3)

    @staticmethod
    def fwd(f, mu):
        return torch.roll(f, -1, 3 - mu)

    @staticmethod
    def bwd(f, mu):
        return torch.roll(f, 1, 3 - mu)


def _mul(a, b):
    r = a[..., :, 0, None] * b[..., 0, None, :]
    for k in (1, 2):
        r = r + a[..., :, k, None] * b[..., k, None, :]
    return r


def _dag(a):
    return a.conj().transpose(-1, -2)


def _unitary(rows):
    n = rows.shape[:-2]
    return _su3(rows[..., :2, :].reshape(-1, 2, 3)).reshape(*n, 3, 3)


def _star(lat, u, g, ndir):
    w = torch.zeros_like(g)
    for mu in range(ndir):
        w = w + _mul(u[..., mu, :, :], _dag(lat.fwd(g, mu)))
        w = w + lat.bwd(_dag(_mul(g, u[..., mu, :, :])), mu)
    return w


def _or_halfsweep(lat, u, g, parity, omega, ndir):
    old = g
    w = _star(lat, u, g, ndir)
    h = g.clone()
    for a, b in ((0, 1), (0, 2), (1, 2)):
        x = _mul(h, w)
        v0 = x[..., a, a].real + x[..., b, b].real
        v3 = x[..., b, b].imag - x[..., a, a].imag
        v1 = -x[..., a, b].imag - x[..., b, a].imag
        v2 = x[..., b, a].real - x[..., a, b].real
        n = torch.sqrt(v0 * v0 + v1 * v1 + v2 * v2 + v3 * v3)
        p, q = torch.complex(v0, v3) / n, torch.complex(v2, v1) / n
        ra, rb = h[..., a, :].clone(), h[..., b, :].clone()
        h[..., a, :] = p[..., None] * ra + q[..., None] * rb
        h[..., b, :] = p.conj()[..., None] * rb - q.conj()[..., None] * ra
    one = torch.eye(3, dtype=torch.complex128, device="cuda")
    r = _mul(h, _dag(old)) - one
    new = _unitary(_mul(one + omega * r + 0.5 * omega * (omega - 1) * _mul(r, r), old))
    return torch.where((lat.parity == parity)[..., None, None], new, old)


def _functional(lat, u, g, ndir):
    x = _mul(g, _star(lat, u, g, ndir))
    tr = x.diagonal(dim1=-2, dim2=-1).sum(-1)
    ah = 0.5 * (x - _dag(x))
    ah = ah - (1j * tr.imag / 3)[..., None, None] * torch.eye(3, device="cuda")
    d = (ah.abs() ** 2).sum((-1, -2))
    slices = d.sum((1, 2, 3)) / (3.0 * lat.V / lat.lt)
    dada = float(d.mean())
    return {"F": float(tr.real.sum()) / (2 * ndir * lat.V), "dAdA": dada,
            "maxdAdA": float(d.max()), "theta": dada / 3, "theta_slice_max": float(slices.max())}


def _host(m):
    return torch.view_as_real(m.contiguous()).reshape(-1, 3, 3, 2).cpu().numpy()


def exact(case, seed):
    c = case
    if c["kind"] in ("thermalize", "anneal", "batch"):
        return None  # a chain of random draws, or which of many maxima is reached
    v = _volume(c)
    if c["kind"] == "solve" and (c["precision"] != "double" or v > 6000):
        return None
    if c["kind"] == "sweeps" and v * c["n"] > 2.2e7:
        return None
    lat = _Lattice(c)
    ndir = 3 if c["gauge"] == "coulomb" else 4
    u, g = lat.u(_links(c, seed)), lat.g(_start(c, seed))
    if c["kind"] == "fix":
        f = _functional(lat, u, g, ndir)
        for mu in range(4):
            u[..., mu, :, :] = _mul(_mul(g, u[..., mu, :, :].clone()), _dag(lat.fwd(g, mu)))
        plaq = 0.0
        for nu in range(3):
            for mu in range(nu + 1, 4):
                a = _mul(u[..., mu, :, :], lat.fwd(u[..., nu, :, :], mu))
                b = _mul(u[..., nu, :, :], lat.fwd(u[..., mu, :, :], nu))
                plaq += float((a * b.conj()).real.sum()) / 3
        p = u[0, ..., 3, :, :]
        for t in range(1, lat.lt):
            p = _mul(p, u[t, ..., 3, :, :])
        loop = complex(p.diagonal(dim1=-2, dim2=-1).sum(-1).mean()) / 3
        return {"functional": f, "plaq": plaq / (6 * v), "polyakov": [loop.real, loop.imag],
                "links": _host(u)}
    if c["kind"] == "sweeps":
        for _ in range(c["n"]):
            for parity in (0, 1):
                g = _or_halfsweep(lat, u, g, parity, 1.7, ndir)
        return {"functional": _functional(lat, u, g, ndir), "g": _host(g)}
    it = 0
    for parity in (0, 1):
        g = _or_halfsweep(lat, u, g, parity, 1.7, ndir)
    f = _functional(lat, u, g, ndir)
    while f["theta"] >= c["eps"] and it < 2000:
        for _ in range(c["checkinterval"]):
            for parity in (0, 1):
                g = _or_halfsweep(lat, u, g, parity, 1.7, ndir)
        it += c["checkinterval"]
        f = _functional(lat, u, g, ndir)
    return {"F": f["F"], "iterations": None, "sweeps": None, "g": _host(g)}
