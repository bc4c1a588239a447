"""The workloads this framework is measured on: lattice-gauge update and measurement calls as a
simulation program makes them, through the public classes of klft_b200.

Kinds of case (``kind``):

* ``measure``    plaquette, temporal and planar Wilson loops of a resident configuration
* ``analyse``    the same for a stored configuration, which comes from host memory first
* ``run``        run_metropolis: sweeps with interval measurements (plaquette, planar loops), then the
                 configuration is fetched
* ``cycles``     one sweep and one measurement per cycle, then the configuration is fetched
* ``hmc``        HMC trajectories with accept/reject, then the configuration is fetched
* ``integrate``  molecular dynamics from given momenta: links and momenta after it
* ``batch``      PTBC replicas and independent chains advanced together
* ``serve``      a burst of mixed jobs through the job server
"""
import numpy as np
import torch

import klft_b200
from klft_b200.serve import Server, poisson_jobs

# beta, spread of the input links about the identity (plaquettes of thermalised size) and proposal width
BETA = {1: 2.0, 2: 2.3, 3: 6.0}
SPREAD = {1: 0.35, 2: 0.25, 3: 0.15}
DELTA = {1: 0.1, 2: 0.3, 3: 0.1}
NCOMP = {1: 1, 2: 3, 3: 8}
EPS, NHITS = 0.25, 10


def listed():
    return [
        # one observable of a small lattice between two steps of a user's own loop: latency alone
        dict(name="plaquette_su2_8x4", kind="measure", nc=2, L="8,8,8,8", precision="fp64", pairs="", planes="", planar=""),
        # klft's small plain-method run: sweeps of tiny lattices, measured every ten
        dict(name="run_u1_8x4", kind="run", nc=1, L="8,8,8,8", precision="fp64", proposal="reference", nsweeps=100,
             interval=10, planes="0x1,1x2,3x2", planar="2x2,3x3,4x3"),
        # klft's own SU(2) run on a ragged box
        dict(name="run_su2_ragged", kind="run", nc=2, L="12,8,10,20", precision="fp64", proposal="reference",
             nsweeps=40, interval=10, planes="0x3,1x3,2x3", planar="1x1,2x2,3x4,4x6"),
        # klft's own SU(3) proposals, double precision as klft computes
        dict(name="run_su3_16x4", kind="run", nc=3, L="16,16,16,16", precision="fp64", proposal="reference",
             nsweeps=11, interval=5, planes="0x3,1x3,2x3", planar="1x1,2x2,3x3,4x4"),
        # the headline workload: SU(3) 32^4 sweep + plaquette + 64 temporal loops a cycle, FP32 links
        dict(name="cycles_su3_32x4_mixed", kind="cycles", nc=3, L="32,32,32,32", precision="mixed", proposal="exp",
             ncycles=10, pairs="8*8"),
        # its double-precision form on a finite-temperature box
        dict(name="cycles_su3_fp64", kind="cycles", nc=3, L="16,16,16,32", precision="fp64", proposal="exp",
             ncycles=10, pairs="4*4"),
        # static-potential measurement with long loops, double precision
        dict(name="loops_su3_fp64", kind="measure", nc=3, L="24,24,24,48", precision="fp64", pairs="8*12",
             planes="0x1,0x2,1x2", planar="4*4"),
        # a stored 32^4 configuration taken from host memory and measured
        dict(name="analyse_su3_32x4_mixed", kind="analyse", nc=3, L="32,32,32,32", precision="mixed", pairs="8*8",
             planes="", planar=""),
        # the HMC workload: SU(2) 24^4, 20 leapfrog steps a trajectory
        dict(name="hmc_su2_24x4_mixed", kind="hmc", nc=2, L="24,24,24,24", precision="mixed", integrator="leapfrog",
             nsteps=20, tau=0.2, ntraj=4),
        # SU(3) molecular dynamics in double precision
        dict(name="integrate_su3_16x4_fp64", kind="integrate", nc=3, L="16,16,16,16", precision="fp64",
             integrator="omelyan", nsteps=10, tau=0.5),
        # PTBC replicas and SU(2) chains of several extents in one batch
        dict(name="batch_ptbc", kind="batch", nrep=8, L="16,16,16,16", precision="mixed", nchains=16, emax=24, ncycles=10),
        # a burst of jobs at the server, mixed groups, dimensions and algorithms
        dict(name="serve_burst", kind="serve", njobs=12, emax=14, sweeps=60, trajectories=6, precision="mixed"),
    ]


def _extents(rng, nd, volume):
    """nd even extents >= 4 whose product is near `volume`."""
    L = []
    for d in range(nd):
        mean = max(4.0, volume ** (1.0 / (nd - d)))
        x = mean * rng.uniform(0.75, 1.35) if d < nd - 1 else mean
        L.append(max(4, min(64, 2 * round(x / 2))))
        volume = max(1.0, volume / L[-1])
    rng.shuffle(L)
    return L


def _grid(rng, L, most):
    """All loops up to an a x b that fits half the lattice, in the 'a*b' form of a pair list."""
    n = min(L)
    a = rng.randint(1, max(1, min(n // 2, most)))
    b = rng.randint(1, max(1, min(L[-1] // 2, 12, 120 // a)))
    return "%d*%d" % (a, b)


def draw(rng):
    kind = rng.choice(["measure", "analyse", "run", "run", "cycles", "hmc", "integrate", "batch", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "serve":
        return dict(kind=kind, njobs=rng.randint(4, 12), emax=rng.choice([8, 10, 12, 14]), sweeps=rng.randint(50, 60),
                    trajectories=rng.randint(3, 6), precision=precision)
    if kind == "batch":
        e = [rng.choice([4, 6, 8, 10, 12, 14]) for _ in range(4)]
        return dict(kind=kind, nrep=rng.randint(2, 8), L=",".join(map(str, e)), precision=precision,
                    nchains=rng.randint(1, 16), emax=rng.choice([8, 12, 16, 20]), ncycles=rng.randint(3, 10))
    nc = rng.choice([1, 2, 3])
    nd = rng.choice([2, 3, 4, 4, 4])
    top = {"measure": 17.0, "analyse": 18.0, "run": 15.0, "cycles": 17.0, "hmc": 16.0, "integrate": 16.0}[kind]
    L = _extents(rng, nd, 2.0 ** rng.uniform(6.0 if nd < 4 else 8.0, min(top, 6.0 * nd)))
    c = dict(kind=kind, nc=nc, L=",".join(map(str, L)), precision=precision)
    if kind in ("measure", "analyse"):
        mu, nu = rng.sample(range(nd), 2)
        c.update(pairs=rng.choice(["", _grid(rng, L, 8)]), planes="%dx%d" % (mu, nu),
                 planar=rng.choice(["", "2x2,3x3,4x3", "1x1,2x5"]))
    elif kind == "run":
        c.update(proposal=rng.choice(["reference", "exp"]) if nc == 3 else "reference", nsweeps=rng.randint(11, 40),
                 interval=rng.choice([5, 10]), planes=rng.choice(["", "0x1", "1x0"]), planar=_grid(rng, L, 4))
    elif kind == "cycles":
        c.update(proposal=rng.choice(["reference", "exp"]) if nc == 3 else "reference", ncycles=rng.randint(2, 10),
                 pairs=_grid(rng, L, 8))
    elif kind == "hmc":
        c.update(integrator=rng.choice(["leapfrog", "omelyan", "reference"]), nsteps=rng.randint(8, 20),
                 tau=round(rng.uniform(0.1, 0.5), 2), ntraj=rng.randint(1, 4))
    else:
        c.update(integrator=rng.choice(["leapfrog", "omelyan", "reference"]), nsteps=rng.randint(5, 12),
                 tau=round(rng.uniform(0.1, 0.5), 2))
    return c


# ------------------------------------------------------------------ inputs
def _list(text):
    """'4,6,8' -> [4, 6, 8]."""
    return [int(x) for x in text.split(",")]


def _pairs(text):
    """'2x3,4x4' -> [(2, 3), (4, 4)]; '2*3' -> every (l, t) with l <= 2, t <= 3."""
    if not text:
        return []
    if "*" in text:
        a, b = (int(x) for x in text.split("*"))
        return [(i, j) for i in range(1, a + 1) for j in range(1, b + 1)]
    return [tuple(int(x) for x in p.split("x")) for p in text.split(",")]


def _links(L, nc, precision, seed):
    """Random links near the identity, complex128 [site, mu, i, j] on the GPU; for the mixed form
    their stored rows hold FP32 values."""
    n = int(np.prod(L)) * len(L)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    s = SPREAD[nc]
    dev = dict(device="cuda", dtype=torch.float64)
    low = (lambda z: z.to(torch.complex64).to(torch.complex128)) if precision == "mixed" else (lambda z: z)
    if nc == 1:
        p = s * torch.randn(n, generator=gen, **dev)
        u = low(torch.complex(torch.cos(p), torch.sin(p))).view(n, 1, 1)
    elif nc == 2:
        q = s * torch.randn(4, n, generator=gen, **dev)
        q[0] += 1.0
        q /= q.square().sum(0).sqrt()
        a, b = low(torch.complex(q[0], q[1])), low(torch.complex(q[2], q[3]))
        u = torch.stack([a, b, -b.conj(), a.conj()], -1).view(n, 2, 2)
    else:
        r = s * torch.randn(2, 3, 2, n, generator=gen, **dev)
        r[0, 0, 0] += 1.0
        r[1, 1, 0] += 1.0
        z = torch.complex(r[:, :, 0], r[:, :, 1])
        r0 = z[0] / z[0].abs().square().sum(0).sqrt()
        r1 = z[1] - (r0.conj() * z[1]).sum(0) * r0
        r1 = r1 / r1.abs().square().sum(0).sqrt()
        r0, r1 = low(r0), low(r1)
        r2 = torch.stack([r0[1] * r1[2] - r0[2] * r1[1], r0[2] * r1[0] - r0[0] * r1[2],
                          r0[0] * r1[1] - r0[1] * r1[0]]).conj()
        u = torch.stack([r0, r1, r2]).permute(2, 0, 1).contiguous()
    return u.view(n // len(L), len(L), nc, nc)


def _momenta(L, nc, precision, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    p = torch.randn(int(np.prod(L)), len(L), NCOMP[nc], generator=gen, device="cuda", dtype=torch.float64)
    return p.float().double() if precision == "mixed" else p


def _field(L, nc, precision, seed):
    g = klft_b200.GaugeField(L, nc, precision, "cold", seed)
    u = _links(L, nc, precision, seed).cpu().numpy()
    g.upload(u)
    g.set_stream(seed, 0)
    return g, u


def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    if kind == "serve":
        rng = np.random.default_rng(seed)
        jobs = [j for _, j in poisson_jobs(c["njobs"], 1.0, 2024, (8, c["emax"]), (50, c["sweeps"]),
                                           (2, c["trajectories"]), c["precision"])]
        for j in jobs:
            j.seed = int(rng.integers(1, 2 ** 62))
        return dict(c, server=Server(), jobs=jobs)
    L = _list(c["L"])
    c["L"] = L
    if kind == "batch":
        rng = np.random.default_rng(c["nchains"])  # the extents belong to the case, the links to the seed
        evens = np.arange(8, c["emax"] + 1, 4)
        b, fields = klft_b200.Batch(), []
        for r in range(c["nrep"]):
            g = klft_b200.GaugeField(L, 3, c["precision"], "hot", seed + r)
            g.set_stream(seed, r)
            g.set_defect(min(4, min(L[1:])), (0, 0, 0), 1.0)
            b.add(g, BETA[3], 0.0, NHITS, "exp", EPS)
            fields.append(g)
        b.set_ptbc(list(range(c["nrep"])), [1.0 - r / max(1, c["nrep"] - 1) for r in range(c["nrep"])], BETA[3], seed)
        for k in range(c["nchains"]):
            e = [int(x) for x in rng.choice(evens, size=4)]
            g = klft_b200.GaugeField(e, 2, c["precision"], "hot", seed + 1000 + k)
            g.set_stream(seed, 1000 + k)
            b.add(g, float(rng.uniform(2.2, 2.6)), DELTA[2], NHITS, "reference", 0.0)
            fields.append(g)
        return dict(c, batch=b, fields=fields, out=[_host(g.shape()) for g in fields])
    g, u = _field(L, c["nc"], c["precision"], seed)
    c.update(g=g, beta=BETA[c["nc"]], delta=DELTA[c["nc"]])
    for k in ("pairs", "planes", "planar"):
        if k in c:
            c[k] = _pairs(c[k])
    if kind == "analyse":
        c["u"] = u
    if kind == "integrate":
        g.set_momenta(_momenta(L, c["nc"], c["precision"], seed).cpu().numpy())
    if kind in ("run", "cycles", "hmc", "integrate"):
        c["out"] = _host(g.shape())
    return c


def _host(shape):
    """The buffer in which a program takes its configurations, its pages touched."""
    a = np.empty(shape, dtype=np.complex128)
    a.fill(0)
    return a


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "serve":
        ids = [s["server"].submit(j) for j in s["jobs"]]
        got = s["server"].wait(ids)
        return [np.array([r["status"], r["plaquette"], r["acceptance"], r["mean_exp_mdH"], r["mean_dH"], r["link_updates"]]
                         + r["wilson"], dtype=np.float64) for r in (got[i] for i in ids)]
    if kind == "batch":
        acc, plaq, lab, _ = s["batch"].run(s["ncycles"])
        return [acc, plaq, lab] + [g.download(o) for g, o in zip(s["fields"], s["out"])]
    g = s["g"]
    if kind in ("measure", "analyse"):
        if kind == "analyse":
            g.upload(s["u"])
        out = [g.plaquette()]
        if s["pairs"]:
            out.append(g.wilson_loop_temporal(s["pairs"]))
        if s["planar"]:
            out += [g.wilson_loop_mu_nu(mu, nu, s["planar"]) for mu, nu in s["planes"]]
        return out
    if kind == "run":
        acc, plaq, _, wm, _ = g.run_metropolis_measured(s["beta"], s["delta"], NHITS, s["nsweeps"], s["interval"],
                                                         s["proposal"], EPS, True, (), s["planes"],
                                                         s["planar"] if s["planes"] else ())
        return [acc, plaq, wm, g.download(s["out"])]
    if kind == "cycles":
        acc, plaq, w, _ = g.run_cycles(s["beta"], s["delta"], NHITS, s["ncycles"], s["proposal"], EPS, True, s["pairs"])
        return [acc, plaq, w, g.download(s["out"])]
    if kind == "hmc":
        dH, acc = g.hmc(s["beta"], s["tau"], s["nsteps"], s["ntraj"], s["integrator"])
        return [dH, acc, g.download(s["out"])]
    g.hmc_integrate(s["beta"], s["tau"], s["nsteps"], s["integrator"])
    return [g.momenta(), g.download(s["out"])]


# ------------------------------------------------------------------ necessary work
MUL = {1: 6, 2: 28, 3: 198}  # flops of one product of two links


def _sweep(nc, nd, links, nhits, precision):
    """Bytes and flops of one sweep: each link read and written once; its staple, then nhits proposals
    with one product and one trace each."""
    b = 2 * links * _link_bytes(nc, precision)
    return b, links * (4 * (nd - 1) * MUL[nc] + nhits * (2 * MUL[nc] + 60) + 2 * MUL[nc])


def _link_bytes(nc, precision):
    return {1: 8, 2: 16, 3: 48}[nc] if precision == "mixed" else 16 * nc * nc


def _loops(nc, V, pairs, planes):
    """Flops of the loops in `planes` planes: a product per line step and a trace per pair."""
    lmax = max([p[0] for p in pairs], default=0)
    return planes * V * ((lmax + 2) * MUL[nc] + len(pairs) * 4 * nc * nc)


def work(case):
    c, kind = case, case["kind"]
    if kind == "serve":
        b = f = 0.0
        for _, j in poisson_jobs(c["njobs"], 1.0, 2024, (8, c["emax"]), (50, c["sweeps"]), (2, c["trajectories"]),
                                 c["precision"]):
            links = j.volume * len(j.extents)
            if j.kind == "metropolis":
                x, y = _sweep(j.nc, len(j.extents), links, j.nhits, c["precision"])
                b, f = b + x * j.nsweeps, f + y * j.nsweeps
            else:
                x, y = _hmc(j.nc, len(j.extents), links, c["precision"], j.integrator, j.nsteps)
                b, f = b + x * j.ntraj, f + y * j.ntraj
        return {"bytes": b, "flops": f}
    L = _list(c["L"])
    nd, V = len(L), int(np.prod(L))
    if kind == "batch":
        rng = np.random.default_rng(c["nchains"])
        evens = np.arange(8, c["emax"] + 1, 4)
        vols = []
        for _ in range(c["nchains"]):
            vols.append(int(np.prod(rng.choice(evens, size=4))))
            rng.uniform(2.2, 2.6)
        b1, f1 = _sweep(3, 4, 4 * V * c["nrep"], NHITS, c["precision"])
        b2, f2 = _sweep(2, 4, 4 * sum(vols), NHITS, c["precision"])
        host = 16 * 4 * (9 * V * c["nrep"] + 4 * sum(vols))
        return {"bytes": c["ncycles"] * (b1 + b2) + host, "flops": c["ncycles"] * (f1 + f2)}
    nc, precision = c["nc"], c["precision"]
    links = V * nd
    field, host = links * _link_bytes(nc, precision), links * 16 * nc * nc
    plaq = V * nd * (nd - 1) / 2 * (2 * MUL[nc] + 4 * nc * nc)
    pairs = _pairs(c.get("pairs", ""))
    if kind in ("measure", "analyse"):
        planar, planes = _pairs(c["planar"]), _pairs(c["planes"])
        f = plaq + _loops(nc, V, pairs, nd - 1) + (_loops(nc, V, planar, len(planes)) if planar else 0)
        return {"bytes": field + (host if kind == "analyse" else 0), "flops": f}
    if kind in ("run", "cycles"):
        sweeps = c["nsweeps"] if kind == "run" else c["ncycles"]
        nmeas = (c["nsweeps"] - 1) // c["interval"] if kind == "run" else sweeps
        b, f = _sweep(nc, nd, links, NHITS, precision)
        m = plaq + _loops(nc, V, pairs, nd - 1)
        if kind == "run" and c["planes"]:
            m += _loops(nc, V, _pairs(c["planar"]), len(_pairs(c["planes"])))
        return {"bytes": sweeps * b + nmeas * field + host, "flops": sweeps * f + nmeas * m}
    b, f = _hmc(nc, nd, links, precision, c["integrator"], c["nsteps"])
    n = c.get("ntraj", 1)
    return {"bytes": n * b + host, "flops": n * f}


def _hmc(nc, nd, links, precision, integrator, nsteps):
    """One trajectory: each force reads links and momenta and writes momenta, each link step reads both
    and writes links."""
    ub, pb = links * _link_bytes(nc, precision), links * NCOMP[nc] * (4 if precision == "mixed" else 8)
    nf, nu = {"reference": (nsteps + 2, nsteps + 1), "leapfrog": (nsteps + 1, nsteps),
              "omelyan": (3 * nsteps, 2 * nsteps)}[integrator]
    force = 4 * (nd - 1) * MUL[nc] + MUL[nc]
    return nf * (ub + 2 * pb) + nu * (2 * ub + pb), links * (nf * force + nu * (MUL[nc] + 150))


# ------------------------------------------------------------------ values in 64 bits
def _lattice(u, L):
    """[site, mu, i, j] -> [x_{nd-1}, ..., x_0, mu, i, j] (x0 runs fastest)."""
    return u.view(*reversed(L), *u.shape[1:])


def _up(t, nd, d, k=1):
    """t(x + k e_d)."""
    return torch.roll(t, -k, dims=nd - 1 - d)


def _mul(a, b):
    return sum(a[..., :, k, None] * b[..., None, k, :] for k in range(a.shape[-1]))


def _dag(a):
    return a.conj().transpose(-1, -2)


def _retr(a, b):
    """Sum over sites of Re Tr a b^+."""
    return float((a.real * b.real + a.imag * b.imag).sum())


def _plaquette(u, nd, nc, V):
    s = 0.0
    for mu in range(nd):
        for nu in range(mu + 1, nd):
            a, b = u[..., mu, :, :], u[..., nu, :, :]
            s += _retr(_mul(a, _up(b, nd, mu)), _mul(b, _up(a, nd, nu)))
    return s / (V * nd * (nd - 1) / 2 * nc)


def _wilson(u, nd, nc, V, mu, nu, pairs):
    def lines(d, n):
        a = u[..., d, :, :]
        got = [None, a]
        for k in range(1, n):
            got.append(_mul(got[-1], _up(a, nd, d, k)))
        return got
    x, y = lines(mu, max(p[0] for p in pairs)), lines(nu, max(p[1] for p in pairs))
    return np.array([_retr(_mul(x[a], _up(y[b], nd, mu, a)), _mul(y[b], _up(x[a], nd, nu, b))) / (V * nc)
                     for a, b in pairs])


def _generators(nc):
    if nc == 1:
        return torch.ones(1, 1, 1, dtype=torch.complex128, device="cuda")
    if nc == 2:
        t = [[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]]
    else:
        r = 1 / 3 ** 0.5
        t = [[[0, 1, 0], [1, 0, 0], [0, 0, 0]], [[0, -1j, 0], [1j, 0, 0], [0, 0, 0]], [[1, 0, 0], [0, -1, 0], [0, 0, 0]],
             [[0, 0, 1], [0, 0, 0], [1, 0, 0]], [[0, 0, -1j], [0, 0, 0], [1j, 0, 0]], [[0, 0, 0], [0, 0, 1], [0, 1, 0]],
             [[0, 0, 0], [0, 0, -1j], [0, 1j, 0]], [[r, 0, 0], [0, r, 0], [0, 0, -2 * r]]]
    return torch.tensor(t, dtype=torch.complex128, device="cuda")


def _integrate(c, L, u, p):
    """U' = exp(i dt p_a t_a) U and p' = p - dt (beta/Nc) Im Tr(t_a U S), in the integrator's order."""
    nd, nc = len(L), c["nc"]
    t, bnc, dt = _generators(nc), BETA[nc] / nc, c["tau"] / c["nsteps"]

    def kick(h):
        for mu in range(nd):
            a, s = u[..., mu, :, :], 0
            for nu in range(nd):
                if nu != mu:
                    b = u[..., nu, :, :]
                    s = s + _mul(_up(b, nd, mu), _dag(_mul(b, _up(a, nd, nu))))
                    low = _up(_mul(_dag(_mul(a, _up(b, nd, mu))), b), nd, nu, -1)
                    s = s + low
            m = _mul(a, s)
            for i in range(len(t)):
                p[..., mu, i] -= h * bnc * sum((t[i, j, k] * m[..., k, j]).imag for j in range(nc) for k in range(nc))

    def move(h):
        for mu in range(nd):
            q = sum(p[..., mu, i, None, None] * t[i] for i in range(len(t))) * (1j * h)
            e = torch.eye(nc, dtype=torch.complex128, device="cuda").expand_as(q)
            x = e
            for n in range(24, 0, -1):  # Horner's scheme of the exponential's series
                x = e + _mul(q, x) / n
            u[..., mu, :, :] = _mul(x, u[..., mu, :, :])

    n = c["nsteps"]
    if c["integrator"] == "reference":
        steps = [(kick, dt / 2), (move, dt)] + [(kick, dt), (move, dt)] * n + [(kick, dt / 2)]
    elif c["integrator"] == "leapfrog":
        steps = [(kick, dt / 2)] + [(move, dt), (kick, dt)] * (n - 1) + [(move, dt), (kick, dt / 2)]
    else:
        lam = 0.1931833275037836
        steps = [(kick, lam * dt), (move, dt / 2), (kick, (1 - 2 * lam) * dt), (move, dt / 2), (kick, lam * dt)] * n
    for f, h in steps:
        f(h)


def exact(case, seed):
    """In 64 bits by plain torch: observables and molecular dynamics.  A Markov chain has no value apart
    from the random stream that its library draws, so runs, cycles, trajectories, batches and jobs have none."""
    c, kind = dict(case), case["kind"]
    if kind not in ("measure", "analyse", "integrate"):
        return None
    L = _list(c["L"])
    nd, nc, V = len(L), c["nc"], int(np.prod(L))
    flat = _links(L, nc, c["precision"], seed)
    u = _lattice(flat, L)
    if kind == "integrate":
        p = _momenta(L, nc, c["precision"], seed)
        _integrate(c, L, u, _lattice(p, L))
        return [p.cpu().numpy(), flat.cpu().numpy()]
    out = [_plaquette(u, nd, nc, V)]
    pairs, planar = _pairs(c["pairs"]), _pairs(c["planar"])
    if pairs:
        out.append(sum(_wilson(u, nd, nc, V, mu, nd - 1, pairs) for mu in range(nd - 1)) / (nd - 1))
    if planar:
        out += [_wilson(u, nd, nc, V, mu, nu, planar) for mu, nu in _pairs(c["planes"])]
    return out
