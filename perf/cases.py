"""The work this framework is timed on: calls that a simulation program makes, over the sizes it is used at.

Five kinds of case.  "density": the CIC density of device arrays.  "run": a stretch of the main loop (particles from the
host, some steps, particles back), the framework's main use.  "batch": the same for many small boxes side by side.  "solve":
one scalar-field solve of a given density.  "power": the P(k) output of a snapshot.  prepare() makes particles and densities
with torch from the seed (Zel'dovich displacements of a random field); exact() restates each path in plain FP64 torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "mg-glam-durham_b200"))
import mgglam_b200 as mg  # noqa: E402

OM, OML, OMB = 0.3089, 0.6911, 0.0486
FR, DGP, SYM, KMF, CSF = 1, 2, 3, 4, 5
PLAIN, MIXED = mg.PREC_PLAIN, mg.PREC_MIXED


def listed():
    def run(name, ngrid, nrow, steps, model=FR, precision=PLAIN, early=True, **kw):
        return dict(name=name, kind="run", ngrid=ngrid, nrow=nrow, steps=steps, model=model, n=kw.get("n", 1),
                    precision=precision, cycle=kw.get("cycle", "V"), early=early, cell=kw.get("cell", 1.0))

    def solve(name, ngrid, model, precision, cycle, cell=1.0, n=1):
        return dict(name=name, kind="solve", ngrid=ngrid, model=model, n=n, precision=precision, cycle=cycle, cell=cell)

    return [
        # a halo or lens plane tool that wants one small density: launches and latency count
        dict(name="density_64", kind="density", ngrid=64, np=29791),
        # the largest density of that entry point, a ragged particle count
        dict(name="density_256", kind="density", ngrid=256, np=2048383),
        # the small test box of the plain path, many short launches
        run("run_fr_64", 64, 31, 8),
        # the 40-step regression run's box (F5, 128^3 particles on a 256^3 mesh)
        run("run_fr_256", 256, 128, 4),
        # a Newtonian control run (scalar field off), clustered late particles, NROW not a power of two
        run("run_newton_512", 512, 250, 6, model=0, early=False),
        # the mid-size production box of the precision form
        run("run_fr_512", 512, 256, 4, precision=MIXED, early=False),
        # the headline box: F5, 512^3 particles on a 1024^3 mesh
        run("run_fr_1024", 1024, 512, 3, precision=MIXED),
        # parameter-space sampling: many 128^3 meshes side by side
        dict(name="batch_8x128", kind="batch", boxes=8, ngrid=128, nrow=64, steps=3, model=FR, n=1, precision=MIXED,
             cycle="V", early=True, cell=1.0),
        # one solve of each other solver family, different cycles and both forms
        solve("solve_dgp_512", 512, DGP, MIXED, "V", 0.5),
        solve("solve_kmf_256", 256, KMF, PLAIN, "V", 0.5),
        solve("solve_sym_256", 256, SYM, PLAIN, "W", 0.5),
        # the P(k) output of a snapshot, NROW not a power of two
        dict(name="power_512", kind="power", ngrid=512, nrow=300, precision=PLAIN, early=False, cell=1.0),
    ]


def draw(rng):
    kind = rng.choice(["density", "run", "run", "run", "batch", "solve", "solve", "power"])
    if kind == "density":
        ngrid = rng.choice([16, 32, 64, 128, 256])
        most = min(2097152, ngrid ** 3)
        return dict(kind=kind, ngrid=ngrid, np=int(math.exp(rng.uniform(math.log(most / 64), math.log(most)))))
    precision, cell = rng.choice([PLAIN, MIXED]), rng.choice([0.5, 1.0, 2.0])
    if kind == "power":
        ngrid = rng.choice([64, 128, 256, 512])
        return dict(kind=kind, ngrid=ngrid, nrow=rng.randint(ngrid // 4, 5 * ngrid // 8), precision=precision,
                    early=rng.random() < 0.5, cell=cell)
    model = rng.choice([FR, FR, DGP, SYM, KMF, CSF])
    n, cycle = (rng.choice([0, 1, 1, 2]) if model == FR else 1), rng.choice(["V", "V", "F", "W"])
    if kind == "solve":
        # F and W cycles leave the mean of the other models' fields, which their equations hardly fix, to rounding
        cycle = cycle if model in (FR, SYM) else "V"
        return dict(kind=kind, ngrid=rng.choice([32, 64, 128, 256, 512]), model=model, n=n, precision=precision,
                    cycle=cycle, cell=cell)
    c = dict(kind=kind, model=model, n=n, precision=precision, cycle=cycle, early=rng.random() < 0.5, cell=cell)
    if kind == "batch":
        c.update(boxes=rng.randint(2, 8), ngrid=rng.choice([32, 64, 128]), steps=rng.randint(1, 3), model=FR, n=1)
    else:
        c.update(ngrid=rng.choice([32, 64, 128, 256, 512]), steps=rng.randint(1, 5))
        if rng.random() < 0.2:
            c.update(model=0, n=1)
    c["nrow"] = rng.randint(c["ngrid"] // 4, c["ngrid"] // 2)
    return c


# ------------------------------------------------------------------- inputs ----
def _gaussian(n, gen, slope, cut):
    """A random field on n^3 cells as its half spectrum (amplitude ~ k^slope below `cut` of the Nyquist wavenumber), and k."""
    f = torch.fft.rfftn(torch.randn(n, n, n, generator=gen, device="cuda"))
    k = [torch.fft.fftfreq(n, 1.0 / n, device="cuda"), torch.fft.rfftfreq(n, 1.0 / n, device="cuda")]
    kz, ky, kx = k[0][:, None, None], k[0][None, :, None], k[1][None, None, :]
    k2 = kx * kx + ky * ky + kz * kz
    k2[0, 0, 0] = 1.0
    f *= k2 ** (slope / 2) * torch.exp(-k2 / (cut * n / 2) ** 2)
    f[0, 0, 0] = 0
    return f, (kx, ky, kz), k2


def _times(case):
    """AEXPN and ASTEP: the start of the 100-step schedule, or late in a run."""
    return (0.02, 0.002) if case["early"] else (0.6, 0.01)


def _particles(case, seed):
    """Positions in [1, NGRID+1) and velocities on the host (pinned): a lattice displaced by a random field, a fraction of a
    cell rms early on and several cells (crossed shells, dense knots) late."""
    nrow, ng = case["nrow"], case["ngrid"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f, ks, k2 = _gaussian(nrow, gen, -0.9, 0.7)
    a, da = _times(case)
    rms = (0.15 if case["early"] else 3.0) * ng / nrow / 2
    xconst = da / math.sqrt((a + da / 2) * (OM + OML * (a + da / 2) ** 3)) / (a + da / 2)
    out = []
    side = (torch.arange(nrow, device="cuda", dtype=torch.float32) + 0.5) * (ng / nrow)
    norm = None
    for axis, k in enumerate(ks):
        d = torch.fft.irfftn(f * (k / k2) * 1j, s=(nrow, nrow, nrow))
        norm = norm or float(rms / d.std())
        d *= norm
        shape = [(1, 1, nrow), (1, nrow, 1), (nrow, 1, 1)][axis]
        # damped towards the two faces, where a last-bit difference would put a particle on the other side of the box
        d *= (torch.minimum(side, ng - side) / (8 * rms)).clamp(max=1).reshape(shape)
        x = torch.remainder(side.reshape(shape) + d, ng) + 1
        x[x >= ng + 1] = float(np.nextafter(np.float32(ng + 1), np.float32(0)))
        out.append((x.reshape(-1), (d * (da / a / xconst)).reshape(-1)))
    host = [torch.empty(nrow ** 3, dtype=torch.float32, pin_memory=True) for _ in range(6)]
    for h, d in zip(host, [x for x, _ in out] + [v for _, v in out]):
        h.copy_(d)
    return host


def _density(case, seed):
    """A lognormal density contrast, as clustered as a late snapshot on cells of about 1 Mpc/h."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ng = case["ngrid"]
    g = torch.fft.irfftn(_gaussian(ng, gen, -0.6, 0.6)[0], s=(ng, ng, ng))
    s = 0.5 if case["n"] == 2 else 1.2
    d = torch.exp(g * (s / g.std()) - s * s / 2)
    return (d / d.mean() - 1).contiguous()


def _background():
    """Background rows (a, phi, dphi/dN, -, aH/H0, -) of the k-mouflage and coupled models, smooth in a."""
    a = np.geomspace(1e-3, 1.0026, 20000)
    h = np.sqrt(OM / a + OML * a * a)
    phi = {KMF: -1.06 * a / (1 + 0.58 * a), CSF: 2.91 * a ** 0.15}
    dphi = {KMF: -1.06 * a / (1 + 0.58 * a) ** 2, CSF: 2.91 * 0.15 * a ** 0.15}
    return {m: np.stack([a, phi[m], dphi[m], 0 * a, h, 0 * a], axis=1) for m in (KMF, CSF)}


_BG = _background()


def _config(case):
    model = case.get("model", 0)
    # three cycles a solve, as the F5 run takes early on: the exit test cannot make the work depend on rounding
    return mg.make_config(case["ngrid"], case.get("nrow", 1), case["ngrid"] * case["cell"], om=OM, oml=OML, omb=OMB,
                          mg_flag=int(model > 0), mg_model=model or FR, fr_n=case.get("n", 1), fr0=-1e-5,
                          cycle=case.get("cycle", "V"), iter_count_max=3, precision=case["precision"], kmf_beta=0.2,
                          kmf_lambda=1.475, csf_lambda=0.917)


def _box(case):
    box = mg.Box(_config(case))
    if case.get("model") in _BG:
        box.set_background(_BG[case["model"]])
    return box


def _ptr(t):
    return mg._fptr(t.numpy())


def _like(parts):
    return [torch.empty_like(p, pin_memory=True) for p in parts]


# -------------------------------------------------------------------- cases ----
def prepare(case, seed):
    kind = case["kind"]
    if kind == "density":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        # half spread evenly, half in clumps
        x = torch.rand(3, case["np"], generator=gen, device="cuda")
        m = case["np"] // 2
        centre = torch.rand(3, 16, generator=gen, device="cuda")
        pick = torch.randint(0, 16, (m,), generator=gen, device="cuda")
        x[:, :m] = torch.remainder(centre[:, pick] + 0.02 * torch.randn(3, m, generator=gen, device="cuda"), 1.0)
        ng = case["ngrid"]
        x = (x * ng + 1).clamp(max=float(np.nextafter(np.float32(ng + 1), np.float32(0)))).contiguous()
        return dict(case=case, x=x, fi=torch.empty(ng, ng, ng, device="cuda"))
    if kind == "solve":
        box = _box(case)
        d = _density(case, seed).cpu().numpy()
        box.upload_grid(mg.GRID_FI, d)
        box.set_time(0.7, 0.01)
        return dict(case=case, box=box, out=torch.empty(d.size, dtype=torch.float32, pin_memory=True))
    boxes = [_box(case) for _ in range(case.get("boxes", 1))]
    parts = [_particles(case, seed * 16 + i) for i in range(len(boxes))]
    if kind == "power":
        for b, p in zip(boxes, parts):
            b.set_time(*_times(case))
            b.upload_particles(*[t.numpy() for t in p])
    return dict(case=case, boxes=boxes, parts=parts, out=[_like(p) for p in parts])


def _named(parts, ekin):
    return dict(zip(("x", "y", "z", "vx", "vy", "vz"), parts), ekin=ekin)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "density":
        x, fi = state["x"], state["fi"]
        mg.density_noalloc(x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), case["np"], case["ngrid"], fi.data_ptr())
        return fi
    if kind == "solve":
        box = state["box"]
        box.scalar_field(1)
        box._check(box.lib.mgg_download_grid(box.h, mg.GRID_FI2, _ptr(state["out"])))
        return state["out"]
    boxes, parts, out = state["boxes"], state["parts"], state["out"]
    if kind == "power":
        return boxes[0].power(True)
    a, da = _times(case)
    for b, p in zip(boxes, parts):
        b._check(b.lib.mgg_upload_particles(b.h, *[_ptr(t) for t in p], b.np))
    states = [b.new_state(a, da) for b in boxes]
    if kind == "batch":
        for _ in range(case["steps"]):
            mg.step_batch(boxes, states)
        ekin = [s.ekin for s in states]
    else:
        _, e = boxes[0].run_steps(states[0], case["steps"])
        ekin = [e[-1]]
    for b, o in zip(boxes, out):
        b._check(b.lib.mgg_download_particles(b.h, *[_ptr(t) for t in o], b.np))
    got = [_named(o, e) for o, e in zip(out, ekin)]
    return got if kind == "batch" else got[0]


def work(case):
    """Bytes: the particles read and written once a step, the density, field and potential written once and read once where
    the next routine needs all of them.  Operations: the transforms, the solve's sweeps, the particles."""
    n3 = float(case["ngrid"]) ** 3
    if case["kind"] == "density":
        return dict(bytes=12.0 * case["np"] + 4 * n3, flops=40.0 * case["np"])
    mgc = 3 * 8 * 1.14 * 15 * n3 * {"V": 1, "F": 1.5, "W": 2}[case.get("cycle", "V")]   # cycles, sweeps, levels, operations
    if case["kind"] == "solve":
        return dict(bytes=8 * n3, flops=mgc)
    npart = float(case["nrow"]) ** 3
    fft = 2.5 * n3 * math.log2(n3)
    if case["kind"] == "power":
        return dict(bytes=12 * npart + 8 * n3, flops=fft + 40 * npart + 10 * n3)
    mgon = case["model"] > 0
    b = 60 * npart + (24 if mgon else 16) * n3
    f = 2 * fft + 300 * npart + (mgc if mgon else 0)
    k = case["steps"] * case.get("boxes", 1)
    return dict(bytes=k * b, flops=k * f)


def tolerance(case):
    """About four times what the path's two forms show against each other and against exact(): FP32 grids and particles; the
    velocities of an early run are differences of a nearly uniform potential."""
    if case["kind"] == "density":
        return dict(rel=3e-7, max=1e-6)
    if case["kind"] == "power":
        return dict(rel=4e-6, max=2e-5)
    if case["kind"] == "solve":
        return dict(rel=8e-6, max=2e-5)
    return dict(rel=2e-5, max=2e-4)


# -------------------------------------------------------------------- exact ----
def exact(case, seed):
    kind = case["kind"]
    if case["ngrid"] >= 1024:
        return None   # over 20 s, and the FP64 grids are 8.6 GB each
    if kind == "density":
        return _cic(prepare(case, seed)["x"].double(), case["ngrid"])
    if kind == "solve":
        s = _Solver(case, 0.7)
        u = s.solve(_density(case, seed).double(), s.background()).reshape(-1)
        return u / s.ubg if case["model"] == FR else u   # f(R): handed out relative to the background
    got = []
    for i in range(case.get("boxes", 1)):
        p = [t.cuda().double() for t in _particles(case, seed * 16 + i)]
        got.append(_power(case, p) if kind == "power" else _steps(case, p))
    return got if kind == "batch" else got[0]


def _nodes(x, n):
    """The eight CIC nodes (flat index, weight) of positions in [1, n+1)."""
    i = [t.long() for t in x]
    d = [t - k for t, k in zip(x, i)]
    for m in range(8):
        w, q = 1.0, 0
        for axis, bit in ((2, m >> 2), (1, m >> 1 & 1), (0, m & 1)):
            w = w * (d[axis] if bit else 1 - d[axis])
            q = q * n + torch.remainder(i[axis] - 1 + bit, n)
        yield q, w


def _chunks(npart, size=1 << 24):
    return [slice(k, min(k + size, npart)) for k in range(0, npart, size)]


def _cic(x, n):
    npart = x[0].numel()
    rho = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    for c in _chunks(npart):
        for q, w in _nodes([t[c] for t in x], n):
            rho.index_add_(0, q, w)
    return (rho * (n ** 3 / npart) - 1).reshape(n, n, n)


def _poisson(d, a):
    n = d.shape[0]
    g = 2 * torch.cos(2 * math.pi * torch.arange(n, dtype=torch.float64, device="cuda") / n)
    lam = g[:, None, None] + g[None, :, None] + g[None, None, : n // 2 + 1] - 6
    lam[0, 0, 0] = 1.0
    return torch.fft.irfftn(torch.fft.rfftn(d) / lam, s=(n, n, n)) * (1.5 * OM / a)


def _power(case, p):
    n = case["ngrid"]
    f = torch.fft.rfftn(_cic(p[:3], n)) / n ** 3
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    kx = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
    r = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kx ** 2)
    w = torch.full_like(kx, 2.0)
    w[0] = w[-1] = 1.0
    w = w.expand_as(r).reshape(-1).clone()
    w[0] = 0
    b = (r + 0.5).long().clamp(min=1).reshape(-1)
    bins = [torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, b, v)[1 : n // 2 + 1]
            for v in (w, w * r.reshape(-1), w * f.abs().square().reshape(-1))]
    box = n * case["cell"]
    return dict(k=bins[1] / bins[0] * (2 * math.pi / box), nmodes=bins[0], pk=bins[2] / bins[0] * box ** 3,
                klog=None, nmodeslog=None, pklog=None)


def _bg(model, a, value, column):
    """The background table between the first row past a and the one before it."""
    t = _BG[model]
    i = max(1, int(np.searchsorted(t[:, 0], a)))
    return t[i - 1, column] + (t[i, column] - t[i - 1, column]) / (t[i, 0] - t[i - 1, 0]) * (value - t[i - 1, 0])


def _steps(case, p):
    """The main loop in FP64."""
    n, model = case["ngrid"], case["model"]
    a, da = _times(case)
    factor, u = da / a, None
    wpar = n ** 3 / p[0].numel()
    for step in range(case["steps"]):
        phi = _cic(p[:3], n)
        s = _Solver(case, a) if model else None
        if s:
            if u is None:
                u = s.background()
            elif model == SYM and a >= s.astar:
                u = s.background()
            elif model == FR:
                u = u * s.ubg
            if model != SYM or a >= s.astar:
                u = s.solve(phi, u)
            if model == FR:
                u = u / s.ubg   # kept relative to the background between steps
        phi = _poisson(phi, a)
        factv = 1.0
        if da < factor / 1.25 * a and a < 0.3:
            da, factv = 1.5 * da, 1.2
        if s:
            phi = phi + s.fifth(u)
        ah = a + da / 2
        pc = -math.sqrt(a / (OM + OML * a ** 3)) * da * 0.5 / factv
        xc = da / math.sqrt(ah * (OM + OML * ah ** 3)) / ah
        boost, fric = 1.0, 0.0
        if model in _BG:
            beta = s.beta
            pc = -da * 0.5 / factv / _bg(model, a, a, 4)
            xc = da / (ah * ah * _bg(model, ah, ah, 4))
            boost = math.exp(beta * _bg(model, ah, a, 1))
            fric = -beta * _bg(model, a, a, 2) / a
        elif model == SYM and a > s.astar:
            fric = -9 * OM * s.xi ** 2 * math.sqrt(1 - (s.astar / a) ** 3)
        ekin = 0.0
        grad = [(torch.roll(phi, -1, ax) - torch.roll(phi, 1, ax)).reshape(-1) for ax in (2, 1, 0)]
        for c in _chunks(p[0].numel()):
            x, acc = [t[c] for t in p[:3]], [0.0, 0.0, 0.0]
            cell = ((x[2].long() - 1) * n + x[1].long() - 1) * n + x[0].long() - 1
            for q, w in _nodes(x, n):
                acc = [t + w * g[q] for t, g in zip(acc, grad)]
            for k in range(3):
                v = p[3 + k][c]
                f = fric * u.reshape(-1)[cell] if model == SYM and fric else fric
                v = v + f * v * (da / factv) + boost * pc * acc[k]
                p[3 + k][c] = v
                p[k][c] = torch.remainder(x[k] + v * xc - 1, n) + 1
                ekin += float(v.square().sum()) * wpar
        a = a + da
        ekin = ekin / 2 / ah ** 2
    return _named(p, torch.tensor(ekin, dtype=torch.float64))


def _sum6(u):
    return sum(torch.roll(u, s, ax) for ax in range(3) for s in (-1, 1))


def _halve(f):
    n = f.shape[0] // 2
    return f.reshape(n, 2, n, 2, n, 2).mean((1, 3, 5))


def _double(c):
    for ax in range(3):
        lo, hi = 0.75 * c + 0.25 * torch.roll(c, 1, ax), 0.75 * c + 0.25 * torch.roll(c, -1, ax)
        c = torch.stack([lo, hi], ax + 1).flatten(ax, ax + 1)
    return c


def _cubic(P, Q):
    """The largest real root of u^3 + P u + Q, in closed form and refined."""
    d0, d1 = -3 * P, 27 * Q
    cc = d1 * d1 - 4 * d0 ** 3
    t = 0.5 * (d1 + torch.where(d1 >= 0, 1.0, -1.0) * cc.clamp(min=0).sqrt())
    c = torch.sign(t) * t.abs() ** (1 / 3)
    one = -(c + d0 / c) / 3
    sq = d0.clamp(min=0).sqrt()
    three = -(2 / 3) * sq * torch.cos(torch.acos((0.5 * d1 / sq ** 3).clamp(-1, 1)) / 3 + 2 * math.pi / 3)
    u = torch.where(cc >= 0, one, three)
    for _ in range(2):
        u = u - ((u * u + P) * u + Q) / (3 * u * u + P)
    return u


class _Solver:
    """The FAS multigrid solve (two red-black sweeps around each coarse correction) in FP64, every cell of a colour from the
    field before that colour's sweep."""

    def __init__(self, case, a):
        self.model, self.n, self.cycle, self.a = case["model"], case["n"], case["cycle"], a
        self.c = 2997.92458 * case["ngrid"] / (case["ngrid"] * case["cell"])
        self.lmax = int(math.log2(case["ngrid"]))
        self.beta = 0.2 if self.model == KMF else -0.2
        if self.model == FR:
            self.rbg = 3 * (OM / a ** 3 + 4 * OML)
            self.fbg = -1e-5 * (3 * (OM + 4 * OML) / self.rbg) ** (self.n + 1)
            self.ubg = abs(self.fbg) ** (1 / (self.n + 1))
        if self.model == DGP:
            orc = 0.25
            b = 1 + (0.5 * OM / a ** 3 + OML) / math.sqrt(orc * (OM / a ** 3 + OML))
            self.alpha = 3 * b * a * a * 4 * orc
            self.dcoef = self.alpha * OM / b / a
        if self.model == SYM:
            self.astar, self.xi = 0.5, 1 / 2997.92458
            self.thick, self.mass = (self.astar / a) ** 3, 0.5 * (a / (self.c * self.xi)) ** 2
        if self.model in _BG:
            self.phibar, self.dphi, self.hub = (_bg(self.model, a, a, k) for k in (1, 2, 4))
        if self.model == KMF:
            self.k3 = 3 * (0.5 / (a * 1.475) ** 2) ** 2
            self.dot2 = (self.dphi * self.hub) ** 2
            self.src = 3 * self.beta * OM / a * math.exp(self.beta * self.phibar)
        if self.model == CSF:
            self.src, self.al = 3 * OM / a, 0.1
            self.vamp = -self.al * 0.917 ** 2 * a * a

    def background(self):
        v = 0.0
        if self.model == FR:
            v = self.ubg
        elif self.model == SYM and self.a > self.astar:
            v = math.sqrt(1 - self.thick)
        return torch.full((1 << self.lmax,) * 3, v, dtype=torch.float64, device="cuda")

    def fifth(self, u):
        if self.model == FR:
            return -(self.c ** 2) * 0.5 * self.fbg * u ** (self.n + 1)
        if self.model == SYM:
            return 3 * self.xi ** 2 * OM * self.c ** 2 / self.astar ** 3 * u * u
        return u * {DGP: 0.5, KMF: self.beta * self.c, CSF: self.beta}[self.model]

    def _phi(self, u):
        p = self.phibar + u / self.c ** 2
        return p, self.beta * torch.exp(self.beta * p), self.vamp / p ** (1 + self.al)

    def _second(self, u):
        """First and second differences of the 19-point stencil."""
        up, lo = [torch.roll(u, -1, ax) for ax in (2, 1, 0)], [torch.roll(u, 1, ax) for ax in (2, 1, 0)]
        first = [p - m for p, m in zip(up, lo)]
        pair = [p + m for p, m in zip(up, lo)]
        cross = [torch.roll(first[i], -1, ax) - torch.roll(first[i], 1, ax) for i, ax in ((0, 1), (0, 0), (1, 0))]
        return first, pair, cross

    def _kmf(self, u, d, h2):
        f, s, x = self._second(u)
        t = (f[0] ** 2 + f[1] ** 2 + f[2] ** 2) / (4 * h2)
        lap = s[0] + s[1] + s[2]
        e = sum(f[i] ** 2 * (3 * s[i] - lap) for i in range(3)) / 12
        e = (e + (x[0] * f[0] * f[1] + x[1] * f[0] * f[2] + x[2] * f[1] * f[2]) / 8) / h2 ** 2
        sig1 = 1 + self.k3 * (7 / 3) * t * t + self.k3 * self.dot2 ** 2
        return lap, (self.src * d - self.k3 * 4 * self.c * t * e) / sig1

    def operator(self, u, d, h2):
        """The equation's left side at every cell; the spacing squared h2."""
        if self.model == FR:
            w = u ** (self.n + 1)
            return (_sum6(w) - 6 * w) * (self.c ** 2 * math.copysign(1, self.fbg) / h2) + OM / self.a * d - \
                self.rbg * self.a ** 2 / 3 * (self.ubg / u - 1)
        if self.model == KMF:
            lap, src = self._kmf(u, d, h2)
            return (lap - 6 * u) / h2 * self.c - src
        if self.model == DGP:
            _, s, x = self._second(u)
            s = [t - 2 * u for t in s]
            sig = (s[0] ** 2 + s[1] ** 2 + s[2] ** 2 - s[0] * s[1] - s[0] * s[2] - s[1] * s[2]) * (2 / 3 / h2 ** 2)
            sig = sig + (x[0] ** 2 + x[1] ** 2 + x[2] ** 2) * (0.125 / h2 ** 2) + self.dcoef * d
            root = torch.sqrt(self.alpha ** 2 + 8 / 3 * sig)
            return (s[0] + s[1] + s[2]) / h2 - 0.75 * (root - self.alpha)
        lap = (_sum6(u) - 6 * u) / h2
        if self.model == SYM:
            return lap - self.mass * ((self.thick * (d + 1) - 1) * u + u ** 3)
        p, A, V = self._phi(u)
        _, A0, V0 = self._phi(torch.zeros((), dtype=torch.float64, device="cuda"))
        return lap - self.src * (A * (d + 1) - A0) - (V - V0)

    def update(self, u, d, tau, h2):
        """The new value of every cell from its neighbours."""
        if self.model == FR:
            f2 = h2 / (self.c ** 2 * math.copysign(1, self.fbg)) / 6
            q2 = self.rbg * self.a ** 2 * f2 / 3
            P, Q = -OM / self.a * f2 * d - q2 + f2 * tau - _sum6(u ** (self.n + 1)) / 6, q2 * self.ubg
            if self.n == 0:
                r = torch.sqrt(P * P - 4 * Q)
                return torch.where(P <= 0, 0.5 * (r - P), -2 * Q / (P + r))
            if self.n == 1:
                return _cubic(P, torch.full_like(P, Q))
            v = (-P).clamp(min=0) ** (1 / 3) + (-Q) ** 0.25   # right of the quartic's positive root
            for _ in range(12):
                v = v - (v * (v ** 3 + P) + Q) / (4 * v ** 3 + P)
            return v
        if self.model == SYM:
            f4 = 2 * (self.c * self.xi / self.a) ** 2
            P = self.thick * (d + 1) - 1 + 6 * f4 / h2
            return _cubic(P, f4 * tau - f4 / h2 * _sum6(u))
        if self.model == KMF:
            lap, src = self._kmf(u, d, h2)
            return (lap - (tau + src) * (h2 / self.c)) / 6
        L = self.operator(u, d, h2) - tau
        if self.model == DGP:
            return u + L * (h2 / 6)
        p, A, V = self._phi(u)
        slope = -6 / h2 - self.src * (d + 1) * self.beta * A / self.c ** 2 + (1 + self.al) * V / self.c ** 2 / p
        return u - L / slope

    def _smooth(self, u, d, tau, h2):
        i = torch.arange(u.shape[0], device="cuda")
        colour = (i[:, None, None] + i[None, :, None] + i) % 2
        for _ in range(2):
            for c in (0, 1):
                u = torch.where(colour == c, self.update(u, d, tau, h2), u)
        return u

    def _cycle(self, level, u, d, tau, kind):
        h2 = 4.0 ** level
        u = self._smooth(u, d, tau, h2)
        if self.lmax - level <= 1:
            return u
        for turn in range(1 if kind == "V" else 2):
            ru, dc = _halve(u), _halve(d)
            rr = _halve(self.operator(u, d, h2) - tau)
            tc = self.operator(ru, dc, 4 * h2) - rr
            uc = self._cycle(level + 1, ru, dc, tc, "V" if kind == "F" and turn else kind)
            t = u + _double(uc - ru)
            if self.model in (FR, SYM):
                t = torch.where(t > 0, t, u)
            elif self.model == CSF:
                t = torch.where(self.phibar + t / self.c ** 2 > 0, t, u)
            u = self._smooth(t, d, tau, h2)
        return u

    def solve(self, d, u, cycles=3):
        tau = torch.zeros((), dtype=torch.float64, device="cuda")
        for _ in range(cycles):
            u = self._cycle(0, u, d, tau, self.cycle)
            if float(self.operator(u, d, 1.0).square().mean()) <= 1e-16:
                break
        return u
