"""The work that users of this library have it do, as measurable cases.

Every case is one call pattern of a user's program on inputs made from a seed:
a shot (the time loop over all steps, its reports, traces and snapshot planes),
the reference's own loop of routine calls, a 2D run, an ensemble of uneven 2D
models, a reciprocity batch over one medium, and a misfit gradient.  Grids,
layers, absorbers and recorders are those of the tests and of bench.py, or
generic.  ``exact`` restates the scheme in 64 bits with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

# depth(top) rho vp vs qp qs of the four-layer model of the tests and benchmarks
LAYERS = [(0.0, 2.7, 5.5, 3.2, 300.0, 150.0), (5.0, 2.8, 6.0, 3.5, 500.0, 250.0),
          (18.0, 2.9, 6.7, 3.9, 600.0, 300.0), (30.0, 3.3, 7.8, 4.5, 1000.0, 500.0)]
FQ_MIN, FQ_MAX, FQ_REF = 0.05, 2.0, 1.0
AIR = 3            # cells of air above the free surface
MO = 1e16
UC = 1e-15
EPS = 1.1920929e-07
DEVICE = "cuda"


def listed():
    shot = dict(kind="shot3d", dx=0.5, nm=3, random=False, precision="f32", nsrc=1, calls=False, planes=False)
    return [
        # a test-sized shot: launches, reports and small transfers
        dict(shot, name="shot3d_small", nx=40, ny=36, nz=32, na=8, nt=60, nst=6, report=10),
        # the plain forward configuration (192 x 192 x 96, absorber 20), with two snapshot planes
        dict(shot, name="shot3d_plain", nx=192, ny=192, nz=96, na=20, nt=200, nst=16, report=50, planes=True),
        # a Fortran driver's loop: one call per routine of the time step, odd sizes
        dict(shot, name="calls3d_odd", nx=101, ny=87, nz=61, na=10, nt=40, nst=9, report=10, calls=True),
        # the large heterogeneous run: random medium, eight sources, many stations
        dict(shot, name="shot3d_large", nx=512, ny=512, nz=256, na=32, nt=20, nst=256, report=10, dx=0.2, nsrc=8,
             random=True, planes=True),
        # memory variables stored in BF16
        dict(shot, name="shot3d_bf16", nx=384, ny=384, nz=192, na=32, nt=20, nst=64, report=10, dx=0.2, nsrc=8,
             random=True, planes=True, precision="bf16r"),
        # single 2D runs: the smallest member of an ensemble, odd sizes, and the largest
        dict(kind="psv", name="psv_small", nx=256, nz=128, na=20, nt=300, dx=0.1, nm=3, nst=16),
        dict(kind="sh", name="sh_odd", nx=517, nz=259, na=20, nt=200, dx=0.1, nm=3, nst=16),
        dict(kind="psv", name="psv_large", nx=2048, nz=1024, na=20, nt=60, dx=0.1, nm=3, nst=16),
        # an ensemble of uneven 2D models in one launch per half step
        dict(kind="ensemble", name="ensemble_psv", n=24, nx0=256, nx1=1024, nz0=128, nz1=512, na=20, nt=60, dx=0.1,
             nm=3, nst=16),
        # reciprocity: single forces at the stations over one shared medium
        dict(kind="forces", name="forces_batch", n=9, nx=144, ny=160, nz=80, na=16, nt=30, dx=0.5, nm=3, nst=6),
        # misfit gradients for vp, vs, rho: a test-sized one, and the benchmark's grid
        dict(kind="gradient", name="gradient_small", nx=64, ny=60, nz=48, na=8, nt=100, dx=0.5, nm=3, nst=16, ckpt=25),
        dict(kind="gradient", name="gradient_large", nx=256, ny=256, nz=128, na=20, nt=60, dx=0.25, nm=3, nst=64,
             ckpt=20),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["shot3d", "shot3d", "psv", "sh", "ensemble", "forces", "gradient"])
    if kind == "shot3d":
        nx, ny, nz = size(40, 448), size(36, 448), size(32, 224)
        na = rng.randint(6, min(32, (min(nx, ny) - 12) // 2, nz // 3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, na=na, nt=rng.randint(15, 60), nst=rng.randint(4, 200), report=10,
                    dx=rng.choice([0.2, 0.5]), nm=rng.choice([3, 3, 3, 2, 1, 0]), random=rng.random() < 0.5,
                    precision=rng.choice(["f32", "f32", "f32", "bf16r", "f16r"]), nsrc=rng.randint(1, 8),
                    calls=rng.random() < 0.25, planes=rng.random() < 0.5)
    if kind in ("psv", "sh"):
        return dict(kind=kind, nx=size(128, 2048), nz=size(64, 1024), na=rng.randint(8, 20), nt=rng.randint(50, 200),
                    dx=0.1, nm=rng.choice([3, 3, 2, 1, 0]), nst=rng.randint(4, 32))
    if kind == "ensemble":
        nx0, nz0 = size(128, 512), size(64, 256)
        return dict(kind=kind, n=rng.randint(4, 32), nx0=nx0, nx1=size(nx0 + 1, 1100), nz0=nz0, nz1=size(nz0 + 1, 560),
                    na=rng.randint(8, 20), nt=rng.randint(30, 60), dx=0.1, nm=3, nst=rng.randint(4, 16))
    if kind == "forces":
        return dict(kind=kind, n=rng.randint(3, 12), nx=size(56, 160), ny=size(56, 160), nz=size(40, 96),
                    na=rng.randint(6, 12), nt=rng.randint(15, 40), dx=0.5, nm=3, nst=rng.randint(3, 8))
    return dict(kind=kind, nx=size(48, 200), ny=size(48, 200), nz=size(40, 112), na=rng.randint(6, 12),
                nt=rng.randint(60, 90), dx=rng.choice([0.25, 0.5]), nm=3, nst=rng.randint(4, 48),
                ckpt=rng.randint(10, 40))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dt(c):
    return 0.04 * c["dx"]


def _beg(n, dx):
    return -(n // 2) * dx


def _centre(i, beg, dx):
    """Coordinate of the centre of cell i."""
    return beg + (i - 0.5) * dx


def _random(c, seed):
    """The random part of a 3D or 2D case: source and station cells, moments,
    rise times (cells away from the absorber and the recorder's edges)."""
    g = np.random.default_rng([seed, 17])
    na, ny = c["na"], c.get("ny", 1)
    cells = lambda n, nmax: [int(v) for v in g.integers(na + 4, nmax - na - 2, n)]
    nsrc = c.get("nsrc", 1)
    kmax = c["nz"] - na - 2
    src = dict(i=cells(nsrc, c["nx"]), j=cells(nsrc, ny) if ny > 1 else [1] * nsrc,
               k=[int(v) for v in g.integers(AIR + 5, max(kmax, AIR + 6), nsrc)],
               m=g.uniform(-1.0, 1.0, (nsrc, 6)), trise=[float(v) for v in g.uniform(8.0, 20.0, nsrc) * c["dx"] / 4.0])
    st = dict(i=cells(c["nst"], c["nx"]), j=cells(c["nst"], ny) if ny > 1 else [1] * c["nst"])
    if c["kind"] == "gradient":
        # a shallow source over the anomaly in the middle, stations within reach of its waves
        at = lambda n, r, num: [int(v) for v in n // 2 + g.integers(-r, r + 1, num)]
        src.update(i=at(c["nx"], 3, nsrc), j=at(ny, 3, nsrc), k=[int(v) for v in g.integers(AIR + 4, AIR + 9, nsrc)])
        st = dict(i=at(c["nx"], 8, c["nst"]), j=at(ny, 8, c["nst"]))
    return src, st


def _params(c, src, st, **kw):
    from openswpc_b200.params import Layer, Params, Source, Station

    dx, nx, ny, nz = c["dx"], c["nx"], c.get("ny", 1), c["nz"]
    xb, yb, zb = _beg(nx, dx), _beg(ny, dx) if ny > 1 else 0.0, -AIR * dx
    y = lambda j: _centre(j, yb, dx) if ny > 1 else 0.0
    sources = [Source(_centre(i, xb, dx), y(j), _centre(k, zb, dx), 0.0, tr, mo=MO, mxx=m[0], myy=m[1], mzz=m[2],
                      myz=m[3], mxz=m[4], mxy=m[5])
               for i, j, k, m, tr in zip(src["i"], src["j"], src["k"], src["m"].tolist(), src["trise"])]
    stations = [Station(_centre(i, xb, dx), y(j), 0.5 * dx, f"s{n}", "fsb")
                for n, (i, j) in enumerate(zip(st["i"], st["j"]))]
    return Params(nx=nx, ny=ny, nz=nz, nt=c["nt"], dx=dx, dy=dx, dz=dx, dt=_dt(c), na=c["na"], nm=c["nm"], xbeg=xb,
                  ybeg=yb, zbeg=zb, fq_min=FQ_MIN, fq_max=FQ_MAX, fq_ref=FQ_REF,
                  layers=[Layer(*row) for row in LAYERS], sources=sources, stations=stations, ntdec_w=1,
                  **{"ntdec_r": c.get("report", 10), **kw})


def _field(gen, shape, amp, coarse=5):
    """A smooth seeded field (wavelengths of several cells) on the GPU."""
    small = [max(2, -(-s // coarse) + 1) for s in shape]
    x = torch.randn(1, 1, *small, generator=gen, device=DEVICE)
    return amp * F.interpolate(x, size=tuple(shape), mode="trilinear" if len(shape) == 3 else "bilinear",
                               align_corners=True)[0, 0]


def _wavefield(c, seed, n, amp=1e-3):
    """Initial velocities over the memory box: a wavefield that already fills
    the grid, zero in the ghost cells and the air."""
    gen = torch.Generator(DEVICE).manual_seed(seed * 7 + 3)
    inner = (c["ny"], c["nx"], c["nz"]) if c.get("ny", 1) > 1 else (c["nx"], c["nz"])
    out = []
    for _ in range(n):
        v = _field(gen, inner, amp)
        v[..., :AIR] = 0.0
        out.append(F.pad(v, (3, 3) * len(inner)))
    return out


def _xi(c, seed):
    """The random medium of a heterogeneous run: 5 % perturbations over the memory box."""
    if not c.get("random"):
        return None
    gen = torch.Generator(DEVICE).manual_seed(seed * 7 + 5)
    shape = (c["ny"] + 6, c["nx"] + 6, c["nz"] + 6)
    return (_field(gen, shape, 0.03, 12) + _field(gen, shape, 0.02, 4)).clamp_(-0.12, 0.12).contiguous()


def _member_cases(c, seed):
    g = np.random.default_rng([seed, 29])
    return [dict(c, kind="psv", nx=int(g.integers(c["nx0"], c["nx1"] + 1)), nz=int(g.integers(c["nz0"], c["nz1"] + 1)))
            for _ in range(c["n"])]


def _forces(c, seed):
    """(station index, component) of each member of a reciprocity batch."""
    return [((m // 3) % c["nst"], "xyz"[m % 3]) for m in range(c["n"])]


def _prepare2d(c, seed):
    from openswpc_b200.swpc2d import Swpc2D

    src, st = _random(c, seed)
    run_ = Swpc2D(_params(c, src, st, sw_wav_u=True), c["kind"])
    for f, v in zip([n for n in run_.field_ids if n[0] == "V"], _wavefield(c, seed, 2 if c["kind"] == "psv" else 1)):
        run_.upload(run_.field_ids[f], v.cpu().numpy())
    return run_


def prepare(case, seed):
    c = case
    if c["kind"] in ("psv", "sh"):
        return dict(case=c, run=_prepare2d(c, seed))
    if c["kind"] == "ensemble":
        from openswpc_b200.swpc2d import Batch2D

        runs = [_prepare2d(m, seed * 64 + n) for n, m in enumerate(_member_cases(c, seed))]
        return dict(case=c, runs=runs, batch=Batch2D(runs))
    from openswpc_b200.swpc3d import ForceBatch3D, Swpc3D

    src, st = _random(c, seed)
    if c["kind"] == "forces":
        p = _params(c, dict(src, i=[]), st, green_mode=True, green_trise=3.0 * c["dx"])
        base = Swpc3D(p, medium_on_device=True)
        base.record()
        return dict(case=c, base=base, batch=ForceBatch3D(base, [(p.stations[s], q) for s, q in _forces(c, seed)]))
    if c["kind"] == "gradient":
        from openswpc_b200.adjoint import Misfit3D
        from openswpc_b200.swpc3d import lhm_model

        p = _params(c, src, st)
        vp, vs, rho, qp, qs = lhm_model(p)
        prob = Misfit3D(p, vp, vs, rho, qp, qs, np.zeros((c["nst"], 3, c["nt"]), np.float32), ckpt=c["ckpt"],
                        slot_memory="auto")
        model = [torch.from_numpy(a).to(DEVICE) for a in (vp, vs, rho)]
        true = model[1] * (1.0 + _anomaly(c))
        prob.misfit(model[0], true, model[2])
        prob.obs = prob.solver.waveforms()
        # the model of the iteration: the layers with small perturbations everywhere
        gen = torch.Generator(DEVICE).manual_seed(seed * 7 + 9)
        model = [(m * (1.0 + _field(gen, m.shape, 0.01))).requires_grad_(True) for m in model]
        return dict(case=c, problem=prob, model=model)
    planes = dict(snaps={"fs_v", "xz_v"}, ntdec_s=10, y0_xz=_centre(c["ny"] // 2, _beg(c["ny"], c["dx"]), c["dx"])) \
        if c["planes"] else {}
    run_ = Swpc3D(_params(c, src, st, **planes), xi=_xi(c, seed), medium_on_device=True, precision=c["precision"])
    for n, v in enumerate(_wavefield(c, seed, 3)):
        run_.upload(n, v.cpu().numpy())
    return dict(case=c, run=run_)


def _anomaly(c):
    """The shear-velocity anomaly of the true model: a Gaussian blob in the middle, near the surface."""
    ax = [torch.arange(n + 6, device=DEVICE, dtype=torch.float32) for n in (c["ny"], c["nx"], c["nz"])]
    mid = (c["ny"] / 2, c["nx"] / 2, AIR + 10)
    r2 = sum(((a - m).view([-1 if q == d else 1 for q in range(3)]) / (0.15 * (n + 6))) ** 2
             for d, (a, m, n) in enumerate(zip(ax, mid, (c["ny"], c["nx"], c["nz"]))))
    return 0.08 * torch.exp(-r2)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    from openswpc_b200 import _lib

    c = state["case"]
    if c["kind"] in ("psv", "sh"):
        r = state["run"]
        r.run(1, c["nt"])
        return {"v": r.waveforms(_lib.WAV_V), "u": r.waveforms(_lib.WAV_U), "vmax": r.kernel__vmax(),
                "fields": [r.download(i) for n, i in r.field_ids.items() if n[0] == "V"]}
    if c["kind"] == "ensemble":
        state["batch"].run(1, c["nt"])
        return [r.waveforms(_lib.WAV_V) for r in state["runs"]]
    if c["kind"] == "forces":
        b = state["batch"]
        b.run(1, c["nt"])
        return [b.waveforms(m) for m in range(c["n"])]
    if c["kind"] == "gradient":
        from openswpc_b200.adjoint import waveform_misfit

        for m in state["model"]:
            m.grad = None
        J = waveform_misfit(*state["model"], state["problem"])
        J.backward()
        return {"misfit": J.detach(), "grad": [m.grad for m in state["model"]]}
    r = state["run"]
    if c["calls"]:
        # the loop of a driver that calls the time step's routines itself
        reports = []
        for it in range(1, c["nt"] + 1):
            if it % c["report"] == 0:
                reports.append((it, r.kernel__vmax() * np.float32(r.UC) * np.float32(r.M0)))
            r.wav__store(it)
            if c["planes"]:
                r.snap__write(it)
            r.kernel__update_stress()
            r.absorb__update_stress()
            r.source__stressglut(it)
            r.global__comm_stress()
            r.kernel__update_vel()
            r.absorb__update_vel()
            r.global__comm_vel()
    else:
        reports = r.run(1, c["nt"])
    out = {"v": r.waveforms(_lib.WAV_V), "vmax": np.array([v for _, v in reports])}
    if c["planes"]:
        out["fs"] = r.snapshots("fs_v")
        out["xz"] = r.snapshots("xz_v")
    if c["nx"] * c["ny"] * c["nz"] <= 1 << 20:
        out["fields"] = [r.download(_lib.F_VX + q) for q in range(3)]
    return out


def work(case):
    """Bytes that cross HBM and operations of one pass: per step the state read
    and written once (V, S and memory variables in the interior; V, S and the
    absorber's auxiliaries elsewhere) and the medium read once."""
    c = case
    nm = c["nm"]
    if c["kind"] in ("psv", "sh", "ensemble"):
        nv, ns, naux, nmed, fl = (1, 2, 4, 3, 40) if c["kind"] == "sh" else (2, 3, 8, 5, 110)
        dims = [(c["nx"], c["nz"])] if c["kind"] != "ensemble" else \
            [((c["nx0"] + c["nx1"]) // 2, (c["nz0"] + c["nz1"]) // 2)] * c["n"]
        by = flops = 0
        for nx, nz in dims:
            inner = (nx - 2 * c["na"]) * (nz - c["na"])
            edge = nx * nz - inner
            by += 4 * (inner * (2 * (nv + ns * (1 + nm)) + nmed) + edge * (2 * (nv + ns + naux) + nmed - 1))
            flops += fl * nx * nz
        return {"bytes": by * c["nt"], "flops": flops * c["nt"]}
    inner = (c["nx"] - 2 * c["na"]) * (c["ny"] - 2 * c["na"]) * (c["nz"] - c["na"])
    edge = c["nx"] * c["ny"] * c["nz"] - inner
    rb = 2 if c.get("precision", "f32") != "f32" else 4
    members = c["n"] if c["kind"] == "forces" else 1
    by = members * (inner * (72 + 12 * nm * rb) + edge * 216) + inner * 40 + edge * 32
    flops = members * (inner + edge) * 280
    if c["kind"] == "gradient":
        # the adjoint step reads and writes as much, keeps and reads the forward V and divergences, and adds eight sums
        by, flops = 2 * by + inner * (48 + 64), 2.4 * flops
    return {"bytes": by * c["nt"], "flops": flops * c["nt"]}


# ---------------------------------------------------------------------------
# the scheme in 64 bits
# ---------------------------------------------------------------------------
def _relaxation(nm):
    """Relaxation times and zeta of the constant-Q fit over FQ_MIN..FQ_MAX."""
    oa, ob = 2 * math.pi * FQ_MIN, 2 * math.pi * FQ_MAX
    if nm == 0:
        return [], 0.0
    ts = [1 / math.sqrt(oa * ob)] if nm == 1 else [1 / (oa * (ob / oa) ** (m / (nm - 1))) for m in range(nm)]
    i0 = sum((math.log(1 + (ob * t) ** 2) - math.log(1 + (oa * t) ** 2)) / (2 * t) for t in ts)
    p = lambda w, t: math.atan(w * t) - w * t / (1 + (w * t) ** 2)
    i1 = sum((p(ob, t) - p(oa, t)) / (2 * t) for t in ts)
    i2 = 0.0
    for m in range(nm):
        for q in range(m + 1, nm):
            a, b = ts[m], ts[q]
            i2 += a * b / (b * b - a * a) * (math.atan(ob * a) / a - math.atan(ob * b) / b - math.atan(oa * a) / a
                                             + math.atan(oa * b) / b)
    return ts, i0 / (i1 + 2 * i2)


def _profile(x, n, beg, dx, na, fcut, dt):
    """ADE-CFS coefficients of one axis at coordinates x."""
    h, end = na * dx, beg + n * dx
    r0 = 10.0 ** (-(math.log10(na) - 1) / math.log10(2.0) - 3.0)
    d0 = -(1 / (2 * h)) * 2 * 6.0 * math.log(r0)
    a0 = math.pi * fcut
    r = torch.where(x <= beg + h, beg + h - x, torch.where(x >= end - h, x - (end - h), torch.zeros_like(x))).abs() / h
    d, a, b = d0 * r, a0 * (1 - r), 1 + 6.0 * r * r
    den = 1 + dt / 2 * (a + d / b)
    return ((1 + dt / 2 * a) / b / den, -1 / b / den, (1 - dt / 2 * (a + d / b)) / den, d / b / den)


class _Scheme:
    """The staggered-grid step in float64 on arrays (j, i, k) or (i, k) over
    the memory box; the last axis is z, the one before it x, the first y."""

    def __init__(self, c, fcut, model=None, xi=None):
        self.c, self.dt, self.nm = c, _dt(c), c["nm"]
        dx, na = c["dx"], c["na"]
        self.n = dict(x=c["nx"], z=c["nz"], **({"y": c["ny"]} if c.get("ny", 1) > 1 else {}))
        self.axes = [a for a in "yxz" if a in self.n]
        self.dim = {a: d for d, a in enumerate(self.axes)}
        f64 = dict(dtype=torch.float64, device=DEVICE)
        shape = [self.n[a] + 6 for a in self.axes]
        view = lambda v, a: v.view([-1 if q == a else 1 for q in self.axes])
        idx = {a: torch.arange(-2, self.n[a] + 4, device=DEVICE) for a in self.axes}
        zc = (idx["z"].double() - 0.5) * dx - AIR * dx
        # the layered model, perturbed by xi
        rho, vp, vs, qp, qs = (torch.zeros(shape, **f64) for _ in range(5))
        for top, *row in LAYERS:
            below = (zc >= top).expand(shape)
            for dst, v in zip((rho, vp, vs, qp, qs), row):
                dst[below] = v
        air = (zc < 0).expand(shape)
        if xi is not None:
            x = xi.double()
            rho, vp, vs = rho * (1 + 0.8 * x), vp * (1 + x), vs * (1 + x)
        if model is not None:
            vp, vs, rho = model
        else:
            rho, vp, vs = rho.masked_fill(air, 0.001), vp.masked_fill(air, 0.0), vs.masked_fill(air, 0.0)
        qp, qs = qp.masked_fill(air, 10.0), qs.masked_fill(air, 10.0)
        mu, m2 = rho * vs * vs, rho * vp * vp
        # the absorber copies the medium of the kernel region's edge
        def edge(f):
            for a in self.axes:
                lo = na + 1 if a != "z" else -2
                f = f.index_select(self.dim[a], idx[a].clamp(lo, self.n[a] - na) + 2)
            return f
        ts, zeta = _relaxation(self.nm)
        taup, taus = self.nm * zeta / edge(qp), self.nm * zeta / edge(qs)
        ratio = lambda v: torch.where(v.detach() > 0, v / v.detach().clamp_min(1e-30), torch.ones_like(v))
        grad = model is not None
        up = lambda f, *r: edge(f).detach() * math.prod(r) if grad else edge(f)
        mu = up(mu, ratio(vs), ratio(vs), ratio(rho)) if grad else edge(mu)
        m2 = up(m2, ratio(vp), ratio(vp), ratio(rho)) if grad else edge(m2)
        rho = edge(rho).detach() + (rho - rho.detach()) if grad else edge(rho)
        if self.nm:
            w = 2 * math.pi * FQ_REF
            cc = sum(complex(0, w * t) / (1 - complex(0, w * t)) for t in ts) / self.nm
            chi = lambda tau: 1 / torch.real(1 / torch.sqrt(1 - cc * tau.to(torch.complex128)))
            mu, m2 = mu / chi(taus) ** 2, m2 / chi(taup) ** 2
        self.inner = inner = torch.ones(shape, dtype=torch.bool, device=DEVICE)
        for a in self.axes:
            ok = idx[a] <= self.n[a] - na
            inner &= view(ok & (idx[a] >= (na + 1 if a != "z" else 1)), a)
        fix = lambda f: torch.where(inner, f, f.detach()) if grad else f
        sh = lambda f, *ax: torch.roll(f, [-1] * len(ax), [self.dim[a] for a in ax])
        mean4 = lambda a, b: (lambda m, p, q, r: 4 * m * p * q * r / (m * p * q + m * p * r + m * q * r + p * q * r + EPS))(
            mu, sh(mu, a), sh(mu, b), sh(mu, a, b))
        mean2 = lambda a: 2 * mu * sh(mu, a) / (mu + sh(mu, a) + EPS)
        cut = self.cut
        if c["kind"] == "sh":
            self.mus = {"xy": cut(mean2("x")), "yz": cut(mean2("z"))}
            self.b = {"y": cut(1 / rho)}
        else:
            pairs = ("yz", "xz", "xy") if "y" in self.n else ("xz",)
            self.mus = {q: cut(fix(mean4(*q))) for q in pairs}
            self.b = {a: cut(fix(2 / (rho + sh(rho, a)))) for a in self.axes}
        self.mu, self.m2 = cut(fix(mu)), cut(fix(m2))
        zero = torch.zeros((), **f64)
        inn = cut(inner)
        self.taup, self.taus = torch.where(inn, cut(taup), zero), torch.where(inn, cut(taus), zero)
        dt = self.dt
        self.c1 = [(2 * t - dt) / (2 * t + dt) for t in ts]
        self.c2 = [2 / (2 * t + dt) / self.nm for t in ts]
        self.d1 = [2 * t / (2 * t - dt) for t in ts]
        d2 = sum(dt / (2 * t - dt) for t in ts) / self.nm if self.nm else 0.0
        self.tp1, self.ts1 = 1 + self.taup * (1 + d2), 1 + self.taus * (1 + d2)
        self.visco = inn
        # 4th order inside the region, 2nd order in the absorber and around the free surface
        k = idx["z"][3:-3]
        fourth = inn & (k > AIR + 2)
        self.e0 = torch.where(fourth, 9 / 8, 1.0).double() / dx
        self.e1 = torch.where(fourth, 1 / 24, 0.0).double() / dx
        self.g = {}
        for a in self.axes:
            beg = -AIR * dx if a == "z" else _beg(self.n[a], dx)
            x = (idx[a][3:-3].double() - 0.5) * dx + beg
            for t, xx in (("c", x), ("e", x + dx / 2)):
                self.g[a + t] = [view(v, a) for v in _profile(xx, self.n[a], beg, dx, na, fcut, dt)]

    def cut(self, f, off=None):
        """The cells 1..n of an array over the memory box, shifted by off."""
        for d, a in enumerate(self.axes):
            o = (off or {}).get(a, 0)
            f = f.narrow(d, 3 + o, self.n[a])
        return f

    def diff(self, f, a, fwd):
        at = lambda o: self.cut(f, {a: o})
        if fwd:
            return (at(1) - at(0)) * self.e0 - (at(2) - at(-1)) * self.e1
        return (at(0) - at(-1)) * self.e0 - (at(1) - at(-2)) * self.e1

    def pml(self, aux, key, prof, d, ahead=False):
        """The stretched derivative; the auxiliary advances (before its use in SH's stress update)."""
        x, y, z, w = self.g[prof]
        old = aux.get(key, 0.0)
        new = z * old + w * d * self.dt
        aux[key] = torch.where(self.visco, torch.zeros_like(new), new)
        return torch.where(self.visco, d, x * d + y * (aux[key] if ahead else old))

    def pad(self, f):
        return F.pad(f, (3, 3) * len(self.axes))

    def memory(self, R, key, f, s):
        """Memory variables of one component with source f; s plus their sum."""
        if not self.nm:
            return s
        R[key] = [self.c1[m] * R[key][m] - self.c2[m] * f * self.dt if key in R else -self.c2[m] * f * self.dt
                  for m in range(self.nm)]
        return s + sum(self.d1[m] * R[key][m] for m in range(self.nm))

    def stress(self, V, S, R, aux):
        dt, ahead = self.dt, self.c["kind"] == "sh"
        # in the absorber the stretched derivatives take the plain ones' place
        D = lambda v, a, fwd: self.pml(aux, f"{a}V{v}", a + ("e" if fwd else "c"), self.diff(V[v], a, fwd), ahead)
        out = {}
        if not ahead:
            dn = {a: D(a, a, False) for a in self.axes}
            tot = sum(dn.values())
            for a in self.axes:
                rest = tot - dn[a]
                s = self.m2 * self.tp1 * tot - 2 * self.mu * self.ts1 * rest
                f = self.m2 * self.taup * tot - 2 * self.mu * self.taus * rest
                out[a + a] = self.memory(R, a + a, f, s)
        for q, mu in self.mus.items():
            d = D(q[1], q[0], True) + D(q[0], q[1], True) if not ahead else D("y", q.replace("y", ""), True)
            out[q] = self.memory(R, q, mu * self.taus * d, mu * self.ts1 * d)
        return {q: S[q] + self.pad(v * dt) if q in S else self.pad(v * dt) for q, v in out.items()}

    def velocity(self, V, S, aux):
        out = {}
        for a in self.b:
            d = 0.0
            for q in self.axes:
                name = a + a if q == a else "".join(sorted(a + q))
                d = d + self.pml(aux, f"{q}S{name}{a}", q + ("e" if q == a else "c"),
                                 self.diff(S[name], q, q == a))
            out[a] = V[a] + self.pad(self.b[a] * d * self.dt)
        return out


def _kupper(t, tr):
    return 3 * math.pi * math.sin(math.pi * t / tr) ** 3 / (4 * tr) if 0 <= t <= tr else 0.0


def _cell(s, k, i, j):
    return (j + 2, i + 2, k + 2) if "y" in s.n else (i + 2, k + 2)


def _glut(s, src, S, it):
    """Stress drop of the moment tensors at it - 1/2."""
    nsrc = len(src["i"])
    vol = s.c["dx"] ** len(s.axes)
    S = {q: v.clone() for q, v in S.items()}
    for n in range(nsrc):
        i, j, k, m = src["i"][n], src["j"][n], src["k"][n], src["m"][n]
        drop = _kupper((it - 0.5) * s.dt, src["trise"][n]) / nsrc * s.dt / vol
        comp = dict(zip(("xx", "yy", "zz", "yz", "xz", "xy"), m))
        for q in S:
            if q[0] == q[1]:
                S[q][_cell(s, k, i, j)] -= comp[q] * drop
                continue
            low = [a for a in q if a in s.n]
            cells = [(k - dk * ("z" in low), i - di * ("x" in low), j - dj * ("y" in low))
                     for dk in (0, 1) for di in (0, 1) for dj in (0, 1)]
            cells = sorted(set(cells))
            for cell in cells:
                S[q][_cell(s, *cell)] -= comp[q] * drop / len(cells)
    return S


def _traces(s, st, V, scale):
    """Velocity at the stations (first cell below the surface), vertical up."""
    k = AIR + 1
    if "y" in s.n:
        ix = (torch.tensor(st["j"], device=DEVICE) + 2, torch.tensor(st["i"], device=DEVICE) + 2)
        at = lambda f, dk=0, di=0, dj=0: f[ix[0] + dj, ix[1] + di, k + 2 + dk]
        return torch.stack([at(V["x"]) + at(V["x"], di=-1), at(V["y"]) + at(V["y"], dj=-1),
                            -(at(V["z"]) + at(V["z"], dk=-1))], 1) / 2 * scale
    ix = torch.tensor(st["i"], device=DEVICE) + 2
    if "y" in V:
        return V["y"][ix, k + 2][:, None] * scale
    return torch.stack([V["x"][ix, k + 2] + V["x"][ix - 1, k + 2], -(V["z"][ix, k + 2] + V["z"][ix, k + 1])], 1) / 2 * scale


def _vmax(s, V, scale):
    na, c = s.c["na"], s.c
    k, m = AIR + 1 + 2, na + 5
    box = [slice(m + 1 + 2, s.n[a] - m + 3) for a in s.axes[:-1]]
    order = [a for a in "xyz" if a in V]
    return torch.stack([V[a][tuple(box) + (k,)].abs().amax() * scale for a in order])


def _shot(s, src, st, V, nt, moment, report=0, planes=False, force=None):
    """The time loop: (traces (nst, ncmp, nt), displacement, reports, planes, final V)."""
    S, R, aS, aV = {}, {}, {}, {}
    tr, us, rep, fs, xz = [], [], [], [], []
    u = 0.0
    for it in range(1, nt + 1):
        if report and it % report == 0:
            rep.append(_vmax(s, V, UC * moment))
        t = _traces(s, st, V, moment * UC * 1e9)
        u = u + t * s.dt
        tr.append(t)
        us.append(u)
        if planes and (it - 1) % 10 == 0:
            v = torch.stack([s.cut(V[a]) for a in "xyz"]) * UC * moment
            fs.append(v[..., AIR].clone())
            xz.append(v[:, s.c["ny"] // 2 - 1].transpose(1, 2).clone())
        S = s.stress(V, S, R, aV)
        if src is not None:
            S = _glut(s, src, S, it)
        V = s.velocity(V, S, aS)
        if force is not None:
            V = force(V, it)
    return torch.stack(tr, -1), torch.stack(us, -1), rep, fs, xz, V


def exact(case, seed):
    c = case
    if c["kind"] == "gradient":
        return _exact_gradient(c, seed) if c["nx"] * c["ny"] * c["nz"] * c["nt"] <= 30_000_000 else None
    with torch.no_grad():
        if c["kind"] == "ensemble":
            return [_exact2d(m, seed * 64 + n)["v"] for n, m in enumerate(_member_cases(c, seed))]
        if c["kind"] in ("psv", "sh"):
            return _exact2d(c, seed)
        src, st = _random(c, seed)
        if c["kind"] == "forces":
            return _exact_forces(c, seed, st)
        s = _Scheme(c, max(1 / t for t in src["trise"]), xi=_xi(c, seed))
        moment = MO * len(src["i"])
        V = dict(zip("xyz", (v.double() for v in _wavefield(c, seed, 3))))
        tr, _, rep, fs, xz, V = _shot(s, src, st, V, c["nt"], moment, c["report"], c["planes"])
        out = {"v": tr, "vmax": torch.stack(rep)}
        if c["planes"]:
            out["fs"], out["xz"] = torch.stack(fs), torch.stack(xz)
        if c["nx"] * c["ny"] * c["nz"] <= 1 << 20:
            out["fields"] = [V[a] for a in "xyz"]
        return out


def _exact2d(c, seed):
    src, st = _random(c, seed)
    s = _Scheme(c, max(1 / t for t in src["trise"]))
    names = "xz" if c["kind"] == "psv" else "y"
    V = dict(zip(names, (v.double() for v in _wavefield(c, seed, len(names)))))
    tr, u, _, _, _, V = _shot(s, src, st, V, c["nt"], MO * len(src["i"]))
    return {"v": tr, "u": u, "vmax": None, "fields": [V[a] for a in names]}


def _exact_forces(c, seed, st):
    trise = 3.0 * c["dx"]
    s = _Scheme(c, 1 / trise)
    out = []
    for n, q in _forces(c, seed):
        i, j, k = st["i"][n], st["j"][n], AIR + 1

        def force(V, it, q=q, cell=(k, i, j)):
            f = _kupper(it * s.dt, trise) * s.dt / c["dx"] ** 3 / 2
            V = dict(V)
            V[q] = V[q].clone()
            for d in (0, 1):
                k1, i1, j1 = cell[0] - d * (q == "z"), cell[1] - d * (q == "x"), cell[2] - d * (q == "y")
                V[q][_cell(s, k1, i1, j1)] += s.b[q][j1 - 1, i1 - 1, k1 - 1] * f
            return V

        V = {a: torch.zeros([s.n[b] + 6 for b in s.axes], dtype=torch.float64, device=DEVICE) for a in "xyz"}
        # green's functions are recorded for a unit moment
        out.append(_shot(s, None, st, V, c["nt"], 1.0, force=force)[0])
    return out


def _exact_gradient(c, seed):
    from torch.utils.checkpoint import checkpoint

    src, st = _random(c, seed)
    fcut = max(1 / t for t in src["trise"])
    shape = (c["ny"] + 6, c["nx"] + 6, c["nz"] + 6)
    zc = (torch.arange(-2, c["nz"] + 4, device=DEVICE).double() - 0.5) * c["dx"] - AIR * c["dx"]
    base = [torch.zeros(shape, dtype=torch.float64, device=DEVICE) for _ in range(3)]
    for top, rho, vp, vs, *_ in LAYERS:
        for f, v in zip(base, (vp, vs, rho)):
            f[..., zc >= top] = v
    base[2][..., zc < 0] = 0.001
    zero = {a: torch.zeros(shape, dtype=torch.float64, device=DEVICE) for a in "xyz"}
    moment = MO * len(src["i"])
    with torch.no_grad():
        true = [base[0], base[1] * (1.0 + _anomaly(c).double()), base[2]]
        obs = _shot(_Scheme(c, fcut, model=true), src, st, dict(zero), c["nt"], moment)[0]
    gen = torch.Generator(DEVICE).manual_seed(seed * 7 + 9)
    model = [(m * (1.0 + _field(gen, m.shape, 0.01).double())).requires_grad_(True) for m in base]
    s = _Scheme(c, fcut, model=model)
    J = 0.0
    state = (dict(zero), {}, {}, {}, {})

    def segment(it0, it1, state):
        V, S, R, aS, aV = (dict(d) for d in state)
        j = 0.0
        for it in range(it0, it1):
            r = _traces(s, st, V, moment * UC * 1e9) - obs[..., it - 1]
            j = j + 0.5 * (r * r).sum()
            S = _glut(s, src, s.stress(V, S, R, aV), it)
            V = s.velocity(V, S, aS)
        return j, (V, S, R, aS, aV)

    for it0 in range(1, c["nt"] + 1, 10):
        j, state = checkpoint(segment, it0, min(it0 + 10, c["nt"] + 1), state, use_reentrant=False)
        J = J + j
    grads = torch.autograd.grad(J, model)
    return {"misfit": J.detach(), "grad": [g.detach() for g in grads]}
