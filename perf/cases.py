"""The work a user of this framework has it do, as measurable cases.

A case is a dict of plain values.  Kinds:

  step   one solver context: set_state, `steps` TVD-RK3 steps, get_state
         (device tensors), the loop of a resident solve
  batch  an ensemble of uneven boxes of several schemes advanced together
  serve  requests with host states submitted to a Server and collected
  rhs    one right-hand side of a given state (the drop-in for a host code
         that integrates by itself)
  ops    the operator plug-ins on a (nz, ny, nx) field with explicit halos:
         reconstruction in both upwind directions, and for explicit schemes
         the differential and the Runge-Kutta stage as well
  diag   statistics and shell spectra of a state, as logged between steps

listed() holds fixed cases, draw() more of the same ranges.  prepare() builds
the inputs (seeded turbulence-like fields) and the handles, run() is one pass
through the public entry points, exact() the same results in plain 64-bit
torch, work() the bytes and operations a pass cannot do without.
"""

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "nuc3d-cartisian_b200" / "python"))
import nuc3d_b200 as nb  # noqa: E402

CFL = 0.5
REYNOLDS = 400.0
# operations per cell and reconstruction direction (both signs, five equations)
DIR_FLOPS = {"weno5js": 728, "weno5z": 808, "crweno5": 1000, "hccs": 1100, "weno7js": 1900}
VISC_FLOPS, PRIM_FLOPS = 267, 20


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # the smallest box of the ensembles: launches and latency count
        dict(name="step_js_32", kind="step", nx=32, ny=32, nz=32, scheme="weno5js",
             precision="fp64", steps=10),
        # an ordinary laminar-to-turbulent box with extents no tile divides
        dict(name="step_z_ragged", kind="step", nx=97, ny=61, nz=45, scheme="weno5z",
             precision="fp64", steps=4),
        # the headline: decaying turbulence at 256^3, WENO5-Z, FP64
        dict(name="step_z_256", kind="step", nx=256, ny=256, nz=256, scheme="weno5z",
             precision="fp64", steps=2),
        # the same box in mixed precision
        dict(name="step_z_256_mixed", kind="step", nx=256, ny=256, nz=256, scheme="weno5z",
             precision="mixed", steps=2),
        # compact reconstruction: a tridiagonal line solve per direction
        dict(name="step_cr_192", kind="step", nx=192, ny=192, nz=192, scheme="crweno5",
             precision="fp64", steps=1),
        # forced turbulence with the hybrid compact scheme, mixed precision
        dict(name="step_hccs_forced", kind="step", nx=160, ny=160, nz=160, scheme="hccs",
             precision="mixed", steps=1, forced=True),
        # seventh order on an elongated box
        dict(name="step_w7_box", kind="step", nx=192, ny=96, nz=80, scheme="weno7js",
             precision="fp64", steps=2),
        # an uneven ensemble, one launch per kernel class for all boxes
        dict(name="batch_20", kind="batch", boxes=20, lo=32, hi=96, layout=7, precision="fp64",
             steps=2),
        # a request stream of small solves through the server
        dict(name="serve_6", kind="serve", boxes=6, lo=32, hi=64, layout=3, precision="mixed",
             steps=4),
        # the right-hand side alone, for a host integrator
        dict(name="rhs_js_128", kind="rhs", nx=128, ny=128, nz=128, scheme="weno5js",
             precision="fp64"),
        # the operator plug-ins of the compact scheme
        dict(name="ops_cr_192", kind="ops", nx=192, ny=128, nz=96, scheme="crweno5"),
        # what a solve logs between steps
        dict(name="diag_128", kind="diag", nx=128, ny=128, nz=128, scheme="weno5z"),
    ]


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["rhs", "ops", "diag", "batch"])
    if kind == "batch":
        lo = _extent(rng, 24, 48)
        return dict(kind=kind, boxes=rng.randint(4, 24), lo=lo, hi=lo + rng.randint(8, 56),
                    layout=rng.randrange(1000), precision=rng.choice(["fp64", "mixed"]),
                    steps=rng.randint(1, 2))
    scheme = rng.choice(["weno5z", "weno5z", "weno5js", "weno5js", "crweno5", "hccs", "weno7js"])
    most = 256 if scheme in ("weno5z", "weno5js") else 160
    n = [_extent(rng, 24, most) for _ in range(3)]
    case = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], scheme=scheme)
    if kind == "step":
        case["precision"] = rng.choice(["fp64", "fp64", "mixed"])
        case["steps"] = rng.randint(1, 2)
    elif kind == "rhs":
        case["precision"] = "fp64"
    return case


# ------------------------------------------------------------------ inputs --
def _field(nx, ny, nz, seed):
    """Conserved state (5, nz, ny, nx) of a turbulent-like flow at turbulent
    Mach number 0.3 (sound speed 1): solenoidal Fourier modes with an energy
    spectrum peaked at k = 3, density and pressure fluctuations of a few per
    cent."""
    rng = random.Random(int(seed))
    dev = torch.device("cuda")
    ax = [torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
          for n in (nx, ny, nz)]
    u = torch.zeros(3, nz, ny, nx, device=dev, dtype=torch.float64)
    s = torch.zeros(2, nz, ny, nx, device=dev, dtype=torch.float64)
    kmax = 7
    for m in range(28):
        k = [0, 0, 0]
        while not 1 <= sum(c * c for c in k) <= kmax * kmax:
            k = [rng.randint(-kmax, kmax) for _ in range(3)]
        kk = math.sqrt(sum(c * c for c in k))
        amp = kk ** 1.0 * math.exp(-(kk / 3.0) ** 2 / 2) + 0.02
        a = [rng.gauss(0, 1) for _ in range(3)]
        dot = sum(x * y for x, y in zip(a, k)) / kk ** 2
        d = [x - dot * y for x, y in zip(a, k)]  # perpendicular to k
        ph = rng.uniform(0, 2 * math.pi)
        e = [torch.polar(torch.ones_like(x), c * x) for x, c in zip(ax, k)]
        plane = (e[2] * complex(math.cos(ph), math.sin(ph)))[:, None] * e[1][None, :]
        wave = plane.real[:, :, None] * e[0].real - plane.imag[:, :, None] * e[0].imag
        for i in range(3):
            u[i].add_(wave, alpha=amp * d[i])
        s[m % 2].add_(wave, alpha=amp)
    u *= 0.3 / math.sqrt(3.0) / u.square().mean().sqrt()
    s /= s.square().mean(dim=(1, 2, 3), keepdim=True).sqrt()
    rho = 1.0 + 0.02 * s[0]
    p = (1.0 + 0.03 * s[1]) / 1.4
    q = torch.empty(5, nz, ny, nx, device=dev, dtype=torch.float64)
    q[0] = rho
    q[1:4] = rho * u
    q[4] = p / 0.4 + 0.5 * rho * u.square().sum(0)
    return q


def _desc(case, **more):
    d = dict(nx=case["nx"], ny=case["ny"], nz=case["nz"], mach=1.0, reynolds=REYNOLDS,
             scheme=(nb.SCHEMES[case["scheme"]],) * 3,
             precision=nb.MIXED if case.get("precision") == "mixed" else nb.FP64)
    if case.get("forced"):
        d.update(forcing=nb.FORCING_BAND, forcing_amp=0.02, forcing_k=2.0)
    d.update(more)
    return nb.BoxDesc(**d)


def _boxes(case):
    """The boxes of a batch or request mix: uneven edges, three schemes."""
    rng = random.Random(1000 + case["layout"])
    return [dict(nx=rng.randint(case["lo"], case["hi"]), ny=rng.randint(case["lo"], case["hi"]),
                 nz=rng.randint(case["lo"], case["hi"]), precision=case["precision"],
                 scheme=("weno5js", "weno5z", "crweno5")[b % 3], steps=case["steps"])
            for b in range(case["boxes"])]


def _operands(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    q = _field(nx, ny, nz, seed)
    h = 4 if case["scheme"] in ("hccs", "weno7js") else 3
    f = q[1].contiguous()
    return q, f, f[..., -h:].contiguous(), f[..., :h].contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = nb.Batch(nb.MIXED if case["precision"] == "mixed" else nb.FP64)
        ids, q, out = [], [], []
        for n, box in enumerate(_boxes(case)):
            bid = b.add(_desc(box))
            b.set_cfl(bid, CFL)
            ids.append(bid)
            q.append(_field(box["nx"], box["ny"], box["nz"], seed * 100 + n))
            out.append(torch.empty_like(q[-1]))
        return dict(case=case, batch=b, ids=ids, q=q, out=out)
    if kind == "serve":
        srv = nb.Server(nb.MIXED if case["precision"] == "mixed" else nb.FP64)
        boxes = _boxes(case)
        q = [_field(x["nx"], x["ny"], x["nz"], seed * 100 + n).cpu().numpy()
             for n, x in enumerate(boxes)]
        return dict(case=case, server=srv, descs=[_desc(x) for x in boxes], q=q)
    if kind == "ops":
        q, f, hl, hr = _operands(case, seed)
        s = dict(case=case, f=f, hl=hl, hr=hr,
                 faces=torch.empty(2, *f.shape[:2], f.shape[2] + 1, device=f.device,
                                   dtype=f.dtype))
        if case["scheme"] not in ("crweno5", "hccs"):
            s.update(q=q, ui=q * 1.01, rhs=q * 0.5, diff=torch.empty_like(f),
                     h3l=f[..., -3:].contiguous(), h3r=f[..., :3].contiguous())
        return s
    q = _field(case["nx"], case["ny"], case["nz"], seed)
    s = dict(case=case, q=q, solver=nb.Solver(_desc(case)))
    if kind != "diag":
        s["out"] = torch.empty_like(q)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["solver"].set_state(list(s["q"]))
        s["solver"].step(case["steps"], CFL, stats=False)
        s["solver"].get_state(list(s["out"]))
        return s["out"]
    if kind == "batch":
        b = s["batch"]
        for i, q in zip(s["ids"], s["q"]):
            b.set_state(i, list(q))
        b.step(case["steps"])
        for i, o in zip(s["ids"], s["out"]):
            b.get_state(i, list(o))
        return s["out"]
    if kind == "serve":
        srv = s["server"]
        tickets = [srv.submit(d, case["steps"], CFL, q0=list(q), want_state=True)
                   for d, q in zip(s["descs"], s["q"])]
        return [np.stack(srv.wait(t)["state"]) for t in tickets]
    if kind == "rhs":
        s["solver"].set_state(list(s["q"]))
        dt = s["solver"].rhs(list(s["out"]))
        return s["out"], dt
    if kind == "diag":
        s["solver"].set_state(list(s["q"]))
        return (np.array(list(s["solver"].stats().values())), s["solver"].spectra())
    sch = nb.SCHEMES[case["scheme"]]
    for k, up in enumerate((1, -1)):
        nb.reconstruct(sch, up, nb.QUIRKS_REFERENCE, s["f"], s["hl"], s["hr"], s["faces"][k])
    if "q" not in s:
        return s["faces"]
    nb.differential(nb.CD6, 3, 2 * math.pi / case["nx"], s["f"], s["h3l"], s["h3r"], s["diff"])
    nb.tvdrk3_stage(1, 1e-3, list(s["rhs"]), list(s["q"]), list(s["ui"]))
    return s["faces"], s["diff"], s["ui"]


def _step_work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    per = 3 * (3 * DIR_FLOPS[case["scheme"]] + VISC_FLOPS + PRIM_FLOPS)
    # input and output once, and per step: stage 1 reads u_n and writes u1,
    # stages 2 and 3 read u_n and u_k and write u_k+1
    return dict(bytes=n * (160 + 320 * case["steps"]), flops=n * case["steps"] * per)


def work(case):
    kind = case["kind"]
    if kind == "step":
        return _step_work(case)
    if kind in ("batch", "serve"):
        w = [_step_work(b) for b in _boxes(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "rhs":
        return dict(bytes=80 * n,
                    flops=n * (3 * DIR_FLOPS[case["scheme"]] + VISC_FLOPS + PRIM_FLOPS))
    if kind == "diag":
        # a state read; seven real transforms of n points, the gradients and sums
        return dict(bytes=40 * n, flops=n * (7 * 2.5 * math.log2(n) + 200))
    flops = n * DIR_FLOPS[case["scheme"]] / 5
    if case["scheme"] in ("crweno5", "hccs"):
        return dict(bytes=n * 24, flops=flops)
    return dict(bytes=n * (24 + 16 + 160), flops=flops + n * 40)


# ------------------------------------------------------- the same in 64 bits --
def _c(axis, f):
    """axis moved last, contiguous"""
    return f.movedim(axis, -1).contiguous()


def _betas(f, quirk2=None):
    d = [f[0] - 2 * f[1] + f[2], f[1] - 2 * f[2] + f[3], f[2] - 2 * f[3] + f[4]]
    if quirk2 is not None:
        d[2] = torch.where(quirk2, f[2] - f[3], d[2])
    e = [f[0] - 4 * f[1] + 3 * f[2], f[1] - f[3], 3 * f[2] - 4 * f[3] + f[4]]
    return [13 / 12 * a * a + b * b / 4 for a, b in zip(d, e)]


def _weno5(f, scheme, quirk2=None):
    b = _betas(f, quirk2)
    c = (0.1, 0.6, 0.3)
    if scheme == "weno5z":
        tau = (b[2] - b[0]).abs()
        a = [ck * (1 + (tau / (bk + 1e-40)) ** 2) for ck, bk in zip(c, b)]
    else:
        a = [ck / (1e-6 + bk) ** 2 for ck, bk in zip(c, b)]
    q = [f[0] / 3 - 7 / 6 * f[1] + 11 / 6 * f[2], -f[1] / 6 + 5 / 6 * f[2] + f[3] / 3,
         f[2] / 3 + 5 / 6 * f[3] - f[4] / 6]
    return (a[0] * q[0] + a[1] * q[1] + a[2] * q[2]) / (a[0] + a[1] + a[2])


def _weno7(f, eps):
    co = ((547, -3882, 4642, -1854, 7043, -17246, 7042, 11003, -9402, 2107),
          (267, -1642, 1602, -494, 2843, -5966, 1922, 3443, -2522, 547),
          (547, -2522, 1922, -494, 3443, -5966, 1602, 2843, -1642, 267),
          (2107, -9402, 7042, -1854, 11003, -17246, 4642, 7043, -3882, 547))
    b = []
    for s, k in enumerate(co):
        x = f[s:s + 4]
        b.append(x[0] * (k[0] * x[0] + k[1] * x[1] + k[2] * x[2] + k[3] * x[3])
                 + x[1] * (k[4] * x[1] + k[5] * x[2] + k[6] * x[3])
                 + x[2] * (k[7] * x[2] + k[8] * x[3]) + k[9] * x[3] * x[3])
    q = [(-3 * f[0] + 13 * f[1] - 23 * f[2] + 25 * f[3]) / 12,
         (f[1] - 5 * f[2] + 13 * f[3] + 3 * f[4]) / 12,
         (-f[2] + 7 * f[3] + 7 * f[4] - f[5]) / 12,
         (3 * f[3] + 13 * f[4] - 5 * f[5] + f[6]) / 12]
    tau = (b[0] - b[3]).abs()
    a = [c / 35 * (1 + (tau / (eps + bk)) ** 2) for c, bk in zip((1, 12, 18, 4), b)]
    return sum(x * y for x, y in zip(a, q)) / sum(a)


def _thomas(a, b, c, d):
    """Tridiagonal systems along dimension 0."""
    n = d.shape[0]
    cp, dp = torch.empty_like(d), torch.empty_like(d)
    cp[0], dp[0] = c[0] / b[0], d[0] / b[0]
    for i in range(1, n):
        den = b[i] - a[i] * cp[i - 1]
        cp[i] = c[i] / den
        dp[i] = (d[i] - a[i] * dp[i - 1]) / den
    for i in range(n - 2, -1, -1):
        dp[i] -= cp[i] * dp[i + 1]
    return dp


def _faces(scheme, sign, ext, n, quirk=True):
    """Face values 0..n along the last axis from cells -4..n+3."""
    def cell(o):
        return ext[..., 4 + o:5 + o + n]
    order = list(range(-4, 3)) if sign > 0 else list(range(3, -4, -1))
    if scheme == "weno7js":
        return _weno7([cell(o) for o in order], 1e-20)
    f = [cell(o) for o in order[1:6]]
    m = torch.arange(n + 1, device=ext.device)
    if scheme == "weno5js":
        return _weno5(f, scheme)
    if scheme == "weno5z":
        return _weno5(f, scheme, (m >= 3) & (m <= n - 3) if quirk and sign > 0 else None)
    h = 4 if scheme == "hccs" else 3
    out = _weno7([cell(o) for o in order], 1e-40) if h == 4 else _weno5(f, "weno5js")
    b = _betas(f)
    c = (0.2, 0.5, 0.3)
    if h == 3:
        al = [ck / (1e-6 + bk) ** 2 for ck, bk in zip(c, b)]
    else:
        tau = (b[2] - b[0]).abs()
        al = [ck * (1 + (tau / (bk + 1e-40)) ** 2) for ck, bk in zip(c, b)]
    s = al[0] + al[1] + al[2]
    w = [x / s for x in al]
    lo, di, hi = (2 * w[0] + w[1]) / 3, (w[0] + 2 * (w[1] + w[2])) / 3, w[2] / 3
    rh = (w[0] * f[1] + (5 * (w[0] + w[1]) + w[2]) * f[2] + (w[1] + 5 * w[2]) * f[3]) / 6
    if h == 4:
        x2 = (s - 1) ** 2
        q7 = (-f[0] + 19 * f[1] + 239 * f[2] + 159 * f[3] + 4 * f[4]) / 420
        x2 = torch.where(1 + x2 < 2, torch.zeros_like(x2), x2)
        r = 1 / (1 + x2)  # keeps the rows' scale near one
        g = x2 * r
        lo, di, hi, rh = lo * g + 2 / 7 * r, di * g + 4 / 7 * r, hi * g + r / 7, rh * g + q7 * r
    if sign < 0:
        lo, hi = hi, lo
    fixed = (m == h) | (m == n - h)
    lo, hi = (x.masked_fill(fixed, 0.0) for x in (lo, hi))
    di = di.masked_fill(fixed, 1.0)
    rh = torch.where(fixed, out, rh)
    sl = slice(h, n - h + 1)
    x = _thomas(*(_c(-1, t[..., sl]).movedim(-1, 0).contiguous() for t in (lo, di, hi, rh)))
    out = out.clone()
    out[..., sl] = x.movedim(0, -1)
    return out


def _deriv(f, axis, dx):
    def d(o):
        return torch.roll(f, -o, axis) - torch.roll(f, o, axis)
    return (0.75 * d(1) - 0.15 * d(2) + d(3) / 60) / dx


def _prims(q):
    rho, u = q[0], q[1:4] / q[0]
    p = ((q[4] - 0.5 * rho * u.square().sum(0)) * 0.4).abs()
    return u, p, (1.4 * p / rho).sqrt(), 1.4 * p / rho


def _mu(t):
    s = 110.4 / 288.0
    return (1 + s) / (t + s) * t.pow(1.5) / REYNOLDS


def _rhs(case, q):
    """dQ/dt = -result; and dt of the CFL-free step."""
    n = (case["nx"], case["ny"], case["nz"])
    dx = [2 * math.pi / x for x in n]
    u, p, c, t = _prims(q)
    out = torch.zeros_like(q)
    for d in range(3):
        axis = 2 - d
        lam = u[d].abs() + c
        for e in range(5):
            f = u[d] * (q[e] + p if e == 4 else q[e])
            if e == 1 + d:
                f = f + p
            tot = 0.0
            for sign in (1, -1):
                s = _c(axis, 0.5 * (f + sign * lam * q[e]))
                ext = torch.cat([s[..., -4:], s, s[..., :4]], -1)
                tot = tot + _faces(case["scheme"], sign, ext, n[d])
            out[e] += ((tot[..., 1:] - tot[..., :-1]) / dx[d]).movedim(-1, axis)
    g = [[_deriv(x, 2 - d, dx[d]) for d in range(3)] for x in (u[0], u[1], u[2], t)]
    mu = _mu(t)
    div = g[0][0] + g[1][1] + g[2][2]
    tau = [[None] * 3 for _ in range(3)]
    for i in range(3):
        for j in range(i, 3):
            # the reference's off-diagonal stresses carry the divergence too
            tau[i][j] = tau[j][i] = mu * (g[i][j] + g[j][i] - 2 / 3 * div)
    kap = mu / (0.4 * 0.72)
    for d in range(3):
        for i in range(3):
            out[1 + i] -= _deriv(tau[i][d], 2 - d, dx[d])
        en = sum(u[i] * tau[i][d] for i in range(3)) + kap * g[3][d]
        out[4] -= _deriv(en, 2 - d, dx[d])
    if case.get("forced"):
        out[1:5] -= _band(u, 0.02, 2.0)
    # the z maximum is folded into y and z left out (reference behaviour)
    ex = (u[0].abs() + c).max()
    ey = torch.maximum((u[1].abs() + c).max(), (u[2].abs() + c).max())
    return out, 1 / (ex / dx[0] + ey / dx[1])


def _wavenumbers(shape, dev):
    k = []
    for a, n in enumerate(shape):
        w = torch.arange(n, device=dev, dtype=torch.float64)
        w = torch.where(w >= n / 2, w - n, w)
        k.append(w.view([-1 if b == a else 1 for b in range(3)]).expand(shape))
    return k[2], k[1], k[0]


def _solenoidal(u):
    k = _wavenumbers(u.shape[1:], u.device)
    mag0 = (k[0] ** 2 + k[1] ** 2 + k[2] ** 2).sqrt()
    mag = torch.where(mag0 < 1e-6, torch.ones_like(mag0), mag0)
    f = [torch.fft.fftn(x) / x.numel() for x in u]
    ku = sum(a * b for a, b in zip(k, f)) / mag
    return k, mag0, mag, f, [f[i] - ku * k[i] / mag for i in range(3)]


def _band(u, rate, kf):
    _, mag0, _, _, s = _solenoidal(u)
    band = (mag0 > 0) & (mag0 <= kf + 1e-12)
    eb = sum(0.5 * x.abs().square()[band].sum() for x in s)
    f = [torch.fft.ifftn(torch.where(band, x * (rate / (2 * eb)), torch.zeros_like(x))).real
         * x.numel() for x in s]
    fu = sum(a * b for a, b in zip(f, u))
    return torch.stack(f + [fu - fu.mean()])


def _steps(case, q):
    for _ in range(case["steps"]):
        r, dt = _rhs(case, q)
        dt = dt * CFL
        q1 = q - dt * r
        q2 = 0.75 * q + 0.25 * (q1 - dt * _rhs(case, q1)[0])
        q = q / 3 + 2 / 3 * (q2 - dt * _rhs(case, q2)[0])
    return q


def _stats(case, q):
    n = (case["nx"], case["ny"], case["nz"])
    u, _, c, t = _prims(q)
    g = [[_deriv(x, 2 - d, 2 * math.pi / n[d]) for d in range(3)] for x in u]
    w = (g[2][1] - g[1][2], g[0][2] - g[2][0], g[1][0] - g[0][1])
    om2 = w[0] ** 2 + w[1] ** 2 + w[2] ** 2
    u2 = u.square().sum(0)
    q2 = (g[0][0] * g[1][1] + g[0][0] * g[2][2] + g[1][1] * g[2][2] - g[0][1] * g[1][0]
          - g[0][2] * g[2][0] - g[1][2] * g[2][1])
    div = g[0][0] + g[1][1] + g[2][2]
    out = [x.mean() for r in g for x in r] + [x.mean() for x in w]
    out += [om2.mean() / 2, q2.mean(), sum(a * b for a, b in zip(w, u)).mean(),
            (0.5 * q[0] * u2).mean()]
    ur, dv = (u2 / 3).mean(), sum(g[i][i] ** 2 for i in range(3)).mean() / 3
    s3 = sum(g[i][i] ** 3 for i in range(3)).mean() / 3
    mu = (_mu(t) * REYNOLDS).mean()
    lam = (ur / dv).sqrt()
    rho = q[0].mean()
    out += [ur.sqrt(), (3 * ur).sqrt() / c.mean(), dv.sqrt(), mu,
            ur.sqrt() * lam * rho / mu * REYNOLDS, lam, rho, lam / ur.sqrt(), s3 / dv ** 1.5,
            (_mu(t) * (om2 + 4 / 3 * div * div)).mean()]
    return torch.stack(out)


def _shells(mag, keep, values, kmax):
    idx = torch.where((mag - mag.floor()) - 0.5 <= 0, mag.floor(), mag.floor() + 1).long()
    out = []
    for v in values:
        h = torch.zeros(kmax + 1, device=v.device, dtype=torch.float64)
        out.append(h.index_add_(0, idx[keep], v[keep])[:kmax])
    return out


def _spectra(case, q):
    n = (case["nx"], case["ny"], case["nz"])
    kmax = min(n) // 2
    u, p, _, _ = _prims(q)
    g = [[_deriv(x, 2 - d, 2 * math.pi / n[d]) for d in range(3)] for x in u]
    w = (g[2][1] - g[1][2], g[0][2] - g[2][0], g[1][0] - g[0][1])
    k, _, mag, f, s = _solenoidal(u)
    comp = [a - b for a, b in zip(f, s)]
    # i k x s / |k| with the reference's sign of the second component
    x = [(k[1] * (1j * s[2]) - k[2] * (1j * s[1])) / mag,
         -(k[0] * (1j * s[2]) - k[2] * (1j * s[0])) / mag,
         (k[0] * (1j * s[1]) - k[1] * (1j * s[0])) / mag]

    def energy(v):
        return 0.5 * sum(a.abs().square() for a in v)
    kin = [energy(f), energy(comp), energy(s), energy([0.5 * (a - b) for a, b in zip(s, x)]),
           energy([0.5 * (a + b) for a, b in zip(s, x)])]
    rows = _shells(mag, mag < kmax, kin, kmax)
    scal = [sum(a * b for a, b in zip(w, u)), sum(a * a for a in w) * 0.5, q[0], p]
    i, j, l = (torch.arange(m, device=q.device, dtype=torch.float64) for m in n)
    k0 = l.view(-1, 1, 1) ** 2 + j.view(1, -1, 1) ** 2 + i.view(1, 1, -1) ** 2
    keep = k0 < kmax * kmax
    rows += _shells(k0.sqrt(), keep,
                    [(torch.fft.fftn(v) / v.numel()).abs().square() for v in scal], kmax)
    return torch.stack(rows)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        return [_steps(b, _field(b["nx"], b["ny"], b["nz"], seed * 100 + n))
                for n, b in enumerate(_boxes(case))]
    if kind == "ops":
        q, f, _, _ = _operands(case, seed)
        ext = torch.cat([f[..., -4:], f, f[..., :4]], -1)
        faces = torch.stack([_faces(case["scheme"], s, ext, case["nx"]) for s in (1, -1)])
        if case["scheme"] in ("crweno5", "hccs"):
            return faces
        return (faces, _deriv(f, 2, 2 * math.pi / case["nx"]),
                0.75 * q + 0.25 * (-(q * 0.5) * 1e-3 + q * 1.01))
    q = _field(case["nx"], case["ny"], case["nz"], seed)
    if kind == "step":
        return _steps(case, q)
    if kind == "rhs":
        r, dt = _rhs(case, q)
        return r, float(dt)
    return _stats(case, q), _spectra(case, q)
