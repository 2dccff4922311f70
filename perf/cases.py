"""The workloads this library's speed is judged on, through its public Python entry points.

Each case is a plain dict.  ``prepare`` makes what a user's program holds before the call (models,
gathers, an open session), ``run`` is one pass, ``exact`` the same outputs in 64-bit torch and
``work`` the bytes and operations a pass cannot do without.  Time axes are shorter than a
production survey's (every time step costs the same), the grids, shot counts, storage types and
options are those of the library's configurations and tests.

Kinds:
  forward   rtm_forward: one shot modelled in one call, host arrays in and out
  model     Session.model: the gathers of a batch of shots (mode 0)
  migrate   Session.run: source pass, reconstruction, receiver pass, imaging, stacking; the
            images read back.  mode 0 models its own gathers and returns them too
  field     recorded shots: set_gather_raw (resampling, mute) of every shot, then Session.run
  resample  interp_gather: F-K and sinc resampling of one recorded shot
"""
import math

import numpy as np
import torch

import gubingluo_b200 as G

DEV = "cuda" if torch.cuda.is_available() else "cpu"
PI = 3.1415926535897932
# half-order h = 1..10 staggered-grid coefficients (Liu and Yang's optimised table), the
# library's defaults
TABLE = [
    [1.0],
    [0.1129042e+1, -0.4301412e-1],
    [0.1185991e+1, -0.7249965e-1, 0.6301572e-2],
    [0.1217990e+1, -0.9382142e-1, 0.1507536e-1, -0.1700324e-2],
    [0.1236607e+1, -0.1082265e+0, 0.2343440e-1, -0.5033546e-2, 0.6817483e-3],
    [0.1247662e+1, -0.1175538e+0, 0.2997970e-1, -0.8719078e-2, 0.2215897e-2, -0.3462075e-3],
    [0.1254799e+1, -0.1238928e+0, 0.3494371e-1, -0.1208897e-1, 0.4132531e-2, -0.1197110e-2, 0.2122227e-3],
    [0.1259312e+1, -0.1280347e+0, 0.3841945e-1, -0.1473229e-1, 0.5924913e-2, -0.2248618e-2, 0.7179226e-3,
     -0.1400855e-3],
    [0.1262502e+1, -0.1310244e+0, 0.4103928e-1, -0.1686807e-1, 0.7530520e-2, -0.3345071e-2, 0.1380367e-2,
     -0.4808410e-3, 0.1023759e-3],
    [0.1264748e+1, -0.1331606e+0, 0.4296909e-1, -0.1851897e-1, 0.8861071e-2, -0.4347073e-2, 0.2076101e-2,
     -0.9164925e-3, 0.3437446e-3, -0.7874250e-4],
]

DEFAULTS = dict(kind="migrate", nx=401, nz=201, d=10.0, npml=40, nt=400, dt=1e-3, fdom=20.0, shots=1, layout=2,
                mode=1, strips="fp32", gathers="fp32", accum=0, graph=0, extra=0, smooth=0, pmlsmooth=0, depth=2,
                narrow=0, wide=0, traces=0, factor=0)


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a single shot modelled in one call, as an interactive program does to look at a
        # gather: the session is opened, run and closed inside the call
        _case("forward, one small shot", kind="forward", nx=401, nz=201, nt=300),
        # the modelling half of a survey: 16 shots' gathers over one model
        _case("model 16 shots", kind="model", nx=601, nz=301, npml=40, nt=500, shots=16, mode=0),
        # the smallest migration that is run in earnest: one shot of the layered model with its
        # whole record; launches and latency count
        _case("migrate one small shot", nx=401, nz=201, nt=2000),
        # one shot of the 1701 x 351 survey per call with the time loops as graphs, as a shot
        # queue does that hands out single shots
        _case("migrate one shot, graph", nx=1701, nz=351, d=12.5, npml=50, nt=500, fdom=15.0, graph=1, depth=1),
        # a few shots of uneven windows with odd sizes: modelled and migrated (mode 0), smoothed
        # PML zone and migration model
        _case("model and migrate 6 odd windows", nx=1203, nz=277, d=10.0, npml=37, nt=400, shots=6, layout=1, mode=0,
              narrow=211, wide=623, smooth=3, pmlsmooth=1, depth=0),
        # the 64-shot full-spread survey in one batch, fp32 throughout
        _case("migrate 64 shots", nx=1701, nz=351, d=12.5, npml=50, nt=240, fdom=15.0, shots=64, depth=1),
        # shots of drawn apertures (2-8 km) with fp16 strips and gathers and fp64 totals
        _case("migrate 40 apertures, fp16", nx=3201, nz=801, d=10.0, npml=40, nt=160, dt=8e-4, shots=40, layout=1,
              strips="fp16", gathers="fp16", accum=3, narrow=201, wide=801),
        # a large grid at 5 m, few shots, fp64 accumulation
        _case("migrate 4 large grids, fp64", nx=4001, nz=1201, d=5.0, npml=60, nt=120, dt=4e-4, fdom=25.0, shots=4,
              strips="bf16", gathers="fp16", accum=1, depth=4),
        # an off-end line: unilateral windows to the right of the source, medium batch
        _case("migrate 12 off-end shots", nx=1401, nz=331, d=10.0, npml=32, nt=500, shots=12, layout=3, narrow=481,
              wide=481, depth=0),
        # all imaging conditions, the drop-in call's default
        _case("migrate 8 shots, all conditions", nx=801, nz=301, npml=40, nt=300, shots=8, extra=1, depth=0),
        # recorded shots: 241 traces every 25 m at 2 ms onto 12.5 m and 1 ms, then migrated
        _case("16 recorded shots", kind="field", nx=1701, nz=351, d=12.5, npml=50, nt=800, fdom=15.0, shots=16,
              traces=241, factor=2, depth=1),
        # one recorded shot resampled by itself (host arrays in and out)
        _case("resample one shot", kind="resample", nx=481, nt=4000, d=12.5, traces=241, factor=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    limit = _cell_steps(_case(nx=1701, nz=351, npml=50, nt=240, shots=64))
    while True:
        kind = rng.choice(["migrate"] * 7 + ["model", "forward", "field", "resample"])
        d = rng.choice([5.0, 7.5, 10.0, 12.5])
        dt = {5.0: 4e-4, 7.5: 6e-4, 10.0: 8e-4, 12.5: 1e-3}[d]
        if kind == "resample":
            traces = _log(rng, 40, 400)
            factor = rng.choice([2, 2, 3, 4])
            nx = (traces - 1) * factor + 1
            return _case(kind=kind, nx=nx, nt=rng.choice([2, 2, 1, 3]) * _log(rng, 300, 2000), d=d, dt=dt,
                         traces=traces, factor=factor)
        c = _case(kind=kind, nx=_log(rng, 150, 3201), nz=_log(rng, 100, 1001), d=d, dt=dt,
                  npml=rng.choice([20, 32, 40, 50, 60, 80, rng.randrange(16, 81)]), nt=_log(rng, 80, 800),
                  fdom=rng.choice([12.0, 15.0, 20.0, 25.0]), shots=_log(rng, 1, 64), depth=rng.choice([0, 1, 2, 4]))
        if kind == "forward":
            c.update(shots=1, nt=min(c["nt"], 400))
        elif kind == "model":
            c.update(mode=0)
        elif kind == "field":
            c["nt"] = 2 * ((c["nt"] + 1) // 2)
            c.update(factor=2, traces=min(241, max(30, c["nx"] // 6)), shots=min(c["shots"], 24), depth=0)
        else:
            c.update(layout=rng.choice([1, 2, 2, 2, 3, 4]), mode=rng.choice([0, 1, 1, 1]),
                     strips=rng.choice(["fp32", "fp32", "fp16", "bf16"]), graph=rng.choice([0, 0, 0, 1]),
                     gathers=rng.choice(["fp32", "fp32", "fp16", "bf16"]), accum=rng.choice([0, 0, 1, 2, 3]),
                     smooth=rng.choice([0, 0, 2]))
            if c["accum"] == 0 and rng.random() < 0.15:
                c["extra"] = 1
        if c["layout"] != 2:
            wide = min(c["nx"], 901)
            c.update(wide=wide, narrow=rng.randrange(max(100, wide // 4), wide + 1) if wide > 110 else wide)
            if c["shots"] <= 8 and c["nx"] * c["nz"] < 4e5:   # model preparation on the host
                c["pmlsmooth"] = rng.choice([0, 1])
        if _cell_steps(c) <= limit:
            return c


# ---- geometry and inputs ------------------------------------------------------------------
def _survey(c):
    return G.SurveyConfig(nx=c["nx"], nz=c["nz"], nt=c["nt"], dx=c["d"], dz=c["d"], dt=float(np.float32(c["dt"])),
                          npml=c["npml"], fdom=c["fdom"], alp=float(np.float32(1.0 / c["d"])), layout=c["layout"],
                          spx0=_column(c, 1) * c["d"], spz0=2 * c["d"], dspx=_stride(c) * c["d"],
                          offsetmax=(c["wide"] - 1) * c["d"] if c["wide"] else 0.0, mode=c["mode"],
                          medium_flag=c["pmlsmooth"], ismth=c["smooth"], direct=_direct(c),
                          mute=2 if c["kind"] == "field" else 1, receiver_depth=c["depth"])


def _direct(c):
    """Length of the direct-wave mute in periods: at most a quarter of the (short) record."""
    return float(np.float32(min(1.5, round(0.25 * c["nt"] * c["dt"] * c["fdom"], 3))))


def _options(c):
    return G.RunOptions(strip_precision=c["strips"], gather_precision=c["gathers"], accum_fp64=c["accum"],
                        use_graph=c["graph"], extra_images=c["extra"])


def _stride(c):
    room = c["nx"] - (c["factor"] * (c["traces"] - 1) + 1 if c["kind"] == "field" else 0)
    return max(1, room // (c["shots"] + 1))


def _column(c, shot):
    """Model column of a shot's source."""
    first = c["factor"] * max(1, _stride(c) // c["factor"]) if c["kind"] == "field" else max(1, _stride(c) // 2)
    step = c["factor"] * max(1, _stride(c) // c["factor"]) if c["kind"] == "field" else _stride(c)
    return min(first // 2 * 2 + (shot - 1) * step, c["nx"] - 1)


def _aperture(c, shot):
    """Columns of a shot's window in layouts 1, 3 and 4."""
    span = c["wide"] - c["narrow"]
    w = c["narrow"] + (span * ((shot * 37) % 16)) // 15 if span else c["wide"]
    return w | 1 if c["layout"] == 1 else w


def _window(c, shot):
    """(first column, last column, source column in the window, first receiver column, receivers)."""
    col = _column(c, shot)
    if c["kind"] == "field":
        x1 = col
        x2 = col + c["factor"] * (c["traces"] - 1)
        return x1, x2, 0, 0, x2 - x1 + 1
    if c["layout"] == 2:
        return 0, c["nx"] - 1, col, 0, c["nx"]
    w = _aperture(c, shot)
    if c["layout"] == 1:
        x1, x2 = max(0, col - (w - 1) // 2), min(c["nx"] - 1, col + (w - 1) // 2)
    elif c["layout"] == 3:
        x1, x2 = col, min(c["nx"] - 1, col + w - 1)
    else:
        x1, x2 = max(0, col - w + 1), col
    return x1, x2, col - x1, 0, x2 - x1 + 1


def _shot_geometry(c, shot):
    x1, x2, src, rec, nrec = _window(c, shot)
    g = G.Geometry()
    p = c["npml"]
    g.nx1, g.nx2, g.nxlength, g.noffset = x1, x2, x2 - x1 + 1, rec
    g.nsx, g.nsz, g.nxpad, g.nzpad = p + src, p + 2, x2 - x1 + 1 + 2 * p, c["nz"] + 2 * p
    g.rz, g.rx0, g.nrec = p + c["depth"], p + rec, nrec
    return g


def _shots(c):
    if c["layout"] == 2 or c["kind"] == "field":
        return list(range(1, c["shots"] + 1))
    # windows of one column are no shots: sources too near the edge are left out
    return [k for k in range(1, c["shots"] + 1) if _window(c, k)[1] - _window(c, k)[0] >= 40] or [1]


def _models(c, seed):
    """True and migration velocity and the density: a gradient with smooth random structure and
    layers, the migration model smoother."""
    rng = np.random.default_rng(1000003 * (seed % 1000003) + 17)
    nz, nx = c["nz"], c["nx"]
    zz = np.arange(nz)[:, None] / nz
    xx = np.arange(nx)[None, :] / nx
    smooth = 1700.0 + 1300.0 * zz + 0 * xx
    for _ in range(6):
        kx, kz, ph = rng.uniform(1, 6), rng.uniform(1, 6), rng.uniform(0, 2 * PI)
        smooth = smooth + rng.uniform(20, 60) * np.sin(2 * PI * (kx * xx + kz * zz) + ph)
    true = smooth.copy()
    for _ in range(5):
        z0, dip = rng.uniform(0.15, 0.95), rng.uniform(-0.2, 0.2)
        true = np.where(zz > z0 + dip * xx, true + rng.uniform(40, 160), true)
    rho = 1900.0 + 0.1 * true
    return (np.clip(true, 1500, 4500).astype(np.float32), np.clip(smooth, 1500, 4500).astype(np.float32),
            rho.astype(np.float32))


def _events(nt, dt, offsets, fdom, seed):
    """A band-limited gather [nt][traces]: a direct wave and hyperbolic reflections with the
    Ricker wavelet, and a little noise."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = torch.rand(16, 3, generator=g, device=DEV)
    t = torch.arange(nt, device=DEV)[:, None] * dt
    x = torch.as_tensor(np.asarray(offsets, np.float32), device=DEV)[None, :]
    out = 1e-3 * torch.randn(nt, x.shape[1], generator=g, device=DEV)
    for k in range(16):
        t0, v = float(u[k, 0]) * nt * dt * 0.9, 1600.0 + 1500.0 * float(u[k, 1])
        a = ((t - torch.sqrt(t0 * t0 + (x / v) ** 2) - 1.0 / fdom) * (PI * fdom)) ** 2
        out += (float(u[k, 2]) - 0.3) * (1 - 2 * a) * torch.exp(-a)
    return np.ascontiguousarray(out.cpu().numpy(), dtype=np.float32)


def _raw_shape(c):
    """Samples and sampling interval of the recorded traces."""
    if c["kind"] == "resample" and c["nt"] % 2:
        return c["nt"], c["dt"]      # resampled in x only
    return c["nt"] // 2, 2 * c["dt"]


def _gathers(c, seed):
    out = []
    for k in _shots(c):
        x1, x2, src, rec, nrec = _window(c, k)
        if c["kind"] == "field":
            nt0, dt0 = _raw_shape(c)
            out.append(_events(nt0, dt0, np.arange(c["traces"]) * c["factor"] * c["d"], c["fdom"], seed * 131 + k))
        else:
            out.append(_events(c["nt"], c["dt"], (np.arange(nrec) + rec - src) * c["d"], c["fdom"], seed * 131 + k))
    return out


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    if c["kind"] == "resample":
        nt0, dt0 = _raw_shape(c)
        return dict(c=c, dt0=dt0, obs=_events(nt0, dt0, np.arange(c["traces"]) * c["factor"] * c["d"], c["fdom"], seed))
    s, o, shots = _survey(c), _options(c), _shots(c)
    true, smooth, rho = _models(c, seed)
    st = dict(c=c, s=s, o=o, shots=shots, true=true, rho=rho)
    if c["kind"] == "forward":
        return st
    geoms = None if c["layout"] == 2 and c["kind"] != "field" else [_shot_geometry(c, k) for k in shots]
    vp = true if c["mode"] == 0 else smooth
    ss = st["ss"] = G.Session(s, o, shots, vp, rho, vp_mig=smooth if c["mode"] == 0 and c["kind"] == "migrate" else None,
                              rho_mig=rho if c["mode"] == 0 and c["kind"] == "migrate" else None, geometries=geoms)
    if c["mode"] == 1:
        st["gathers"] = _gathers(c, seed)
        if c["kind"] == "migrate":
            for k, g in enumerate(st["gathers"]):
                ss.set_gather(k, g)
    if c["kind"] != "model":
        ss.prepare(0, len(shots))
    return st


def run(st):
    c = st["c"]
    if c["kind"] == "resample":
        return G.interp_gather(st["obs"], c["nx"], c["nt"], float(np.float32(c["dt"])), float(np.float32(st["dt0"])), 1)
    if c["kind"] == "forward":
        return dict(zip(("p", "vx", "vz", "gather"), G.forward(st["s"], st["o"], 1, st["true"], st["rho"], c["nt"])))
    ss = st["ss"]
    if c["kind"] == "model":
        ss.model()
        return [ss.gather(k) for k in range(len(st["shots"]))]
    ss.reset_images()
    if c["kind"] == "field":
        for k, g in enumerate(st["gathers"]):
            ss.set_gather_raw(k, g, float(np.float32(_raw_shape(c)[1])), 1)
    ss.run()
    out = dict(ss.images())
    if c["extra"]:
        out.update(ss.images_extra())
    if c["mode"] == 0:
        out["gathers"] = [ss.gather(k) for k in range(len(st["shots"]))]
    return out


# ---- what a pass cannot do without ----------------------------------------------------------
def _sizes(c):
    """(padded cells, interior cells, strip cells, receivers) summed over the shots."""
    p = c["npml"]
    cells = inner = strips = recs = 0
    for k in _shots(c):
        x1, x2, _, _, nrec = _window(c, k)
        n = x2 - x1 + 1
        cells += (n + 2 * p) * (c["nz"] + 2 * p)
        inner += n * c["nz"]
        strips += 40 * (n + c["nz"])
        recs += nrec
    return cells, inner, strips, recs


def _cell_steps(c):
    cells, inner, _, _ = _sizes(c)
    passes = 1 if c["kind"] in ("forward", "model") else 2
    return (passes * cells + (inner if passes == 2 else 0)) * c["nt"]


def work(case):
    c = dict(DEFAULTS, **case)
    if c["kind"] == "resample":
        nt0 = _raw_shape(c)[0]
        n = nt0 * c["traces"]
        m = c["nt"] * c["nx"]
        return {"bytes": 4.0 * (n + m), "flops": 5.0 * 3 * n * c["factor"] ** 2 * math.log2(max(2, n)) + 42.0 * m}
    cells, inner, strips, recs = _sizes(c)
    nt = c["nt"]
    # per cell and step of a propagation: p, vx, vz read and written, 1/rho and kappa read, four
    # derivatives of 10 taps (3 operations each) and the updates
    full, b, f = 32.0 * cells, 0.0, 130.0 * cells
    if c["kind"] in ("forward", "model"):
        return {"bytes": nt * (full + 4.0 * recs), "flops": nt * f}
    sb = 4.0 if c["strips"] == "fp32" else 2.0
    acc = 8.0 if c["accum"] in (1, 2) else 4.0
    b = 2 * full + 32.0 * inner                      # source and receiver passes, reconstruction
    b += 2 * sb * strips                             # strips written and read
    b += (4.0 * acc + 4.0) * inner                   # g1 and illum read and written, ps read
    b += (4.0 if c["gathers"] == "fp32" else 2.0) * recs * (1 + (c["mode"] == 0))
    if c["extra"]:
        b += (4 * 8.0 + 8 * 4.0) * inner
    return {"bytes": nt * b, "flops": nt * (2 * f + 134.0 * inner)}


# ---- the same in 64 bits ---------------------------------------------------------------------
def _taps(first):
    """[11][20] tap weights of half-orders 0..10; the taps start at offset -10 + first (pressure
    0: v[n+i-1] - v[n-i]; velocity 1: p[n+i] - p[n+1-i])."""
    t = torch.zeros(11, 20, dtype=torch.float64)
    for r, row in enumerate(TABLE, 1):
        for i, w in enumerate(row, 1):
            w = float(np.float32(w))
            t[r, 10 + i - 1] += w
            t[r, 10 - i] -= w
    return t


class _Deriv:
    """Derivative along the last axis, half-order per output node, as a product of column blocks
    with small banded matrices."""

    BLOCK = 96

    def __init__(self, n, order, first):
        self.n, self.first = n, first
        nb = -(-n // self.BLOCK)
        w = torch.zeros(nb, self.BLOCK + 19, self.BLOCK, dtype=torch.float64)
        t = _taps(first)
        for k in range(n):
            b, o = divmod(k, self.BLOCK)
            w[b, o:o + 20, o] = t[int(order[k])]
        self.w, self.nb = w.to(DEV), nb

    def __call__(self, f):
        lead = f.shape[:-1]
        f = f.reshape(-1, self.n)
        f = torch.nn.functional.pad(f, (10 - self.first, self.nb * self.BLOCK + 9 + self.first - self.n))
        blocks = f.unfold(1, self.BLOCK + 19, self.BLOCK).transpose(0, 1)
        out = torch.bmm(blocks, self.w).transpose(0, 1).reshape(f.shape[0], -1)[:, :self.n]
        return out.reshape(*lead, self.n)


class _Edge:
    """The pressure derivative along the last axis on lines where the order is also bounded by the
    distance across (the outer ten lines of each side)."""

    def __init__(self, n, across):
        self.n = n
        lines = [k for k in range(across) if min(k, across - 1 - k) < 10]
        self.lines = torch.tensor(lines, device=DEV)
        along = torch.tensor([min(k, n - 1 - k, 10) for k in range(n)])
        bound = torch.tensor([min(k, across - 1 - k, 10) for k in lines])
        self.w = _taps(0)[torch.minimum(along[None, :], bound[:, None])].to(DEV)   # [lines, n, 20]

    def __call__(self, f):   # f [..., lines, n]
        return (torch.nn.functional.pad(f, (10, 9)).unfold(-1, 20, 1) * self.w).sum(-1)


class _Grid:
    """One window size: derivatives and damping of its padded grid."""

    def __init__(self, c, X, vmax):
        p, d, dt = c["npml"], c["d"], float(np.float32(c["dt"]))
        Z = c["nz"] + 2 * p
        self.X, self.Z, self.p, self.dt, self.h = X, Z, p, dt, dt / d
        T = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV)  # noqa: E731
        vo = lambda n: [min(k + 1, n - 1 - k, 10) for k in range(n)]  # noqa: E731
        po = lambda n: [min(k, n - 1 - k, 10) for k in range(n)]  # noqa: E731
        self.vx_d, self.vz_d = _Deriv(X, vo(X), 1), _Deriv(Z, vo(Z), 1)
        self.px_d, self.pz_d = _Deriv(X, po(X), 0), _Deriv(Z, po(Z), 0)
        self.px_e, self.pz_e = _Edge(X, Z), _Edge(Z, X)
        d0 = 1.5 * vmax * math.log(1e10) / (p * d)

        def profile(n, half):
            k = np.arange(n, dtype=np.float64)
            left = np.where(k < p, p - k - half, 0.0)
            right = np.where(k >= n - p, k - n + p + 1 - half, 0.0)
            return d0 * ((left + right) / p) ** 2

        def factors(prof):
            c1 = 1.0 - 0.5 * dt * prof
            return T(c1), T(1.0 / (2.0 - c1))

        self.ax, self.bx = factors(profile(X, 0.0))
        self.az, self.bz = (t[:, None] for t in factors(profile(Z, 0.0)))
        self.avx, self.bvx = factors(np.append(profile(X - 1, 0.5), 0.0))
        self.avz, self.bvz = (t[:, None] for t in factors(np.append(profile(Z - 1, 0.5), 0.0)))
        kx, kz = torch.arange(X, device=DEV), torch.arange(Z, device=DEV)[:, None]
        inx, inz = (kx >= p) & (kx < X - p), (kz >= p) & (kz < Z - p)
        self.inner = inx & inz
        self.live = (kx > 0) & (kx < X - 1) & (kz > 0) & (kz < Z - 1)
        self.rvx = inz & (kx >= p) & (kx <= X - p - 2)
        self.rvz = inx & (kz >= p) & (kz <= Z - p - 2)

    def dz(self, op, f):
        return op(f.transpose(-1, -2)).transpose(-1, -2)

    def div(self, vx, vz):
        ex, ez = self.px_d(vx), self.dz(self.pz_d, vz)
        ex[..., self.px_e.lines, :] = self.px_e(vx[..., self.px_e.lines, :])
        cols = self.pz_e.lines
        ez[..., :, cols] = self.pz_e(vz[..., :, cols].transpose(-1, -2)).transpose(-1, -2)
        return ex * self.h, ez * self.h

    def forward(self, w, ir, ka):
        w["vx"] = (self.avx * w["vx"] - self.vx_d(w["p"]) * self.h * ir) * self.bvx
        w["vz"] = (self.avz * w["vz"] - self.dz(self.vz_d, w["p"]) * self.h * ir) * self.bvz
        w["vx"][..., :, self.X - 1] = 0
        w["vz"][..., self.Z - 1, :] = 0
        ex, ez = self.div(w["vx"], w["vz"])
        ex, ez = ex * ka, ez * ka
        band = self.live & ~self.inner
        w["sx"] = torch.where(band, (self.ax * w["sx"] - ex) * self.bx, w["sx"])
        w["sz"] = torch.where(band, (self.az * w["sz"] - ez) * self.bz, w["sz"])
        w["p"] = torch.where(self.inner, w["p"] - (ex + ez), torch.where(band, w["sx"] + w["sz"], w["p"]))

    def strips(self, w):
        p, X, Z = self.p, self.X, self.Z
        r, q = slice(p, Z - p), slice(p, X - p)
        return [w["vx"][:, r, p - 10:p], w["vx"][:, r, X - p - 1:X - p + 9], w["vz"][:, p - 10:p, q],
                w["vz"][:, Z - p - 1:Z - p + 9, q], w["p"][:, r, p - 10:p], w["p"][:, r, X - p:X - p + 10],
                w["p"][:, p - 10:p, q], w["p"][:, Z - p:Z - p + 10, q]]

    def backward(self, w, ir, ka, later, now):
        for dst, src in zip(self.strips(w)[:4], later[:4]):
            dst.copy_(src)
        w["vx"] += torch.where(self.rvx, self.vx_d(w["p"]) * self.h * ir, 0.0)
        w["vz"] += torch.where(self.rvz, self.dz(self.vz_d, w["p"]) * self.h * ir, 0.0)
        for dst, src in zip(self.strips(w)[4:], now[4:]):
            dst.copy_(src)
        ex, ez = self.px_d(w["vx"]) * self.h * ka, self.dz(self.pz_d, w["vz"]) * self.h * ka
        w["p"] += torch.where(self.inner, ex + ez, 0.0)


def _field(B, g):
    return {k: torch.zeros(B, g.Z, g.X, dtype=torch.float64, device=DEV) for k in ("p", "vx", "vz", "sx", "sz")}


def _pad(v, x1, x2, p):
    return np.pad(v[:, x1:x2 + 1].astype(np.float64), p, mode="edge")


def _mute(c, gather, v2, shot):
    """Zero every trace up to the direct wave's end."""
    x1, x2, src, rec, nrec = _window(c, shot)
    p, d = c["npml"], np.float32(c["d"])
    dt, f = np.float32(c["dt"]), np.float32(c["fdom"])
    nw = int(np.float32(_direct(c)) / (f * dt))
    row = np.sqrt(v2[p + c["depth"], p + rec:p + rec + nrec].astype(np.float32)).astype(np.float64)
    at = float(np.sqrt(np.float32(v2[p + 2, p + src])))
    vt = (0.482 * (1.0 / row + 1.0 / at)).astype(np.float32)
    k = np.arange(nrec) + rec - src
    dist = np.sqrt((k * k).astype(np.float32) * (d * d) + np.float32((c["depth"] - 2) ** 2) * (d * d)).astype(np.float32)
    cut = np.minimum((dist * vt * np.float32(1.0 / float(dt))).astype(np.int64) + nw, c["nt"])
    out = gather.copy()
    out[np.arange(c["nt"])[:, None] <= cut[None, :]] = 0
    return out


def _resample(obs, nx, nt, dt, dt0):
    """F-K interpolation in x (general beyond-alias form), then a 21-tap Kaiser-windowed sinc."""
    nt0, nx0 = obs.shape
    a = torch.as_tensor(obs, device=DEV).to(torch.float64).T.contiguous()     # [nx0][nt0]
    if nx > nx0:
        lx = (nx - 1) // (nx0 - 1)
        nf = 1 + nt0 // 2
        K = torch.fft.fft2(a)[:, :nf]
        S = torch.fft.fft2(a, s=(lx * nx0, lx * nt0))
        fold = S.reshape(lx, nx0, lx * nt0).sum(0) / lx
        eps = float(fold.abs().max()) * 1e-5
        H = S[:, :nf] / (fold[:, :nf] + eps).repeat(lx, 1)
        H = torch.where(H.abs() > lx * lx, torch.full_like(H, lx), H)
        g = torch.fft.ifft(H * K.repeat(lx, 1), dim=0, norm="forward")[:nx]
        full = torch.zeros(nx, nt0, dtype=torch.complex128, device=DEV)
        full[:, :nf] = g
        for k in range(nf, nt0):
            full[:, k] = g[:, nt0 - k].conj()
        a = torch.fft.ifft(full, dim=1, norm="forward").real.contiguous()
    a = a[:nx].T.cpu().numpy()                                               # [nt0][nx]
    if nt <= nt0:
        return a[:nt]
    dt, dt0 = np.float32(dt), np.float32(dt0)
    wk = np.i0(2.0 * np.sqrt(np.maximum(0.0, 1 - ((np.arange(21) - 10) / 10.0) ** 2))) / np.i0(2.0)
    out = np.zeros((nt, nx))
    for it in range(nt):
        mid = int(np.float32(it + 1) * dt / dt0)
        lo, hi = max(0, mid - 10), min(nt0 - 1, mid + 10)
        shift = 21 - (hi - lo + 1) if lo <= 10 else 0
        u = it * float(dt) / float(dt0) - np.arange(lo, hi + 1)
        out[it] = (np.sinc(u) * wk[shift:shift + hi - lo + 1]) @ a[lo:hi + 1]
    return out


def exact(case, seed):
    c = dict(DEFAULTS, **case)
    if c["kind"] == "resample":
        st = prepare(case, seed)
        return _resample(st["obs"], c["nx"], c["nt"], c["dt"], st["dt0"])
    shots = _shots(c)
    sizes = len({_window(c, k)[1] - _window(c, k)[0] for k in shots})
    # smoothed models are prepared by the library's own iterations, and the weights of the other
    # imaging conditions switch on the signs of rounded products: no 64-bit value for those
    steps = c["nt"] * (3 if c["kind"] in ("migrate", "field") else 1)
    if c["smooth"] or c["pmlsmooth"] or _cell_steps(c) * 4e-11 * 8 + steps * sizes * 3e-3 > 60:
        return None
    true, smooth, rho = _models(c, seed)
    gathers = _gathers(c, seed) if c["mode"] == 1 and c["kind"] in ("migrate", "field") else None
    p, d, dt, nt = c["npml"], c["d"], float(np.float32(c["dt"])), c["nt"]
    wt = (PI * c["fdom"] * np.abs(np.arange(nt) * dt - 1.0 / c["fdom"])) ** 2
    wavelet = (1.0 - 2.0 * wt) * np.exp(-wt)
    alp = float(np.float32(1.0 / d))
    T = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV)  # noqa: E731
    img = {k: np.zeros((c["nz"], c["nx"])) for k in ("image1", "image2s", "image2m", "illum")}
    recorded, last = [None] * len(shots), {}
    groups = {}
    for j, k in enumerate(shots):
        x1, x2 = _window(c, k)[:2]
        groups.setdefault(x2 - x1 + 1, []).append((j, k))
    parts = [m[i:i + 16] for m in groups.values() for i in range(0, len(m), 16)]
    fwd_model = true if c["mode"] == 0 or c["kind"] == "forward" else smooth
    for members in parts:
        B = len(members)
        wins = [_window(c, k) for _, k in members]
        vf = [_pad(fwd_model, w[0], w[1], p) for w in wins]
        vb = [_pad(smooth, w[0], w[1], p) for w in wins]
        rh = [_pad(rho, w[0], w[1], p) for w in wins]
        X = vf[0].shape[1]
        g = _Grid(c, X, float(vf[0].max()))
        same = c["layout"] == 2 and c["kind"] != "field"
        pick = (lambda a: T(a[0])[None]) if same else (lambda a: T(np.stack(a)))
        ir, kf = 1.0 / pick(rh), pick(rh) * pick(vf) ** 2
        kb = pick(rh) * pick(vb) ** 2
        zz, xx = np.arange(g.Z)[:, None] - (p + 2), np.arange(X)[None, :]
        src = T(np.stack([dt * np.exp(-alp * alp * d * d * ((xx - p - w[2]) ** 2 + zz ** 2)) for w in wins]))
        rz = p + c["depth"]
        cols = [slice(p + w[3], p + w[3] + w[4]) for w in wins]
        w, saved = _field(B, g), []
        rec = [torch.zeros(nt, wi[4], dtype=torch.float64, device=DEV) for wi in wins]
        for it in range(nt):
            g.forward(w, ir, kf)
            w["p"] += src * float(wavelet[it])
            if c["mode"] == 0 or c["kind"] == "forward":
                for b in range(B):
                    rec[b][it] = w["p"][b, rz, cols[b]]
            if steps > nt:
                saved.append([s.clone() for s in g.strips(w)])
        for b, (j, _) in enumerate(members):
            recorded[j] = rec[b].cpu().numpy()
        if c["kind"] == "forward":
            last = {"p": w["p"][0].cpu().numpy(), "vx": w["vx"][0, :, :X - 1].cpu().numpy(),
                    "vz": w["vz"][0, :g.Z - 1].cpu().numpy()}
        if steps == nt:
            continue
        data = []
        for b, (j, k) in enumerate(members):
            if c["mode"] == 0:
                seis = recorded[j]
            elif c["kind"] == "field":
                seis = _resample(gathers[j], wins[b][4], nt, c["dt"], _raw_shape(c)[1])
            else:
                seis = gathers[j].astype(np.float64)
            data.append(T(_mute(c, seis, (vb if c["kind"] == "field" else vf)[b] ** 2, k)))
        back, w = w, _field(B, g)
        back["vx"].zero_()
        back["vz"].zero_()

        def inject(it):
            for b in range(B):
                w["p"][b, rz, cols[b]] = dt * data[b][it]

        inject(nt - 1)
        inner = (slice(None), slice(p, g.Z - p), slice(p, X - p))
        g1 = torch.zeros_like(w["p"][inner])
        il = torch.zeros_like(g1)
        for it in range(nt - 2, -1, -1):
            g.backward(back, ir, kb, saved[it + 1], saved[it])
            back["p"] -= src * float(wavelet[it])
            g.forward(w, ir, kb)
            inject(it)
            ps = back["p"][inner]
            g1 += ps * w["p"][inner]
            il += ps * ps
        n = X - 2 * p
        nwin = 50
        while 2 * nwin >= n:
            nwin -= 3
        k = np.arange(n)
        taper = np.where(k < nwin, np.exp(-0.0036 * (nwin - k) ** 2.0), 1.0)
        taper = np.where(k >= n - nwin, np.exp(-0.0036 * (k - n + nwin + 1) ** 2.0), taper)
        for b, wi in enumerate(wins):
            gg, ii = g1[b].cpu().numpy() * taper, il[b].cpu().numpy() * taper
            at = (slice(None), slice(wi[0], wi[1] + 1))
            img["image1"][at] += gg
            img["image2m"][at] += gg
            img["image2s"][at] += gg / (ii + 1e-6)
            img["illum"][at] += ii
    if c["kind"] == "forward":
        return dict(last, gather=recorded[0])
    if c["kind"] == "model":
        return recorded
    out = dict(img)
    if c["extra"]:
        out.update({k: None for k in G.Session.EXTRA_IMAGES})
    if c["mode"] == 0:
        out["gathers"] = recorded
    return out
