"""Cases of the engine's performance measurement.

A case is one piece of work that a user of the engine has it do through the
public Python layer: advance a deck by some RK4 steps, read the observables
the deck's output schedule asks for and take a snapshot of the state, or run
the discrete adjoint forward and backward, or advance a batched sweep.

`exact` restates the same runs in plain torch, 64-bit, without the engine.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The engine's Python package (its folder name is not an identifier)."""
    if "goferro_b200" not in sys.modules:
        path = os.path.join(_ROOT, "go-ferro_b200")
        spec = importlib.util.spec_from_file_location("goferro_b200", os.path.join(path, "__init__.py"),
                                                      submodule_search_locations=[path])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["goferro_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["goferro_b200"]


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # Ferromagnetic film with per-stage FFT magnetostatics.
        # The smallest grid (the finite-difference copy of the adjoint study),
        # <m> written after every step as the reference's loop does: latency
        # and launches.
        dict(name="fm_32x32x8_fp64", kind="fm", nx=32, ny=32, nz=8, precision="fp64", steps=20, every=1),
        # The benchmark's FM + magnetostatics film, both arithmetic forms.
        dict(name="fm_64x64x16_fp64", kind="fm", nx=64, ny=64, nz=16, precision="fp64", steps=40, every=40),
        dict(name="fm_64x64x16_mixed", kind="fm", nx=64, ny=64, nz=16, precision="mixed", steps=40, every=40),
        # A film whose sides are not powers of two.
        dict(name="fm_120x90x20_fp64", kind="fm", nx=120, ny=90, nz=20, precision="fp64", steps=20, every=20),
        # Ferroelectric TDGL + electrostriction + elastodynamics + FDTD:
        # one sweep-sized instance, a ragged grid, and the headline 128^3 run
        # in both forms.
        dict(name="fe_48x48x32_mixed", kind="fe", nx=48, ny=48, nz=32, precision="mixed", steps=20, every=20),
        dict(name="fe_75x61x37_fp64", kind="fe", nx=75, ny=61, nz=37, precision="fp64", steps=10, every=10),
        dict(name="fe_128x128x128_fp64", kind="fe", nx=128, ny=128, nz=128, precision="fp64", steps=4, every=4),
        dict(name="fe_128x128x128_mixed", kind="fe", nx=128, ny=128, nz=128, precision="mixed", steps=4, every=4),
        # Magnetoelastic film on a substrate under vacuum + FDTD, the
        # benchmark's coupled film in both forms.
        dict(name="me_128x128x96_fp64", kind="me", nx=128, ny=128, nz=96, precision="fp64", steps=4, every=4),
        dict(name="me_128x128x96_mixed", kind="me", nx=128, ny=128, nz=96, precision="mixed", steps=4, every=4),
        # Gradients of a band response of <m_x>: forward and backward run of
        # the adjoint on the adjoint study's 256x256x32 film (FP32 form).
        dict(name="adjoint_256x256x32_mixed", kind="adjoint", nx=256, ny=256, nz=32, precision="mixed", steps=12, every=6),
        # Batched sweep: instances of uneven grids advanced by one graph.
        dict(name="sweep_12_mixed", kind="sweep", precision="mixed", steps=10, every=10,
             grids="32x32x32,96x96x24,48x48x32,64x64x32,32x32x32,64x64x32,48x48x32,96x96x24,64x64x32,32x32x32,48x48x32,96x96x24"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(v, factors=(2, 3, 5)):
    """The next size at or below v that FFT users pick (factors 2, 3 and 5)."""
    while True:
        r = v
        for f in factors:
            while r % f == 0:
                r //= f
        if r == 1:
            return v
        v -= 1


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["fm", "fm", "fe", "fe", "me", "adjoint", "sweep"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "fm":
        # most users pick smooth sides; a few take what the film measures
        sm = (lambda v: v) if rng.random() < 0.25 else _smooth
        c = dict(kind=kind, nx=sm(_log_int(rng, 24, 256)), ny=sm(_log_int(rng, 24, 192)), nz=sm(_log_int(rng, 4, 32)),
                 precision=prec)
        c["steps"] = max(4, min(40, int(2.6e6 / (c["nx"] * c["ny"] * c["nz"]))))
        c["every"] = rng.choice([1, c["steps"]])
        return c
    if kind in ("fe", "me"):
        nz = _log_int(rng, 16 if kind == "me" else 10, 120)
        nx = _log_int(rng, 24, 128)
        ny = max(nz, _log_int(rng, 24, 128))
        if rng.random() < 0.5:
            nx, ny, nz = nx // 16 * 16 or 16, (ny + 15) // 16 * 16, nz // 16 * 16 or 16
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=prec)
        c["steps"] = max(4, min(20, int(2.0e6 / (nx * ny * nz))))
        c["every"] = c["steps"]
        return c
    if kind == "adjoint":
        c = dict(kind=kind, nx=_smooth(_log_int(rng, 32, 256)), ny=_smooth(_log_int(rng, 32, 192)),
                 nz=_smooth(_log_int(rng, 8, 32)), precision="mixed" if rng.random() < 0.7 else "fp64")
        c["steps"] = 12
        c["every"] = rng.choice([4, 6])
        return c
    sizes = ["32x32x32", "48x48x32", "64x64x32", "96x96x24"]
    return dict(kind=kind, precision="mixed", steps=10, every=10,
                grids=",".join(rng.choice(sizes) for _ in range(rng.randint(3, 12))))


# --------------------------------------------------------------------------
# decks
# --------------------------------------------------------------------------
def _tilted(rng, shape, inside, max_deg=1.0):
    th = np.deg2rad(max_deg) * rng.random(shape)
    ph = 2.0 * np.pi * rng.random(shape)
    return np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)]) * inside[None]


def _wave(d, rng):
    """An acoustic pulse in flight: ~1 pm displacement with a lateral ripple,
    and the velocity it moves with."""
    x = (np.arange(d.nx) + 0.5)[:, None, None] / d.nx
    y = (np.arange(d.ny) + 0.5)[None, :, None] / d.ny
    z = (np.arange(d.nz) + 0.5)[None, None, :] / d.nz
    zc, w = rng.uniform(0.3, 0.7), rng.uniform(0.1, 0.25)
    solid = (d.material_cell() != 0)
    u = []
    for _ in range(3):
        a, b, ph = rng.uniform(0.3, 1.0), rng.uniform(0.1, 0.3), rng.uniform(0.0, 2 * np.pi)
        u.append(1e-12 * a * np.exp(-0.5 * ((z - zc) / w) ** 2) * (1.0 + b * np.cos(2 * np.pi * (x + y) + ph)) * solid)
    d.u0 = np.stack(u)
    d.v0 = -4e3 * np.gradient(d.u0, d.dz, axis=3)
    return d


def _fe_deck(D, nx, ny, nz, rng, steps):
    d = D.preset_ferroelectric(nx=nx, ny=ny, nz=nz, steps=steps)
    d.p0 = rng.uniform(-1e-3, 1e-3, (3, nx, ny, nz))
    d.q0 = np.zeros_like(d.p0)
    return _wave(d, rng)


def _decks(case, seed):
    """The deck of a case (a list of them for a sweep), made from the seed."""
    D = _package().decks
    rng = np.random.default_rng([int(seed), 20241203])
    kind = case["kind"]
    if kind == "sweep":
        out = []
        for g in case["grids"].split(","):
            nx, ny, nz = (int(v) for v in g.split("x"))
            d = _fe_deck(D, nx, ny, nz, rng, 8000)
            # z-polarised Gaussian x sine sheet current, 10-500 kV/cm, 0.5-3 THz
            d.jf_type = 6
            d.jf_freq = rng.uniform(0.5e12, 3e12)
            d.jf_sigma = 8000 * d.dt / 10.0
            d.jf_amp *= 10.0 ** rng.uniform(1.0, math.log10(500.0)) / 100.0
            out.append(d)
        return out
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "fm":
        d = D.preset_fm_demag(nx=nx, ny=ny, nz=nz, steps=4000)
        d.m0 = _tilted(rng, (nx, ny, nz), d.material_cell() != 0)
    elif kind == "fe":
        d = _fe_deck(D, nx, ny, nz, rng, 40000)
    elif kind == "me":
        # the benchmark's layer stack, 56 : 32 : 8 of 96
        sub = max(5, round(nz * 56 / 96))
        film = min(nz - sub, max(2, round(nz * 32 / 96)))
        d = D.preset_magnetoelastic(nx=nx, ny=ny, nz=nz, sub=sub, film=film)
        d.m0 = _tilted(rng, (nx, ny, nz), d.material_cell() == 2)
        _wave(d, rng)
    elif kind == "adjoint":
        # free magnetoelastic film, 1 T bias, Liao boundary at k = 0
        d = D.preset_fm_demag(nx=nx, ny=ny, nz=nz, steps=case["steps"])
        d.Hext_table = None
        d.Hext_stat = (0.0, 0.0, 1.0 / D.MU0)
        d.materials = [D.yig(1e-3, magnetoelastic=True)]
        d.elastic = d.elasto_back = d.elasto_on = True
        d.abc_1D, d.liao_w = False, 0.5
        d.m0 = _tilted(rng, (nx, ny, nz), d.material_cell() != 0)
    else:
        raise ValueError(kind)
    return d


def _adjoint_inputs(case, seed, n, mu0):
    rng = np.random.default_rng([int(seed), 20241208])
    nw = 256
    alpha = 1e-3 * (1.0 + 0.1 * rng.random(n))
    tt = (np.arange(nw) + 0.5) / nw
    wave = (1e-3 / mu0) * np.sin(2 * np.pi * 8 * tt) * np.exp(-((tt - 0.3) / 0.1) ** 2) * rng.uniform(0.5, 1.5)
    return alpha, wave


def _trace_cotangent(tr):
    """d loss / d <m_x>(t) of the in-phase response of the trace at its first
    seven harmonics (a lock-in reading of the band)."""
    n = np.arange(tr.size)
    return sum(2.0 / k * np.cos(2 * np.pi * k * n / tr.size + 0.3 * k) for k in range(1, 8))


# --------------------------------------------------------------------------
# the runs
# --------------------------------------------------------------------------
_SNAPSHOT = {"fm": ("m",), "fe": ("p", "q", "u", "v", "Ex", "Ey", "Ez", "Hx", "Hy", "Hz"),
             "me": ("m", "u", "v", "Ex", "Ey", "Ez", "Hx", "Hy", "Hz"), "sweep": ("p", "q", "u", "Ez", "Hx")}
_OBS = {"fm": ("m",), "fe": ("p", "u"), "me": ("m", "u"), "sweep": ("p",)}


def _buffers(eng, names):
    out = {}
    for f in names:
        dims, count = eng.field_dims(f)
        nc = count // (dims[0] * dims[1] * dims[2])
        out[f] = torch.empty(((nc,) if nc > 1 else ()) + tuple(dims), dtype=torch.float64, device="cuda")
    return out


def prepare(case, seed):
    gf = _package()
    kind = case["kind"]
    if kind == "sweep":
        decks = _decks(case, seed)
        engines = [gf.Engine.from_params(d, device=0, precision=case["precision"]) for d in decks]
        batch = gf.Batch(engines, autotune=True)
        # a sweep of up to twelve instances keeps a snapshot of the first two
        bufs = [_buffers(e, _SNAPSHOT["sweep"]) for e in engines[:2]]
        return dict(case=case, engines=engines, batch=batch, bufs=bufs,
                    streams=[torch.cuda.ExternalStream(e.stream()) for e in engines])
    d = _decks(case, seed)
    eng = gf.Engine.from_params(d, device=0, precision=case["precision"])
    st = dict(case=case, eng=eng, stream=torch.cuda.ExternalStream(eng.stream()))
    if kind == "adjoint":
        alpha, wave = _adjoint_inputs(case, seed, d.n, gf.decks.MU0)
        adj = gf.Adjoint(eng, wave.size, case["every"])
        adj.set_alpha(alpha)
        adj.set_waveform(wave)
        st.update(adj=adj)
    else:
        st["bufs"] = _buffers(eng, _SNAPSHOT[kind])
        st["probe"] = (case["nx"] // 2, case["ny"] // 2, case["nz"] // 2)
    return st


def _snapshot(eng, bufs, stream, single):
    """The engine's fields into device buffers; a mixed-form run keeps FP32
    snapshots (the resolution its state has)."""
    fields = _package().FIELD
    for f, b in bufs.items():
        rc = eng.lib.gf_download_device(eng.h, fields[f], ctypes.c_void_p(b.data_ptr()), b.numel())
        if rc != 0:
            raise RuntimeError("gf_download_device: %d" % rc)
    if not single:
        return dict(bufs)
    with torch.cuda.stream(stream):
        return {f: b.float() for f, b in bufs.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    single = case["precision"] == "mixed"
    ftype = np.float32 if single else np.float64
    if kind == "adjoint":
        adj = state["adj"]
        tr = adj.forward(case["steps"])
        gw, ga = adj.backward(_trace_cotangent(tr))
        return {"trace": tr.astype(ftype), "grad_wave": gw.astype(ftype), "grad_alpha": ga.astype(ftype)}
    if kind == "sweep":
        state["batch"].advance(case["steps"])
        state["batch"].synchronize()
        out = {"snapshots": [_snapshot(e, b, s, single) for e, b, s in zip(state["engines"], state["bufs"], state["streams"])]}
        out["P"] = np.stack([e.average("p") for e in state["engines"]]).astype(ftype)
        return out
    eng = state["eng"]
    rows = []
    for _ in range(case["steps"] // case["every"]):
        eng.advance(case["every"])
        if len(rows) + 1 < case["steps"] // case["every"]:
            rows.append(np.concatenate([eng.average(o) for o in _OBS[kind]]))
    out = _snapshot(eng, state["bufs"], state["stream"], single)
    rows.append(np.concatenate([eng.average(o) for o in _OBS[kind]]))
    rows = np.stack(rows)
    for q, o in enumerate(_OBS[kind]):
        out["<%s>" % o] = rows[:, 3 * q:3 * q + 3].astype(ftype)
    if kind in ("fe", "me"):
        e, h = eng.probe_em(*state["probe"])
        out["probe_E"], out["probe_H"] = e.astype(ftype), h.astype(ftype)
    return out


def work(case):
    """Bytes: every RK stage reads the state it starts from and writes the one
    it ends with once (a stage's stencils need its neighbours' stage values,
    and the state is larger than the chip), plus the snapshot.  The adjoint
    does a forward run and, backward, each step's stages again and their
    transposes."""
    es = 4.0 if case["precision"] == "mixed" else 8.0
    kind = case["kind"]
    if kind == "sweep":
        cells = 0
        for g in case["grids"].split(","):
            a, b, c = (int(v) for v in g.split("x"))
            cells += a * b * c
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    # state scalars per cell, flops per cell and stage
    scal, fl = {"fm": (3.0, 350.0), "fe": (18.0, 600.0), "me": (13.0, 400.0), "adjoint": (9.0, 700.0),
                "sweep": (18.0, 600.0)}[kind]
    passes = 3.0 if kind == "adjoint" else 1.0
    return {"bytes": cells * es * scal * (case["steps"] * 4 * 2 * passes + 1.0), "flops": cells * fl * 4 * case["steps"] * passes}


# --------------------------------------------------------------------------
# the same runs in plain torch, 64-bit
# --------------------------------------------------------------------------
_MU0, _E0, _C0 = 1.256637061e-6, 8.854187817e-12, 2.99792458e8


def _newell_f(x, y, z):
    r = torch.sqrt(x * x + y * y + z * z)
    tiny = 1e-300

    def ash(a, b, c):
        return torch.asinh(a / torch.sqrt(b * b + c * c + tiny))
    return (0.5 * y * (z * z - x * x) * ash(y, x, z) + 0.5 * z * (y * y - x * x) * ash(z, x, y)
            - x * y * z * torch.atan2(y * z * torch.sign(x), torch.abs(x) * r) + (2 * x * x - y * y - z * z) * r / 6.0)


def _newell_g(x, y, z):
    r = torch.sqrt(x * x + y * y + z * z)
    tiny = 1e-300

    def ash(a, b, c):
        return torch.asinh(a / torch.sqrt(b * b + c * c + tiny))

    def at(a, b, c):
        return torch.atan2(a * b * torch.sign(c), torch.abs(c) * r)
    return (x * y * z * ash(z, x, y) + y / 6.0 * (3 * z * z - y * y) * ash(x, y, z) + x / 6.0 * (3 * z * z - x * x) * ash(y, x, z)
            - z ** 3 / 6.0 * at(x, y, z) - z * y * y / 2.0 * at(x, z, y) - z * x * x / 2.0 * at(y, z, x) - x * y * r / 3.0)


def _demag_spectra(shape, h, dev):
    """Spectra of the six distinct cell-averaged demagnetising tensor
    components (Newell, Williams and Dunlop, J. Geophys. Res. 98, 9551, 1993)
    on wrapped offsets below half the period."""
    axes, oks = [], []
    for n in shape:
        a = torch.arange(n, device=dev, dtype=torch.float64)
        half = n // 2
        axes.append(torch.where(a <= half - 1, a, a - n))
        oks.append((a <= half - 1) | (a >= n - half + 1))
    ok = oks[0][:, None, None] & oks[1][None, :, None] & oks[2][None, None, :]
    # the differences are taken in units of the cell so that the far field keeps its digits
    s = h[0]
    X, Y, Z = torch.meshgrid(axes[0] * (h[0] / s), axes[1] * (h[1] / s), axes[2] * (h[2] / s), indexing="ij")
    d = [v / s for v in h]
    w = {0: 2.0, 1: -1.0, -1: -1.0}

    def table(fn, perm):
        c = (X, Y, Z)
        c = [c[p] for p in perm]
        dd = [d[p] for p in perm]
        acc = torch.zeros_like(X)
        for i in w:
            for j in w:
                for k in w:
                    acc += w[i] * w[j] * w[k] * fn(c[0] + i * dd[0], c[1] + j * dd[1], c[2] + k * dd[2])
        acc /= 4 * math.pi * d[0] * d[1] * d[2]
        return torch.fft.rfftn(torch.where(ok, acc, torch.zeros_like(acc)))
    N = {}
    for q, p in (("xx", (0, 1, 2)), ("yy", (1, 2, 0)), ("zz", (2, 0, 1))):
        N[q] = table(_newell_f, p)
    for q, p in (("xy", (0, 1, 2)), ("yz", (1, 2, 0)), ("zx", (2, 0, 1))):
        N[q] = table(_newell_g, p)
    return N


def _demag(N, M):
    k = [torch.fft.rfftn(M[a]) for a in range(3)]
    hx = k[0] * N["xx"] + k[1] * N["xy"] + k[2] * N["zx"]
    hy = k[0] * N["xy"] + k[1] * N["yy"] + k[2] * N["yz"]
    hz = k[0] * N["zx"] + k[1] * N["yz"] + k[2] * N["zz"]
    return -torch.stack([torch.fft.irfftn(v, s=M[0].shape) for v in (hx, hy, hz)])


def _up(f, d):
    return torch.roll(f, -1, d)


def _dn(f, d):
    return torch.roll(f, 1, d)


class _Model:
    """A layered deck (periodic x and y, open z) with constant materials per
    layer; the damping can be a per-cell field."""

    def __init__(self, d, dev):
        self.d, self.dev = d, dev
        self.h = (d.dx, d.dy, d.dz)
        self.shape = (d.nx, d.ny, d.nz)
        mc = torch.from_numpy(d.material_cell().astype(np.int64)).to(dev)
        self.solid = mc != 0

        def tab(fn, vac=0.0):
            t = torch.tensor([vac] + [float(fn(m)) for m in d.materials], dtype=torch.float64, device=dev)
            return t[mc]
        self.fm, self.fe = tab(lambda m: m.fm) > 0, tab(lambda m: m.fe) > 0
        self.has_fm, self.has_fe = bool(self.fm.any()), bool(self.fe.any())
        self.c11, self.c12, self.c44 = tab(lambda m: m.c11), tab(lambda m: m.c12), tab(lambda m: m.c44)
        self.rrho = tab(lambda m: 1.0 / m.density)
        self.er, self.cond = tab(lambda m: m.er, 1.0), tab(lambda m: m.cond)
        self.Ms = tab(lambda m: m.Ms if m.fm else 0.0)
        self.Aex = tab(lambda m: m.Aex if m.fm else 0.0)
        self.K1c = tab(lambda m: m.K1 / _MU0 / m.Ms if m.fm else 0.0)
        self.B1c = tab(lambda m: -1.5 * m.lam100 * (m.c11 - m.c12) / _MU0 / m.Ms if m.fm else 0.0)
        self.B2c = tab(lambda m: -3.0 * m.lam111 * m.c44 / _MU0 / m.Ms if m.fm else 0.0)
        self.exc = tab(lambda m: 2.0 / _MU0 / m.Ms if m.fm else 0.0)
        self.gyro, self.alpha = tab(lambda m: m.gyro if m.fm else 0.0), tab(lambda m: m.alpha if m.fm else 0.0)
        self.l100, self.l111 = tab(lambda m: m.lam100 if m.fm else 0.0), tab(lambda m: m.lam111 if m.fm else 0.0)
        self.Q11, self.Q12, self.Q44 = tab(lambda m: m.Q11), tab(lambda m: m.Q12), tab(lambda m: m.Q44)
        for m in d.materials:
            if m.stiff_damping or m.mass_damping or m.K2 or m.iDMI or (m.fm and m.aniso_type != 1):
                raise ValueError("not covered")
        self.N = _demag_spectra(self.shape, self.h, dev) if (self.has_fm and d.magnetostatics) else None
        fe = [m for m in d.materials if m.fe]
        self.fem = fe[0] if fe else None
        # free z faces (face f between cells f-1 and f; both ends free) and
        # the two-cell masks of the x, y faces
        zf = torch.zeros((d.nx, d.ny, d.nz + 1), dtype=torch.float64, device=dev)
        zf[..., 1:-1] = (self.solid[..., 1:] & self.solid[..., :-1]).double()
        self.zface = zf
        self.xface = (self.solid & _dn(self.solid, 0)).double()
        self.yface = (self.solid & _dn(self.solid, 1)).double()
        ez = torch.zeros((d.nx, d.ny, d.nz + 1), dtype=torch.float64, device=dev)
        self.fmz = ez.clone()
        self.fmz[..., 1:-1] = (self.fm[..., 1:] & self.fm[..., :-1]).double()
        self.fez = ez.clone()
        self.fez[..., 1:-1] = (self.fe[..., 1:] & self.fe[..., :-1]).double()
        if d.elastic:
            m0 = [m for m in [self._mat(0)] if m][0]
            mt = self._mat(d.nz - 1)
            self.vs = (math.sqrt(m0.c11 / m0.density), math.sqrt(m0.c44 / m0.density))
            self.vt = (math.sqrt(mt.c11 / mt.density), math.sqrt(mt.c44 / mt.density)) if mt else (0.0, 0.0)
        if d.em:
            n0, n1 = self._mat(0), self._mat(d.nz - 1)
            self.cb, self.ct = _C0 / math.sqrt(n0.er if n0 else 1.0), _C0 / math.sqrt(n1.er if n1 else 1.0)
            self.edge = [self._edge(c) for c in range(3)]

    def _mat(self, k):
        z = 0
        for n, q in self.d.layers:
            if z <= k < z + n:
                return self.d.materials[q - 1] if q else None
            z += n
        return None

    # cells around an E edge of component c, padded to the edge's z extent
    def _four(self, f, c):
        if c == 2:
            return [f, _dn(f, 0), _dn(f, 1), _dn(_dn(f, 0), 1)]
        t = 1 - c
        g = torch.zeros(self.shape[:2] + (self.shape[2] + 1,), dtype=torch.float64, device=self.dev)
        lo, hi = g.clone(), g.clone()
        hi[..., :-1], lo[..., 1:] = f, f
        return [hi, lo, _dn(hi, t), _dn(lo, t)]

    def _edge(self, c):
        er = sum(self._four(self.er, c)) / 4.0
        er = torch.where(er == 0, torch.ones_like(er), er)
        cond = sum(self._four(self.cond, c)) / 4.0
        cnt = sum(self._four(self.fe.double(), c))
        return er, cond, torch.clamp(cnt, min=1.0)

    # -- magnetisation ----------------------------------------------------
    def h_demag(self, m):
        return _demag(self.N, m * self.Ms) if self.N is not None else torch.zeros_like(m)

    def dm(self, m, hs, hext, strain, alpha, Hc=None):
        H = hs + hext.reshape(3, 1, 1, 1)
        ex = torch.zeros_like(m)
        for dd, mask in ((1, self.fm & _dn(self.fm, 0)), (2, self.fm & _dn(self.fm, 1))):
            g = (m - _dn(m, dd)) * mask.double() / self.h[dd - 1] ** 2
            ex = ex + (_up(g, dd) - g)
        g = torch.zeros((3,) + self.fmz.shape, dtype=torch.float64, device=self.dev)
        g = torch.nn.functional.pad(m[..., 1:] - m[..., :-1], (1, 1)) * self.fmz / self.h[2] ** 2
        ex = ex + (g[..., 1:] - g[..., :-1])
        H = H + self.exc * self.Aex * ex
        x, y, z = m
        H = H + torch.stack([-2 * self.K1c * (y * y + z * z) * x, -2 * self.K1c * (x * x + z * z) * y, -2 * self.K1c * (x * x + y * y) * z])
        if strain is not None:
            e = strain
            H = H - 2 * torch.stack([self.B1c * e[0] * x + self.B2c * (e[5] * y + e[4] * z),
                                     self.B1c * e[1] * y + self.B2c * (e[5] * x + e[3] * z),
                                     self.B1c * e[2] * z + self.B2c * (e[4] * x + e[3] * y)])
        if Hc is not None:
            H = H + Hc
        p = torch.cross(m, H, dim=0)
        q = torch.cross(m, p, dim=0)
        pre = -self.gyro * self.d.dt / (1 + alpha * alpha) * self.fm
        return pre * p + alpha * pre * q

    # -- elasticity -------------------------------------------------------
    def grads(self, u):
        gx = (u - _dn(u, 1)) * self.xface / self.h[0]
        gy = (u - _dn(u, 2)) * self.yface / self.h[1]
        gz = torch.nn.functional.pad(u[..., 1:] - u[..., :-1], (1, 1)) * self.zface / self.h[2]
        T = [gx + _up(gx, 1), gy + _up(gy, 2), gz[..., 1:] + gz[..., :-1]]     # T[d][a]
        return gx, gy, gz, T

    def strain(self, T):
        return torch.stack([T[0][0] / 2, T[1][1] / 2, T[2][2] / 2, (T[2][1] + T[1][2]) / 4, (T[2][0] + T[0][2]) / 4, (T[1][0] + T[0][1]) / 4])

    def eigen(self, m, p):
        e = [torch.zeros(self.shape, dtype=torch.float64, device=self.dev) for _ in range(6)]
        if not self.d.elasto_back:
            return e
        pairs = ((1, 2), (0, 2), (1, 0))
        if m is not None:
            for a in range(3):
                e[a] = e[a] + 1.5 * self.l100 * (m[a] * m[a] - 1.0 / 3.0)
                e[3 + a] = e[3 + a] + 1.5 * self.l111 * m[pairs[a][0]] * m[pairs[a][1]]
        if p is not None:
            s = p * p
            for a in range(3):
                b, c = pairs[a]
                e[a] = e[a] + self.Q11 * s[a] + self.Q12 * (s[b] + s[c])
                e[3 + a] = e[3 + a] + self.Q44 * p[b] * p[c]
        return e

    def force(self, u, e0):
        gx, gy, gz, T = self.grads(u)
        c11, c12, c44 = self.c11, self.c12, self.c44

        def normal(g, d):
            b, c = [q for q in range(3) if q != d]
            return c11 * (g - e0[d]) + c12 * (T[b][b] / 2 - e0[b] + T[c][c] / 2 - e0[c])

        def shear(g, d, a):
            # stress component (d, a) of a face normal to d: own gradient du_a/dx_d, cell mean of du_d/dx_a
            q = {(0, 1): 5, (0, 2): 4, (1, 2): 3}[(min(d, a), max(d, a))]
            return c44 * 2 * ((T[a][d] + 2 * g) / 4 - e0[q])
        f = [0.0, 0.0, 0.0]
        for d, g, mask in ((0, gx, self.xface), (1, gy, self.yface)):
            for a in range(3):
                fn = (lambda gg: normal(gg, d)) if a == d else (lambda gg, a=a: shear(gg, d, a))
                hi = fn(g[a])                      # the cell above the face
                lo = _dn(fn(_up(g[a], d)), d)      # the cell below it
                s = 0.5 * (hi + lo) * mask
                f[a] = f[a] + (_up(s, d) - s) / self.h[d]
        for a in range(3):
            fn = (lambda gg: normal(gg, 2)) if a == 2 else (lambda gg, a=a: shear(gg, 2, a))
            hi = torch.nn.functional.pad(fn(gz[a][..., :-1]), (0, 1))
            lo = torch.nn.functional.pad(fn(gz[a][..., 1:]), (1, 0))
            s = 0.5 * (hi + lo) * self.zface
            f[a] = f[a] + (s[..., 1:] - s[..., :-1]) / self.h[2]
        return torch.stack(f) * self.solid, T

    # -- polarisation -----------------------------------------------------
    def dq(self, p, q, strain, e0, Ec):
        t = self.fem
        lap = 0.0
        for dd, mask in ((1, self.fe & _dn(self.fe, 0)), (2, self.fe & _dn(self.fe, 1))):
            g = (p - _dn(p, dd)) * mask.double() / self.h[dd - 1] ** 2
            lap = lap + (_up(g, dd) - g)
        g = torch.nn.functional.pad(p[..., 1:] - p[..., :-1], (1, 1)) * self.fez / self.h[2] ** 2
        lap = lap + (g[..., 1:] - g[..., :-1])
        tv1 = 2 * (t.c11 * t.Q11 + 2 * t.c12 * t.Q12)
        tv2 = 2 * (t.c11 * t.Q12 + t.c12 * t.Q11 + t.c12 * t.Q12)
        tv3 = 4 * t.c44 * t.Q44
        s = p * p
        e = [e0[a] - strain[a] for a in range(6)]
        sh = {(0, 1): 5, (0, 2): 4, (1, 2): 3}
        out = []
        for a in range(3):
            b, c = [v for v in range(3) if v != a]
            sa, sb, sc = s[a], s[b], s[c]
            F = (2 * t.a1 * p[a] + 4 * t.a11 * sa * p[a] + 2 * t.a12 * (sb + sc) * p[a] + 6 * t.a111 * sa * sa * p[a]
                 + 4 * t.a112 * sa * p[a] * (sb + sc) + 2 * t.a112 * (sb * sb + sc * sc) * p[a] + 2 * t.a123 * p[a] * sb * sc
                 + 8 * t.a1111 * sa ** 3 * p[a] + 2 * t.a1112 * p[a] * (sb ** 3 + sc ** 3 + 3 * sa * sa * (sb + sc))
                 + 4 * t.a1122 * sa * p[a] * (sb * sb + sc * sc) + 2 * t.a1123 * p[a] * sb * sc * (2 * sa + sb + sc))
            F = F + (tv1 * e[a] + tv2 * (e[b] + e[c])) * p[a]
            for o in (b, c):
                F = F + tv3 * e[sh[(min(a, o), max(a, o))]] * p[o]
            F = F - t.G11 * lap[a] + t.fe_damping * q[a]
            if Ec is not None:
                F = F - Ec[a]
            out.append(-self.d.dt / t.fe_mass * F)
        return torch.stack(out) * self.fe

    # -- Maxwell ----------------------------------------------------------
    # E: Ex, Ey (nx, ny, nz+1), Ez (nx, ny, nz); H: Hx, Hy (nx, ny, nz), Hz (nx, ny, nz+1)
    def e_cell(self, E):
        x = E[0] + _up(E[0], 1)
        y = E[1] + _up(E[1], 0)
        z = E[2] + _up(E[2], 0)
        return torch.stack([(x[..., 1:] + x[..., :-1]) / 4, (y[..., 1:] + y[..., :-1]) / 4, (z + _up(z, 1)) / 4])

    def h_cell(self, H):
        return torch.stack([(H[0] + _up(H[0], 0)) / 2, (H[1] + _up(H[1], 1)) / 2, (H[2][..., 1:] + H[2][..., :-1]) / 2])

    def dE(self, E, H, q, jf):
        d, h = self.d, self.h
        pad = torch.nn.functional.pad
        cx = (H[2] - _dn(H[2], 1)) / h[1] - pad(H[1][..., 1:] - H[1][..., :-1], (1, 1)) / h[2]
        cy = pad(H[0][..., 1:] - H[0][..., :-1], (1, 1)) / h[2] - (H[2] - _dn(H[2], 0)) / h[0]
        cz = (H[1] - _dn(H[1], 0)) / h[0] - (H[0] - _dn(H[0], 1)) / h[1]
        out = []
        for c, curl in enumerate((cx, cy, cz)):
            er, cond, cnt = self.edge[c]
            rhs = curl - cond * E[c]
            if jf is not None and c == jf[0]:
                rhs = rhs - sum(self._four(jf[1], c)) / 4.0
            if q is not None:
                rhs = rhs - sum(self._four(q[c] * self.solid, c)) / cnt
            v = d.dt / _E0 / er * rhs
            if c < 2:
                v = v.clone()
                v[..., 0] = 0.0
                v[..., -1] = 0.0
            out.append(v)
        return out

    def dH(self, E, dm):
        h = self.h
        c = [(_up(E[2], 1) - E[2]) / h[1] - (E[1][..., 1:] - E[1][..., :-1]) / h[2],
             (E[0][..., 1:] - E[0][..., :-1]) / h[2] - (_up(E[2], 0) - E[2]) / h[0],
             (_up(E[1], 0) - E[1]) / h[0] - (_up(E[0], 1) - E[0]) / h[1]]
        out = []
        for a in range(3):
            v = -self.d.dt / _MU0 * c[a]
            if dm is not None:
                M, fm = dm[a] * self.Ms, self.fm.double()
                if a < 2:
                    cnt = torch.clamp(fm + _dn(fm, a), min=1.0)
                    v = v - (M + _dn(M, a)) / cnt
                else:
                    def ends(f):
                        return torch.cat([f[..., :1], f], -1), torch.cat([f, f[..., -1:]], -1)
                    (m1, m2), (f1, f2) = ends(M), ends(fm)
                    v = v - (m1 + m2) / torch.clamp(f1 + f2, min=1.0)
            out.append(v)
        return out

    def mur(self, X, O, half):
        dz, dt = self.h[2], self.d.dt * (0.5 if half else 1.0)
        kt, kb = (dz - self.ct * dt) / (dz + self.ct * dt), (dz - self.cb * dt) / (dz + self.cb * dt)
        for c in range(2):
            O[c][..., -1] = X[c][..., -2] + kt * (X[c][..., -1] - O[c][..., -2])
            O[c][..., 0] = X[c][..., 1] + kb * (X[c][..., 0] - O[c][..., 1])

    # -- one step ---------------------------------------------------------
    def step(self, S, n, hext, alpha, wave=None):
        """S: dict of the state; n: 0-based step.  Returns the new state."""
        d, dt = self.d, self.d.dt
        t = (n + 1) * dt
        keys = [k for k in ("m", "p", "q", "u", "v", "E", "H") if k in S]
        as_list = {k: (list(S[k]) if k in "EH" else [S[k]]) for k in keys}
        X = as_list
        cur = {k: list(v) for k, v in X.items()}
        acc = {k: [0.0] * len(v) for k, v in X.items()}
        Hs = S.get("Hs")
        for s in range(4):
            m, p, q = (cur[k][0] if k in cur else None for k in ("m", "p", "q"))
            D = {}
            strain = e0 = None
            if d.elastic:
                u, v = cur["u"][0], cur["v"][0]
                e0 = self.eigen(m, p)
                f, T = self.force(u, e0)
                strain = self.strain(T)
                D["u"], D["v"] = [v * dt], [f * (dt * self.rrho)]
            if m is not None:
                he = hext if wave is None else hext + torch.nn.functional.pad(wave.reshape(1), (0, 2))
                D["m"] = [self.dm(m, Hs, he, strain if d.elasto_on else None, alpha, self.h_cell(cur["H"]) if d.em and d.em_back_M else None)]
            if p is not None:
                D["q"] = [self.dq(p, q, strain, e0, self.e_cell(cur["E"]) if d.em and d.em_back_P else None)]
                D["p"] = [q * dt]
            if d.em:
                jf = None
                if d.jf:
                    tj = t - dt if s == 0 else (t - 0.5 * dt if s < 3 else t)
                    if d.jf_type == 4:
                        val = d.jf_amp * math.exp(-(tj - 5 * d.jf_freq) ** 2 / (2 * d.jf_freq ** 2))
                    else:
                        val = d.jf_amp * math.exp(-(tj - 5 * d.jf_sigma) ** 2 / (2 * d.jf_sigma ** 2)) * math.sin(2 * math.pi * d.jf_freq * tj)
                    box = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
                    box[d.jf_lo[0]:d.jf_hi[0] + 1, d.jf_lo[1]:d.jf_hi[1] + 1, d.jf_lo[2]:d.jf_hi[2] + 1] = val
                    jf = ("xyz".index(d.jf_comp), box)
                D["E"] = self.dE(cur["E"], cur["H"], q if d.em_fromP and p is not None else None, jf)
                D["H"] = self.dH(cur["E"], D["m"][0] if d.em_fromM and m is not None else None)
            new = {}
            for k in keys:
                for a in range(len(X[k])):
                    acc[k][a] = acc[k][a] + D[k][a] * (1.0 / 6.0 if s in (0, 3) else 1.0 / 3.0)
                new[k] = [X[k][a] + (D[k][a] * (1.0 if s == 2 else 0.5) if s < 3 else acc[k][a]) for a in range(len(X[k]))]
            if d.elastic:
                self._u_boundary(S, X, new, s, t)
            if d.em:
                self.mur(X["E"], new["E"], s < 2)
            cur = new
            if "m" in cur and not d.em and self.N is not None:
                Hs = self.h_demag(cur["m"][0])
        out = {k: (v if k in "EH" else v[0]) for k, v in cur.items()}
        out["Hs"], out["hist"] = Hs, S.get("hist", [])
        if d.elastic and not d.abc_1D:
            out["hist"] = [S["u"][..., 1:5]] + list(S["hist"])[:2]
        return out

    def _u_boundary(self, S, X, new, s, t):
        d = self.d
        u = new["u"][0]
        if d.abc_1D:
            dz, h = d.dz, (0.5 * d.dt if s < 2 else d.dt)
            x = X["u"][0]
            parts = [u[..., 0], u[..., -1]]
            for side, vs in ((0, self.vs), (1, self.vt)):
                k = torch.tensor([(dz - vs[i] * h) / (dz + vs[i] * h) for i in (1, 1, 0)], dtype=torch.float64, device=self.dev).reshape(3, 1, 1)
                b, i = (0, 1) if side == 0 else (-1, -2)
                parts[side] = x[..., i] + k * (x[..., b] - u[..., i])
            new["u"][0] = torch.cat([parts[0][..., None], u[..., 1:-1], parts[1][..., None]], -1)
        elif s == 3:
            w = d.liao_w
            x = X["u"][0]
            z = torch.zeros_like(x[..., 0])
            hist = list(S["hist"])
            v = (4 * w + 2 * (1 - w)) * x[..., 1]
            for r, (c, pl) in enumerate(((-(6 * w + (1 - w)), 1), (4 * w, 2), (-w, 3))):
                v = v + c * (hist[r][..., pl] if r < len(hist) else z)
            new["u"][0] = torch.cat([v[..., None], u[..., 1:]], -1)
            self.last = v
        else:
            # stages 1-3 put the last full update's value back on plane 0 of the step-start u
            last = getattr(self, "last", None)
            if last is not None:
                X["u"][0] = torch.cat([last[..., None], X["u"][0][..., 1:]], -1)
            elif len(S["hist"]) == 0:
                X["u"][0] = torch.cat([torch.zeros_like(X["u"][0][..., :1]), X["u"][0][..., 1:]], -1)
        if d.strain_pulse:
            tl = t - 0.5 * d.dt if s < 2 else t
            vs = self.vs[0] if d.strain_comp == "z" else self.vs[1]
            val = d.amp_gauss * vs / 2.0 / math.pi / d.sigma_gauss * (math.cos(2 * math.pi * d.sigma_gauss * tl) - 1)
            c = "xyz".index(d.strain_comp)
            on = self.solid[..., d.strain_z]
            u = new["u"][0].clone()
            u[c, :, :, d.strain_z] = torch.where(on, torch.full_like(u[c, :, :, 0], val), u[c, :, :, d.strain_z])
            new["u"][0] = u

    def start(self):
        d, dev = self.d, self.dev

        def arr(a):
            return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)  # noqa: E731
        S = {"hist": []}
        nx, ny, nz = self.shape
        if self.has_fm:
            S["m"] = arr(d.m0)
            S["Hs"] = self.h_demag(S["m"])
        if self.has_fe:
            S["p"], S["q"] = arr(d.p0), arr(d.q0)
        if d.elastic:
            S["u"], S["v"] = (z(3, nx, ny, nz) if a is None else arr(a) for a in (d.u0, d.v0))
        if d.em:
            S["E"] = [z(nx, ny, nz + 1), z(nx, ny, nz + 1), z(nx, ny, nz)]
            S["H"] = [z(nx, ny, nz), z(nx, ny, nz), z(nx, ny, nz + 1)]
        return S

    def hext(self, n):
        d = self.d
        if d.Hext_table is None:
            return torch.tensor(d.Hext_stat, dtype=torch.float64, device=self.dev)
        # the row held during step n: the index moves on when t - dt passes the row's time
        idx, t = 0, 0.0
        for _ in range(n + 1):
            t += d.dt
            if idx < len(d.Hext_table) and t - d.dt > d.Hext_table[idx, 0]:
                idx += 1
        return torch.tensor(d.Hext_table[idx, 1:4], dtype=torch.float64, device=self.dev)


def _wrap(f, axes):
    for a in axes:
        f = torch.cat([f, f.narrow(a, 0, 1)], a)
    return f


def _fields(S, names):
    """The engine's field layout: Yee arrays repeat plane 0 at the far x / y end."""
    yee = {"Ex": ("E", 0, (1,)), "Ey": ("E", 1, (0,)), "Ez": ("E", 2, (0, 1)), "Hx": ("H", 0, (0,)), "Hy": ("H", 1, (1,)), "Hz": ("H", 2, ())}
    out = {}
    for f in names:
        out[f] = _wrap(S[yee[f][0]][yee[f][1]], yee[f][2]) if f in yee else S[f]
    return out


def _means(model, S, obs):
    d = {"m": model.fm, "p": model.fe, "u": torch.ones_like(model.fm)}
    return {o: (S[o].sum(dim=(1, 2, 3)) / d[o].sum()).cpu().numpy() for o in obs}


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if dev == "cpu" and kind != "sweep" and case["nx"] * case["ny"] * case["nz"] * case["steps"] > 4e5:
        return None
    if kind == "adjoint":
        return _exact_adjoint(case, seed, dev)
    if kind == "sweep":
        snaps, P = [], []
        for q, d in enumerate(_decks(case, seed)):
            M = _Model(d, dev)
            S = M.start()
            for n in range(case["steps"]):
                S = M.step(S, n, None, None)
            if q < 2:
                snaps.append(_fields(S, _SNAPSHOT["sweep"]))
            P.append(_means(M, S, ("p",))["p"])
        return {"snapshots": snaps, "P": np.stack(P)}
    M = _Model(_decks(case, seed), dev)
    S = M.start()
    rows = {o: [] for o in _OBS[kind]}
    for n in range(case["steps"]):
        S = M.step(S, n, M.hext(n) if M.has_fm else None, M.alpha)
        if (n + 1) % case["every"] == 0:
            for o, v in _means(M, S, _OBS[kind]).items():
                rows[o].append(v)
    out = _fields(S, _SNAPSHOT[kind])
    for o, v in rows.items():
        out["<%s>" % o] = np.stack(v)
    if kind in ("fe", "me"):
        i, j, k = case["nx"] // 2, case["ny"] // 2, case["nz"] // 2
        out["probe_E"] = M.e_cell(S["E"])[:, i, j, k].cpu().numpy()
        out["probe_H"] = M.h_cell(S["H"])[:, i, j, k].cpu().numpy()
    return out


def _exact_adjoint(case, seed, dev):
    """Reverse-mode differentiation of the same steps, one step's graph at a time."""
    d = _decks(case, seed)
    M = _Model(d, dev)
    N = case["steps"]
    al, wv = _adjoint_inputs(case, seed, d.n, _MU0)
    alpha = torch.from_numpy(al).to(dev).reshape(M.shape)
    wave = torch.from_numpy(wv).to(dev)
    hx = M.hext(0)
    nfm = float(M.fm.sum())
    with torch.no_grad():
        S = M.start()
        states, tr = [S], [S["m"][0].sum() / nfm]
        for n in range(N):
            M.last = S["u"][..., 0] if n else None
            S = M.step(S, n, hx, alpha, wave[(n * wave.numel()) // N])
            states.append(S)
            tr.append(S["m"][0].sum() / nfm)
    tr = torch.stack(tr).cpu().numpy()
    g = _trace_cotangent(tr)
    gw, ga = torch.zeros_like(wave), torch.zeros_like(alpha)
    inj = M.fm.double() / nfm
    lam = {k: torch.zeros_like(states[N][k]) for k in ("m", "u", "v")}
    pend = {}
    for n in range(N - 1, -1, -1):
        lam["m"][0] += g[n + 1] * inj
        for k, v in pend.pop(n + 1, {}).items():
            lam["u"][..., 1:5] += v
        S0 = states[n]
        a = alpha.clone().requires_grad_(True)
        seg = (n * wave.numel()) // N
        w = wave[seg].clone().requires_grad_(True)
        leaf = {k: S0[k].clone().requires_grad_(True) for k in ("m", "u", "v")}
        hist = [h.clone().requires_grad_(True) for h in S0["hist"]]
        T = dict(S0)
        T.update(leaf)
        T["hist"] = hist
        T["Hs"] = M.h_demag(leaf["m"])
        M.last = leaf["u"][..., 0] if n else None
        with torch.enable_grad():
            O = M.step(T, n, hx, a, w)
            loss = sum((O[k] * lam[k]).sum() for k in ("m", "u", "v"))
            args = [leaf["m"], leaf["u"], leaf["v"], a, w] + hist
            gr = torch.autograd.grad(loss, args, allow_unused=True)
        lam = {k: (v if v is not None else torch.zeros_like(leaf[k])) for k, v in zip(("m", "u", "v"), gr[:3])}
        ga += gr[3]
        gw[seg] += gr[4]
        for r, v in enumerate(gr[5:]):
            if v is not None:
                # hist[r] holds planes 1-4 of the step-start u of step n-1-r
                slot = pend.setdefault(n - 1 - r, {})
                slot["u"] = slot["u"] + v if "u" in slot else v
    return {"trace": tr, "grad_wave": gw.cpu().numpy(), "grad_alpha": ga.cpu().numpy().ravel()}
