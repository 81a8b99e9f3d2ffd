"""The calls that a user of the simulation engine makes, as measurable cases.

A case names one public entry point, its sizes, its number type and its
arithmetic.  ``listed()`` holds the fixed cases, ``draw()`` gives further ones
of the same ranges, ``prepare()`` builds what a program holds before the call,
``run()`` is one call, ``exact()`` the same result from plain torch in 64 bits,
``work()`` the bytes and operations that no implementation can do without.

Entry points (field ``call``):

* ``simulate``  one ``homs.simulate`` on host arrays: upload, run, signal back;
* ``blocks``    one ``homs.run_blocks`` on host arrays from a given spin state;
* ``plan``      one run of a prepared plan, signal and final state left on the
                device (the C interface with device pointers);
* ``resident``  ``homs.simulate`` of a new sequence on a phantom that is kept
                on the device;
* ``reduce``    the standalone coil reduction on device arrays;
* ``kspace``    ``homs.get_kspace``, the encoding export, on host arrays.

Sequences (field ``seq``): ``spiral`` is a hard 90-degree pulse, a partition
blip and a spiral readout per interleave; ``trloop`` a windowed-sinc slab pulse,
a spiral readout and a recovery delay per repetition; ``gre`` a windowed-sinc
pulse, prewinders, a Cartesian readout and spoilers per repetition.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "highordermrisim.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import homs  # noqa: E402
from homs import _lib  # noqa: E402

GAMMA = homs.GAMMA
FOV = 0.2  # m


# --------------------------------------------------------------------------- the cases

def _sim(name, call, seq, nx, ny, nz, nc, nrep, nadc, dwell, precision, arithmetic, mask="1111", nrf=2):
    return {"name": name, "call": call, "seq": seq, "nx": nx, "ny": ny, "nz": nz, "nc": nc, "nrep": nrep,
            "nadc": nadc, "dwell": dwell, "precision": precision, "arithmetic": arithmetic, "mask": mask, "nrf": nrf}


def listed():
    return [
        # A first try or a unit test of a user's own sequence: launch and set-up latency.
        _sim("blocks_tiny_f64", "blocks", "spiral", 10, 10, 10, 8, 1, 200, 1e-5, "f64", "plain"),
        # The call with default parameters (FP32, plain) on a 64 x 64 slice and one ideal coil.
        _sim("simulate_2d_1coil_f32", "simulate", "spiral", 64, 64, 1, 1, 1, 2048, 5e-6, "f32", "plain"),
        # The default arithmetic on an ordinary multi-coil slice, four interleaves of 10,000 samples.
        _sim("simulate_2d_8coil_f32", "simulate", "spiral", 200, 200, 1, 8, 4, 10000, 1e-6, "f32", "plain", "1110"),
        # The same slice prepared once and run many times in FP64 (parameter studies).
        _sim("plan_2d_8coil_f64", "plan", "spiral", 200, 200, 1, 8, 4, 10000, 1e-6, "f64", "plain", "1110"),
        # FP64 verification runs of a 3D 32-coil acquisition on a coarse grid with odd sides.
        _sim("plan_3d_32coil_f64", "plan", "spiral", 33, 33, 11, 32, 4, 9500, 1e-6, "f64", "plain"),
        # The 3D 32-coil production run: 350,000 spins, 38,000 samples, split arithmetic.
        _sim("plan_3d_32coil_split", "plan", "spiral", 100, 100, 35, 32, 4, 9500, 1e-6, "f64", "split"),
        # A one-off 3D simulation of FP32 data in split arithmetic: the phantom crosses and is prepared each time.
        _sim("simulate_3d_16coil_split", "simulate", "spiral", 48, 48, 24, 16, 1, 8000, 2e-6, "f32", "split"),
        # A served request on a phantom that stays on the device.
        _sim("resident_2d_8coil_split", "resident", "spiral", 61, 61, 1, 8, 1, 5000, 2e-6, "f32", "split"),
        # A 3D TR loop: 35 shaped pulses, each followed by a readout and a recovery delay.
        _sim("plan_trloop_32coil_split", "plan", "trloop", 100, 100, 8, 32, 35, 2000, 4e-6, "f64", "split", "1111", 400),
        # A Cartesian gradient-echo train: many shaped pulses, short readouts, FP32.
        _sim("plan_gre_8coil_f32", "plan", "gre", 173, 173, 1, 8, 48, 128, 1e-5, "f32", "plain", "1111", 64),
        # The coil reduction of stored states, as the reference's stand-alone kernel is used.
        {"name": "reduce_64x32_f64", "call": "reduce", "ns": 200000, "nadc": 64, "nc": 32, "precision": "f64"},
        # Encoding of a whole 3D TR loop for a reconstruction.
        {"name": "kspace_trloop_f64", "call": "kspace", "seq": "trloop", "nrep": 35, "nadc": 9500, "dwell": 1e-6,
         "nrf": 400, "precision": "f64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["blocks", "simulate", "simulate", "plan", "plan", "plan", "resident", "gre", "trloop", "reduce",
                       "reduce", "kspace"])
    if call == "reduce":
        ns, nc = _log_int(rng, 2000, 200000), rng.choice([1, 3, 8, 12, 16, 31, 32])
        return {"call": "reduce", "ns": ns, "nadc": _log_int(rng, 16, 96 if ns * nc < 4e6 else 64), "nc": nc,
                "precision": rng.choice(["f32", "f64"])}
    if call == "kspace":
        return {"call": "kspace", "seq": "trloop", "nrep": rng.randint(4, 35), "nadc": _log_int(rng, 500, 9500),
                "dwell": rng.choice([1e-6, 2e-6, 4e-6]), "nrf": rng.randint(50, 400),
                "precision": rng.choice(["f32", "f64"])}
    precision = rng.choice(["f32", "f64"])
    arithmetic = rng.choice(["plain", "plain", "split"])
    mask = rng.choice(["1111", "1111", "1110", "0110", "0000", "0100"])
    nc = rng.choice([1, 4, 8, 12, 16, 24, 32])
    dwell = rng.choice([1e-6, 2e-6, 5e-6])
    if call == "blocks":
        return _drawn(call, "spiral", _log_int(rng, 100, 4000), rng, nc, 1, _log_int(rng, 32, 1000), dwell, precision,
                      arithmetic, mask, 2)
    if call == "gre":
        return _drawn("plan", "gre", _log_int(rng, 3000, 30000), rng, min(nc, 16), rng.randint(8, 48),
                      rng.choice([64, 96, 128]), 1e-5, precision, arithmetic, mask, rng.randint(24, 64))
    if call == "trloop":
        return _drawn("plan", "trloop", _log_int(rng, 5000, 80000), rng, nc, rng.randint(4, 35), _log_int(rng, 200, 2000),
                      4e-6, precision, "split", mask, rng.randint(100, 400))
    if call == "resident":
        return _drawn(call, "spiral", _log_int(rng, 1000, 60000), rng, nc, 1, _log_int(rng, 1000, 8000), dwell, precision,
                      "split", mask, 2)
    # simulate and plan: the plain arithmetic up to the listed slices, the split one up to a coarse volume
    top = 40000 if arithmetic == "plain" else 150000
    ns = _log_int(rng, 2000, top)
    nrep = rng.randint(1, 4)
    nadc = _log_int(rng, 1000, 9500)
    while ns * nrep * nadc * (nc + 8) > (1.8e10 if arithmetic == "plain" else 1.5e11):
        nadc //= 2
    return _drawn(call, "spiral", ns, rng, nc, nrep, nadc, dwell, precision, arithmetic, mask, 2)


def _drawn(call, seq, ns, rng, nc, nrep, nadc, dwell, precision, arithmetic, mask, nrf):
    """A 2D or 3D grid of about ``ns`` spins."""
    nz = 1 if rng.random() < 0.5 else max(2, int(round(ns ** (1 / 3) / 2)))
    nx = max(2, int(round(math.sqrt(ns / nz))))
    ny = max(2, int(round(ns / nz / nx)))
    c = _sim("", call, seq, nx, ny, nz, nc, nrep, nadc, dwell, precision, arithmetic, mask, nrf)
    del c["name"]
    return c


# --------------------------------------------------------------------------- inputs

def _rng(seed):
    return np.random.Generator(np.random.PCG64(int(seed)))


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid(c):
    dx = FOV / c["nx"]
    i = (np.arange(c["nx"]) - (c["nx"] - 1) / 2) * dx
    j = (np.arange(c["ny"]) - (c["ny"] - 1) / 2) * dx
    k = (np.arange(c["nz"]) - (c["nz"] - 1) / 2) * dx
    z, y, x = np.meshgrid(k, j, i, indexing="ij")
    return x.ravel(), y.ravel(), z.ravel()


def _coils(rng, x, y, z, nc):
    """Gaussian receive profiles around a hemisphere, one seeded phase per coil."""
    if nc == 1:
        return np.ones((x.shape[0], 1), np.complex128)
    k = np.arange(nc) + 0.5
    r, phi = np.sqrt(1 - (k / nc) ** 2), np.pi * (1 + 5 ** 0.5) * k
    centre = torch.tensor(0.14 * np.stack([r * np.cos(phi), r * np.sin(phi), k / nc]), device=_dev())
    phase = torch.tensor(rng.uniform(0, 2 * np.pi, nc), device=_dev())
    p = torch.tensor(np.stack([x, y, z]), device=_dev())
    d2 = sum((p[a][None, :] - centre[a][:, None]) ** 2 for a in range(3))
    g = torch.exp(-d2 / (2 * 0.08 ** 2))
    return torch.polar(g, phase[:, None].expand_as(g).contiguous()).cpu().numpy().T  # column-major (ns, nc)


def _phantom(c, rng):
    """Voxels of an ellipsoid with ordinary tissue values; outside it the density is zero."""
    x, y, z = _grid(c)
    n = x.shape[0]
    half = 0.45 * c["nz"] * FOV / c["nx"]
    inside = (x / 0.09) ** 2 + (y / 0.09) ** 2 + (0.0 if c["nz"] == 1 else (z / half) ** 2) <= 1.0
    rho = rng.uniform(0.5, 1.0, n) * inside
    T1, T2 = rng.uniform(0.5, 2.0, n), rng.uniform(0.03, 0.2, n)
    dw = 2 * np.pi * rng.normal(0.0, 30.0, n)
    csm = _coils(rng, x, y, z, c["nc"])
    obj = homs.HO_Phantom(x=x, y=y, z=z, rho=rho, T1=T1, T2=T2, dw=dw, csm=csm)
    return obj.astype(np.float32) if c["precision"] == "f32" else obj


def _spiral(nadc, dwell, kmax, rot):
    """Archimedean spiral of 30 mT/m peak gradient, at the sample times."""
    T = nadc * dwell
    s = np.arange(1, nadc + 1) / nadc
    w = math.sqrt(max((GAMMA * 30e-3 * T / kmax) ** 2 - 1.0, 0.0))  # radians over the readout
    g = kmax / T * (1 + 1j * w * s) * np.exp(1j * (w * s + rot)) / GAMMA
    return g.real, g.imag


class _Sections:
    """Sampled sections one after the other; each shares its first node with the section before."""

    def __init__(self):
        self.dt, self.g, self.b1, self.adc, self.exc = [], [np.zeros((3, 1))], [np.zeros(1, complex)], [np.zeros(1, bool)], []

    def add(self, dt, gx=0.0, gy=0.0, gz=0.0, b1=0.0, adc=False, exc=False):
        n = dt.shape[0]
        full = lambda v, t: np.broadcast_to(np.asarray(v, t), (n,)).copy()  # noqa: E731
        self.dt.append(dt)
        self.g.append(np.stack([full(v, float) for v in (gx, gy, gz)]))
        self.b1.append(full(b1, complex))
        self.adc.append(full(adc, bool))
        self.exc.append(full(exc, bool))

    def pulse(self, dt, b1, gz=0.0):
        """B1 ``b1[i]`` over interval i (the value of its first node)."""
        self.b1[-1][-1] = b1[0]
        self.add(dt, gz=gz, b1=np.concatenate([b1[1:], [0.0]]), exc=True)

    def sinc(self, flip_deg, dur, n, slab):
        tc = (np.arange(n) + 0.5) * dur / n - dur / 2
        env = np.sinc(4.0 / dur * tc) * (0.5 + 0.5 * np.cos(2 * np.pi * tc / dur))
        gsel = 4.0 / dur / (GAMMA * slab)
        self.pulse(np.full(n, dur / n), (flip_deg / 360.0) / (GAMMA * env.sum() * dur / n) * env, gz=gsel)
        self.add(np.full(10, dur / 20), gz=-gsel)


def _sequence(c, rng):
    """The sampled sequence, and the intervals at which a pulse's centre falls."""
    s = _Sections()
    centres, at = [], 0
    kmax = c.get("nx", 100) / (2 * FOV)
    for r in range(c["nrep"]):
        if c["seq"] == "spiral":
            amp = 0.25 / (GAMMA * 1e-4)
            s.pulse(np.full(c["nrf"], 1e-4 / c["nrf"]), np.full(c["nrf"], amp))
            s.add(np.full(10, 1e-5), gz=((r % 4) - 1.5) / (0.07 * GAMMA * 1e-4) if c["nz"] > 1 else 0.0)
            gx, gy = _spiral(c["nadc"], c["dwell"], kmax, r * np.pi / 2)
            s.add(np.full(c["nadc"], c["dwell"]), gx=gx, gy=gy, adc=True)
        elif c["seq"] == "trloop":
            s.sinc(15.0, 2e-3, c["nrf"], 0.04)
            s.add(np.full(10, 1e-5), gz=((r % 8) - 3.5) / (0.05 * GAMMA * 1e-4))
            gx, gy = _spiral(c["nadc"], c["dwell"], kmax, r * np.pi / 2)
            s.add(np.full(c["nadc"], c["dwell"]), gx=gx, gy=gy, adc=True)
            s.add(np.full(200, 1e-3))
        else:
            s.sinc(30.0, 1.6e-3, c["nrf"], 0.005)
            k = 2 * kmax / c["nx"] * ((r % c["nx"]) - c["nx"] / 2)
            s.add(np.full(8, 5e-5), gx=-kmax / (GAMMA * 4e-4), gy=k / (GAMMA * 4e-4))
            s.add(np.full(c["nadc"], c["dwell"]), gx=2 * kmax / (GAMMA * c["nadc"] * c["dwell"]), adc=True)
            s.add(np.full(20, 1e-4), gx=12e-3, gy=-k / (GAMMA * 2e-3), gz=15e-3)
        centres.append(at + c["nrf"] // 2)
        at = sum(d.shape[0] for d in s.dt)
    dt = np.concatenate(s.dt)
    t = np.concatenate([[0.0], np.cumsum(dt)])
    g = np.concatenate(s.g, axis=1)
    # measured fields: three seeded sinusoids per term, plus the nominal gradients in the first order
    h = np.zeros((16, t.shape[0]))
    for k in range(16):
        a = (1e-6, 1e-3, 5e-3, 20e-3)[0 if k == 0 else 1 if k < 4 else 2 if k < 9 else 3] / 3
        for _ in range(3):
            h[k] += a * rng.uniform(0.5, 1.0) * np.sin(2 * np.pi * rng.uniform(50, 500) * t + rng.uniform(0, 2 * np.pi))
    h[1:4] += g
    seq = homs.HO_DiscreteSequence(t, dt=dt, gx=g[0], gy=g[1], gz=g[2], b1=np.concatenate(s.b1),
                                   adc=np.concatenate(s.adc), excitation=np.concatenate(s.exc), h=h)
    return (seq.astype(np.float32) if c["precision"] == "f32" else seq), centres


def _state(c, obj, rng):
    """A spin state left by an earlier part of a sequence."""
    m = rng.uniform(0.1, 0.9, len(obj)) * np.exp(2j * np.pi * rng.uniform(0, 1, len(obj))) * obj.rho
    z = rng.uniform(-0.5, 0.9, len(obj)) * obj.rho
    f32 = c["precision"] == "f32"
    return homs.Mag(m.astype(np.complex64 if f32 else np.complex128), z.astype(np.float32 if f32 else np.float64))


def _inputs(c, seed):
    rng = _rng(seed)
    obj = _phantom(c, rng)
    seq, _ = _sequence(c, rng)
    return obj, seq, (_state(c, obj, rng) if c["call"] == "blocks" else None)


def _reduce_inputs(c, seed):
    g = torch.Generator(device=_dev()).manual_seed(int(seed))
    rt, ct = (torch.float32, torch.complex64) if c["precision"] == "f32" else (torch.float64, torch.complex128)
    make = lambda n: torch.view_as_complex(torch.randn(n, c["ns"], 2, generator=g, device=_dev(), dtype=rt)).to(ct)  # noqa: E731
    return make(c["nadc"]), make(c["nc"])  # column-major (ns, n): one row per column


# --------------------------------------------------------------------------- one call

class _Held:
    """What a program keeps between calls; closed with the program's last reference."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for k in ("plan", "resident"):
            if k in self.__dict__:
                try:
                    self.__dict__[k].close()
                except Exception:
                    pass


_SHARED = {}


def _context():
    if "ctx" not in _SHARED:
        _SHARED["ctx"] = homs.Context(0)
    return _SHARED["ctx"]


def prepare(case, seed):
    c = dict(case)
    if c["call"] == "reduce":
        states, csm = _reduce_inputs(c, seed)
        return _Held(c=c, ctx=_context(), states=states, csm=csm,
                     sig=torch.empty(c["nc"], c["nadc"], dtype=states.dtype, device=states.device))
    if c["call"] == "kspace":
        seq, centres = _sequence(c, _rng(seed))
        return _Held(c=c, ctx=_context(), seq=seq, starts=centres, signs=[0] * len(centres))
    obj, seq, state = _inputs(c, seed)
    params = {"sim_method": homs.BlochHighOrder(c["mask"]), "precision": c["precision"],
              "homs_precision": c["arithmetic"]}
    s = _Held(c=c, ctx=_context(), obj=obj, seq=seq, state=state, params=params)
    if c["call"] == "blocks":
        s.parts, s.excitation = homs.get_sim_ranges(seq)
    elif c["call"] == "resident":
        s.resident = homs.ResidentPhantom(obj, c["precision"], c["arithmetic"], context=s.ctx)
    elif c["call"] == "plan":
        s.plan = homs.prepare_simulation(obj, seq, sim_params=params, context=s.ctx)
        rt, ct = (torch.float32, torch.complex64) if c["precision"] == "f32" else (torch.float64, torch.complex128)
        s.sig = torch.empty(c["nc"], s.plan.nadc, dtype=ct, device="cuda")
        s.xy = torch.empty(len(obj), dtype=ct, device="cuda")
        s.z = torch.empty(len(obj), dtype=rt, device="cuda")
        s.out = _lib.State(s.xy.data_ptr(), s.z.data_ptr(), _lib.HOMS_DEVICE)
    return s


def run(s):
    c = s.c
    if c["call"] == "simulate":
        return homs.simulate(s.obj, s.seq, sim_params=s.params, context=s.ctx)
    if c["call"] == "resident":
        return homs.simulate(s.resident, s.seq, sim_params=s.params, context=s.ctx)
    if c["call"] == "blocks":
        return homs.run_blocks(s.obj, s.seq, s.parts, s.excitation, s.params["sim_method"], c["precision"],
                               c["arithmetic"], s.state, s.ctx)
    if c["call"] == "plan":
        _lib.check(_lib.load().homs_plan_run(s.plan.handle, s.sig.data_ptr(), _lib.HOMS_DEVICE, ctypes.byref(s.out)),
                   s.ctx.handle)
        return s.sig, s.xy, s.z
    if c["call"] == "reduce":
        dt = _lib.HOMS_F32 if c["precision"] == "f32" else _lib.HOMS_F64
        _lib.check(_lib.load().homs_coil_reduce(s.ctx.handle, dt, c["ns"], c["nadc"], c["nc"], s.states.data_ptr(),
                                                c["ns"], s.csm.data_ptr(), c["ns"], s.sig.data_ptr(), c["nadc"]),
                   s.ctx.handle)
        return s.sig
    return homs.get_kspace(s.seq, s.starts, s.signs, context=s.ctx, precision=c["precision"])


# --------------------------------------------------------------------------- what it takes

def _nodes(c):
    tail = {"spiral": 10, "trloop": 10 + 10 + 200, "gre": 10 + 8 + 20}[c["seq"]]
    return 1 + c["nrep"] * (c["nrf"] + c["nadc"] + tail)


def work(case):
    c = dict(case)
    b = 4 if c["precision"] == "f32" else 8
    if c["call"] == "reduce":
        return {"bytes": 2 * b * (c["ns"] * (c["nadc"] + c["nc"]) + c["nadc"] * c["nc"]),
                "flops": 8 * c["ns"] * c["nadc"] * c["nc"]}
    n, nadc = _nodes(c), c["nrep"] * c["nadc"]
    if c["call"] == "kspace":
        return {"bytes": 21 * b * n + 19 * 8 * (n + nadc), "flops": 19 * 4 * (n + nadc)}
    ns = c["nx"] * c["ny"] * c["nz"]
    m = c["mask"]
    terms = 3 + (m[0] == "1") + 5 * (m[2] == "1") + 7 * (m[3] == "1") + 1
    nrf = c["nrep"] * c["nrf"]
    moved = b * ns * (7 + 2 * c["nc"]) + b * n * (8 + 16) + 2 * b * nadc * c["nc"] + 3 * b * ns
    # per spin and sample: the field terms, a cosine, a sine, a decay factor, a complex product, the coils;
    # per spin and pulse node: the rotation and the relaxation
    return {"bytes": moved, "flops": ns * nadc * (2 * terms + 10 + 8 * c["nc"]) + 60 * ns * nrf}


# --------------------------------------------------------------------------- the same in 64 bits

def _basis(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    r2 = x2 + y2 + z2
    return torch.stack([torch.ones_like(x), x, y, z, x * y, z * y, 3 * z2 - r2, x * z, x2 - y2, 3 * y * x2 - y2 * y,
                        x * z * y, (5 * z2 - r2) * y, 5 * z2 * z - 3 * z * r2, (5 * z2 - r2) * x, x2 * z - y2 * z,
                        x2 * x - 3 * x * y2])


def exact(case, seed):
    c = dict(case)
    dev = _dev()
    f64 = lambda v: torch.as_tensor(np.asarray(v), device=dev).to(torch.float64)  # noqa: E731
    if c["call"] == "reduce":
        states, csm = _reduce_inputs(c, seed)
        return csm.to(torch.complex128) @ states.to(torch.complex128).T
    if c["call"] == "kspace":
        return _exact_kspace(c, seed)
    obj, seq, state = _inputs(c, seed)
    x, y, z, rho, T1, T2, dw = (f64(getattr(obj, k)) for k in ("x", "y", "z", "rho", "T1", "T2", "dw"))
    csm = torch.as_tensor(np.asarray(obj.csm), device=dev).to(torch.complex128)
    m = c["mask"]
    h, dt = f64(seq.h).clone(), f64(seq.dt)
    if m[1] == "0":
        h[1:4] = torch.stack([f64(seq.gx), f64(seq.gy), f64(seq.gz)])
    for rows, on in ((slice(0, 1), m[0]), (slice(4, 9), m[2]), (slice(9, 16), m[3])):
        if on == "0":
            h[rows] = 0
    basis = _basis(x, y, z)  # 16 x ns
    xy = torch.zeros(len(obj), dtype=torch.complex128, device=dev) if state is None else \
        torch.as_tensor(state.xy, device=dev).to(torch.complex128)
    mz = rho.clone() if state is None else f64(state.z)
    b1 = np.asarray(seq.b1, np.complex128)
    g = torch.stack([f64(seq.gx), f64(seq.gy), f64(seq.gz)])
    dts = np.asarray(seq.dt, np.float64)
    adc = np.asarray(seq.adc, bool)
    on = np.asarray(seq.excitation, bool)
    cuts = [0, *(np.flatnonzero(on[1:] != on[:-1]) + 1), on.shape[0]]
    sig = []
    for lo, hi in zip(cuts[:-1], cuts[1:]):
        pulse = on[lo]
        if pulse:
            B0 = torch.einsum("ks,kn->ns", basis[1:4], g[:, lo:hi]) + dw / (2 * math.pi * GAMMA)
            for n in range(lo, hi):
                bz, bt, d = B0[n - lo], complex(b1[n]), float(dts[n])
                B = torch.sqrt(abs(bt) ** 2 + bz * bz)
                half = -math.pi * GAMMA * B * d
                u = torch.where(B > 0, torch.sin(half) / torch.where(B > 0, B, torch.ones_like(B)), torch.zeros_like(B))
                al = torch.complex(torch.cos(half), -bz * u)
                be = torch.complex(bt.imag * u, -bt.real * u)
                xyn = 2 * al.conj() * be * mz + al.conj() ** 2 * xy - be ** 2 * xy.conj()
                mz = (al.abs() ** 2 - be.abs() ** 2) * mz - 2 * (al * be * xy.conj()).real
                e1 = torch.exp(-d / T1)
                xy, mz = xyn * torch.exp(-d / T2), mz * e1 + rho * (1 - e1)
            continue
        trap = torch.cumsum(0.5 * (h[:, lo:hi] + h[:, lo + 1:hi + 1]) * dt[lo:hi], 1)  # 16 x intervals
        tt = torch.cumsum(dt[lo:hi], 0)
        want = torch.as_tensor(np.flatnonzero(adc[lo + 1:hi + 1]), device=dev)
        turns = lambda q: -GAMMA * (trap[:, q].T @ basis) - tt[q][:, None] * (dw / (2 * math.pi))  # noqa: E731
        step = max(1, int(2.5e8 // len(obj)))
        for a in range(0, want.shape[0], step):
            q = want[a:a + step]
            th = turns(q)
            th = 2 * math.pi * (th - torch.round(th))
            sig.append((torch.polar(torch.exp(-tt[q][:, None] / T2), th) * xy) @ csm)
        last = torch.tensor([hi - lo - 1], device=dev)
        th = turns(last)[0]
        xy = xy * torch.polar(torch.exp(-tt[-1] / T2), 2 * math.pi * (th - torch.round(th)))
        e1 = torch.exp(-tt[-1] / T1)
        mz = mz * e1 + rho * (1 - e1)
    sig = torch.cat(sig)  # nadc x nc
    if c["call"] == "plan":
        return sig.T.contiguous(), xy, mz
    if c["call"] == "blocks":
        return sig.cpu().numpy(), xy.cpu().numpy(), mz.cpu().numpy()
    return sig.cpu().numpy()[:, :, None]


def _exact_kspace(c, seed):
    seq, starts = _sequence(c, _rng(seed))
    a = lambda v: np.asarray(v, np.float64)  # noqa: E731
    dt, t = a(seq.dt), a(seq.t)
    cols = np.concatenate([[a(seq.gx), a(seq.gy), a(seq.gz)], a(seq.h)])
    k = np.cumsum(0.5 * (cols[:, :-1] + cols[:, 1:]) * dt, axis=1)
    # every pulse is an excitation: the integral restarts at its centre
    base = np.zeros_like(k)
    for i, st in enumerate(starts):
        end = starts[i + 1] if i + 1 < len(starts) else k.shape[1]
        base[:, st:end] = k[:, st - 1:st]
    k = (GAMMA * (k - base)).T
    knots = t[:-1] + dt
    q = t[np.asarray(seq.adc, bool)]
    n = np.searchsorted(knots, q, side="right") - 1
    lo = np.clip(n, 0, k.shape[0] - 2)
    w = (q - knots[lo]) / (knots[lo + 1] - knots[lo])
    kq = k[lo] + w[:, None] * (k[lo + 1] - k[lo])
    kq[n < 0] = 0.0
    kq[q > knots[-1]] = 0.0
    return k[:, :3], kq[:, :3], k[:, 3:], kq[:, 3:]
