"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the named ones and ``draw(rng)`` more of the
same ranges; ``prepare`` makes what a program holds before the call (inputs from the seed, a
resident simulation where the program keeps one), ``run`` is one pass through the public entry
points, ``exact`` the same outputs from a plain FP64 torch restatement of the scheme, and ``work``
the bytes and operations a pass cannot do without.

The kinds of call, by their entry point:

* ``solve``    one whole ``kspace_first_order`` call on host arrays: set-up, the time loop and the
               sensor's pressure series back on the host.
* ``reverse``  one whole time-reversal ``kspace_first_order`` call: boundary data in, the final
               pressure field out.
* ``axisym``   one whole ``kspace_first_order_as`` call.
* ``step``     a resident ``Simulation``: ``advance`` a number of time steps, then look at the
               pressure field (a frame of a movie, a check on convergence, a checkpoint).
* ``elastic``  the same for the elastic stress-velocity solvers.
* ``batch``    ``solve_batch`` on independent 2D simulations of mixed sizes.

The library steps in FP32 and the whole-solve entry points widen what they recorded to float64 on
the way out.  ``run`` hands those values on as the FP32 numbers they are, so that an output's type
says what precision it was computed in; ``Simulation.pressure`` returns FP32 by itself.
"""

import math
import os
import sys
import warnings

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-wave-julia_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

# The whole-solve entry points warn on every call that the solve is FP32.
warnings.filterwarnings("ignore", message="kwave_b200 steps fields and FFTs in FP32")

DX = 1e-4
STEPS_NO_END = 50_000_000  # a resident simulation's Nt: it is advanced as long as its program runs


def listed():
    """Sizes and options from this repository's own workloads, benchmark and tests: the 128^2 ring,
    the 512^2 absorbing medium, the 256^3 nonlinear piston, the mixed 2D batch (sides 128-1024),
    the serving stream's 3D sides (64-192, of any 2/3/5-smooth length), the elastic solid."""
    return [
        # the smallest call there is: a 1D line, all latency and launches
        dict(name="solve1d_512", kind="solve", nx=512, steps=1000, medium="layered", source="p0", sensor="line"),
        # the first thing a new user runs: a disc source in a homogeneous 2D medium, a ring of sensors
        dict(name="solve2d_128", kind="solve", nx=128, ny=128, steps=689, medium="homogeneous", source="p",
             sensor="ring"),
        # photoacoustic reconstruction: time reversal of the data on a planar sensor
        dict(name="reverse2d_256", kind="reverse", nx=256, ny=256, steps=500, medium="homogeneous"),
        # the ordinary 2D study: heterogeneous tissue with power-law absorption, aggregates everywhere
        dict(name="step2d_512", kind="step", nx=512, ny=512, steps=200, medium="absorbing", source="p0",
             record="p_max,p_rms"),
        # homogeneous absorbing water or tissue with dispersion (the :stokes branch), on a plain rectangle
        dict(name="step2d_stokes_384x320", kind="step", nx=384, ny=320, steps=200, medium="stokes", source="p"),
        # a grid cut to an anatomy and not to a power of two
        dict(name="step2d_ragged_810x450", kind="step", nx=810, ny=450, steps=200, medium="absorbing", source="p"),
        # a fine 2D study
        dict(name="step2d_1024", kind="step", nx=1024, ny=1024, steps=200, medium="absorbing", source="p"),
        # a small 3D volume of no particular size
        dict(name="step3d_ragged_120x108x100", kind="step", nx=120, ny=108, nz=100, steps=200, medium="absorbing",
             source="p"),
        # an ordinary 3D volume
        dict(name="step3d_160", kind="step", nx=160, ny=160, nz=160, steps=100, medium="absorbing", source="p"),
        # the largest: 256^3 heterogeneous nonlinear ultrasound, a piston source, the volume's peak pressure
        dict(name="step3d_256_nonlinear", kind="step", nx=256, ny=256, nz=256, steps=200, medium="nonlinear",
             source="ux", record="p_max"),
        # shear waves in a heterogeneous solid
        dict(name="elastic3d_128", kind="elastic", nx=128, ny=128, nz=128, steps=100),
        # many independent simulations at once
        dict(name="batch2d_12", kind="batch", count=12, lo=128, hi=1024, steps=300),
    ]


def _smooth_side(rng, lo, hi):
    """A side in [lo, hi], spread over its logarithm: mostly 2/3/5-smooth, as users pick them, and
    one in five as it comes."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.2:
        return n
    return min(_smooth_sides(lo, hi), key=lambda m: abs(m - n))


def _smooth_sides(lo, hi):
    out = []
    for n in range(lo, hi + 1):
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    kind = rng.choice(["solve", "solve", "step", "step", "step", "step3", "step3", "step3", "reverse", "axisym",
                       "elastic", "batch"])
    if kind == "solve":
        if rng.random() < 0.3:
            return dict(kind="solve", nx=_smooth_side(rng, 128, 2048), steps=rng.randint(300, 1500),
                        medium=rng.choice(["homogeneous", "layered"]), source="p0", sensor="line")
        return dict(kind="solve", nx=_smooth_side(rng, 64, 512), ny=_smooth_side(rng, 64, 512),
                    steps=rng.randint(200, 900), medium=rng.choice(["homogeneous", "absorbing", "stokes"]),
                    source=rng.choice(["p", "p0"]), sensor="ring")
    if kind == "step":
        return dict(kind="step", nx=_smooth_side(rng, 64, 1024), ny=_smooth_side(rng, 64, 1024),
                    steps=rng.randint(50, 300), medium=rng.choice(["homogeneous", "absorbing", "stokes", "nonlinear"]),
                    source=rng.choice(["p", "p0", "ux"]), record=rng.choice(["", "p_max", "p_max,p_rms"]))
    if kind == "step3":
        return dict(kind="step", nx=_smooth_side(rng, 48, 192), ny=_smooth_side(rng, 48, 192),
                    nz=_smooth_side(rng, 48, 192), steps=rng.randint(30, 120),
                    medium=rng.choice(["homogeneous", "absorbing", "absorbing", "stokes", "nonlinear"]),
                    source=rng.choice(["p", "p0", "ux"]), record=rng.choice(["", "p_max"]))
    if kind == "reverse":
        return dict(kind="reverse", nx=_smooth_side(rng, 64, 512), ny=_smooth_side(rng, 64, 512),
                    steps=rng.randint(200, 900), medium=rng.choice(["homogeneous", "absorbing"]))
    if kind == "axisym":
        return dict(kind="axisym", nx=_smooth_side(rng, 64, 512), ny=_smooth_side(rng, 64, 512),
                    steps=rng.randint(200, 900), medium=rng.choice(["homogeneous", "absorbing"]), source="p",
                    sensor="ring")
    if kind == "elastic":
        if rng.random() < 0.5:
            return dict(kind="elastic", nx=_smooth_side(rng, 64, 512), ny=_smooth_side(rng, 64, 512),
                        steps=rng.randint(50, 300))
        return dict(kind="elastic", nx=_smooth_side(rng, 48, 128), ny=_smooth_side(rng, 48, 128),
                    nz=_smooth_side(rng, 48, 128), steps=rng.randint(30, 100))
    return dict(kind="batch", count=rng.randint(4, 12), lo=64, hi=rng.choice([512, 1024]), steps=rng.randint(100, 300))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------

def _shape(case):
    return tuple(case[k] for k in ("nx", "ny", "nz") if k in case)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _random_field(gen, shape, sigma, lo, hi):
    """Gaussian random field: white noise filtered with a Gaussian of `sigma` points, mapped onto [lo, hi]."""
    w = torch.randn(shape, generator=gen, device=_device(), dtype=torch.float64)
    k2 = torch.zeros((), device=_device(), dtype=torch.float64)
    for ax, n in enumerate(shape):
        kv = 2 * math.pi * torch.fft.fftfreq(n, device=_device(), dtype=torch.float64)
        k2 = k2 + (kv ** 2).reshape([n if a == ax else 1 for a in range(len(shape))])
    f = torch.fft.ifftn(torch.fft.fftn(w) * torch.exp(-k2 * sigma ** 2 / 2)).real
    f = (f - f.min()) / (f.max() - f.min())
    return (lo + (hi - lo) * f).cpu().numpy()


def _tone_burst(dt, freq, cycles):
    n = int(round(cycles / freq / dt))
    t = np.arange(n) * dt
    burst = np.sin(2 * math.pi * freq * t) * np.exp(-((t - cycles / freq / 2) / (1 / (2 * freq))) ** 2 / 2)
    return np.append(burst, 0.0)  # a short signal holds its last value


def _ball(shape, centre, radius):
    d2 = np.zeros((1,) * len(shape))
    for ax, n in enumerate(shape):
        d2 = d2 + ((np.arange(n) - centre[ax]) ** 2).reshape([n if a == ax else 1 for a in range(len(shape))])
    return d2 <= radius ** 2


def _inputs(case, seed):
    """Everything a simulation is given, as numbers and numpy arrays."""
    shape = _shape(case)
    D = len(shape)
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(rng.integers(1 << 40)))
    dx = 2e-4 if D == 3 else DX
    q = dict(shape=shape, dx=dx, steps=case["steps"], pml=min(10 if D == 3 else 20, min(shape) // 4))
    ctr = [int(rng.integers(n // 3, n - n // 3)) for n in shape]
    if case["kind"] == "elastic":
        s = 5.0 * min(shape) / 256
        q["cp"] = _random_field(gen, shape, s, 2600.0, 3200.0)
        q["cs"] = _random_field(gen, shape, s, 1100.0, 1600.0)
        q["rho"] = _random_field(gen, shape, s, 1600.0, 2100.0)
        q["dt"] = 0.3 * dx / 3200.0
        q["p0"] = 1e5 * _ball(shape, ctr, 4.0)
        q["s_mask"] = np.zeros(shape, dtype=bool)
        q["s_mask"][tuple(n // 4 for n in shape)] = True
        q["sxx"] = 1e4 * _tone_burst(q["dt"], 3e6, 3)[None, :]
        return q
    m = case["medium"]
    if m in ("homogeneous", "stokes"):
        q["c"], q["rho"] = float(rng.uniform(1480, 1520)), float(rng.uniform(990, 1010))
    elif m == "layered":
        at = int(rng.integers(shape[0] // 2, 3 * shape[0] // 4))
        q["c"], q["rho"] = np.full(shape, 1500.0), np.full(shape, 1000.0)
        q["c"][at:], q["rho"][at:] = 1650.0, 1100.0
    else:
        q["c"] = _random_field(gen, shape, 5.0, 1400.0, 1600.0)
        q["rho"] = _random_field(gen, shape, 5.0, 900.0, 1100.0)
    if m == "stokes":
        q["alpha"] = (0.75, 1.5, "stokes")
    elif m == "absorbing":
        q["alpha"] = (0.75, float(rng.uniform(1.05, 1.9)), "no_dispersion")
    elif m == "nonlinear":
        q["alpha"] = (0.5, 1.1, "no_dispersion")
        q["BonA"] = np.where(_ball(shape, ctr, min(shape) / 12), 9.0, 5.0)
    q["dt"] = 0.3 * dx / float(np.max(q["c"]))
    if case["kind"] == "reverse":
        # data of a planar sensor at x = pml + 1: the arrivals of a few point absorbers
        mask = np.zeros(shape, dtype=bool)
        mask[q["pml"] + 1, q["pml"]: shape[1] - q["pml"]] = True
        t = np.arange(case["steps"]) * q["dt"]
        data = np.zeros((int(mask.sum()), case["steps"]))
        ys = np.flatnonzero(mask[q["pml"] + 1])
        for _ in range(6):
            px, py = rng.uniform(0.3, 0.8) * shape[0], rng.uniform(0.2, 0.8) * shape[1]
            r = dx * np.sqrt((px - q["pml"] - 1) ** 2 + (py - ys) ** 2)
            a = (t[None, :] - r[:, None] / 1500.0) / 1.5e-7
            data += rng.uniform(0.5, 1.5) * -a * np.exp(-a * a / 2) / np.sqrt(r[:, None] / dx)
        q["mask"], q["data"] = mask, 1e3 * data
        return q
    src = case["source"]
    if src == "p0":
        q["p0"] = 1e6 * _ball(shape, ctr, 5.0)
    elif src == "p":
        q["p_mask"] = _ball(shape, ctr, 0.5 if D == 3 else 4.0)
        q["p"] = 1e5 * np.tile(_tone_burst(q["dt"], float(rng.uniform(0.8e6, 2.5e6)), 4), (int(q["p_mask"].sum()), 1))
    else:
        half = max(1, min(shape[1:]) // 16)
        q["u_mask"] = np.zeros(shape, dtype=bool)
        q["u_mask"][(q["pml"] + 1,) + tuple(slice(n // 2 - half, n // 2 + half) for n in shape[1:])] = True
        q["ux"] = 0.5 * np.tile(_tone_burst(q["dt"], 1e6, 3), (int(q["u_mask"].sum()), 1))
    if case.get("sensor") == "line":
        q["mask"] = np.zeros(shape, dtype=bool)
        q["mask"][q["pml"]:: 4] = True
    elif case.get("sensor") == "ring":
        # around the source, near enough for its wave to pass every point of it
        r = min(0.25 * min(shape), 0.15 * case["steps"])
        q["mask"] = _ball(shape, ctr, r) & ~_ball(shape, ctr, r - 1)
    return q


def _batch(case, seed):
    """The simulations of a batch: sides spread over [lo, hi], each a `solve` of its own."""
    import random
    rng = random.Random(seed * 7919 + 17)
    # sides follow from the case alone, so that another seed is the same work on other inputs
    sides = random.Random(case["count"] * 1000003 + case["lo"] * 101 + case["hi"] + case["steps"])
    out = []
    for i in range(case["count"]):
        sub = dict(kind="solve", nx=_smooth_side(sides, case["lo"], case["hi"]),
                   ny=_smooth_side(sides, case["lo"], case["hi"]), steps=case["steps"], medium="absorbing",
                   source="p", sensor="ring")
        out.append((sub, rng.randrange(1 << 40)))
    return out


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------

def _api(kb, case, q):
    """(kgrid, medium, source, sensor, kwargs) of this package for the inputs q."""
    args = []
    for n in q["shape"]:
        args += [n, q["dx"]]
    g = kb.KWaveGrid(*args)
    g.dt = q["dt"]
    g.Nt = STEPS_NO_END if case["kind"] in ("step", "elastic") else q["steps"]
    kw = dict(pml_size=q["pml"])
    if case["kind"] == "elastic":
        return (g, kb.ElasticMedium(sound_speed_compression=q["cp"], sound_speed_shear=q["cs"], density=q["rho"]),
                kb.ElasticSource(p0=q["p0"], s_mask=q["s_mask"], sxx=q["sxx"]), kb.KWaveSensor(), kw)
    med = dict(sound_speed=q["c"], density=q["rho"], BonA=q.get("BonA"))
    if "alpha" in q:
        med.update(alpha_coeff=q["alpha"][0], alpha_power=q["alpha"][1], alpha_mode=q["alpha"][2])
    src = {k: q[k] for k in ("p0", "p_mask", "p", "u_mask", "ux") if k in q}
    sen = {}
    if case.get("record"):
        sen = dict(mask=np.ones(q["shape"], dtype=bool), record=case["record"].split(","))
    elif "mask" in q:
        sen = dict(mask=q["mask"], record=["p"])
        if "data" in q:
            sen["time_reversal_boundary_data"] = q["data"]
    return g, kb.KWaveMedium(**med), kb.KWaveSource(**src), kb.KWaveSensor(**sen), kw


def prepare(case, seed):
    import kwave_b200 as kb
    if case["kind"] == "batch":
        return dict(kind="batch", kb=kb, jobs=[_api(kb, sub, _inputs(sub, s)) for sub, s in _batch(case, seed)])
    args = _api(kb, case, _inputs(case, seed))
    st = dict(kind=case["kind"], kb=kb, steps=case["steps"])
    if case["kind"] in ("step", "elastic"):
        g, med, src, sen, kw = args
        st["sim"] = kb.Simulation(g, med, src, sen, **kw)
    else:
        st["args"] = args
    return st


def _f32(a):
    return np.asarray(a, dtype=np.float32)


def run(state):
    kb, kind = state["kb"], state["kind"]
    if kind in ("step", "elastic"):
        state["sim"].advance(state["steps"])
        return {"p": state["sim"].pressure()}
    if kind == "batch":
        return [_f32(o["p"]) for o in kb.solve_batch(state["jobs"])]
    g, med, src, sen, kw = state["args"]
    solve = kb.kspace_first_order_as if kind == "axisym" else kb.kspace_first_order
    out = solve(g, med, src, sen, **kw)
    return {"p_final": _f32(out["p_final"])} if kind == "reverse" else {"p": _f32(out["p"])}


# ---------------------------------------------------------------------------------------------
# the same in plain FP64
# ---------------------------------------------------------------------------------------------

def _along(v, ax, D):
    return v.reshape([-1 if a == ax else 1 for a in range(D)])


def _k(n, d):
    m = np.arange(n)
    return np.where(m < (n + 1) // 2, m, m - n) * (2 * math.pi / (n * d))


class _Scheme:
    """Grid operators of the staggered k-space scheme in FP64."""

    def __init__(self, q):
        dev = _device()
        self.D, self.shape, self.dt, self.dx = len(q["shape"]), q["shape"], q["dt"], q["dx"]
        T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        D, dx, npml = self.D, self.dx, q["pml"]
        self.T = T
        self.ik, self.pml, self.pml_sg = {}, [], []
        for ax, n in enumerate(self.shape):
            k = _k(n, dx)[: n // 2 + 1]
            for sg in (1, -1):
                self.ik[ax, sg] = _along(T(1j * k * np.exp(sg * 1j * k * dx / 2)), ax, D)
            for stag, to in ((0.0, self.pml), (0.5, self.pml_sg)):
                v = np.ones(n)
                for i in range(1, npml + 1):
                    e = math.exp(-(2.0 * ((npml - i + 1 - stag) / npml) ** 4) * self.dt)
                    v[i - 1] = v[n - i] = e
                to.append(_along(T(v), ax, D))

    def grad(self, f, ax, sg):
        return torch.fft.irfft(torch.fft.rfft(f, dim=ax) * self.ik[ax, sg], n=self.shape[ax], dim=ax)

    def zeros(self):
        return torch.zeros(self.shape, device=_device(), dtype=torch.float64)

    def stagger(self, rho, ax):
        return rho if not torch.is_tensor(rho) else (rho + torch.roll(rho, -1, ax)) / 2


def _smooth_p0(s, p0):
    r = p0.to(torch.complex128)
    for ax, n in enumerate(s.shape):
        i = np.arange(n)
        w = 0.42 - 0.5 * np.cos(2 * math.pi * i / (n - 1)) + 0.08 * np.cos(4 * math.pi * i / (n - 1))
        r = torch.fft.ifft(torch.fft.fft(r, dim=ax) * _along(s.T(np.roll(w, n // 2)), ax, s.D), dim=ax)
    r = r.real
    return r * (p0.abs().max() / r.abs().max())


def _points(mask):
    """A mask's points, first axis fastest."""
    idx = np.argwhere(np.transpose(mask))[:, ::-1]
    return tuple(torch.as_tensor(np.ascontiguousarray(idx[:, a]), device=_device()) for a in range(mask.ndim))


def _exact_fluid(case, q):
    s = _Scheme(q)
    D, dt, T = s.D, s.dt, s.T
    val = lambda v: T(v) if isinstance(v, np.ndarray) else v
    c, rho0, bona = val(q["c"]), val(q["rho"]), val(q["BonA"]) if "BonA" in q else None
    c_ref = float(np.mean(q["c"]))
    k2 = torch.zeros((), device=_device(), dtype=torch.float64)
    for ax, n in enumerate(s.shape):
        k2 = k2 + _along(T(_k(n, s.dx) ** 2), ax, D)
    # the half spectrum of a transform over all axes whose last axis is halved
    kk = torch.sqrt(k2)[..., : s.shape[-1] // 2 + 1]
    a = c_ref * kk * dt / 2
    mul = torch.where(a == 0, torch.ones_like(a), torch.sin(a) / torch.where(a == 0, torch.ones_like(a), a))
    mul2 = None
    if "alpha" in q:
        coeff, y, mode = q["alpha"]
        np_ = coeff * (1e-2 / (20 * math.log10(math.e))) * (2 * math.pi * 1e6) ** (-y)
        f = 2 * np_ * c_ref ** (y - 1)
        if mode == "stokes" and not torch.is_tensor(c):
            mul2 = mul * (f * math.tan(math.pi * y / 2)) * torch.where(kk > 0, kk, torch.ones_like(kk)) ** (y - 1)
            mul2 = torch.where(kk > 0, mul2, torch.zeros_like(mul2))
        mul = mul * (1 - f * kk ** y)
    rsg = [s.stagger(rho0, ax) for ax in range(D)]
    p, u, rho = s.zeros(), [s.zeros() for _ in range(D)], [s.zeros() for _ in range(D)]
    prev = s.zeros()
    tr = T(q["data"]) if "data" in q else None
    pts = _points(q["mask"]) if "mask" in q else None
    at = lambda v, idx: v[idx] if torch.is_tensor(v) else v
    if "p0" in q:
        p = _smooth_p0(s, T(q["p0"]))
        for ax in range(D):
            rho[ax] = p / (D * c ** 2)
            u[ax] = -dt / (2 * rsg[ax]) * s.grad(p, ax, 1)
    p_idx = _points(q["p_mask"]) if "p_mask" in q else None
    u_idx = _points(q["u_mask"]) if "u_mask" in q else None
    p_sig = T(q["p"]) if "p" in q else None
    u_sig = T(q["ux"]) if "ux" in q else None
    if case["kind"] == "axisym":
        n = s.shape[1]
        r = np.abs((np.arange(n) - (n - 1) / 2) * s.dx)
        inv_r = _along(T(1 / np.where(r == 0, s.dx / 2, r)), 1, D)
    eos = (lambda r: r * (1 + bona / 2 * r / rho0)) if bona is not None else (lambda r: r)
    dims = tuple(range(D))
    series = []
    for t in range(q["steps"]):
        if tr is not None:
            for ax in range(D):
                rho[ax][pts] = tr[:, q["steps"] - 1 - t] / (D * at(c, pts) ** 2)
        for ax in range(D):
            u[ax] = s.pml_sg[ax] * (s.pml_sg[ax] * u[ax] - dt / rsg[ax] * s.grad(p, ax, 1))
        if u_idx is not None:
            u[0][u_idx] += u_sig[:, min(t, u_sig.shape[1] - 1)]
        for ax in range(D):
            g = s.grad(u[ax], ax, -1)
            if case["kind"] == "axisym" and ax == 1:
                g = g + u[1] * inv_r
            rho[ax] = s.pml[ax] * (s.pml[ax] * rho[ax] - dt * rho0 * g)
        if p_idx is not None:
            for ax in range(D):
                rho[ax][p_idx] += p_sig[:, min(t, p_sig.shape[1] - 1)] / (D * at(c, p_idx) ** 2)
        tot = sum(rho[1:], rho[0])
        F = torch.fft.rfftn(c ** 2 * eos(tot), dim=dims) * mul
        if mul2 is not None:
            F = F - torch.fft.rfftn(c ** 2 * (eos(tot) - eos(prev)) / dt, dim=dims) * mul2
            prev = tot
        p = torch.fft.irfftn(F, s=s.shape, dim=dims)
        if pts is not None and tr is None:
            series.append(p[pts])
    if case["kind"] == "reverse":
        return {"p_final": p.permute(*reversed(range(D))).reshape(-1).cpu().numpy()}
    if case["kind"] == "step":
        return {"p": p.cpu().numpy()}
    return {"p": torch.stack(series, dim=1).cpu().numpy()}


def _exact_elastic(q):
    s = _Scheme(q)
    D, dt, T = s.D, s.dt, s.T
    rho0, cp, cs = T(q["rho"]), T(q["cp"]), T(q["cs"])
    lam, mu = rho0 * (cp ** 2 - 2 * cs ** 2), rho0 * cs ** 2
    rsg = [s.stagger(rho0, ax) for ax in range(D)]
    v = [s.zeros() for _ in range(D)]
    sig = {(i, j): s.zeros() for i in range(D) for j in range(i, D)}
    of = lambda i, j: sig[min(i, j), max(i, j)]
    for i in range(D):
        sig[i, i] = -T(q["p0"])
    idx, src = _points(q["s_mask"]), T(q["sxx"])
    for t in range(q["steps"]):
        for j in range(D):
            acc = sum(s.grad(of(d, j), d, 1) for d in range(D))
            v[j] = s.pml_sg[j] * (s.pml_sg[j] * v[j] + dt / rsg[j] * acc)
        g = [[s.grad(v[j], d, -1) for d in range(D)] for j in range(D)]
        div = sum(g[i][i] for i in range(D))
        for i in range(D):
            sig[i, i] = s.pml[i] * (s.pml[i] * sig[i, i] + dt * (lam * div + 2 * mu * g[i][i]))
            for j in range(i + 1, D):
                sig[i, j] = s.pml[i] * s.pml[j] * (sig[i, j] + dt * mu * (g[i][j] + g[j][i]))
        sig[0, 0][idx] += src[:, min(t, src.shape[1] - 1)]
    return {"p": (-sum(sig[i, i] for i in range(D)) / D).cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_fluid(sub, _inputs(sub, s))["p"] for sub, s in _batch(case, seed)]
    q = _inputs(case, seed)
    return _exact_elastic(q) if case["kind"] == "elastic" else _exact_fluid(case, q)


# ---------------------------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------------------------

def work(case):
    """Per time step, each field of the state read once and written once and each array of the
    medium read once (FP32); five N log2 N operations a complex transform of N points."""
    if case["kind"] == "batch":
        each = [work(sub) for sub, _ in _batch(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    shape = _shape(case)
    D, n = len(shape), float(np.prod(shape))
    lg = sum(math.log2(v) for v in shape)
    if case["kind"] == "elastic":
        words = 2 * (D + D * (D + 1) // 2) + 3
        flops = 2 * D * 5 * lg + 20 * D * D
    else:
        words = 2 * (2 * D + 1)
        words += {"homogeneous": 0, "stokes": 2, "layered": 2, "absorbing": 2, "nonlinear": 3}[case["medium"]]
        words += sum({"p_max": 2, "p_rms": 4}[r] for r in case.get("record", "").split(",") if r)
        flops = 10 * lg + (10 if case["medium"] == "stokes" else 5) * lg + 20 * D
    return {"bytes": 4.0 * words * n * case["steps"], "flops": flops * n * case["steps"]}
