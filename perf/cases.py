"""Performance cases of the hydro pass: what programs that use this library have it do.

A case is a plain dict: what is run (``path``), on which particles (``field``, ``n``), in which form. ``listed()``
holds the fixed ones, ``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` makes the inputs and
the handle a program has in hand before the call, ``run(state)`` is one pass through the public entry points,
``work`` and ``tolerance`` say what the pass cannot do without and how far two correct implementations differ,
and ``exact`` is the same pass in plain 64-bit torch, where that is quick.

Paths:
  host     HydroPass.upload / density, hydro_gradient_calc, hydro_force / download: the call for call drop-in of
           a host code that keeps its particles in host memory
  calls    the same with device arrays in and out (gz_upload_device, gz_download_device): one step of a program
           whose particles live on the GPU
  graph    device arrays in and out around hydro_pass(graph=True): the three passes as one CUDA graph
  replay   hydro_pass(graph=True, restage=True) on the resident inputs, device arrays out: the throughput loop
  subset   density, gradients and force of an active list between two full steps (individual timesteps), the
           grid and the kernel lengths of the last step in place, device arrays out
  step     DeviceStep.step(): timestep, kick, drift, pass, kick, all on the device
  kicks    gz_timestep, gz_kick, gz_drift, gz_kick on the caller's arrays, without a pass
  sums     gz_density_sums_noalloc: the density sums at given kernel lengths for callers that cannot allocate
"""
import ctypes as C
import math

import numpy as np
import torch

from gizmo_b200 import abi, ics
from gizmo_b200.hydro import HydroPass, drift, kick, timestep
from gizmo_b200.step import DeviceStep

VOL = ics.VOLNORM
TIMEBASE = 2.0 ** -40
FIELDS = abi.OUTPUT_FIELDS
FORCE = ("accel", "dudt", "vsig", "dtmass", "dmass", "gravwork")


def listed():
    return [
        # the smallest call: one box of a batch, in the default form, from host arrays
        {"name": "tube_4k_host", "path": "host", "field": "tube", "n": 4096, "mixed": False},
        # the point blast of the reference's own test suite, 32^3, replayed: launch latency
        {"name": "sedov_32k_replay", "path": "replay", "field": "sedov", "n": 32768, "mixed": True},
        # a driven-turbulence box of ordinary size, not a power of two, in the FP64 form
        {"name": "lognormal_110k_calls", "path": "calls", "field": "lognormal", "n": 110003, "mixed": False, "sigma": 1.5},
        # a clustered MFV set, FP64, as a graph
        {"name": "plummer_1m_graph", "path": "graph", "field": "plummer", "n": 1000003, "mixed": False},
        # turbulence at 128^3, mixed: the second headline configuration
        {"name": "lognormal_2m_replay", "path": "replay", "field": "lognormal", "n": 2097152, "mixed": True, "sigma": 1.5},
        # the clustered headline configuration at half its particles (three states fit one GPU)
        {"name": "plummer_8m_replay", "path": "replay", "field": "plummer", "n": 8388608, "mixed": True},
        # a batch of independent boxes of mixed size in one set
        {"name": "boxes_64_graph", "path": "graph", "field": "boxes", "boxes": 64, "n": 700000, "mixed": True},
        # a short active list of the deepest timestep bins: few targets, scattered
        {"name": "subset_1pct_mixed", "path": "subset", "field": "lognormal", "n": 2097152, "mixed": True, "sigma": 2.0, "fraction": 0.01},
        # a tenth of the cells active, MFV and FP64
        {"name": "subset_10pct_fp64", "path": "subset", "field": "plummer", "n": 1048576, "mixed": False, "fraction": 0.1},
        # a whole step on the device
        {"name": "step_64k_mfm", "path": "step", "field": "tube", "n": 64000, "mixed": False},
        # the half-step kernels around the pass of a large MFV set
        {"name": "kicks_4m_mfv", "path": "kicks", "field": "plummer", "n": 4194304, "mixed": False},
        # the call for hosts that own the device memory
        {"name": "sums_20k_noalloc", "path": "sums", "field": "plummer", "n": 20000, "mixed": False},
    ]


def draw(rng):
    """One more case: path and form at random, sizes spread over the logarithm of each path's range."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["host", "calls", "graph", "replay", "replay", "subset", "step", "kicks", "sums"])
    field = rng.choice(["sedov", "tube", "lognormal", "plummer"])
    top = {"host": 20000, "calls": 1000000, "graph": 4000000, "replay": 4000000, "subset": 3000000, "step": 500000,
           "kicks": 8000000, "sums": 50000}[path]
    low = {"subset": 50000, "kicks": 10000, "sums": 1000}.get(path, 1500)
    if path == "subset":
        field = rng.choice(["lognormal", "plummer"])
    if path in ("kicks", "sums"):
        field = rng.choice(["lognormal", "plummer"])
    if path == "step":
        field = "tube"
    if path == "graph" and rng.random() < 0.5:
        field, top, low = "boxes", 2000000, 20000
    c = {"path": path, "field": field, "n": size(low, top), "mixed": rng.random() < 0.5 and path not in ("kicks", "sums")}
    if field == "lognormal":
        c["sigma"] = round(rng.uniform(1.0, 2.0), 2)
    if field == "boxes":
        c["boxes"] = max(2, min(300, int(c["n"] / size(2000, 20000))))
    if path == "subset":
        c["fraction"] = round(math.exp(rng.uniform(math.log(0.002), math.log(0.3))), 4)
    return c


# ---------------------------------------------------------------- particles
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Rand:
    def __init__(self, seed):
        self.dev = _device()
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(seed)

    def u(self, *shape, lo=0.0, hi=1.0):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device=self.dev, dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device=self.dev, dtype=torch.float64)


def _lattice(n1, r):
    """n1^3 cells, +-0.1 spacing of jitter, and kernel lengths within 5% of the lattice's."""
    g = (torch.arange(n1, device=r.dev, dtype=torch.float64) + 0.5) / n1
    pos = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    pos = torch.remainder(pos + r.u(n1 ** 3, 3, lo=-0.1, hi=0.1) / n1, 1.0)
    h = (32.0 / (VOL * n1 ** 3)) ** (1 / 3) * r.u(n1 ** 3, lo=0.95, hi=1.05)
    return pos, h


def _tube(n, r):
    """A shock tube of random orientation and states on the lattice nearest to n cells."""
    n1 = max(8, round(n ** (1 / 3)))
    pos, h = _lattice(n1, r)
    nrm = r.normal(3)
    left = (pos - 0.5) @ (nrm / nrm.norm()) < 0
    a = r.u(4).tolist()
    side = left.double()
    rho = 0.125 + 0.875 * (a[1] + (a[0] - a[1]) * side)
    u = (0.1 + 0.9 * (a[3] + (a[2] - a[3]) * side)) / (2.0 / 3.0 * rho)
    return pos, torch.zeros_like(pos), rho / n1 ** 3, u, h


def _sedov(n, r):
    """A point blast: energy 1 on the 32 cells nearest the centre, in a cold lattice."""
    n1 = max(8, round(n ** (1 / 3)))
    pos, h = _lattice(n1, r)
    d, near = torch.topk((pos - 0.5).norm(dim=1), 33, largest=False)
    q = d[:32] / d[32]
    w = torch.where(q < 0.5, 1 + 6 * (q - 1) * q * q, 2 * (1 - q) ** 3).clamp(min=1e-3)
    u = torch.full((n1 ** 3,), 1e-5, device=r.dev, dtype=torch.float64)
    u[near[:32]] += n1 ** 3 * w / w.sum()
    return pos, torch.zeros_like(pos), torch.full_like(u, 1.0 / n1 ** 3), u, h


def _field_k(ng, dev):
    k = torch.fft.fftfreq(ng, d=1.0 / ng, device=dev, dtype=torch.float64)
    kz = torch.fft.rfftfreq(ng, d=1.0 / ng, device=dev, dtype=torch.float64)
    return torch.stack(torch.broadcast_tensors(k[:, None, None], k[None, :, None], kz[None, None, :]))


def _lognormal(n, r, sigma):
    """Supersonic turbulence: a log-normal density field with P(k) ~ k^-3, solenoidal velocities P(k) ~ k^-4 at
    Mach 2, near-isothermal gas. The kernel lengths come from the field the particles were drawn from, averaged
    over as many cells as hold the wanted neighbours: within about 10% of the converged ones."""
    ng = 128 if n > 200000 else 64
    K = _field_k(ng, r.dev)
    k2 = (K ** 2).sum(0)
    k2[0, 0, 0] = 1.0

    def noise(slope, *lead):
        a = k2 ** (slope / 4.0)
        a[0, 0, 0] = 0.0
        return torch.complex(r.normal(*lead, *k2.shape), r.normal(*lead, *k2.shape)) * a

    d = torch.fft.irfftn(noise(-3.0), s=(ng, ng, ng))
    rho = torch.exp(d / d.std() * sigma)
    rho = rho / rho.sum()
    cum = torch.cumsum(rho.reshape(-1), 0)
    cell = torch.searchsorted(cum, r.u(n) * cum[-1]).clamp(max=ng ** 3 - 1)
    c3 = torch.stack([cell // (ng * ng), (cell // ng) % ng, cell % ng], -1)
    pos = torch.remainder((c3 + r.u(n, 3)) / ng, 1.0)
    v = noise(-4.0, 3)
    v = torch.fft.irfftn(v - K * ((K * v).sum(0) / k2), s=(ng, ng, ng))
    vel = v[:, c3[:, 0], c3[:, 1], c3[:, 2]].T.contiguous()
    cs = math.sqrt(1.0001 * 0.0001)
    vel = vel * (2.0 * cs / (vel ** 2).sum(1).mean().sqrt())
    # kernel length: the smallest smoothing of the field whose ball holds 64 expected particles
    want, h, done = 64.0, torch.zeros(n, device=r.dev, dtype=torch.float64), torch.zeros(n, device=r.dev, dtype=torch.bool)
    hat = torch.fft.rfftn(rho)
    for b in [0.0] + [0.5 * 2 ** (k / 2) for k in range(15)]:  # ball radii in cells
        sm = torch.fft.irfftn(hat * torch.exp(-0.1 * k2 * (2 * math.pi * b / ng) ** 2), s=(ng, ng, ng)).clamp(min=1e-12)
        hb = (want / (VOL * n * ng ** 3 * sm[c3[:, 0], c3[:, 1], c3[:, 2]])) ** (1 / 3)
        take = ~done & (hb * ng <= max(1.5 * b, 0.5))
        h[take] = hb[take]
        done |= take
    h = torch.where(done, h, hb).clamp(max=0.2)
    return pos, vel, torch.full((n,), 1.0 / n, device=r.dev, dtype=torch.float64), torch.ones(n, device=r.dev, dtype=torch.float64), h


def _plummer(n, r):
    """90% of the particles in up to 1000 Plummer spheres, 10% uniform at rest; kernel lengths from the density
    the particles were drawn from, within Poisson noise of the converged ones."""
    ns = max(4, min(1000, n // 1000))
    n_bg = n // 10
    ctr = r.u(ns, 3)
    a = torch.exp(r.u(ns, lo=math.log(0.002), hi=math.log(0.02))) * (1000.0 / ns) ** (1 / 3)
    sid = torch.arange(n - n_bg, device=r.dev) % ns
    top = (1 + 1 / 400.0) ** -1.5  # mass inside 20 scale radii
    rr = a[sid] * ((r.u(n - n_bg, lo=1e-9) * top) ** (-2 / 3) - 1).clamp(min=1e-12) ** -0.5
    d = r.normal(n - n_bg, 3)
    pos = torch.remainder(ctr[sid] + d / d.norm(dim=1, keepdim=True) * rr[:, None], 1.0)
    m_s = 0.9 / ns
    vel = r.normal(n - n_bg, 3) * (m_s / (rr ** 2 + a[sid] ** 2).sqrt()).sqrt()[:, None]
    pos = torch.cat([pos, r.u(n_bg, 3)])
    vel = torch.cat([vel, torch.zeros(n_bg, 3, device=r.dev, dtype=torch.float64)])
    mix = torch.randperm(n, generator=r.g, device=r.dev)
    pos, vel = pos[mix].contiguous(), vel[mix].contiguous()
    dens = torch.full((n,), 0.1, device=r.dev)
    p32, c32, a32 = pos.float(), ctr.float(), a.float()
    for b in range(0, n, 1 << 17):  # the spheres' profiles, summed at every particle
        x = p32[b:b + (1 << 17), None, :] - c32[None]
        q = 1 + ((x - x.round()) ** 2).sum(-1) / a32 ** 2
        dens[b:b + (1 << 17)] += (m_s * 3 / (4 * math.pi) / a32 ** 3 * q ** -2.5).sum(-1)
    h = (32.0 / (VOL * n * dens.double())) ** (1 / 3) * r.u(n, lo=0.95, hi=1.05)
    one = torch.ones(n, device=r.dev, dtype=torch.float64)
    return pos, vel, one / n, one * 1e-2, h.clamp(max=0.2)


def _counts(case):
    """Lattice sizes of a box set: log-uniform over a factor of 16 in particles, adding up to about n."""
    rng = np.random.default_rng(case["boxes"])
    w = np.exp(rng.uniform(0, math.log(16.0), case["boxes"]))
    return [max(8, round(float(x) ** (1 / 3))) for x in w / w.sum() * case["n"]]


def _particles(case, seed):
    r = _Rand(seed * 7919 + 13)
    f = case["field"]
    if f == "boxes":
        parts = [(_tube if k % 2 else _sedov)(n1 ** 3, r) for k, n1 in enumerate(_counts(case))]
        pos, vel, mass, u, h = (torch.cat(x) for x in zip(*parts))
    elif f == "lognormal":
        pos, vel, mass, u, h = _lognormal(case["n"], r, case["sigma"])
    else:
        pos, vel, mass, u, h = {"tube": _tube, "sedov": _sedov, "plummer": _plummer}[f](case["n"], r)
    gamma = 1.0001 if f == "lognormal" else 5.0 / 3.0
    cs = (gamma * (gamma - 1) * u).sqrt() + (vel ** 2).sum(1).sqrt()
    dt = torch.pow(2.0, -torch.ceil(-torch.log2(0.2 * h / cs)).clamp(4, 30))  # power-of-two bins
    p = {"pos": pos, "vel": vel, "mass": mass, "u": u, "dt": dt, "h": h, "cond": torch.zeros_like(h)}
    return {k: v.to(torch.float64).contiguous() for k, v in p.items()}  # what the library reads: FP64 rows


def _params(case):
    prec = abi.PRECISION_MIXED if case["mixed"] else abi.PRECISION_FP64
    if case["field"] == "lognormal":
        return ics.make_params(abi.KERNEL_WENDLAND_C2, abi.METHOD_MFM, 1.0001, 64.0, 0.1, prec)
    method = abi.METHOD_MFV if case["field"] == "plummer" else abi.METHOD_MFM
    return ics.make_params(abi.KERNEL_CUBIC, method, 5.0 / 3.0, 32.0, 0.1, prec)


def _n(case):
    if case["field"] == "boxes":
        return sum(k ** 3 for k in _counts(case))
    if case["field"] in ("tube", "sedov"):
        return max(8, round(case["n"] ** (1 / 3))) ** 3
    return case["n"]


# ------------------------------------------------------------------ prepare
def _ptr(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double))


def _upload_device(hp, p):
    g = abi.GzParticles()
    g.n = p["mass"].shape[0]
    for k, v in p.items():
        setattr(g, k, _ptr(v))
    hp._check(hp.lib.gz_upload_device(hp._ctx, C.byref(g)))
    hp.n = int(g.n)


def _timestep_params():
    tp = abi.GzTimestepParams()
    tp.err_tol_int_accuracy, tp.courant_fac = 0.02, 0.2
    tp.max_size_timestep, tp.min_size_timestep, tp.timebase = 1e-2, 0.0, TIMEBASE
    for b in range(abi.TIMEBINS):
        tp.bin_active[b] = 1
    return tp


def _kick_state(case, seed):
    """A set in mid-run: the fields of the half-step kernels, with the spread of a clustered MFV or MFM set."""
    p, r, prm = _particles(case, seed), _Rand(seed * 31 + 7), _params(case)
    n = _n(case)
    one, i64 = torch.ones(n, device=r.dev, dtype=torch.float64), torch.zeros(n, device=r.dev, dtype=torch.int64)
    rho = p["mass"] * 32 / (VOL * p["h"] ** 3)
    cs = (prm.gamma * (prm.gamma - 1) * p["u"]).sqrt()
    s = {"pos": p["pos"], "vel": p["vel"], "u": p["u"], "mass": p["mass"], "mass_true": p["mass"].clone(), "h": p["h"],
         "rho": rho, "pressure": (prm.gamma - 1) * p["u"] * rho, "vel_pred": p["vel"].clone(), "u_pred": p["u"].clone(),
         "accel": r.normal(n, 3) * (cs ** 2 / p["h"])[:, None] * 0.1, "dudt": r.normal(n) * p["u"] * cs / p["h"] * 0.1,
         "divvel": r.normal(n) * cs / p["h"] * 0.1, "vsig": 2 * cs * r.u(n, lo=1.0, hi=2.0), "num_ngb": one * 32 ** (1 / 3),
         "pvel": p["vel"] * 0.9, "dp": torch.zeros_like(p["vel"]), "gravwork": torch.zeros_like(p["vel"]),
         "dmass": r.normal(n) * p["mass"] * 1e-4, "dtmass": r.normal(n) * p["mass"] * cs / p["h"] * 1e-3,
         "tstart": i64, "tend": i64.clone(), "ti_current": i64.clone(), "ti_begstep": i64.clone(), "dt_step": i64.clone(),
         "bin": torch.zeros(n, device=r.dev, dtype=torch.int32), "status": torch.zeros(1, device=r.dev, dtype=torch.int32)}
    return s


def prepare(case, seed):
    path = case["path"]
    st = {"case": case, "path": path, "params": _params(case)}
    if path == "kicks":
        st.update(fields=_kick_state(case, seed), tp=_timestep_params(), ti=0, step=1 << 20,
                  mfv=st["params"].method == abi.METHOD_MFV)
        return st
    p = _particles(case, seed)
    n = st["n"] = p["mass"].shape[0]
    if path == "step":
        st["step"] = DeviceStep(st["params"], _timestep_params(), p["pos"], p["vel"], p["mass"], p["u"], p["h"])
        return st
    st["in"] = p
    if path == "sums":
        st["out"] = {"acc": torch.empty(n, 14, device=_device(), dtype=torch.float64),
                     "pv": torch.empty(n, 3, device=_device(), dtype=torch.float64)}
        return st
    torch.cuda.synchronize()  # the library reads the inputs on its own stream
    hp = st["hp"] = HydroPass(st["params"])
    if case["field"] == "boxes":
        hp.set_boxes([k ** 3 for k in _counts(case)])
    if path == "host":
        st["in"] = {k: v.cpu().numpy() for k, v in p.items()}
        return st
    _upload_device(hp, p)
    hp.full_pass()  # a program in mid-run has taken a step with this handle
    if path == "replay":
        del st["in"]  # the inputs are resident in the context
    if path == "subset":
        cs = math.sqrt(st["params"].gamma * (st["params"].gamma - 1))
        key = p["h"] / (cs * p["u"].sqrt() + (p["vel"] ** 2).sum(1).sqrt())
        k = max(1, int(round(case["fraction"] * n)))
        st["active"] = torch.topk(key, k, largest=False).indices.sort().values.int().cpu().numpy()
        del st["in"]
    st["out"] = {k: torch.zeros((n,) if w == 1 else (n, w), device=_device(), dtype=torch.float64) for k, w in FIELDS}
    st["outputs"] = abi.GzOutputs()
    for k, t in st["out"].items():
        setattr(st["outputs"], k, _ptr(t))
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------- run
def _run_kicks(st):
    f, prm, tp, ti, step, mfv = st["fields"], st["params"], st["tp"], st["ti"], st["step"], st["mfv"]
    sid = torch.cuda.current_stream().cuda_stream
    tp.ti_current = ti
    timestep(prm, tp, {k: f[k] for k in ("accel", "vsig", "h", "num_ngb", "divvel", "mass", "bin", "ti_begstep", "dt_step", "status")}, sid)
    kf = {k: f[k] for k in ("vel", "u", "mass", "accel", "dudt", "vel_pred", "u_pred", "dp", "tstart", "tend")}
    df = {k: f[k] for k in ("pos", "vel_pred", "accel", "divvel", "mass", "rho", "u_pred", "dudt", "h", "pressure", "ti_current", "status")}
    if mfv:
        kf.update({k: f[k] for k in ("mass_true", "dmass", "dtmass", "gravwork")})
        df.update({k: f[k] for k in ("pvel", "dtmass", "mass_true")})
    else:
        df["vel"] = f["vel"]
    f["tstart"].fill_(ti)
    f["tend"].fill_(ti + step // 2)
    kick(prm, kf, 0, TIMEBASE, 0.0, sid)
    drift(prm, df, ti + step, TIMEBASE, 0.0, sid)
    f["tstart"].fill_(ti + step // 2)
    f["tend"].fill_(ti + step)
    kick(prm, kf, 1, TIMEBASE, 0.0, sid)
    st["ti"] = ti + step
    return {k: v for k, v in f.items() if k not in ("tstart", "tend", "accel", "vsig", "num_ngb", "divvel", "pvel", "gravwork", "dtmass")}


def run(st):
    path = st["path"]
    if path == "kicks":
        return _run_kicks(st)
    if path == "step":
        st["step"].step()
        return {k: v for k, v in st["step"].state.items()}
    if path == "sums":
        p, o = st["in"], st["out"]
        lib = abi.load_library()
        rc = lib.gz_density_sums_noalloc(C.byref(st["params"]), st["n"], p["pos"].data_ptr(), p["vel"].data_ptr(),
                                         p["mass"].data_ptr(), p["h"].data_ptr(), o["acc"].data_ptr(), o["pv"].data_ptr(),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(f"gz_density_sums_noalloc: {rc}")
        return o
    hp = st["hp"]
    if path == "host":
        hp.upload(**st["in"])
        hp.full_pass()
        return hp.download([k for k, _ in FIELDS])
    if path in ("calls", "graph"):
        _upload_device(hp, st["in"])
        if path == "calls":
            hp.full_pass()
        else:
            hp.hydro_pass(graph=True)
    elif path == "replay":
        hp.hydro_pass(graph=True, restage=True)
    else:
        hp.full_pass(st["active"])
    hp._check(hp.lib.gz_download_device(hp._ctx, C.byref(st["outputs"])))
    return st["out"]


# --------------------------------------------------------- work, tolerance
def work(case):
    n, path = _n(case), case["path"]
    ngb = 64.0 if case["field"] == "lognormal" else 32.0
    if path == "kicks":
        # every field read once and written once: 60 doubles or integers in, 34 out
        return {"bytes": 8.0 * 94 * n, "flops": 100.0 * n}
    if path == "sums":
        return {"bytes": 8.0 * (8 + 17) * n, "flops": 72.0 * ngb * n}
    act = case.get("fraction", 1.0) * n
    # one density sum at the converged length, one gradient row, one face per pair (a subset: per row entry)
    flops = act * (72.0 * ngb + 60.0 * 1.2 * ngb + 430.0 * 1.2 * ngb * (0.5 if path != "subset" else 1.0))
    outs = sum(w for _, w in FIELDS)
    return {"bytes": 8.0 * (11 * n + outs * n + (94 * n if path == "step" else 0)), "flops": flops}


def tolerance(case):
    """About four times what the same sets differ by with their axes exchanged, which visits the neighbours in
    another order.

    Lattice sets: 8e-15 of the norm in FP64 (8e-14 of a value), 1e-7 (6e-6) where the faces are FP32. Among random
    particles about one cell in a million ends the kernel-length iteration at another length that the iteration
    accepts too (it branches on sums) and carries it into its own fields: 5e-5 of the norm, 0.03 of a value."""
    if case["path"] == "sums":
        return {"rel": 1e-14, "max": 1e-12}
    if case["path"] == "kicks":
        return {"rel": 1e-14, "max": 1e-13, "differ": 0.0}
    if case["field"] in ("plummer", "lognormal"):
        return {"rel": 2e-4, "max": 0.1}
    if case["path"] == "step":  # a few steps carry the sums' rounding on
        return {"rel": 1e-6, "max": 1e-4} if case["mixed"] else {"rel": 1e-11, "max": 1e-9}
    return {"rel": 1e-6, "max": 5e-5} if case["mixed"] else {"rel": 5e-14, "max": 5e-13}


# -------------------------------------------------------------------- exact
def _pairs(pos, reach, sym, box_id=None):
    """(i, j, r) of all pairs with r < reach_i (sym: or r < reach_j), by comparing all with all."""
    n, out = pos.shape[0], []
    for b in range(0, n, 512):
        d = pos[b:b + 512, None, :] - pos[None]
        r2 = ((d - d.round()) ** 2).sum(-1)
        ok = r2 < reach[b:b + 512, None] ** 2
        if sym:
            ok |= r2 < reach[None] ** 2
        out.append(torch.nonzero(ok) + torch.tensor([b, 0], device=pos.device))
    ij = torch.cat(out)
    i, j = ij[:, 0], ij[:, 1]
    d = pos[i] - pos[j]
    d = d - d.round()
    return i, j, d, (d ** 2).sum(-1).sqrt()


def _kernel(cubic, r, h):
    u, hi = r / h, 1 / h
    t = (1 - u).clamp(min=0)
    if cubic:
        w = torch.where(u < 0.5, 1 - 6 * t * u * u, 2 * t ** 3) * (8 / math.pi) * hi ** 3
        dw = torch.where(u < 0.5, u * (18 * u - 12), -6 * t * t) * (8 / math.pi) * hi ** 4
    else:
        w = t ** 4 * (1 + 4 * u) * (21 / (2 * math.pi)) * hi ** 3
        dw = -20 * u * t ** 3 * (21 / (2 * math.pi)) * hi ** 4
    z = torch.zeros_like(w)
    return torch.where(u < 1, w, z), torch.where(u < 1, dw, z)


def _sums(p, cubic, mfv, h, i, j, d, r):
    """The 17 density sums of every particle at its kernel length, [n, 17]."""
    n = h.shape[0]
    k = r < h[i]
    i, j, d, r = i[k], j[k], d[k], r[k]
    w, dw = _kernel(cubic, r, h[i])
    dv = p["vel"][i] - p["vel"][j]
    far = (r > 0).double()
    mw = p["mass"][j] * w
    x = [w, mw, -(3 / h[i] * w + r / h[i] * dw), -dw * (d * dv).sum(-1) / r.clamp(min=1e-300) * far]
    x += [d[:, a] * d[:, b] * w for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))]
    x += [w * d[:, a] for a in range(3)] + [torch.zeros_like(w)]
    x += [mw * p["vel"][j, a] * (1.0 if mfv else 0.0) for a in range(3)]
    return torch.zeros(n, 17, device=h.device, dtype=torch.float64).index_add_(0, i, torch.stack(x, 1))


def _invert(h, ngb, acc):
    """Moment matrix inverse, condition number and face-closure error."""
    V = VOL * h ** 3 / torch.where(ngb > 0, ngb, torch.ones_like(ngb))
    a = acc[:, 4:10]
    raw = torch.stack([a[:, 0], a[:, 3], a[:, 5], a[:, 3], a[:, 1], a[:, 4], a[:, 5], a[:, 4], a[:, 2]], 1).view(-1, 3, 3)
    T = raw * h[:, None, None]
    add = 1.05 * torch.diagonal(T, dim1=1, dim2=2).sum(1) / 3 / 1e4
    eye = torch.eye(3, device=h.device, dtype=torch.float64)
    for _ in range(64):
        inv = torch.linalg.inv_ex(T).inverse
        cn = ((T ** 2).sum((1, 2)) * (inv ** 2).sum((1, 2))).sqrt().div(3).clamp(min=1)
        bad = ~(cn < 1e4)
        if not bad.any():
            break
        T = T + (bad * add)[:, None, None] * eye
        add = add * 1.2
    dx2 = V * torch.diagonal(raw, dim1=1, dim2=2).sum(1)
    Tn = inv * h[:, None, None]
    fce = (2 * V[:, None] * (Tn @ acc[:, 10:13, None])[..., 0]).abs().sum(1) / 3 / (6 * dx2)
    return Tn, cn, fce


def _next_h(prm, it, h, acc, cond, sc):
    """One step of the bracketed kernel-length iteration: (new length, converged). `sc`: the bracket, in place."""
    big = torch.where
    n0 = acc[:, 0]
    drk = acc[:, 2] * h / (3 * n0)
    ngb = n0 * VOL * h ** 3
    drk = big(drk > -0.9, 1 / (1 + drk), torch.ones_like(drk))
    _, cn, fce = _invert(h, ngb, acc)
    cur = sc["cn"]
    corr = big(cur > 100, (1 + (cur - 100) / 1e3).clamp(min=0).sqrt(), torch.ones_like(cur)).clamp(max=2)
    corr = big(fce > 0.35, torch.maximum(corr, (fce / 0.35).clamp(max=2)), corr)
    des, dev = prm.des_num_ngb * corr, prm.max_num_ngb_dev * corr
    if it > 1:
        dev = torch.minimum(0.25 * des, dev * torch.exp(0.1 * torch.log(des / (16 * dev)) * it))
    top = prm.max_kernel_radius
    low, high = ngb < des - dev, ngb > des + dev
    redo = (low & (h < 0.999 * top)) | high
    setmax = (h >= 0.999 * top) & low & (h != top)
    redo = big((h >= 0.999 * top) & low, setmax, redo)
    L, R = sc["left"], sc["right"]
    tight = redo & (L > 0) & (R > 0) & (R - L < 1e-3 * L)
    redo = redo & ~tight
    sc["cn"] = big(redo, cur, cn)
    free = redo & ~setmax
    L = big(free & low, torch.maximum(h, L), L)
    R = big(free & ~low, big((R == 0) | (h < R), h, R), R)
    sc["left"], sc["right"] = L, R
    lr = torch.log(des / ngb) / 3
    # both ends known
    jump = torch.log(R.clamp(min=1e-300) / L.clamp(min=1e-300)) * 0.2 if it > 1 else torch.zeros_like(h)
    var = drk * lr
    if it > 1:
        var = big(var.abs() < jump, big(var < 0, -jump, jump), var)
    two = big(ngb > 1, h * torch.exp(var), 2 * h)
    inside = (two < R) & (two > L)
    inner = two
    if it > 1:
        inner = torch.minimum(inner, R / torch.exp(jump))
        inner = big(inner < L * torch.exp(jump), L * torch.exp(jump), inner)
    outer = (torch.maximum(torch.minimum(two, R), L) * L * R).clamp(min=0) ** (1 / 3)
    two = big(inside, inner, outer)
    # one end known
    slope = big(drk < 1, 0.5 * (drk + 1), drk) if it > 2 else drk
    near = (ngb < 2 * des) & (ngb > 0.1 * des)
    lim = big(ngb > 1, lr, torch.full_like(lr, 1.4))
    fac = lim * slope
    if it >= 4:
        fac = big(drk == 1, fac * 10, fac)
    up = big(near, torch.minimum(fac, lim + 0.231), lim)
    lim_d = lim.clamp(min=-1.535)
    fac_d = lim_d * slope
    if it >= 4:
        fac_d = big(drk == 1, fac_d * 10, fac_d)
    down = big(near, torch.maximum(fac_d, lim_d - 0.231), lim_d)
    new = big((L > 0) & (R > 0), two, h * torch.exp(big(R == 0, up, down)))
    new = big(setmax, torch.full_like(h, top), new).clamp(prm.min_kernel_radius, top)
    return big(redo, new, h), ~redo


def _limit(g, hi, lo, alim, h, tol, dmax=None, cen=None):
    a = g.norm(dim=1)
    c = 1 / (alim * h * a)
    big, small = torch.maximum(hi.abs(), lo.abs()), torch.minimum(hi.abs(), lo.abs())
    f = torch.minimum(small + tol * big, big)
    c = c * f
    if cen is not None:  # positive fields
        fm = torch.minimum(cen, torch.minimum(0.5 * (cen + lo), cen - f).clamp(min=0))
        c = torch.minimum((cen - fm) / dmax / a, c)
    return torch.where((a > 0) & (c < 1), c, torch.ones_like(c))[:, None] * g


def _exact_density(p, prm):
    cubic, mfv = prm.kernel == abi.KERNEL_CUBIC, prm.method == abi.METHOD_MFV
    h, n = p["h"].clone(), p["h"].shape[0]
    built = 1.5 * h
    pairs = _pairs(p["pos"], built, False)
    sc = {k: torch.zeros_like(h) for k in ("left", "right", "cn")}
    todo = torch.ones(n, device=h.device, dtype=torch.bool)
    for it in range(150):
        if (h > built).any():
            built = 1.5 * torch.maximum(h, p["h"])
            pairs = _pairs(p["pos"], built, False)
        acc = _sums(p, cubic, mfv, h, *pairs)
        if not todo.any():
            break
        t = {k: v[todo] for k, v in sc.items()}
        nh, conv = _next_h(prm, it, h[todo], acc[todo], p["cond"][todo], t)
        for k in sc:
            sc[k][todo] = t[k]
        h[todo] = nh
        todo[todo.clone()] = ~conv
    ngb = acc[:, 0] * VOL * h ** 3
    drk = acc[:, 2] * h / (3 * acc[:, 0])
    drk = torch.where(drk > -0.9, 1 / (1 + drk), torch.ones_like(drk))
    Tn, cn, fce = _invert(h, ngb, acc)
    rho = p["mass"] * ngb / (VOL * h ** 3)
    pv = p["vel"] * 0.7 + acc[:, 14:17] * (0.3 / acc[:, 1:2]) if mfv else torch.zeros_like(p["vel"])
    six = torch.stack([Tn[:, 0, 0], Tn[:, 1, 1], Tn[:, 2, 2], Tn[:, 0, 1], Tn[:, 1, 2], Tn[:, 0, 2]], 1)
    return {"h": h, "num_ngb": ngb ** (1 / 3), "drkern": drk, "divvel": acc[:, 3] / acc[:, 0] * drk, "rho": rho,
            "pressure": (prm.gamma - 1) * p["u"] * rho, "nvt": six, "cond": cn, "fce": fce, "pvel": pv}, Tn


def _exact_gradients(p, prm, o, Tn, i, j, d, r):
    n, dev = o["h"].shape[0], p["pos"].device
    q = torch.cat([o["rho"][:, None], o["pressure"][:, None], p["vel"]], 1)
    dq = q[j] - q[i]
    w, _ = _kernel(prm.kernel == abi.KERNEL_CUBIC, r, o["h"][i])
    s = torch.zeros(n, 3, 5, device=dev, dtype=torch.float64).index_add_(0, i, -w[:, None, None] * d[:, :, None] * dq[:, None, :])
    ext = i[:, None].expand(-1, 5)
    hi = torch.zeros(n, 5, device=dev, dtype=torch.float64).scatter_reduce_(0, ext, dq, "amax")
    lo = torch.zeros(n, 5, device=dev, dtype=torch.float64).scatter_reduce_(0, ext, dq, "amin")
    far = torch.zeros(n, device=dev, dtype=torch.float64).scatter_reduce_(0, i, r, "amax")
    g = Tn @ s
    alim = torch.where(o["cond"] > 100, (0.25 + 0.25 * (o["cond"] - 100) / 100).clamp(max=0.5), torch.full_like(far, 0.25))
    dmax = torch.maximum(o["h"], far)
    gv = [_limit(g[:, :, 2 + c], hi[:, 2 + c], lo[:, 2 + c], alim, o["h"], 0.1) for c in range(3)]
    return {"grad_rho": _limit(g[:, :, 0], hi[:, 0], lo[:, 0], alim, o["h"], 0.0, dmax, o["rho"]),
            "grad_p": _limit(g[:, :, 1], hi[:, 1], lo[:, 1], alim, o["h"], 0.1, dmax, o["pressure"]),
            "grad_v": torch.cat(gv, 1)}


def _face_states(qi, gi, qj, gj, di, dj):
    """Pairwise-limited reconstruction at the face: (state from j, state from i)."""
    R, L = qi + (gi * di).sum(-1), qj + (gj * dj).sum(-1)
    lo, hi = torch.minimum(qi, qj), torch.maximum(qi, qj)
    f = 0.5 * (hi - lo)
    top, bot = hi + f, lo - f
    top = torch.where((hi < 0) & (top > 0), hi * hi / (hi - (top - hi)), top)
    bot = torch.where((lo > 0) & (bot < 0), lo * lo / (lo + (lo - bot)), bot)
    med = 0.5 * (qi + qj)
    mx, mn = torch.minimum(med + 0.375 * (hi - lo), top), torch.maximum(med - 0.375 * (hi - lo), bot)
    up = qi < qj
    R = torch.where(up, torch.minimum(torch.maximum(R, bot), mx), torch.maximum(torch.minimum(R, top), mn))
    L = torch.where(up, torch.maximum(torch.minimum(L, top), mn), torch.minimum(torch.maximum(L, bot), mx))
    same = qi == qj
    return torch.where(same, qi, L), torch.where(same, qi, R)


def _star(rl, rr, pl, pr, vl, vr, L2, R2, v_roe, n_, lim, G):
    """Star pressure and contact speed of the MFM face: (P, S) before the iterative solver, (P, S) after it."""
    MR = 1e-56
    cl, cr = (G * pl / rl).sqrt(), (G * pr / rr).sqrt()
    hl = pl / rl + pl / ((G - 1) * rl) + 0.5 * L2
    hr = pr / rr + pr / ((G - 1) * rr) + 0.5 * R2
    cm = torch.maximum(cl, cr)

    def clamp(P, S):
        low = P <= MR
        return torch.where(low, torch.full_like(P, MR), P), torch.where(low, torch.zeros_like(S), S)

    sl, sr = torch.minimum(vl, vr) - cm, torch.maximum(vl, vr) + cm
    wl, wr = rl * (sl - vl), rr * (sr - vr)
    S = ((pr - pl) + wl * vl - wr * vr) / (wl - wr)
    P, S = clamp((pl * wr - pr * wl + wl * wr * (vr - vl)) / (wr - wl), S)
    bad = ~(P <= lim)
    ql, qr = rl.sqrt(), rr.sqrt()
    vroe, h_roe = (v_roe * n_).sum(-1), (ql * hl + qr * hr) / (ql + qr)
    croe = ((G - 1) * (h_roe - 0.5 * (v_roe ** 2).sum(-1))).clamp(min=1e-30).sqrt()
    sr, sl = torch.maximum(vr + cr, vroe + croe), torch.minimum(vl - cl, vroe - croe)
    wr, wl = rr * (sr - vr), -rl * (sl - vl)
    S2 = ((wr * vr + wl * vl) + (pl - pr)) / (wr + wl)
    P2, S2 = clamp(rl * (vl - sl) * (vl - S2) + pl, S2)
    P, S = torch.where(bad, P2, P), torch.where(bad, S2, S)
    bad &= ~(P <= lim)
    rc = (rl + rr) * (cl + cr)
    P3 = 0.5 * ((pl + pr) + (vl - vr) * 0.25 * rc)
    sp = torch.maximum((vl.abs() + cl), (vr.abs() + cr))
    P3, S3 = clamp(P3, torch.minimum(torch.maximum(0.5 * (vr + vl) + 2 * (pl - pr) / rc, -sp), sp))
    P, S = torch.where(bad, P3, P), torch.where(bad, S3, S)
    vac = (vr - vl) > cm
    P, S = torch.where(vac, torch.full_like(P, MR), P), torch.where(vac, torch.zeros_like(S), S)
    again = ~(P <= lim)
    # Newton iteration for the star pressure (Toro's exact solver); separating faces leave a vacuum
    X = (pl + pr) * 0.5
    for _ in range(200):
        def side(p_, r_, c_):
            a = (2 / (G + 1) / r_ / (X + (G - 1) / (G + 1) * p_)).sqrt()
            shock = (X - p_) * a, a * (1 - 0.5 * (X - p_) / ((G - 1) / (G + 1) * p_ + X))
            fan = 2 / (G - 1) * c_ * (torch.pow(X / p_, (G - 1) / (2 * G)) - 1), 1 / (r_ * c_) * torch.pow(X / p_, -(G + 1) / (2 * G))
            return torch.where(X > p_, shock[0], fan[0]), torch.where(X > p_, shock[1], fan[1])
        (fl, zl), (fr, zr) = side(pl, rl, cl), side(pr, rr, cr)
        X = torch.maximum(X - (fl + fr + vr - vl) / (zl + zr), 0.1 * X)
    open_ = 2 / (G - 1) * (cl + cr) - (vr - vl) < 0
    Pe = torch.where(open_, torch.zeros_like(X), X)
    Se = 0.5 * (vl + vr) + 0.5 * (fr - fl)
    return P, S, torch.where(again, Pe, P), torch.where(again, Se, S)


def _exact_force(p, prm, o, i, j, d, r):
    """MFM face fluxes of every pair and their sums. (i, j) hold every pair once."""
    G, cubic = prm.gamma, prm.kernel == abi.KERNEL_CUBIC
    n, dev = o["h"].shape[0], d.device
    m, v, rho, P, h = p["mass"], p["vel"], o["rho"], o["pressure"], o["h"]
    cs, V = (G * P / rho).sqrt(), p["mass"] / rho
    wi, dwi = _kernel(cubic, r, h[i])
    wj, dwj = _kernel(cubic, r, h[j])
    dv = v[i] - v[j]
    vdr = (d * dv).sum(-1)
    vsig = cs[i] + cs[j] - torch.where(vdr < 0, vdr / r, torch.zeros_like(r)) + (cs[i] - cs[j]).abs()
    Vi, Vj = V[i], V[j]
    contrast = (Vi - Vj).abs() / torch.minimum(Vi, Vj) / 3 > 1.25
    mean = Vi * Vj * (wi + wj) / (Vi * wi + Vj * wj)
    wti, wtj = torch.where(contrast, mean, Vi), torch.where(contrast, mean, Vj)
    s = o["nvt"]
    T = torch.stack([s[:, 0], s[:, 3], s[:, 5], s[:, 3], s[:, 1], s[:, 4], s[:, 5], s[:, 4], s[:, 2]], 1).view(-1, 3, 3)
    A = (T[i] @ d[..., None])[..., 0] * (wi * wti)[:, None] + (T[j] @ d[..., None])[..., 0] * (wj * wtj)[:, None]
    crit = 1e6 - o["cond"][i] ** 2
    sph = (o["cond"][j] ** 2 > 1e12 + crit) | ((A * d).sum(-1) < 0)
    fk = -(wti * Vi * dwi + wtj * Vj * dwj) / r
    A = torch.where(sph[:, None], d * fk[:, None], A)
    area = A.norm(dim=1)
    live = area > 0
    nrm = A / torch.where(live, area, torch.ones_like(area))[:, None]
    e = d / r[:, None]
    di, dj = e * (-0.5 * r)[:, None], e * (0.5 * r)[:, None]
    frame = 0.5 * (v[i] + v[j])
    fvi, fvj = (v[i] * nrm).sum(-1), (v[j] * nrm).sum(-1)
    vd = vdr / r
    app = torch.where(vd < 0, vd * vd, torch.zeros_like(vd))
    app = torch.where(fvi < fvj, torch.maximum(app, (fvi - fvj) ** 2), app)
    flat = 0.5 * (o["fce"][i] + o["fce"][j]) > 1
    lim = 1.1 * torch.maximum(P[i] + rho[i] * app, P[j] + rho[j] * app)
    lim = torch.where(flat, torch.maximum(lim, torch.maximum(torch.maximum(P[i], P[j]), 2 * torch.maximum(rho[i], rho[j]) * app)), lim)

    def face(q, g):
        L, R = _face_states(q[i], g[i], q[j], g[j], di, dj)
        return torch.where(flat, q[j], L), torch.where(flat, q[i], R)

    rl, rr = face(rho, o["grad_rho"])
    pl, pr = face(P, o["grad_p"])
    vl, vr = [], []
    for c in range(3):
        g = o["grad_v"][:, 3 * c:3 * c + 3]
        L, R = _face_states(v[i, c] - frame[:, c], g[i], v[j, c] - frame[:, c], g[j], di, dj)
        vl.append(torch.where(flat, v[j, c] - frame[:, c], L))
        vr.append(torch.where(flat, v[i, c] - frame[:, c], R))
    vl, vr = torch.stack(vl, 1), torch.stack(vr, 1)

    def solve(rl, rr, pl, pr, vl, vr, lim):
        ql, qr = rl.sqrt()[:, None], rr.sqrt()[:, None]
        return _star(rl, rr, pl, pr, (vl * nrm).sum(-1), (vr * nrm).sum(-1), (vl ** 2).sum(-1), (vr ** 2).sum(-1),
                     (vl * ql + vr * qr) / (ql + qr), nrm, lim, G)

    P0, S0, PM, SM = solve(rl, rr, pl, pr, vl, vr, lim)
    for k in (1, 2):  # cell-centred states, then the same at rest
        again = (PM < 0) | PM.isnan() | ((PM > 1.4 * lim) if k == 1 else torch.zeros_like(live))
        zero = 1.0 if k == 1 else 0.0
        new = solve(rho[j], rho[i], P[j], P[i], (v[j] - frame) * zero, (v[i] - frame) * zero, (1.4 if k == 1 else 2.0) * lim)
        P0, S0, PM, SM = (torch.where(again, a, b) for a, b in zip(new, (P0, S0, PM, SM)))
    live = live & (PM > 0)
    mom = nrm * P0[:, None]
    en = P0 * S0 + (frame * mom).sum(-1)
    # the entropic switch between the Riemann work and the PdV work of the face
    work_f, rel = PM * area, SM.abs() / torch.minimum(cs[i], cs[j])
    pdv = PM * vd
    old = work_f * (SM + 0.5 * (fvi + fvj))
    new = 0.5 * (dwi * Vi ** 2 * o["drkern"][i] * pdv - dwj * Vj ** 2 * o["drkern"][j] * pdv + work_f * (fvi + fvj))
    c2 = o["cond"][j] ** 2
    prd = P / rho
    tj, ti = -old + work_f * fvj, old - work_f * fvi
    nj, ni = -new + work_f * fvj, new - work_f * fvi
    hot_i, hot_j = prd[i] > 1.001 * prd[j], 1.001 * prd[i] < prd[j]
    one_i, one_j = (tj > 0) | ((tj < 0) & (tj > nj)), (ti > 0) | ((ti < 0) & (ti > ni))
    both = ((tj < 0) & (tj > nj)) | ((ti < 0) & (ti > ni))
    refuse = torch.where(hot_i, one_i, torch.where(hot_j, one_j, both)) & (rel > 1e-3) & (c2 < crit)
    use = ((rel < 0.5) | flat) & (~refuse | (c2 >= crit))
    flux = area * en + torch.where(use, new - old, torch.zeros_like(new))
    flux, mom = torch.where(live, flux, torch.zeros_like(flux)), torch.where(live[:, None], mom * area[:, None], torch.zeros_like(mom))
    acc = torch.zeros(n, 3, device=dev, dtype=torch.float64).index_add_(0, i, mom).index_add_(0, j, -mom)
    en = torch.zeros(n, device=dev, dtype=torch.float64).index_add_(0, i, flux).index_add_(0, j, -flux)
    vs = cs.clone().scatter_reduce_(0, i, vsig, "amax").scatter_reduce_(0, j, vsig, "amax")
    du = (en - (v * acc).sum(-1)) / m
    z = torch.zeros(n, device=dev, dtype=torch.float64)
    return {"accel": acc / m[:, None], "dudt": torch.where(h >= 0.99 * prm.max_kernel_radius, z, du), "vsig": vs,
            "dtmass": z, "dmass": z.clone(), "gravwork": torch.zeros(n, 3, device=dev, dtype=torch.float64)}


def _exact_kicks(case, seed):
    f, prm, tp, step = _kick_state(case, seed), _params(case), _timestep_params(), 1 << 20
    mfv = prm.method == abi.METHOD_MFV
    core = 1.61199 * f["h"] / f["num_ngb"]
    ac = f["accel"].norm(dim=1).clamp(min=1e-30)
    dt = (2 * tp.err_tol_int_accuracy * core / ac).sqrt()
    dt = torch.minimum(dt, tp.courant_fac * core / (0.5 * f["vsig"]))
    dt = torch.minimum(dt, 1.5 / f["divvel"].abs()).clamp(max=tp.max_size_timestep)
    f["bin"] = torch.floor(torch.log2((dt / TIMEBASE).floor())).int()
    f["dt_step"] = torch.pow(2.0, f["bin"].double()).long()

    def half(mode):
        t = step // 2 * TIMEBASE
        if mfv:
            dm = f["dmass"].clone()
            if mode:
                dm = t * f["dtmass"]
                dm = torch.where(dm * f["dmass"] < 0, torch.zeros_like(dm), dm)
                dm = torch.where(dm.abs() > f["dmass"].abs(), f["dmass"], dm)
            on = f["dmass"] != 0
            f["dmass"] = torch.where(on, f["dmass"] - dm, f["dmass"])
            f["mass_true"] = torch.where(on, f["mass_true"] + torch.maximum(dm, -0.99 * f["mass_true"]), f["mass_true"])
            inv = 1 / torch.where(on, f["mass_true"], f["mass"])
        else:
            inv = 1 / f["mass"]
        f["u"] = torch.maximum(f["u"] + f["dudt"] * t, 0.5 * f["u"])
        dp = f["accel"] * (f["mass"] * t)[:, None]
        f["vel"] = f["vel"] + dp * inv[:, None]
        f["dp"] = f["dp"] + dp
        if mode:
            f["vel_pred"], f["u_pred"] = f["vel"].clone(), f["u"].clone()
            f["mass"] = f["mass_true"].clone() if mfv else f["mass"]

    half(0)
    t = step * TIMEBASE
    f["pos"] = f["pos"] + (f["pvel"] if mfv else f["vel"]) * t
    lc = (f["divvel"] * t).clamp(-0.3, 0.3)
    f["vel_pred"] = f["vel_pred"] + f["accel"] * t
    if mfv:
        f["mass"] = torch.maximum(f["mass"] + f["dtmass"] * t, 0.5 * f["mass_true"])
    f["rho"] = f["rho"] * torch.exp(-lc)
    f["u_pred"] = torch.maximum(f["u_pred"] + f["dudt"] * t, 0.5 * f["u_pred"])
    f["h"] = (f["h"] * torch.exp(lc / 3)).clamp(prm.min_kernel_radius, prm.max_kernel_radius)
    f["pressure"] = (prm.gamma - 1) * f["u_pred"] * f["rho"]
    half(1)
    f["ti_current"] = torch.full_like(f["ti_current"], step)
    return {k: v for k, v in f.items() if k not in ("tstart", "tend", "accel", "vsig", "num_ngb", "divvel", "pvel", "gravwork", "dtmass")}


def exact(case, seed):
    """The kicks, the density sums, and one whole pass of up to 40,000 particles; above that comparing all with
    all takes too long. Subsets and steps carry a library state from pass to pass, box sets mix boxes: no value.
    The MFV fluxes of a pass have no value here either (density and gradients do)."""
    path = case["path"]
    if path == "kicks":
        return _exact_kicks(case, seed)
    if path in ("subset", "step") or case["field"] == "boxes" or _n(case) > 40000:
        return None
    prm, p = _params(case), _particles(case, seed)
    if path == "sums":
        acc = _sums(p, prm.kernel == abi.KERNEL_CUBIC, prm.method == abi.METHOD_MFV, p["h"], *_pairs(p["pos"], p["h"], False))
        return {"acc": acc[:, :14].contiguous(), "pv": acc[:, 14:].contiguous()}
    out, Tn = _exact_density(p, prm)
    i, j, d, r = _pairs(p["pos"], out["h"], True)
    k = r > 0
    i, j, d, r = i[k], j[k], d[k], r[k]
    out.update(_exact_gradients(p, prm, out, Tn, i, j, d, r))
    if prm.method == abi.METHOD_MFM:
        k = i < j
        out.update(_exact_force(p, prm, out, i[k], j[k], d[k], r[k]))
    else:
        out.update({k: None for k in FORCE})
    if path == "host":
        out = {k: v if v is None else v.cpu().numpy() for k, v in out.items()}
    return out
