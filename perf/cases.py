"""Workloads of the B200 AWP-ODC-SGT framework for timing and for checking
results: time stepping over the grids, media, components, precisions and
boundaries that SGT jobs use, whole small SGT jobs, and the reciprocity
synthesis of rupture variations.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs and handles a user's program has before the call
  run(state)          one pass through the public entry points
  work(case)          bytes and floating-point operations a pass cannot do without
  exact(case, seed)   what run returns, in 64 bits by plain torch / numpy

A "steps" pass advances a solve that is under way: the wavefield is filled
with a smooth random state, so that the pass works on values a running job
meets, and the source keeps adding to it.  A "job" pass is one whole SGT job
from host arrays to host SGTs.  A "synth" pass is one rupture: its variations
added, synthesised against the resident SGT set, the seismograms back on the
host.
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cybershake-core_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import awp_inputs as ai  # noqa: E402
import awpsgt  # noqa: E402

_WAVE = awpsgt.FIELDS[:9]            # u v w and the six stresses
_MEM = awpsgt.FIELDS[9:15]           # r1..r6
_ND = 20                             # width of the absorbing boundary, as CyberShake runs it
_DH, _DT = 100.0, 0.005
_FL, _FH, _FP = 0.01, 25.0, 0.5


def _steps(name, nx, ny, nz, comps, steps, **kw):
    c = {"kind": "steps", "nx": nx, "ny": ny, "nz": nz, "comps": comps, "steps": steps, "precision": "f32",
         "medium": "layered", "nve": 1, "npc": 0, "subfaults": 0, "monitor": 0, "npts": 1000}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def _job(name, nx, ny, nz, comps, nt, npts, nvar=3):
    c = {"kind": "job", "nx": nx, "ny": ny, "nz": nz, "comps": comps, "nt": nt, "npts": npts, "nvar": nvar}
    if name:
        c["name"] = name
    return c


def _synth(name, nx_f, nz_f, nt, nv, ntout, ncomp, nstf0, nstf1):
    c = {"kind": "synth", "nx_f": nx_f, "nz_f": nz_f, "nt": nt, "nv": nv, "ntout": ntout, "ncomp": ncomp,
         "nstf0": nstf0, "nstf1": nstf1}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest grid of the serving stream, one component: launches and
        # the length of one column march decide, not bandwidth
        _steps("steps_100x100x50_fx", 100, 100, 50, "1", 50, npts=200),
        # the plain single-component FP32 job (homogeneous half-space, 1000 points)
        _steps("steps_160x160x80_fx", 160, 160, 80, "1", 50, medium="homogeneous"),
        # a mid-sized request of the serving stream, sizes that fit no tile
        _steps("steps_251x187x93_fxfy", 251, 187, 93, "12", 20),
        # the batched three-component job on the layered medium
        _steps("steps_400x400x200_fxfyfz", 400, 400, 200, "123", 10, npts=5000),
        # the large two-component job with 16-bit media and memory variables
        _steps("steps_640x640x256_fxfy_f16", 640, 640, 256, "12", 10, precision="f16", npts=5000),
        # FP32 media, 16-bit memory variables within 1e-4 of FP64, largest serving grid
        _steps("steps_500x500x250_fxfy_bfp", 500, 500, 250, "12", 10, precision="bfp"),
        # the elastic scheme, one component, with the stability monitor on
        _steps("steps_333x222x111_fz_elastic", 333, 222, 111, "3", 20, nve=0, monitor=10),
        # the PML boundary (NPC = 1), three components
        _steps("steps_300x280x150_fxfyfz_pml", 300, 280, 150, "123", 10, npc=1),
        # a kinematic rupture of 1600 subfaults radiating into the layered medium
        _steps("steps_320x200x100_rupture", 320, 200, 100, "1", 20, subfaults=1600),
        # a whole short job, host arrays in, SGTs in RWG order out
        _job("job_120x110x60_fxfy", 120, 110, 60, "12", 200, 500),
        # one rupture of an ordinary site: few variations of a small fault
        _synth("synth_12x6_8var", 12, 6, 400, 8, 600, 2, 8, 40),
        # a large rupture: 64 variations of 1024 points
        _synth("synth_32x32_64var", 32, 32, 1500, 64, 2000, 2, 20, 80),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "store", "store", "pml", "elastic", "rupture", "job", "synth"])
    if kind == "job":
        c = _job(None, _logint(rng, 64, 200), _logint(rng, 64, 200), _logint(rng, 32, 100),
                 rng.choice(["1", "2", "3", "12", "123"]), rng.choice([100, 150, 200]), _logint(rng, 100, 2000))
        return c
    if kind == "synth":
        return _synth(None, _logint(rng, 6, 40), _logint(rng, 4, 24), _logint(rng, 200, 1500), _logint(rng, 2, 64),
                      _logint(rng, 300, 2000), rng.choice([1, 2, 2, 3]), 8, rng.choice([40, 80, 120]))
    comps = rng.choice(["1", "2", "3", "12", "13", "123", "123"])
    while True:
        nx, ny, nz = _logint(rng, 64, 640), _logint(rng, 64, 640), _logint(rng, 48, 256)
        updates = nx * ny * nz * len(comps)
        if kind == "pml":
            updates *= 2
        if updates <= 9.0e7:
            break
    steps = 50 if updates < 2.0e6 else (20 if updates < 2.0e7 else 10)
    kw = {"npts": _logint(rng, 100, 3000) if updates > 4.0e6 else 200}
    if kind == "store":
        kw["precision"] = rng.choice(["mixed", "bfp", "f16", "bf16"])
    elif kind == "pml":
        kw["npc"] = 1
    elif kind == "elastic":
        kw["nve"] = 0
        kw["monitor"] = rng.choice([0, 10])
    elif kind == "rupture":
        comps = "1"
        kw["subfaults"] = _logint(rng, 20, 2000)
    else:
        kw["medium"] = rng.choice(["layered", "layered", "homogeneous"])
    return _steps(None, nx, ny, nz, comps, steps, **kw)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed, salt):
    return torch.Generator(device=_dev()).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _smooth(shape, cells, g):
    """Unit-amplitude random field that varies over about `cells` cells."""
    coarse = [max(2, -(-n // cells) + 1) for n in shape]
    t = torch.randn([1, 1] + coarse, generator=g, device=_dev())
    return F.interpolate(t, size=tuple(shape), mode="trilinear", align_corners=True)[0, 0]


def _media(case, seed):
    """Media file image [nz][ny][nx][vp vs rho] on the host."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case.get("medium") == "homogeneous":
        vs = torch.full((nz, ny, nx), 3464.0 * (1.0 + 0.01 * (seed % 7)), device=_dev())
        vp, rho = vs * (6000.0 / 3464.0), torch.full_like(vs, 2700.0)
    else:
        layer = torch.div(torch.arange(nz, device=_dev()) * 8, nz, rounding_mode="floor").float()
        vs = 500.0 * 8.0 ** (layer / 7.0)                     # 8 layers, 500 .. 4000 m/s
        pert = _smooth((nz, ny, nx), 20, _gen(seed, 1)).mul_(0.05).clamp_(-0.15, 0.15)
        vs = vs[:, None, None] * (1.0 + pert)
        vp = 1.73 * vs
        rho = 1740.0 * (vp / 1000.0) ** 0.25
    return torch.stack((vp, vs, rho), dim=-1).cpu().numpy()


def _stf(nst, column, seed):
    """Band-limited source table [nst][6], a sum of sines of seeded phases."""
    rng = np.random.default_rng(seed * 11 + column)
    t = np.arange(nst) * _DT
    s = sum(np.sin(2.0 * np.pi * f * t + rng.uniform(0, 2 * np.pi)) for f in (0.3, 0.5, 0.8, 1.1, 1.7))
    out = np.zeros((nst, 6), np.float32)
    out[:, column] = (1.0e9 * s).astype(np.float32)
    return out


def _rupture(case, seed):
    """Subfault cells (a dipping plane, some cells shared) and their table
    rows [type slip t_rupture t_rise area 0] [strike dip rake 0 0 0]."""
    n, nx, ny, nz = case["subfaults"], case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed + 77)
    along = max(1, min(n, nx - 2 * _ND - 4))
    m = np.arange(n)
    xyz = np.stack([_ND + 3 + m % along, np.full(n, ny // 2), 1 + (m // along) % max(1, nz - _ND - 2)], axis=1)
    xyz[:, 1] += xyz[:, 2] // 4
    xyz[:, 1] = np.minimum(xyz[:, 1], ny)
    k = max(1, n // 50)
    xyz[rng.integers(0, n, k)] = xyz[rng.integers(0, n, k)]
    t = np.zeros((n, 2, 6), np.float32)
    t[:, 0, 0] = 1 + m % 3
    t[:, 0, 1] = rng.uniform(0.5, 2.0, n)
    t[:, 0, 2] = rng.uniform(0.0, 20 * _DT, n)
    t[:, 0, 3] = rng.uniform(20.0, 60.0, n)
    t[:, 0, 4] = 1.0e4
    t[:, 1, 0] = 300.0 + rng.uniform(-5.0, 5.0, n)
    t[:, 1, 1] = rng.uniform(60.0, 90.0, n)
    t[:, 1, 2] = rng.uniform(-180.0, 180.0, n)
    return xyz.astype(np.int32), t


def _igreen(case):
    return tuple(int(x) for x in case["comps"])


def _points(case, seed):
    zmax = max(1, min(case["nz"], 101))
    n = min(case["npts"], case["nx"] * case["ny"] * zmax // 2)
    return ai.sgt_points(case["nx"], case["ny"], zmax, n, seed=int(seed) & 0x7fffffff)


def _source_xyz(case):
    return (case["nx"] // 2, case["ny"] // 2, min(case["nz"] // 2, 21))


def _steps_params(case):
    cells = case["nx"] * case["ny"] * case["nz"] * len(case["comps"])
    nt = 400000 if cells < 4.0e6 else 20000
    kw = dict(nd=_ND, arbc=0.92, fl=_FL, fh=_FH, fp=_FP, socalq=1, nve=case["nve"], ntiskp_sgt=10,
              igreen=_igreen(case), precision=case["precision"], monitor_every=case["monitor"], npc=case["npc"])
    nst = min(nt, 20000)
    if case["subfaults"]:
        nst = 2
        kw["kinematic"] = 1
    return awpsgt.make_params(case["nx"], case["ny"], case["nz"], _DH, _DT, nt, nst=nst, **kw)


def _wave_inputs(case, seed):
    """(component, field name, interior values [nz][ny][nx]) of the state the
    pass starts from."""
    shape = (case["nz"], case["ny"], case["nx"])
    for q in range(len(case["comps"])):
        for f, name in enumerate(_WAVE):
            yield q, name, _smooth(shape, 8, _gen(seed, 100 + 16 * q + f)).mul_(1.0e-3 if f < 3 else 5.0e3)
        if case["nve"] and case["precision"] == "f32":
            for f, name in enumerate(_MEM):
                yield q, name, _smooth(shape, 8, _gen(seed, 109 + 16 * q + f)).mul_(5.0e1)


class _Memory:
    """Device memory of a solver as torch reads it; keeps the solver alive as
    long as a tensor on it lives."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3,
                                         "strides": None}


def _view(solver, name, q):
    """Interior of a device field [nz][ny][nx] (awp_device_field)."""
    ptr, L = solver.device_field(name, q)
    t = torch.as_tensor(_Memory(solver, ptr, (L.nz + 4, L.plane // L.pitch, L.pitch)), device="cuda")
    return t[2:2 + L.nz, 2:2 + L.ny, 8:8 + L.nx]


def _prepare_steps(case, seed):
    p = _steps_params(case)
    s = awpsgt.Solver(p)
    s.load_media(_media(case, seed))
    if case["subfaults"]:
        xyz, tab = _rupture(case, seed)
        s.set_source(0, xyz, tab)
    else:
        for q, ig in enumerate(_igreen(case)):
            s.set_source(q, [_source_xyz(case)], _stf(p.nst, ig - 1, seed))
    s.set_points(_points(case, seed))
    for q, name, v in _wave_inputs(case, seed):
        _view(s, name, q).copy_(v)
    torch.cuda.synchronize()
    out = [_view(s, name, q) for q in range(p.ncomp) for name in _WAVE]
    return {"case": case, "solver": s, "out": out, "nt": p.nt, "done": 0}


def _run_steps(st):
    n = st["case"]["steps"]
    if st["done"] + n > st["nt"]:
        st["solver"].reset()
        st["done"] = 0
    st["solver"].run(n)
    st["done"] += n
    return st["out"]


def _job_params(case):
    return awpsgt.make_params(case["nx"], case["ny"], case["nz"], _DH, _DT, case["nt"], nst=case["nt"] - 1, nd=_ND,
                              arbc=0.92, fl=_FL, fh=_FH, fp=_FP, socalq=1, ntiskp_sgt=10, igreen=_igreen(case))


def _prepare_job(case, seed):
    p = _job_params(case)
    stf = [_stf(p.nst, ig - 1, seed) for ig in _igreen(case)]
    return {"case": case, "params": p, "media": _media(case, seed), "src": _source_xyz(case), "stf": stf,
            "pts": _points(case, seed)}


def _run_job(st):
    with awpsgt.Solver(st["params"]) as s:
        s.load_media(st["media"])
        for q, t in enumerate(st["stf"]):
            s.set_source(q, [st["src"]], t)
        s.set_points(st["pts"])
        s.run(st["params"].nt)
        return [s.sgt_rwg(q, z_source=ig == 3) for q, ig in enumerate(_igreen(st["case"]))]


def _synth_inputs(case, seed):
    """awp_inputs.synth_case with the SGT traces made on the device: damped
    wavelets of seeded frequency, arrival and size."""
    c = ai.synth_case(seed=int(seed), nx_f=case["nx_f"], nz_f=case["nz_f"], nt=12, nv=case["nv"], ntout=case["ntout"],
                      ncomp=case["ncomp"], nstf=(case["nstf0"], case["nstf1"]), drop_frac=0.08)
    nt, npg = case["nt"], len(c.index)
    c.master["nt"] = nt
    c.headers["nt"] = nt
    g = _gen(seed, 5)
    t = torch.arange(nt, device=_dev()) * float(c.dtout)
    c.comps = []
    for _ in range(case["ncomp"]):
        r = torch.rand((3, npg, 6, 1), generator=g, device=_dev())
        x = t - (float(c.dtout) * nt * (0.1 + 0.5 * r[1]))
        amp = 1.0e-9 * (2.0 * r[2] - 1.0)
        c.comps.append((amp * torch.exp(-(x / 3.0) ** 2) * torch.sin(2.0 * math.pi * (0.2 + 0.8 * r[0]) * x)).cpu().numpy())
    return c


def _prepare_synth(case, seed):
    c = _synth_inputs(case, seed)
    s = awpsgt.Synth(c.slon, c.slat, c.dtout, ntout=c.ntout)
    s.set_sgt(c.master, c.index, c.headers, c.comps)
    return {"case": case, "synth": s, "variations": c.variations}


def _run_synth(st):
    s = st["synth"]
    s.clear_variations()
    for v, (pts, pool) in enumerate(st["variations"]):
        s.add_variation(v, pts, pool, borrow=True)
    return s.run()


def prepare(case, seed):
    return {"steps": _prepare_steps, "job": _prepare_job, "synth": _prepare_synth}[case["kind"]](case, seed)


def run(state):
    return {"steps": _run_steps, "job": _run_job, "synth": _run_synth}[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def _step_bytes(case):
    """Bytes of one time step: the state of every cell read and written once
    (it does not stay on the chip from step to step), the media read once."""
    n = len(case["comps"])
    prec = case.get("precision", "f32")
    r = {"f32": 24, "bfp": 14}.get(prec, 12) if case.get("nve", 1) else 0
    media = (5 if case.get("nve", 1) else 3) * (2 if prec in ("f16", "bf16") else 4)
    cells = case["nx"] * case["ny"] * case["nz"]
    b = cells * (n * (2 * 36 + 2 * r) + media)
    if case.get("npc"):
        inner = max(0, case["nx"] - 2 * _ND) * max(0, case["ny"] - 2 * _ND) * max(0, case["nz"] - _ND)
        b += (cells - inner) * n * 2 * 18 * 4           # the split fields of the boundary zones
    return b


def work(case):
    if case["kind"] == "synth":
        pts = case["nx_f"] * case["nz_f"]
        sgt = (case["nx_f"] + 2) * 3 * (case["nz_f"] + 1) * case["ncomp"] * 6 * case["nt"] * 4
        mean = 0.5 * (case["nstf0"] + case["nstf1"])
        traces = 3 if case["ncomp"] == 3 else 2
        return {"bytes": sgt + case["nv"] * (3 * case["ntout"] * 4 + pts * (mean * 4 + 100)),
                "flops": 2.0 * 1.1 * case["nv"] * pts * traces * case["ntout"] * mean}
    cells = case["nx"] * case["ny"] * case["nz"]
    n = len(case["comps"])
    steps = case["steps"] if case["kind"] == "steps" else case["nt"]
    b = steps * _step_bytes(case)
    if case["kind"] == "job":
        b += cells * 12 + n * case["npts"] * 6 * (case["nt"] // 10) * 4
    return {"bytes": b, "flops": 220.0 * cells * n * steps}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------

def _f32(x):
    return float(np.float32(x))


class _Exact:
    """The staggered-grid scheme (4th order in space, 2nd in time, coarse-grained
    memory variables, Cerjan sponge, free surface at k = nz) in 64 bits, one
    component at a time, arrays [nz+4][ny+4][nx+4] with two ghost layers."""

    def __init__(self, case, seed, nt):
        self.nx, self.ny, self.nz = nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.nve = case.get("nve", 1)
        self.dh, self.dt = _f32(_DH), _f32(_DT)
        dev = _dev()
        m = torch.from_numpy(_media(case, seed)).to(dev).flip(0).double()     # k = 1 at the bottom
        vp, vs, rho = (m[..., i].clone() for i in range(3))
        del m
        sq = 0.05 * vs
        pq = 2.0 * sq
        tmax, tmin = 1.0 / (2 * math.pi * _f32(_FL)), 1.0 / (2 * math.pi * _f32(_FH))
        w0, w2 = 2 * math.pi * _f32(_FP), 2 * math.pi * _f32(_FH)
        lw = math.log(w2 / w0)
        vs = vs * (1.0 + lw / (math.pi * sq))
        vp = vp * (1.0 + lw / (math.pi * pq))
        vs = torch.where(vp / vs < 1.45, vp / 1.45, vs)
        mu = 1.0 / (rho * vs * vs)
        lam = 1.0 / (rho * (vp * vp - 2.0 * vs * vs))

        def clamp(a):
            return F.pad(a[None, None], (1,) * 6, mode="replicate")[0, 0]

        self.lam, self.mu, self.d1 = clamp(lam), clamp(mu), clamp(rho)
        for a in (self.mu, self.d1):          # the one corner that padmedia fills with lam
            a[0, 0, nx + 1] = self.lam[1, 1, nx]
        if self.nve:
            t1 = 2.0 / math.pi * math.log(tmax / tmin)
            t2 = 2.0 / math.pi * math.log(w0 * tmin)

            def q(x):
                a = F.pad(t1 / x / (1.0 - t2 / x), (1,) * 6)
                a[nz + 1, 1:-1, 1:-1] = a[nz, 1:-1, 1:-1]
                return a

            self.qp, self.qs = q(pq), q(sq)
            tab = torch.tensor([[[1, 6], [7, 4]], [[8, 3], [2, 5]]], dtype=torch.float64, device=dev)
            tau = torch.exp(0.5 * (math.log(tmax * tmin) + math.log(tmax / tmin) * (2.0 * (tab - 0.5) / 8.0 - 1.0)))
            iz = (nz + 1 - torch.arange(1, nz + 1, device=dev)) & 1
            iy, ix = torch.arange(1, ny + 1, device=dev) & 1, torch.arange(1, nx + 1, device=dev) & 1
            tau = tau[iz][:, iy][:, :, ix] / self.dt
            self.vx1, self.vx2 = 1.0 / (tau + 0.5), tau - 0.5
        alpha = math.sqrt(-math.log(_f32(0.92))) / _ND

        def sponge(n, high):
            f = torch.ones(n, dtype=torch.float64, device=dev)
            for i in range(1, n + 1):
                if i <= _ND:
                    f[i - 1] *= math.exp(-(alpha * (_ND - i + 1)) ** 2)
                if high and i >= n - _ND + 1:
                    f[i - 1] *= math.exp(-(alpha * (_ND - (n - i))) ** 2)
            return f

        self.crj = (sponge(nx, True)[None, None, :] * sponge(ny, True)[None, :, None]) * sponge(nz, False)[:, None, None]

    def new_state(self):
        z = lambda: torch.zeros((self.nz + 4, self.ny + 4, self.nx + 4), dtype=torch.float64, device=_dev())  # noqa: E731
        st = {n: z() for n in _WAVE}
        for n in _MEM if self.nve else ():
            st[n] = torch.zeros((self.nz, self.ny, self.nx), dtype=torch.float64, device=_dev())
        return st

    def inner(self, a, dx=0, dy=0, dz=0):
        return a[2 + dz:2 + dz + self.nz, 2 + dy:2 + dy + self.ny, 2 + dx:2 + dx + self.nx]

    def med(self, a, dx=0, dy=0, dz=0):
        return a[1 + dz:1 + dz + self.nz, 1 + dy:1 + dy + self.ny, 1 + dx:1 + dx + self.nx]

    def diff(self, a, axis, fwd):
        """9/8 and -1/24 difference along an axis, forward (half a cell up) or backward."""
        def at(n):
            o = [0, 0, 0]
            o[axis] = n + (1 if fwd else 0)
            return self.inner(a, *o)
        return (9.0 / 8.0) * (at(0) - at(-1)) - (1.0 / 24.0) * (at(1) - at(-2))

    def mean(self, a, offs):
        s = 0
        for o in offs:
            s = s + self.med(a, *o)
        return s

    def velocity(self, s):
        dth = self.dt / self.dh
        d = self.d1
        fu = dth / (0.25 * self.mean(d, [(0, 0, 0), (0, -1, 0), (0, 0, -1), (0, -1, -1)]))
        fv = dth / (0.25 * self.mean(d, [(0, 0, 0), (1, 0, 0), (0, 0, -1), (1, 0, -1)]))
        fw = dth / (0.25 * self.mean(d, [(0, 0, 0), (1, 0, 0), (0, -1, 0), (1, -1, 0)]))
        du = self.diff(s["xx"], 0, False) + self.diff(s["xy"], 1, False) + self.diff(s["xz"], 2, False)
        dv = self.diff(s["xy"], 0, True) + self.diff(s["yy"], 1, True) + self.diff(s["yz"], 2, False)
        dw = self.diff(s["xz"], 0, True) + self.diff(s["yz"], 1, False) + self.diff(s["zz"], 2, True)
        for n, f, x in (("u1", fu, du), ("v1", fv, dv), ("w1", fw, dw)):
            self.inner(s[n]).add_(f * x).mul_(self.crj)

    def surface(self, s):
        nx, ny, k = self.nx, self.ny, self.nz + 1
        u, v, w = s["u1"], s["v1"], s["w1"]

        def at(a, dx=0, dy=0):
            return a[k, 2 + dy:2 + dy + ny, 2 + dx:2 + dx + nx]

        uf = at(u) - (at(w) - at(w, -1))
        vf = at(v) - (at(w, 0, 1) - at(w))
        xl = 1.0 / self.lam[self.nz, 1:-1, 1:-1]
        x2 = 2.0 / self.mu[self.nz, 1:-1, 1:-1] + xl
        ue = torch.zeros_like(uf)
        ue[:, :-1] = uf[:, 1:]
        vs = torch.zeros_like(vf)
        vs[1:] = vf[:-1]
        wf = w[k - 1, 2:-2, 2:-2] - (xl / x2) * ((ue - uf) + (at(u, 1) - at(u)) + (vf - vs) + (at(v) - at(v, 0, -1)))
        u[k + 1, 2:-2, 2:-2], v[k + 1, 2:-2, 2:-2], w[k + 1, 2:-2, 2:-2] = uf, vf, wf

    def stress(self, s):
        dt, dth, dh1 = self.dt, self.dt / self.dh, 1.0 / self.dh
        eight = [(a, b, c) for a in (0, 1) for b in (0, -1) for c in (0, -1)]
        xl = 8.0 / self.mean(self.lam, eight)
        xm = 8.0 / self.mean(self.mu, eight)
        pair = {"xy": (0, 0, -1), "xz": (0, -1, 0), "yz": (1, 0, 0)}
        u, v, w = s["u1"], s["v1"], s["w1"]
        n = [self.diff(u, 0, True), self.diff(v, 1, False), self.diff(w, 2, False)]
        sh = {"xy": self.diff(u, 1, True) + self.diff(v, 0, False), "xz": self.diff(u, 2, True) + self.diff(w, 0, False),
              "yz": self.diff(v, 2, True) + self.diff(w, 1, True)}
        tr = n[0] + n[1] + n[2]
        if self.nve:
            qpa = 0.125 * self.mean(self.qp, eight)
            h1 = -(xm * (0.125 * self.mean(self.qs, eight)))
            lm = xl + 2.0 * xm
            va = -(qpa * lm * dh1 * tr / 2.0)
        for i, name in enumerate(("xx", "yy", "zz")):
            rest = tr - n[i]
            if self.nve:
                r = s[_MEM[i]]
                new = (self.vx2 * r - h1 * rest * dh1 + va) * self.vx1
                add = dth * (lm * tr - 2.0 * xm * rest) + dt * (r + new)
                s[_MEM[i]] = new
            else:
                add = dth * ((xl + 2.0 * xm) * n[i] + xl * rest)
            self.inner(s[name]).add_(add).mul_(self.crj)
        for i, name in enumerate(("xy", "xz", "yz")):
            x = 2.0 / (self.med(self.mu) + self.med(self.mu, *pair[name]))
            add = x * dth * sh[name]
            if self.nve:
                r = s[_MEM[3 + i]]
                h2 = -(0.5 * (self.med(self.qs) + self.med(self.qs, *pair[name])) * x / 2.0)
                new = (self.vx2 * r + h2 * dh1 * sh[name]) * self.vx1
                add = add + dt * (r + new)
                s[_MEM[3 + i]] = new
            self.inner(s[name]).add_(add).mul_(self.crj)
        k = self.nz + 1
        c = (slice(2, -2), slice(2, -2))
        s["zz"][k + 1][c] = -s["zz"][k][c]
        s["zz"][k + 2][c] = -s["zz"][k - 1][c]
        for name in ("xz", "yz"):
            s[name][k + 1][c] = -s[name][k - 1][c]
            s[name][k + 2][c] = -s[name][k - 2][c]
            s[name][k][c] = 0.0

    def force(self, s, ig, xyz, amp):
        i, j, k = xyz[0], xyz[1], self.nz + 1 - xyz[2]
        s[_WAVE[ig - 1]][k + 1, j + 1, i + 1] += amp * (self.dt / self.dh ** 3) / self.d1[k, j, i]

    def kinematic(self, s, xyz, tab, n):
        tab = tab.astype(np.float64)
        t = n * self.dt - tab[:, 0, 2]
        rise = tab[:, 0, 3]
        a, d, r = (np.radians(tab[:, 1, i]) for i in range(3))
        nv = np.stack([np.sin(d) * np.cos(a), -np.sin(d) * np.sin(a), np.cos(d)])
        dv = np.stack([np.cos(r) * np.sin(a) - np.cos(d) * np.sin(r) * np.cos(a),
                       np.cos(r) * np.cos(a) + np.cos(d) * np.sin(r) * np.sin(a), np.sin(r) * np.sin(d)])
        w = 2 * math.pi / rise
        rate = {1: w * (w * t) * np.exp(-w * t)}
        for kind, c in ((2, 0.3), (3, 0.2)):
            t1 = 0.13 * rise
            t2 = rise - t1
            area = (1.7 - c) * t1 + 1.2 * t1 / math.pi + c * t2
            p, q = t / t1, (t - t1) / t2
            f = np.where(t < t1, 0.7 * (1 - np.cos(np.pi * p)) + 0.6 * np.sin(0.5 * np.pi * p),
                         np.where(t < 2 * t1, 1 - (1 - c) * np.cos(np.pi * p) + c * np.cos(np.pi * q),
                                  c * (1 + np.cos(np.pi * q))))
            rate[kind] = np.where(t < rise, f, 0.0) / area
        kind = tab[:, 0, 0].astype(int)
        sl = np.select([kind == k for k in (1, 2, 3)], [rate[k] for k in (1, 2, 3)])
        sl = np.where(t > 0, sl, 0.0) * tab[:, 0, 1] * tab[:, 0, 4] * (self.dt / self.dh ** 3)
        i, j, k = (torch.from_numpy(np.ascontiguousarray(x)).to(_dev()).long()
                   for x in (xyz[:, 0], xyz[:, 1], self.nz + 1 - xyz[:, 2]))
        sl = torch.from_numpy(sl).to(_dev()) / self.mu[k, j, i]
        for name, a, b in (("xx", 0, 0), ("yy", 1, 1), ("zz", 2, 2), ("xz", 0, 2), ("yz", 1, 2), ("xy", 0, 1)):
            m = torch.from_numpy(nv[a] * dv[b] + nv[b] * dv[a]).to(_dev())
            s[name].index_put_((k + 1, j + 1, i + 1), -sl * m, accumulate=True)


def _exact_steps(case, seed):
    if case["npc"]:
        return None                          # 17 zones of split-field operators
    p = _steps_params(case)
    e = _Exact(case, seed, p.nt)
    out = []
    for q, ig in enumerate(_igreen(case)):
        s = e.new_state()
        for c, name, v in _wave_inputs(case, seed):
            if c == q:
                (e.inner(s[name]) if name in _WAVE else s[name]).copy_(v)
        if case["subfaults"]:
            xyz, tab = _rupture(case, seed)
        else:
            stf = _stf(p.nst, ig - 1, seed)[:, ig - 1].astype(np.float64)
            e.force(s, ig, _source_xyz(case), float(stf[0]))
        for n in range(1, case["steps"] + 1):
            e.velocity(s)
            e.surface(s)
            e.stress(s)
            if case["subfaults"]:
                e.kinematic(s, xyz, tab, n)
            elif n < p.nst:
                e.force(s, ig, _source_xyz(case), float(stf[n]))
        out += [e.inner(s[name]).clone() for name in _WAVE]
    return out


def _exact_job(case, seed):
    p = _job_params(case)
    e = _Exact(case, seed, p.nt)
    pts = torch.from_numpy(np.asarray(_points(case, seed), np.int64)).to(_dev())
    k, j, i = e.nz + 1 - pts[:, 2], pts[:, 1], pts[:, 0]
    lam, mu = e.lam[k, j, i], e.mu[k, j, i]
    a = (1.0 / lam + 1.0 / mu) / (1.0 / mu * (3.0 / lam + 2.0 / mu))
    b = -(1.0 / lam / (2.0 / mu * (3.0 / lam + 2.0 / mu)))
    out = []
    for ig in _igreen(case):
        s = e.new_state()
        stf = _stf(p.nst, ig - 1, seed)[:, ig - 1].astype(np.float64)
        e.force(s, ig, _source_xyz(case), float(stf[0]))
        got = []
        for n in range(1, p.nt + 1):
            e.velocity(s)
            e.surface(s)
            e.stress(s)
            if n < p.nst:
                e.force(s, ig, _source_xyz(case), float(stf[n]))
            if n % 10 == 0:
                xx, yy, zz, xy, xz, yz = (s[c][k + 1, j + 1, i + 1] for c in ("xx", "yy", "zz", "xy", "xz", "yz"))
                # RWG order: XX <- YY, YY <- XX, ZZ, XY, XZ <- -YZ, YZ <- -XZ
                got.append(torch.stack([b * xx + a * yy + b * zz, a * xx + b * yy + b * zz, b * xx + b * yy + a * zz,
                                        mu * xy, -mu * yz, -mu * xz], dim=1))
        img = torch.stack(got, dim=2) * (-2.0 if ig == 3 else 1.0)
        out.append(img.reshape(-1).cpu().numpy())
    return out


def _exact_synth(case, seed):
    """The seismograms by FFT convolution.  The choice of the SGT points and
    the whole-sample shifts follow the 32-bit arithmetic of their definition
    (they are integers); everything else is in 64 bits."""
    c = _synth_inputs(case, seed)
    f = np.float32
    nt, ntout, nv, ncomp = case["nt"], case["ntout"], case["nv"], case["ncomp"]
    sx, sy, h = 8, 10, float(c.h_km)
    ix = np.stack([c.index["xsgt"], c.index["ysgt"], c.index["zsgt"]], 1).astype(np.int64)
    where = {tuple(x): n for n, x in enumerate(ix)}
    p0 = c.variations[0][0]
    npt = len(p0)
    fault = [(20 + a, 40, 1 + b) for a in range(case["nx_f"]) for b in range(case["nz_f"])]
    zs = (p0["dep"].astype(np.float64) / h + 1.5).astype(np.int64)
    brackets = []
    for n in range(npt):
        eq = np.array([fault[n][0], fault[n][1], zs[n]])
        if tuple(eq) in where:
            brackets.append(([where[tuple(eq)]], [1.0]))
            continue
        rng = (ix[:, 0] - sx) ** 2 + (ix[:, 1] - sy) ** 2
        far = (rng > (eq[0] - sx) ** 2 + (eq[1] - sy) ** 2) + 2 * (ix[:, 2] - 1 > eq[2] - 1)
        d = ((ix - eq) ** 2).sum(1).astype(np.float64)
        order = sorted(set(far), key=lambda q: int(np.argmax(far == q)))
        pos = [int(np.flatnonzero(far == q)[np.argmin(d[far == q])]) for q in order]
        w = 1.0 / np.sqrt(d[pos])
        brackets.append((pos, list(w / w.sum())))
    taper = np.ones(nt)
    tap0 = nt - 10
    taper[tap0 + 1:] = 0.5 * (1.0 + np.cos(np.pi / 10 * np.arange(1, nt - tap0)))
    dev = _dev()
    sgt = [torch.from_numpy(x).to(dev).double() * torch.from_numpy(taper).to(dev) for x in c.comps]
    nfft = 1
    while nfft < ntout + max(case["nstf1"], 1):
        nfft *= 2
    hd = c.headers
    out = torch.zeros((nv, 3, ntout), dtype=torch.float64, device=dev)
    for v, (pts, pool) in enumerate(c.variations):
        rows, pos, shift, cof, amp, slip = [], [], [], [], [], []
        nterm = 0
        for n in range(npt):
            a = pts[n]
            bp, bw = brackets[n]
            comps = [m for m in range(3) if a["nt%d" % (m + 1)] > 0]
            if not comps:
                continue
            pbar = f(0)
            for g in bp:
                pbar = f(float(pbar) + math.sqrt(float(f(hd[g]["rho"] / hd[g]["mu"]))))
            pbar = f(pbar / f(len(bp)))
            gft = [f(pbar * hd[g]["cdist"]) for g in bp]
            t0 = [f(max(gft) - x) for x in gft]
            back = f(0)
            for x, w in zip(t0, bw):
                back = f(back - f(x * f(w)))
            back = f(f(back + a["tinit"]) - f(0))
            t0 = [f(x + hd[g]["tst"]) for x, g in zip(t0, bp)]
            dip, rake = math.radians(a["dip"]), math.radians(a["rake"])
            for m in comps:
                u = [float(m == x) for x in range(3)]
                for g, w, ts in zip(bp, bw, t0):
                    H = hd[g]
                    T = math.radians(float(a["stk"]) - float(H["xazim"]))
                    vx, vy, vz = -math.sin(dip) * math.sin(T), math.sin(dip) * math.cos(T), -math.cos(dip)
                    us = u[0] * math.cos(rake) - u[1] * math.sin(rake)
                    ud = u[0] * math.sin(rake) + u[1] * math.cos(rake)
                    un = u[2] * math.sin(dip) - ud * math.cos(dip)
                    ux = -un * math.sin(T) + us * math.cos(T)
                    uy = un * math.cos(T) + us * math.sin(T)
                    uz = -(u[2] * math.cos(dip) + ud * math.sin(dip))
                    lam, mu = float(H["lam"]), float(H["mu"])
                    tr = lam * (vx * ux + vy * uy + vz * uz)
                    cof.append([tr + 2 * mu * vx * ux, tr + 2 * mu * vy * uy, tr + 2 * mu * vz * uz,
                                mu * (vx * uy + vy * ux), mu * (vx * uz + vz * ux), mu * (vy * uz + vz * uy)])
                    amp.append(float(a["area"]) * w / float(H["xmom"]))
                    x = f(f(ts + back) / H["dt"])
                    shift.append(int(float(x) + 0.5) if x >= 0 else int(float(x) - 0.5))
                    rows.append(nterm)
                    pos.append(g)
                o, k = int(a["stf%d" % (m + 1)]), int(a["nt%d" % (m + 1)])
                slip.append((k, o))
                nterm += 1
        if not nterm:
            continue
        S = np.zeros((nterm, nfft))
        for n, (k, o) in enumerate(slip):
            S[n, :k] = float(f(c.dtout)) * pool[o:o + k].astype(np.float64)
        sp = torch.fft.rfft(torch.from_numpy(S).to(dev))
        cof_t = torch.tensor(cof, dtype=torch.float64, device=dev)
        amp_t = torch.tensor(amp, dtype=torch.float64, device=dev)
        azim = math.radians(float(hd[0]["xazim"]))
        idx = torch.arange(ntout, device=dev)[None, :] - torch.tensor(shift, device=dev)[:, None]
        ok = (idx >= 0) & (idx < nt)
        idx = idx.clamp(0, nt - 1)
        pos_t, row_t = torch.tensor(pos, device=dev), torch.tensor(rows, device=dev)
        tot = []
        for q in range(ncomp):
            acc = torch.zeros(nfft // 2 + 1, dtype=torch.complex128, device=dev)
            for b0 in range(0, len(pos), 512):
                b = slice(b0, b0 + 512)
                tr = torch.einsum("nct,nc->nt", sgt[q][pos_t[b]], cof_t[b]) * amp_t[b][:, None]
                tr = torch.where(ok[b], torch.gather(tr, 1, idx[b]), torch.zeros((), dtype=torch.float64, device=dev))
                acc += (torch.fft.rfft(tr, n=nfft) * sp[row_t[b]]).sum(0)
            tot.append(torch.fft.irfft(acc, n=nfft)[:ntout])
        X = tot[0]
        Y = tot[1] if ncomp > 1 else torch.zeros_like(X)
        if ncomp > 2:
            out[v, 0] = -tot[2]
        out[v, 1] = X * math.cos(azim) - Y * math.sin(azim)
        out[v, 2] = X * math.sin(azim) + Y * math.cos(azim)
    return out.cpu().numpy()


def exact(case, seed):
    return {"steps": _exact_steps, "job": _exact_job, "synth": _exact_synth}[case["kind"]](case, seed)
