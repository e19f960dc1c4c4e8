"""Performance cases: the work a user of this framework has it do, through its
public entry points (Solver, Batch and, for the Fortran host, one call per
reference routine).

A case is a grid, its borders and media, its sources and probes, and what one
pass does with it: advance the fields a few steps, advance a batch, transform
a near-field surface, or a whole solve from the problem description to the
probe traces and final fields on the host.  Geometry follows the case's own
`geo` number; the initial fields and the waveform's amplitude follow the seed.

`exact` restates the update in 64 bits with torch alone: curl, CPML,
pole-residue currents, plane waves, dipoles, border conditions, the
frequency-domain volume probe and the near-to-far-field transform.
"""
import ctypes
import math

import numpy as np
import torch

from semba_fdtd_b200 import Solver, _lib
from semba_fdtd_b200.batch import Batch
from semba_fdtd_b200.case import NodalSource, PlaneWave, Problem, Region, Waveform

EPS0 = 8.8541878176203898505e-12
MU0 = 1.2566370614359172954e-6
C0 = 1.0 / math.sqrt(EPS0 * MU0)
ETA0 = math.sqrt(MU0 / EPS0)
DEFAULT = dict(kind="steps", nx=64, ny=64, nz=64, layers=10, order=3.0, borders="pml", media="vacuum", wave=False,
               dipole=False, graded=False, probes=0, steps=32, mode="graph", build="exact", count=1, freqs=0, geo=1)


def listed():
    return [
        # The smallest problems: parity cases and parameter sweeps of a few
        # thousand cells with the reference's default border (Mur).
        dict(name="tiny_mur", nx=20, ny=23, nz=18, layers=0, borders="mur", media="blocks", dipole=True, probes=6,
             steps=16),
        # The plain small benchmark workload: 64^3 vacuum, CPML 10, a plane
        # wave through a TF/SF box, 16 probes.
        dict(name="small_planewave", nx=64, ny=64, nz=64, layers=10, wave=True, probes=16, steps=32),
        # Odd and ragged sizes, another border kind per face (periodic in z).
        dict(name="ragged_borders", nx=93, ny=41, nz=67, layers=7, borders="pml,mur,pec,pmc,periodic,periodic",
             media="blocks", wave=True, dipole=True, probes=9, steps=24, geo=3),
        # The plain mid benchmark workload: 256^3, CPML 12, scatterers inside a
        # plane wave's TF/SF box, 64 probes.
        dict(name="mid_scatterer", nx=256, ny=256, nz=256, layers=12, media="blocks", wave=True, probes=64, steps=8),
        # The headline workload: 512^3 graded mesh, CPML 12, a quarter of the volume
        # in two-pair pole-residue media, a dipole at the centre.
        dict(name="large_dispersive", nx=512, ny=512, nz=512, layers=12, media="dispersive", dipole=True, graded=True,
             probes=8, steps=2),
        # Electric and magnetic pole-residue media on a non-cubic graded grid.
        dict(name="odd_dispersive", nx=203, ny=97, nz=150, layers=9, media="magnetic", dipole=True, graded=True,
             probes=5, steps=8, geo=2),
        # The Fortran host's own loop: one call per reference routine.
        dict(name="host_routines", nx=100, ny=90, nz=110, layers=10, media="blocks", wave=True, probes=4, steps=4,
             mode="routines"),
        # Half steps called by a host that works between them, in the FMA build.
        dict(name="half_steps_fma", nx=160, ny=128, nz=144, layers=8, media="blocks", dipole=True, probes=4, steps=8,
             mode="fused", build="fast"),
        # Fields of a sub-volume at several frequencies (k-maps, SAR-like maps).
        dict(name="frequency_volume", kind="frequency", nx=96, ny=96, nz=96, layers=10, media="blocks", wave=True,
             probes=4, steps=64, freqs=4),
        # Radiation pattern: the surface transform of a run, then the far field.
        dict(name="far_field", kind="far", nx=80, ny=72, nz=64, layers=8, media="blocks", dipole=True, probes=2,
             steps=32, freqs=6),
        # The batched form: uneven instances advanced together.
        dict(name="batched_uneven", kind="batch", nx=32, ny=32, nz=32, layers=8, media="blocks", wave=True, probes=4,
             steps=32, count=10, geo=6),
        # A whole solve: description in, probe traces and final fields out.
        dict(name="whole_solve", kind="solve", nx=72, ny=56, nz=64, layers=10, media="dispersive", dipole=True,
             probes=12, steps=400),
    ]


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["frequency", "far", "batch", "solve"])
    lo, hi = {"steps": (16, 320), "frequency": (24, 120), "far": (24, 90), "batch": (24, 64), "solve": (20, 100)}[kind]

    def edge():
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = dict(kind=kind, nx=edge(), ny=edge(), nz=edge(), layers=rng.randint(4, 12), order=rng.choice([2.0, 3.0]),
             media=rng.choice(["vacuum", "blocks", "dispersive", "magnetic"]), wave=rng.random() < 0.5,
             dipole=rng.random() < 0.7, graded=rng.random() < 0.4, probes=rng.randint(1, 40),
             steps=rng.randint(2, 40), geo=rng.randint(1, 10**6))
    if kind == "steps":
        c["mode"] = rng.choice(["graph", "graph", "graph", "fused", "routines"])
        c["build"] = rng.choice(["exact", "exact", "fast"])
        if rng.random() < 0.4:
            pairs = ["pml,pml", "mur,mur", "pec,pmc", "periodic,periodic", "pml,mur", "pmc,pec"]
            c["borders"] = ",".join(rng.choice(pairs) for _ in range(3))
    if kind == "frequency":
        c["freqs"] = rng.randint(1, 8)
    if kind == "far":
        c["freqs"] = rng.randint(1, 8)
    if kind == "batch":
        c.update(count=rng.randint(2, 10), media=rng.choice(["vacuum", "blocks", "dispersive"]))
    if kind == "solve":
        c["steps"] = rng.randint(60, 500)
        c["dipole"] = c["dipole"] or not c["wave"]
    return c


# -- problems ---------------------------------------------------------------

def _full(case):
    return {**DEFAULT, **case}


def _borders(c):
    b = c["borders"].split(",")
    return tuple(b * 6 if len(b) == 1 else b)


def _axis_steps(n, base, graded, rng):
    if not graded:
        return np.full(n, base, np.float32)
    i = np.arange(n)
    return (base * (1 + 0.5 * np.cos(2 * np.pi * rng.integers(1, 4) * i / n + rng.uniform(0, 6)))).astype(np.float32)


def _poles(rng, scale, strength):
    """One or two conjugate pole pairs: (residues, minus the poles)."""
    res, bp = [], []
    for _ in range(2 if scale == EPS0 else 1):
        w, z = 2 * math.pi * rng.uniform(1e9, 2e10), rng.uniform(0.05, 0.3)
        a = complex(-z * w, w * math.sqrt(1 - z * z))
        r = -strength * rng.uniform(0.3, 0.7) * scale * a
        res += [r, r.conjugate()]
        bp += [-a, -a.conjugate()]
    return np.array(res, np.complex64), np.array(bp, np.complex64)


def _boxes(n, count, rng, lo_frac, hi_frac, margin):
    out = []
    for _ in range(count):
        b = []
        for e in n:
            m = margin + 2
            size = int(rng.integers(max(1, int(e * lo_frac)), max(2, int(e * hi_frac)) + 1))
            size = max(1, min(size, e - 2 * m - 1))
            o = int(rng.integers(m, max(m + 1, e - m - size)))
            b += [o, o + size - 1]
        out.append(b)
    return out


def _problem(c, seed, nsteps=None):
    rng = np.random.default_rng(int(c["geo"]) * 7919 + 13)
    n = (c["nx"], c["ny"], c["nz"])
    des = [_axis_steps(e, 0.002, c["graded"], rng) for e in n]
    dmin = min(float(d.min()) for d in des)
    dt = 0.8 * dmin / (C0 * math.sqrt(3.0))
    inset = max(2, min(15, min(n) // 4))
    regions = []
    if c["media"] == "blocks":
        for q, b in enumerate(_boxes(n, 8, rng, 0.05, 0.2, inset if min(n) > 24 else 2)):
            if q % 4 == 3:
                regions.append(Region(0, np.array([b], np.int32)))
            else:
                regions.append(Region(1, np.array([b], np.int32), eps=float(np.float32(EPS0 * rng.uniform(1, 10))),
                                      sigma=float(np.float32(rng.uniform(0, 0.1)))))
    elif c["media"] in ("dispersive", "magnetic"):
        count = 12 if c["media"] == "magnetic" else 40 if max(n) >= 400 else 24
        for q, b in enumerate(_boxes(n, count, rng, 0.06, 0.25 if max(n) < 400 else 0.33, 1)):
            r = Region(2, np.array([b], np.int32), eps=float(np.float32(EPS0 * rng.uniform(1, 2))))
            if c["media"] == "dispersive" or q % 3 != 1:
                r.residues, r.bpoles = _poles(rng, EPS0, rng.uniform(0.5, 3))
            if c["media"] == "magnetic" and q % 3:
                r.mresidues, r.mbpoles = _poles(rng, MU0, rng.uniform(0.2, 1))
                r.mu = float(np.float32(MU0 * rng.uniform(1, 1.5)))
            regions.append(r)
    amp = 0.5 + (seed % 1009) / 1009.0
    ds = dt / 2
    t = np.arange(int(40 / 0.5))
    pulse = (amp * np.exp(-((t * 0.5 - 14.0) / 5.0) ** 2)).astype(np.float32)
    if c["kind"] == "solve":  # a carrier that lasts as long as the solve, so its final fields are not a residue
        t = np.arange(2 * c["steps"] + 60)
        pulse = (amp * np.sin(2 * np.pi * t / 50.0) * np.minimum(1, t / 100.0)).astype(np.float32)
    waves = []
    if c["wave"]:
        th, ph, psi = rng.uniform(0.3, 2.8), rng.uniform(0, 6), rng.uniform(0, 6)
        th_hat = np.array([math.cos(th) * math.cos(ph), math.cos(th) * math.sin(ph), -math.sin(th)])
        ph_hat = np.array([-math.sin(ph), math.cos(ph), 0.0])
        e = math.cos(psi) * th_hat + math.sin(psi) * ph_hat
        waves.append(PlaneWave((inset,) * 3, tuple(v - inset for v in n), float(np.float32(th)), float(np.float32(ph)),
                               float(np.float32(math.acos(max(-1, min(1, e[2]))))),
                               float(np.float32(math.atan2(e[1], e[0]))), Waveform(pulse, np.float32(ds))))
    nodals = []
    if c["dipole"]:
        p = [v // 2 for v in n]
        nodals.append(NodalSource(True, False, np.array([[p[0], p[0], p[1], p[1], p[2], p[2]]], np.int32),
                                  np.array([[0, 0, 1e-3]], np.float32), Waveform(pulse, np.float32(ds))))
    probes = np.array([[int(rng.integers(0, 6))] + [int(rng.integers(1, e - 1)) for e in n]
                       for _ in range(c["probes"])], np.int32).reshape(-1, 4)
    L = c["layers"]
    return Problem(*n, *des, nsteps=int(c["steps"] if nsteps is None else nsteps), cfl=0.8, pml_layers=(L,) * 6,
                   pml_order=(c["order"],) * 6, pml_refl=(1e-6,) * 6, regions=regions, planewaves=waves, nodals=nodals,
                   probes=probes, borders=_borders(c))


def _instances(c):
    """The cases of a batch's instances: edges spread over a factor of four."""
    rng = np.random.default_rng(int(c["geo"]))
    out = []
    for q in range(c["count"]):
        f = np.exp(rng.uniform(0, math.log(4), 3))
        out.append(dict(c, kind="steps", nx=int(c["nx"] * f[0]), ny=int(c["ny"] * f[1]), nz=int(c["nz"] * f[2]),
                        geo=int(c["geo"]) + q))
    return out


# -- initial fields -----------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _layout(c):
    """(layers below, layers above, cells) per axis and, per component, the
    shape of its Alloc box and its swept range in local indices."""
    b, n = _borders(c), (c["nx"], c["ny"], c["nz"])
    lay = [c["layers"] if k == "pml" else 0 for k in b]
    lo, hi = lay[0::2], lay[1::2]
    half = [[a == f if f < 3 else a != f - 3 for a in range(3)] for f in range(6)]
    top = [[n[a] + hi[a] - half[f][a] + lo[a] + 1 for a in range(3)] for f in range(6)]  # last swept local index
    return lo, hi, n, half, top


def _initial(c, seed):
    """Smooth fields over every component's swept range, [k][j][i]: a few
    standing waves with the amplitudes of a unit plane wave."""
    _, _, _, _, top = _layout(c)
    rng = np.random.default_rng(int(seed) * 31 + 5)
    dev, out = _device(), []
    for f in range(6):
        shape = [top[f][a] for a in (2, 1, 0)]
        v = torch.zeros(shape, dtype=torch.float32, device=dev)
        for _ in range(2):
            ax = [torch.sin(torch.arange(s, device=dev, dtype=torch.float64) * rng.uniform(0.05, 0.6) + rng.uniform(0, 6))
                  .float() for s in shape]
            v += float(rng.uniform(0.3, 1.0)) * ax[0][:, None, None] * ax[1][None, :, None] * ax[2][None, None, :]
        out.append(v if f < 3 else v / ETA0)
    return out


class _Raw:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (int(ptr), False), "version": 3}


def _views(lib, handle):
    """The six components over their Alloc boxes, [k][j][i], as views of device memory."""
    a6 = (_lib.Lim * 6)()
    lib.sgpu_host_info(handle, None, None, a6, None, None)
    lims = [a.tuple() for a in a6]
    rows = max(a[3] - a[2] + 1 for a in lims)
    planes = max(a[5] - a[4] + 1 for a in lims)
    out = []
    for f in range(6):
        p, size = ctypes.c_void_p(), ctypes.c_uint64()
        rc = lib.sgpu_zplane(handle, f, lims[f][4], ctypes.byref(p), ctypes.byref(size))
        if rc:
            raise RuntimeError("sgpu_zplane failed")
        full = torch.as_tensor(_Raw(p.value, (planes, rows, size.value // 4 // rows)), device="cuda")
        a = lims[f]
        out.append(full[:a[5] - a[4] + 1, :a[3] - a[2] + 1, :a[1] - a[0] + 1])
    return out


def _load(views, fields):
    for v, f in zip(views, fields):
        v[1:1 + f.shape[0], 1:1 + f.shape[1], 1:1 + f.shape[2]] = f


# -- the cases ----------------------------------------------------------------

def _time_vector(c):
    """Steps a kept solver may take in all (its time vector's length)."""
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] in ("frequency", "far"):
        return 60000
    return 1000000 if cells < 100000 else 300000 if cells < 4000000 else 20000


def _frequencies(c):
    return [2e9 * (q + 1) for q in range(c["freqs"])]


def _probe_box(c):
    n = (c["nx"], c["ny"], c["nz"])
    return [v for e in n for v in (e // 6, e // 6 + max(1, min(48, 2 * e // 3)) - 1)]


def _movie_box(c):
    return [c["nx"] // 4, 3 * c["nx"] // 4, c["ny"] // 4, 3 * c["ny"] // 4, c["nz"] // 2, c["nz"] // 2]


def _far_box(c):
    return [v for e in (c["nx"], c["ny"], c["nz"]) for v in (3, e - 3)]


_ANGLES = (0.0, 3.0, 0.25, 0.0, 6.0, 0.5)


def _incident(c):
    t = np.arange(64, dtype=np.float32) * np.float32(2e-12)
    return np.stack([t, np.exp(-((t - 5e-11) / 2e-11) ** 2)], 1).astype(np.float32)


def prepare(case, seed):
    c = _full(case)
    if c["kind"] == "solve":
        return {"case": c, "problem": _problem(c, seed)}
    if c["kind"] == "batch":
        limit = 200000
        inst = _instances(c)
        batch = Batch(sum(i["nx"] * i["ny"] * i["nz"] for i in inst) * 400 + (2 << 30), c["count"])
        slots = [batch.add(_problem(i, seed, limit)) for i in inst]
        views = []
        for s, i in zip(slots, inst):
            ctx = ctypes.c_void_p()
            if batch.lib.sgpu_batch_instance(batch._h, s, ctypes.byref(ctx)):
                raise RuntimeError("sgpu_batch_instance failed")
            v = _views(batch.lib, ctx)
            _load(v, _initial(i, seed))
            views += v
        torch.cuda.synchronize()
        return {"case": c, "batch": batch, "out": views}
    s = Solver(_problem(c, seed), variant=c["build"], max_steps=_time_vector(c))
    views = _views(s.lib, s.handle)
    _load(views, _initial(c, seed))
    torch.cuda.synchronize()
    st = {"case": c, "solver": s, "out": views}
    if c["kind"] == "frequency":
        st["fid"] = s.add_freq_probe(False, _probe_box(c), freqs=_frequencies(c))
        st["mid"] = s.add_movie_probe(True, _movie_box(c), every=8, capacity=64)
    if c["kind"] == "far":
        fr = _frequencies(c)
        st["ffid"] = s.add_farfield(_far_box(c), initial=fr[0], final=fr[-1] + 1e8, step=2e9)
        st["incident"] = _incident(c)
    return st


def run(state):
    c = state["case"]
    if c["kind"] == "solve":
        with Solver(state["problem"]) as s:
            traces = s.run()
            return {"probes": traces, "fields": [s.field(f) for f in range(6)]}
    if c["kind"] == "batch":
        state["batch"].advance(c["steps"])
        return {"fields": state["out"]}
    s = state["solver"]
    s.step(c["steps"], mode=c["mode"])
    if c["kind"] == "frequency":
        return {"fields": state["out"], "frequency": s.freq_probe(state["fid"], c["freqs"]),
                "movie": s.movie_frames(state["mid"])[1]}
    if c["kind"] == "far":
        rows = s.farfield_transform(state["ffid"], _ANGLES, state["incident"])
        return {"fields": state["out"], "pattern": [np.ascontiguousarray(rows[:, q]) for q in range(3, 9)]}
    return {"fields": state["out"]}


def _cells(c):
    lo, hi, n, _, _ = _layout(c)
    return [n[a] + lo[a] + hi[a] for a in range(3)]


def work(case):
    """Per step: each field value read and written once with its two-byte
    medium (60 B a cell), 8 B per CPML psi point, 8 B and 32 B per stored pole
    pair for each pole-residue node; the probe's and the transform's own
    accumulators; for a whole solve the fields' way to the host as well."""
    c = _full(case)
    if c["kind"] == "batch":
        parts = [work(dict(i, kind="steps")) for i in _instances(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    e = _cells(c)
    cells = e[0] * e[1] * e[2]
    lo, hi, n, _, _ = _layout(c)
    psi = sum(4 * (lo[a] + hi[a]) * cells // e[a] for a in range(3))  # four corrected components an axis
    nodes = [0, 0]
    if c["media"] in ("dispersive", "magnetic"):
        for r in _problem(c, 0, 1).regions:  # overlaps counted once each: an upper estimate below a few per cent
            b = r.boxes[0]
            v = 3 * int((b[1] - b[0] + 1) * (b[3] - b[2] + 1) * (b[5] - b[4] + 1))
            nodes[0] += v * (len(r.bpoles) // 2)
            nodes[1] += v * (len(r.mbpoles) // 2)
        nodes = [min(nodes[0], 3 * 2 * cells * 0.5), min(nodes[1], 3 * cells * 0.5)]
    byt = 60 * cells + 8 * psi + (4 + 32) * nodes[0] + (8 + 32) * nodes[1]
    flops = 42 * cells + 6 * psi + 30 * (nodes[0] + nodes[1])
    byt, flops = byt * c["steps"], flops * c["steps"]
    if c["kind"] == "solve":
        byt += 24 * cells
    if c["kind"] == "frequency":
        b = _probe_box(c)
        v = 3 * (b[1] - b[0] + 1) * (b[3] - b[2] + 1) * (b[5] - b[4] + 1)
        byt += v * (4 + 32 * c["freqs"]) * c["steps"] + 16 * v * c["freqs"]
        flops += 4 * v * c["freqs"] * c["steps"]
    if c["kind"] == "far":
        face = 2 * sum((e_ - 6) * (f_ - 6) for e_, f_ in ((n[0], n[1]), (n[1], n[2]), (n[0], n[2])))
        byt += 6 * face * (4 + 32 * c["freqs"]) * c["steps"]
        flops += 24 * face * c["freqs"] * c["steps"] + 200 * face * c["freqs"] * 13 * 13
    return {"bytes": float(byt), "flops": float(flops)}


def tolerance(case):
    """Four times the distance seen between this framework's 32-bit results
    and the 64-bit restatement below, over the listed cases and drawn ones: a
    few steps stay within 7e-7 of it, a pattern within 1e-5 (small rows next
    to the surface sums they come from), a whole solve within 3e-5 (rounding
    accumulated over hundreds of steps)."""
    kind = _full(case)["kind"]
    if kind == "solve":
        return {"rel": 1.2e-4, "max": 2e-2}
    if kind == "far":
        return {"rel": 4e-5, "max": 4e-3}
    return {"rel": 4e-6, "max": 5e-4}


# -- the same update in 64 bits ------------------------------------------------

class _Exact:
    """All components in one box of local indices [k][j][i]; component f is
    swept over 1..top[f] on each axis."""

    def __init__(self, c, seed):
        self.c, dev = c, _device()
        self.dev, self.pb = dev, _problem(c, seed)
        self.lo, self.hi, self.n, self.half, self.top = _layout(c)
        self.o = [v + 1 for v in self.lo]
        self.size = [self.n[a] + self.lo[a] + self.hi[a] + 3 for a in range(3)]
        pb = self.pb
        d = []
        for a, v in enumerate((pb.desx, pb.desy, pb.desz)):
            v = np.asarray(v, np.float64)
            d.append(np.concatenate([np.full(self.o[a] + 1, v[0]), v, np.full(self.hi[a] + 3, v[-1])]))  # cell -o-1 first
        self.de = [x[1:1 + s] for x, s in zip(d, self.size)]
        self.dh = [0.5 * (x[1:1 + s] + x[:s]) for x, s in zip(d, self.size)]
        self.dt = 0.8 / (C0 * math.sqrt(sum((1 / x.min()) ** 2 for x in d)))
        self.line = [np.concatenate([[0.0], np.cumsum(np.asarray(v, np.float64))]) for v in (pb.desx, pb.desy, pb.desz)]
        self.ie = [self.vec(1 / x, a) for a, x in enumerate(self.de)]
        self.ih = [self.vec(1 / x, a) for a, x in enumerate(self.dh)]
        self.F = [torch.zeros(self.size[::-1], dtype=torch.float64, device=dev) for _ in range(6)]
        self.media()
        self.cpml()
        self.t = 0.0

    def vec(self, v, a):
        shape = [1, 1, 1]
        shape[2 - a] = -1
        return torch.tensor(np.asarray(v, np.float64), device=self.dev).reshape(shape)

    def sl(self, f, a=None, d=0):
        """Swept box of component f, moved by d along axis a."""
        return tuple(slice(1 + (d if q == a else 0), self.top[f][q] + 1 + (d if q == a else 0)) for q in (2, 1, 0))

    def along(self, v, f, a):
        s = [slice(None)] * 3
        s[2 - a] = slice(1, self.top[f][a] + 1)
        return v[tuple(s)]

    def media(self):
        tab = [(EPS0, 0.0, MU0, 1.0, 10, None), (EPS0, 0.0, MU0, 1.0, 10, None)]  # 0 PEC, 1 vacuum
        prio = torch.tensor([150, 10] + [{1: 20, 2: 40}.get(r.kind, 150) for r in self.pb.regions], device=self.dev)
        self.mi = [torch.ones(self.size[::-1], dtype=torch.uint8, device=self.dev) for _ in range(6)]
        index = []
        for q, r in enumerate(self.pb.regions):
            index.append(0 if r.kind == 0 else q + 2)
        for kind in (0, 1, 2):
            for r, m in zip(self.pb.regions, index):
                if r.kind != kind:
                    continue
                for b in np.asarray(r.boxes):
                    for f in range(6):
                        s = tuple(slice(int(b[2 * a]) + self.o[a], int(b[2 * a + 1]) + self.o[a] + 1 + (not self.half[f][a]))
                                  for a in (2, 1, 0))
                        old = self.mi[f][s]
                        new = prio[m] > prio[old.long()] if f < 3 else prio[m] >= prio[old.long()]
                        self.mi[f][s] = torch.where(new, torch.full_like(old, m), old)
        for face, b in enumerate(_borders(self.c)):
            if b != "pec":
                continue
            a = face // 2
            for f in range(6):
                if (a == f % 3) != (f >= 3):
                    continue
                s = [slice(1, self.top[f][q] + 1) for q in (2, 1, 0)]
                s[2 - a] = slice(1, 2) if face % 2 == 0 else slice(self.top[f][a], self.top[f][a] + 1)
                self.mi[f][tuple(s)] = 0
        dt, count = self.dt, len(self.pb.regions) + 2
        g = np.zeros((4, count))
        g[:, 1] = 1.0, dt / EPS0, 1.0, dt / MU0
        self.disp = []
        for q, r in enumerate(self.pb.regions):
            if r.kind == 0:
                continue
            m = q + 2
            for side, (v, s, res, bp) in enumerate(((r.eps, r.sigma, r.residues, r.bpoles),
                                                    (r.mu, r.sigmam, r.mresidues, r.mbpoles))):
                a = -np.asarray(bp, np.complex128)
                kap, bet = (1 + a * dt / 2) / (1 - a * dt / 2), np.asarray(res, np.complex128) * dt / (1 - a * dt / 2)
                den = 2 * v + bet.real.sum() + s * dt
                g[2 * side:2 * side + 2, m] = (2 * v + bet.real.sum() - s * dt) / den, 2 * dt / den
                if len(a):
                    for f in range(3 * side, 3 * side + 3):
                        w = torch.nonzero((self.mi[f][self.sl(f)] == m).reshape(-1)).reshape(-1)
                        g3 = dt / den * (1 + kap)
                        self.disp.append([f, w, torch.zeros(len(w), dtype=torch.float64, device=self.dev),
                                          [(k, b, x, torch.zeros(len(w), dtype=torch.complex128, device=self.dev))
                                           for k, b, x in zip(kap[::2], bet[::2], g3[::2])]])
        self.g = torch.tensor(g, device=self.dev)

    def cpml(self):
        b, L = _borders(self.c), self.c["layers"]
        self.pb_, self.pc_ = [[None] * 3, [None] * 3], [[None] * 3, [None] * 3]
        for a in range(3):
            for side in range(2):
                x = np.arange(self.size[a]) - self.o[a] + 0.5 * side
                sig = np.zeros(self.size[a])
                for end in range(2):
                    if b[2 * a + end] != "pml":
                        continue
                    depth = (-x if end == 0 else x - self.n[a]) / L
                    edge = self.de[a][0 if end == 0 else -1]
                    top = (0.8 * (self.c["order"] + 1) / (ETA0 * edge) if L in (5, 10) else
                           -math.log(1e-6) * (self.c["order"] + 1) / (2 * ETA0 * L * edge))
                    sig += np.where(depth > 0, top * np.abs(depth) ** self.c["order"], 0)
                pbv = np.exp(-sig * self.dt / EPS0)
                step = (self.dh if side == 0 else self.de)[a]
                self.pb_[side][a] = self.vec(pbv, a)
                self.pc_[side][a] = self.vec(np.where(sig > 0, (pbv - 1) / step, 0.0), a)
        self.psi = {}
        self.mur = {}

    def curl(self, side):
        G, inv = self.g[2 * side:2 * side + 2], (self.ih, self.ie)[side]
        for q in range(3):
            f, s = 3 * side + q, self.sl(3 * side + q)
            m = self.mi[f][s].long()
            g2 = G[1][m]
            v = G[0][m] * self.F[f][s]
            for a, sign in (((q + 1) % 3, 1.0), ((q + 2) % 3, -1.0)):
                o = 3 * (1 - side) + 3 - q - a  # the other field's component of this term
                sg = sign if side == 0 else -sign
                diff = self.F[o][s] - self.F[o][self.sl(f, a, -1)] if side == 0 else self.F[o][self.sl(f, a, 1)] - self.F[o][s]
                term = diff * self.along(inv[a], f, a)
                if "pml" in _borders(self.c)[2 * a:2 * a + 2]:
                    p = self.psi.get((f, a), 0.0)
                    p = self.along(self.pb_[side][a], f, a) * p + diff * self.along(self.pc_[side][a], f, a)
                    self.psi[f, a] = p
                    term = term + p
                v = v + sg * g2 * term
            self.F[f][s] = v

    def poles(self, side):
        for e in self.disp:
            f, w, prev, st = e
            if f // 3 != side:
                continue
            box = self.F[f][self.sl(f)].contiguous().reshape(-1)
            v = box[w]
            for k, b, g3, J in st:
                v = v - 2 * (g3.real * J.real - g3.imag * J.imag)
            d = (v - prev) / self.dt
            e[3] = [(k, b, g3, complex(k) * J + complex(b) * d) for k, b, g3, J in st]
            e[2] = v
            box[w] = v
            self.F[f][self.sl(f)] = box.reshape(self.F[f][self.sl(f)].shape)

    @staticmethod
    def table(wave, t):
        ds, ev = float(wave.dsamples), np.asarray(wave.samples, np.float64)
        k = np.trunc(t / ds).astype(np.int64)
        ok = (k > 0) & (k + 1 <= len(ev) - 1)
        k = np.clip(k, 0, len(ev) - 2)
        return np.where(ok, (ev[k + 1] - ev[k]) / ds * (t - k * ds) + ev[k], 0.0)

    def pos(self, f, a, i):
        ln = self.line[a]
        return 0.5 * (ln[i] + ln[i + 1]) if self.half[f][a] else ln[i]

    def sources(self, side):
        t = self.t + 0.5 * self.dt * side
        for w in self.pb.planewaves:
            p = np.array([math.sin(w.theta) * math.cos(w.phi), math.sin(w.theta) * math.sin(w.phi), math.cos(w.theta)])
            e = np.array([math.sin(w.alpha) * math.cos(w.beta), math.sin(w.alpha) * math.sin(w.beta), math.cos(w.alpha)])
            amp = list(e) + list(np.cross(p, e) / ETA0)
            box = [(w.coor1[a], w.coor2[a]) for a in range(3)]
            d0 = sum(p[a] * self.line[a][max(box[a][0] - 1, 0) if p[a] >= 0 else min(box[a][1] + 1, self.n[a])]
                     for a in range(3))
            for a in range(3):
                for end in range(2):
                    for cc in ((a + 1) % 3, (a + 2) % 3):  # the electric component of the pair
                        hh = 3 + 3 - a - cc
                        f, fld = (cc, hh) if side == 0 else (hh, cc)
                        plane = box[a][end] - (side == 1 and end == 0)
                        at = plane + ((-1 if side == 0 else 1) if end == 0 else 0)
                        sign = (-1.0 if cc == (a + 2) % 3 else 1.0) * (1 if end == 0 else -1)
                        if side == 1:
                            sign = (1.0 if hh - 3 == (a + 2) % 3 else -1.0) * (1 if end == 0 else -1)
                        idx = [np.arange(box[q][0], box[q][1] + (q != cc)) for q in range(3)]
                        idx[a] = np.array([plane])
                        xyz = [self.pos(fld, q, idx[q] if q != a else np.array([at])) for q in range(3)]
                        d = (xyz[0][None, None, :] * p[0] + xyz[1][None, :, None] * p[1] + xyz[2][:, None, None] * p[2]) - d0
                        v = amp[fld] * self.table(w.wave, t - d / C0)
                        inv = float((self.ih if side == 0 else self.ie)[a].reshape(-1)[plane + self.o[a]])
                        s = tuple(slice(int(idx[q][0]) + self.o[q], int(idx[q][-1]) + self.o[q] + 1) for q in (2, 1, 0))
                        self.F[f][s] += torch.tensor(v, device=self.dev) * (sign * inv * float(self.g[2 * side + 1, 1]))
        if side == 0:
            for nd in self.pb.nodals:
                b = nd.boxes[0]
                l = [int(b[2 * a]) + self.o[a] for a in range(3)]
                m = int(self.mi[2][l[2], l[1], l[0]])
                if m:
                    inv = float(self.ih[0].reshape(-1)[l[0]] * self.ih[1].reshape(-1)[l[1]])
                    self.F[2][l[2], l[1], l[0]] -= (float(self.g[1, m]) * inv * float(nd.amp[0][2]) *
                                                    float(self.table2(nd.wave, t)))

    @staticmethod
    def table2(wave, t):
        ds, ev = float(wave.dsamples), np.asarray(wave.samples, np.float64)
        k = int(t / ds)
        return 0.0 if k + 1 > len(ev) - 1 else (ev[k + 1] - ev[k]) / ds * (t - k * ds) + ev[k]

    def borders(self):
        b = _borders(self.c)

        def plane(f, a, i):
            s = [slice(0, self.top[f][q] + 2) for q in (2, 1, 0)]
            s[2 - a] = i
            return tuple(s)

        order = ((0, 2), (0, 1), (1, 0), (1, 2), (2, 0), (2, 1))
        for kind in ("pmc", "periodic"):
            for h, a in order:
                f, t = 3 + h, self.top[3 + h][a]
                for end in range(2):
                    if b[2 * a + end] == kind:
                        out = 0 if end == 0 else t + 1
                        src = (1 if end == 0 else t) if kind == "pmc" else (t if end == 0 else 1)
                        v = self.F[f][plane(f, a, src)].clone()
                        self.F[f][plane(f, a, out)] = -v if kind == "pmc" else v
        new = {}
        for face in range(6):
            a, end = face // 2, face % 2
            if b[face] != "mur":
                continue
            for h in ((a + 1) % 3, (a + 2) % 3):
                f = 3 + h
                s = [slice(1, self.top[f][q] + 1) for q in (2, 1, 0)]
                so = list(s)
                s[2 - a], so[2 - a] = (1, 0) if end == 0 else (self.top[f][a], self.top[f][a] + 1)
                s, so = tuple(s), tuple(so)
                edge = self.dh[a][0 if end == 0 else self.n[a] + self.o[a] + self.hi[a] + 0]
                er = np.array([1.0, 1.0] + [1.0 if r.kind == 0 else r.eps / EPS0 * r.mu / MU0 for r in self.pb.regions])
                cn = edge / (self.dt * C0 / np.sqrt(er))
                cab = torch.tensor((1 - cn) / (1 + cn), device=self.dev)[self.mi[f][s].long()]
                po, pi = self.mur.get((face, h), (0.0, 0.0))
                inner = self.F[f][s].clone()
                outer = pi + cab * (inner - po)
                self.F[f][so] = outer
                new[face, h] = (outer, inner)
        self.mur.update(new)

    def step(self):
        self.curl(0)
        self.poles(0)
        self.sources(0)
        self.curl(1)
        self.poles(1)
        self.sources(1)
        self.borders()
        self.t += self.dt

    def out(self):
        return [self.F[f][tuple(slice(0, self.top[f][a] + 2) for a in (2, 1, 0))] for f in range(6)]

    def box(self, f, b):
        return self.F[f][tuple(slice(b[2 * a] + self.o[a], b[2 * a + 1] + self.o[a] + 1) for a in (2, 1, 0))]


def _far_samples(x, c):
    """Surface samples of one step: per face and tangential E component, E and the H partner on its two planes."""
    b, out = _far_box(c), []
    for a in range(3):
        for end in range(2):
            for cc in ((a + 1) % 3, (a + 2) % 3):
                r = [v for q in range(3) for v in (b[2 * q], b[2 * q + 1] - (q == cc))]
                planes = [b[2 * a + end], b[2 * a + end] - (end == 0), b[2 * a + end] + (end == 1)]
                for k, f in enumerate((cc, 6 - a - cc, 6 - a - cc)):
                    r[2 * a] = r[2 * a + 1] = planes[k]
                    out.append((f, x.box(f, r).clone()))
    return out


def _far_rows(x, c, acc, freqs):
    b, rows = _far_box(c), []
    inc = _incident(c).astype(np.float64)
    th = np.arange(_ANGLES[0], _ANGLES[1] + 1e-6, _ANGLES[2])
    ph = np.arange(_ANGLES[3], _ANGLES[4] + 1e-6, _ANGLES[5])
    T, P = [torch.tensor(v.reshape(-1), device=x.dev) for v in np.meshgrid(th, ph, indexing="ij")]
    for q, fr in enumerate(freqs):
        k0 = 2 * math.pi * fr / C0
        sums = torch.zeros(2, 4, len(T), dtype=torch.complex128, device=x.dev)  # arithmetic, geometric; Lt Lp Nt Np
        i = 0
        for a in range(3):
            for end in range(2):
                for cc in ((a + 1) % 3, (a + 2) % 3):
                    E, H1, H2 = (acc[i + k][q] for k in range(3))
                    i += 3
                    dd = 3 - a - cc  # the magnetic current's axis
                    sign = (-1.0 if cc == (a + 2) % 3 else 1.0) * (1 if end else -1)
                    idx = [np.arange(b[2 * u], b[2 * u + 1] + (u != cc)) for u in range(3)]
                    idx[a] = np.array([b[2 * a + end]])
                    xyz = [torch.tensor(x.pos(cc, u, idx[u]), device=x.dev) for u in range(3)]
                    shape = tuple(len(idx[u]) for u in (2, 1, 0))
                    R = [v.reshape([-1 if 2 - u == k else 1 for k in range(3)]).expand(shape).reshape(-1)
                         for u, v in enumerate(xyz)]
                    area = (x.vec(x.de[cc][idx[cc] + x.o[cc]], cc) * x.vec(x.dh[dd][idx[dd] + x.o[dd]], dd)).expand(shape)
                    area = sign * area.reshape(-1)
                    p1, p2 = torch.angle(H1), torch.angle(H2)
                    pi = math.pi
                    n1 = torch.where((p1 < -pi / 2) & (p2 > pi / 2), p1 - 2 * pi, p1)
                    n2 = torch.where((p2 < -pi / 2) & (p1 > pi / 2), p2 - 2 * pi, p2)
                    geo = torch.polar(torch.sqrt((H1 * H2).abs()), (n1 + n2) / 2)
                    for d0 in range(0, len(T), 32):
                        t, p = T[d0:d0 + 32, None], P[d0:d0 + 32, None]
                        w = torch.exp(1j * k0 * (R[0] * (torch.sin(t) * torch.cos(p)) + R[1] * (torch.sin(t) * torch.sin(p)) +
                                                 R[2] * torch.cos(t)))
                        ft = (torch.cos(t) * torch.cos(p), torch.cos(t) * torch.sin(p), -torch.sin(t))
                        fp = (-torch.sin(p), torch.cos(p), torch.zeros_like(p))
                        M = (w * (E.reshape(-1) * area)).sum(1, keepdim=True)
                        for k, J in enumerate(((H1 + H2) / 2, geo)):
                            N = (w * (J.reshape(-1) * area)).sum(1, keepdim=True)
                            for z, (v, u) in enumerate(((M, dd), (M, dd), (N, cc), (N, cc))):
                                sums[k, z, d0:d0 + 32] += (v * (ft, fp)[z % 2][u]).reshape(-1)
        m = np.arange(1, len(inc))
        dte = inc[1, 0] - inc[0, 0]
        dft = abs((inc[1:, 1] * dte * np.exp(-2j * math.pi * fr * dte * (m - 1))).sum())
        X, Y = sums[:, 1] + ETA0 * sums[:, 2], sums[:, 0] - ETA0 * sums[:, 3]
        rcs = k0 ** 2 / (4 * math.pi * dft ** 2) * (X.abs() ** 2 + Y.abs() ** 2)
        et, ep = -1j * fr / (2 * C0) * X[1], 1j * fr / (2 * C0) * Y[1]
        rows.append(torch.stack([et.abs(), torch.angle(et), ep.abs(), torch.angle(ep), rcs[0], rcs[1]], 1))
    rows = torch.cat(rows).cpu().numpy()
    return [np.ascontiguousarray(rows[:, q]) for q in range(6)]


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "batch":
        return {"fields": [f for i in _instances(c) for f in exact(i, seed)["fields"]]}
    x = _Exact(c, seed)
    if c["kind"] != "solve":
        for f, v in enumerate(_initial(c, seed)):
            x.F[f][x.sl(f)] = v.double()
    freqs = [float(np.float32(v)) for v in _frequencies(c)]
    freq, movie, far, traces = 0.0, [], None, []
    for n in range(c["steps"] + (c["kind"] == "solve")):
        x.step()
        if c["kind"] == "solve":
            traces.append([float(x.F[p[0]][tuple(int(p[1 + a]) + x.o[a] for a in (2, 1, 0))]) for p in x.pb.probes])
        if c["kind"] == "frequency":
            w = torch.tensor([x.dt * np.exp(-2j * math.pi * f * n * x.dt) for f in freqs], device=x.dev)
            v = torch.stack([x.box(f, _probe_box(c)) for f in range(3)])
            freq = freq + w[:, None, None, None, None] * v
            if n % 8 == 0:
                movie.append(torch.stack([x.box(f, _movie_box(c)) for f in range(3, 6)]))
        if c["kind"] == "far":
            sm = _far_samples(x, c)
            far = far or [0.0] * len(sm)
            for i, (f, v) in enumerate(sm):
                w = [x.dt * np.exp(-2j * math.pi * fr * x.dt * (n + 0.5 * (f >= 3))) for fr in freqs]
                far[i] = far[i] + torch.tensor(w, device=x.dev)[:, None, None, None] * v
    if c["kind"] == "solve":
        return {"probes": np.array(traces).reshape(len(traces), c["probes"]),
                "fields": [f.permute(2, 1, 0).contiguous().cpu().numpy() for f in x.out()]}
    if c["kind"] == "frequency":
        return {"fields": x.out(), "frequency": freq.cpu().numpy(), "movie": torch.stack(movie).cpu().numpy()}
    if c["kind"] == "far":
        return {"fields": x.out(), "pattern": _far_rows(x, c, far, freqs)}
    return {"fields": x.out()}
