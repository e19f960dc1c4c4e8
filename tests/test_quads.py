"""The quad half-step kernels at the sizes where a quad can go wrong: widths
around multiples of four and of the 32-cell pitch, CPML slabs that begin and
end inside a quad, grids of one block and a few planes, and both sides of the
line to the TMA ring; what rides in them (source rows, observations) and when
it does not; and the contexts that they hand to other kernels."""
import ctypes
import tempfile
from dataclasses import replace
from pathlib import Path

import numpy as np
import pytest

import oracle
from bits import assert_bits_equal
from semba_fdtd_b200 import Solver, _lib, casegen, read_case

pytestmark = pytest.mark.gpu
_DIR = Path(tempfile.mkdtemp(prefix="semba_quads_"))


def _case(n, layers, boundary="pml", steps=24):
    rng = np.random.default_rng(sum(n) + layers)
    b = casegen._Builder(n, steps, max(layers, 1), boundary=boundary)
    dx = 0.003
    b.steps([dx], [dx], [dx])
    ds = casegen.courant_dt(dx) / 2
    c = [v // 2 for v in n]
    b.nodal(c, (c[0], c[1], c[2] + 1), "dipole.exc", ds, casegen.gaussian_derivative(ds, 8e-12, 40e-12, 0.1e-9))
    mid = b.material({"type": "simple", "relativePermittivity": 3.0, "electricConductivity": 0.05})
    b.bulk(mid, [tuple(x for v in n for x in (v // 3, max(v // 3, 2 * v // 3 - 1)))])
    b.probe("p", "electric", [max(1, v // 2 - 1) for v in n], "xyz")
    return read_case(b.write(_DIR, f"q_{'x'.join(map(str, n))}_{layers}_{boundary}")), rng


@pytest.mark.parametrize("n,layers,boundary", [
    ((5, 6, 7), 1, "pml"), ((6, 5, 4), 2, "pml"), ((7, 9, 5), 3, "pml"), ((8, 4, 6), 4, "pml"), ((13, 5, 6), 7, "pml"),
    ((27, 7, 5), 1, "pml"), ((29, 6, 9), 0, "mur"), ((30, 5, 8), 0, "pec"), ((31, 8, 5), 0, "pmc"),
    ((33, 5, 6), 0, "periodic"), ((61, 40, 37), 5, "pml"), ((97, 3, 5), 2, "pml")])
def test_ragged_quads_equal_the_oracle(n, layers, boundary):
    pb, rng = _case(n, layers, boundary)
    o = oracle.Oracle(pb)
    with Solver(pb) as s:
        for c in range(6):
            f = rng.standard_normal(s.field_shape(c)).astype(np.float32)
            f[0], f[-1], f[:, 0], f[:, -1], f[:, :, 0], f[:, :, -1] = 0, 0, 0, 0, 0, 0
            s.upload_field(c, f)
            o.set_field(c, f.transpose(2, 1, 0))
        assert_bits_equal(s.run(), o.step(pb.nsteps + 1))
        for c in range(6):
            assert_bits_equal(s.field(c), o.field(c), err_msg=f"component {c}")


@pytest.mark.parametrize("mode", ["graph", "fused", "routines", "batch"])
@pytest.mark.parametrize("layers", [4, 8, 12])
def test_both_x_slabs_in_one_quad_equal_the_oracle(layers, mode):
    """Two cells in x: the low slab of Hy and Hz ends on the first cell of a
    quad and the high slab begins on its last, as nowhere else in a grid the
    set-up makes."""
    from semba_fdtd_b200.batch import Batch
    pb, _ = _case((2, 7, 6), layers)
    o = oracle.Oracle(pb)
    want = o.step(pb.nsteps + 1)
    with Solver(pb) as s:
        x0 = s.alloc[0][0]
        for c in (4, 5):
            assert (s.sinpml[c][0] - 1 - x0) // 4 == (s.sinpml[c][1] + 1 - x0) // 4
        if mode != "batch":
            assert_bits_equal(s.run(mode=mode), want)
            got = [s.field(c) for c in range(6)]
    if mode == "batch":
        with Batch(64 << 20, 2) as b:
            slot = b.add(pb)
            b.run_all()
            assert_bits_equal(b.probes(slot), want)
            got = [b.field(slot, c) for c in range(6)]
    for c in range(6):
        assert_bits_equal(got[c], o.field(c), err_msg=f"component {c}")


def _launches(s):
    k = ctypes.c_int()
    s._check(s.lib.sgpu_kernels_per_step(s.handle, ctypes.byref(k)))
    return k.value


@pytest.mark.parametrize("mode,call", [("graph", 1), ("graph", 7), ("graph", 48), ("fused", 1)])
def test_a_wave_that_ends(mode, call):
    """Source rows ride in the half steps once the plane wave is past: calls of
    one step find the first such step, longer ones begin in mid-wave.  A line of
    36 nodes along x lies in one warp's cells, a lane more than it has."""
    n = (41, 26, 23)
    b = casegen._Builder(n, 150, 3)
    b.steps([0.003], [0.003], [0.003])
    ds = casegen.courant_dt(0.003) / 2
    b.planewave([9] * 3, [v - 9 for v in n], 0.7, 1.9, 1.1, 0.4, "gauss.exc", ds, casegen.gaussian(ds, 20e-12, 60e-12, 0.2e-9))
    late = casegen.gaussian_derivative(ds, 0.1e-9, 0.4e-9, 1.2e-9)
    b.nodal([3, 12, 11], [39, 12, 11], "line.exc", ds, late)
    b.nodal([30, 12, 11], [30, 12, 12], "dipole.exc", ds, late)
    b.nodal([9, 10, 9], [9, 10, 14], "hard.exc", ds, late, hard=True)
    b.probe("p", "electric", [v // 2 for v in n], "xyz")
    pb = read_case(b.write(_DIR, "wave_ends"))
    o = oracle.Oracle(pb)
    want = o.step(pb.nsteps + 1)
    seen = []
    with Solver(pb) as s:
        while s.n <= pb.nsteps:
            s.step(min(call, pb.nsteps + 1 - s.n), mode=mode)
            seen.append(_launches(s))
        # with a step a call the probes of the fused mode have launches of their own, which are not counted
        assert seen[0] == 4 and seen[-1] == 2 and seen == sorted(seen, reverse=True), seen
        assert_bits_equal(s.probes(), want)
        for c in range(6):
            assert_bits_equal(s.field(c), o.field(c), err_msg=f"component {c}")


@pytest.mark.parametrize("inset", [2, 5, 9])
def test_rows_and_observers_in_the_half_steps(inset):
    """A TF/SF box from one that fills the grid to a small one (its rows are
    k_sources'), with more point probes than a block of observers, a volume probe
    of each kind and field, and a step count that leaves a remainder after the
    captured steps."""
    n = (41, 26, 23)
    b = casegen._Builder(n, 75, 3)
    b.steps([0.003], [0.003], [0.003])
    ds = casegen.courant_dt(0.003) / 2
    lo, hi = [inset] * 3, [v - inset for v in n]
    b.planewave(lo, hi, 0.7, 1.9, 1.1, 0.4, "gauss.exc", ds, casegen.gaussian(ds, 20e-12, 60e-12, 0.2e-9))
    b.nodal([v // 2 for v in n], [n[0] // 2, n[1] // 2, n[2] // 2 + 1], "dipole.exc", ds,
            casegen.gaussian_derivative(ds, 8e-12, 40e-12, 0.1e-9))
    rng = np.random.default_rng(inset)
    for q in range(25):
        pos = [int(rng.integers(1, v - 1)) for v in n]
        b.probe(f"e{q}", "electric", pos, "xyz")
        b.probe(f"h{q}", "magnetic", pos, "z")
    pb = read_case(b.write(_DIR, f"rows_{inset}"))
    box, freqs = (5, 20, 4, 15, 3, 12), (1e9, 3e9)
    o = oracle.Oracle(pb)
    ids = [o.add_freq_probe(m, box, (2, 1, 3), np.array(freqs, np.float32)) for m in (False, True)]
    with Solver(pb) as s:
        got = [s.add_freq_probe(m, box, (2, 1, 3), freqs) for m in (False, True)]
        mov = [s.add_movie_probe(m, box, every=7, capacity=64) for m in (False, True)]
        assert_bits_equal(s.run(), o.step(pb.nsteps + 1))
        for c in range(6):
            assert_bits_equal(s.field(c), o.field(c), err_msg=f"component {c}")
        for a, r in zip(got, ids):
            assert_bits_equal(s.freq_probe(a, 2), o.freq_probe(r))
        for m, first in zip(mov, (0, 3)):
            n0, frames = s.movie_frames(m)
            assert n0 == 0 and len(frames) == 11
            # the last frame is of step 70: compare with a fresh run to it
            with Solver(pb, kernel_family=0) as w:
                w.step(71)
                for c in range(3):
                    f = w.field(first + c)
                    lo_ = [-a for a in (s.alloc[first + c][0], s.alloc[first + c][2], s.alloc[first + c][4])]
                    want = f[5 + lo_[0]:21 + lo_[0], 4 + lo_[1]:16 + lo_[1], 3 + lo_[2]:13 + lo_[2]].transpose(2, 1, 0)
                    assert_bits_equal(frames[-1][c], np.ascontiguousarray(want))


@pytest.mark.parametrize("n,launches", [((203, 187, 179), 2), ((235, 241, 241), 2), ((235, 242, 241), 4), ((301, 249, 197), 4)])
def test_both_sides_of_the_line_equal_the_oracle(n, launches):
    """Below, on, just above and above the line at 16 Mi padded cells (0.52, 1, 1.004
    and 1.07 times it), where the quads, in which the dipole and the probes ride,
    hand over to the TMA ring; four steps."""
    pb, _ = _case(n, 6)
    pb = replace(pb, nsteps=3)
    o = oracle.Oracle(pb)
    with Solver(pb) as s:
        assert_bits_equal(s.run(), o.step(4))
        assert _launches(s) == launches
        for c in range(6):
            assert_bits_equal(s.field(c), o.field(c), err_msg=f"component {c}")



def test_batch_of_small_and_large_instances():
    """Quads and TMA ring in one batch: an instance above the line next to one
    below it, a join while the large one runs, and a switch of families."""
    from semba_fdtd_b200.batch import Batch
    big, _ = _case((301, 249, 197), 6)
    small, _ = _case((27, 7, 5), 1)
    wide, _ = _case((61, 40, 37), 5)
    pbs = [replace(big, nsteps=5), replace(small, nsteps=9), replace(wide, nsteps=7)]
    want = [oracle.Oracle(pb).step(pb.nsteps + 1) for pb in pbs]
    with Batch(4 << 30, 4) as b:
        slots = [b.add(pbs[0]), b.add(pbs[1])]
        b.advance(2)
        slots.append(b.add(pbs[2]))
        b.advance(2)
        b._check(b.lib.sgpu_batch_set_kernel_family(b._h, 0), "family")
        b.advance(1)
        b._check(b.lib.sgpu_batch_set_kernel_family(b._h, 1), "family")
        b.run_all()
        for s, w in zip(slots, want):
            assert_bits_equal(b.probes(s), w)


@pytest.mark.parametrize("mode", ["graph", "fused"])
def test_sources_listed_while_the_ring_served(mode):
    """The source rows are listed under the wait drill, which keeps the quads
    off, and the steps run after it."""
    pb, _ = _case((41, 26, 23), 3, steps=70)
    o = oracle.Oracle(pb)
    with Solver(pb) as s:
        h = s.handle
        s._check(s.lib.sgpu_set_wait_drill(h, 1))
        s._check(s.lib.sgpu_advance_nodal_e(h, 0))  # lists the rows; no half step, so no wait runs out
        s._check(s.lib.sgpu_set_wait_drill(h, 0))
        for c in range(6):
            s.upload_field(c, np.zeros(s.field_shape(c), np.float32))
        assert_bits_equal(s.run(mode=mode), o.step(pb.nsteps + 1))
        for c in range(6):
            assert_bits_equal(s.field(c), o.field(c), err_msg=f"component {c}")


@pytest.mark.parametrize("calls", ["halves", "steps"])
def test_sources_of_an_instance_stepped_by_its_context(calls):
    """sgpu_batch_instance hands out a context; stepping it applies the sources."""
    from semba_fdtd_b200.batch import Batch
    pb, _ = _case((41, 26, 23), 3, steps=36)
    o = oracle.Oracle(pb)
    o.step(pb.nsteps + 1)
    with Batch(256 << 20, 2) as b:
        slot, ctx = b.add(pb), ctypes.c_void_p()
        b._check(b.lib.sgpu_batch_instance(b._h, slot, ctypes.byref(ctx)), "instance")
        if calls == "steps":
            assert b.lib.sgpu_advance_steps(ctx, 0, pb.nsteps + 1) == 0
        for n in range(pb.nsteps + 1 if calls == "halves" else 0):
            assert b.lib.sgpu_advance_e(ctx, n) == 0
            assert b.lib.sgpu_advance_h(ctx, n) == 0
        assert b.lib.sgpu_synchronize(ctx) == 0
        for c in range(6):
            assert_bits_equal(b.field(slot, c), o.field(c), err_msg=f"component {c}")


def _new_cpml(s, kind):
    """sgpu_init_cpml of a stepping context: the problem's y and z slabs with x
    slabs of other widths, or none at all; coefficients of the usual size."""
    class Desc(ctypes.Structure):
        _fields_ = [("pmlc", (_lib.Lim * 6) * 6)] + [(n, _lib.c_float_p * 3) for n in ("be", "ce", "bm", "cm")]

    d, rng, keep = Desc(), np.random.default_rng(7), []
    widths = {"none": (0, 0), "thin": (1, 2), "wide": (9, 6)}[kind]
    for f in range(6):
        w, q = s.sweep[f], s.sinpml[f]
        boxes = [(*w[:4], w[4], q[4] - 1), (*w[:4], q[5] + 1, w[5]), (*w[:2], w[2], q[2] - 1, *w[4:]),
                 (*w[:2], q[3] + 1, w[3], *w[4:]), (w[0], w[0] + widths[0] - 1, *w[2:]), (w[1] - widths[1] + 1, w[1], *w[2:])]
        for r, b in enumerate(boxes):
            d.pmlc[f][r] = _lib.Lim(*((1, 0, 1, 0, 1, 0) if kind == "none" else b))
    for a, c in enumerate((3, 4, 5)):
        n = s.alloc[c][2 * a + 1] - s.alloc[c][2 * a] + 1
        for name, lo, hi in (("be", 0.3, 0.9), ("ce", -100, 0), ("bm", 0.3, 0.9), ("cm", -100, 0)):
            v = rng.uniform(lo, hi, n).astype(np.float32)
            keep.append(v)
            getattr(d, name)[a] = v.ctypes.data_as(_lib.c_float_p)
    s._check(s.lib.sgpu_init_cpml(s.handle, ctypes.byref(d)), "sgpu_init_cpml")


@pytest.mark.parametrize("mode", ["graph", "fused"])
@pytest.mark.parametrize("kind", ["none", "thin", "wide"])
def test_cpml_set_again_between_steps(kind, mode):
    """The slabs decide how quads are numbered, and so the groups of the source
    rows; the register-marching kernels, which number nothing, are the reference."""
    n = (61, 31, 29)
    b = casegen._Builder(n, 60, 5)
    b.steps([0.003], [0.003], [0.003])
    ds = casegen.courant_dt(0.003) / 2
    wave = casegen.gaussian_derivative(ds, 20e-12, 80e-12, 0.6e-9)
    for q in range(4):  # lines through the slabs and between them
        b.nodal([2, 5 + 5 * q, 4 + 6 * q], [58, 5 + 5 * q, 4 + 6 * q], f"x{q}.exc", ds, wave)
        b.nodal([7 + 13 * q, 9, 8], [7 + 13 * q, 9, 20], f"z{q}.exc", ds, wave)
    b.probe("p", "electric", [v // 2 for v in n], "xyz")
    pb = read_case(b.write(_DIR, "cpml_again"))
    out = []
    for family in (1, 0):
        with Solver(pb, kernel_family=family) as s:
            s.step(20, mode=mode)
            _new_cpml(s, kind)
            s.step(41, mode=mode)
            out.append([s.probes()] + [s.field(c) for c in range(6)])
            assert _launches(s) == (2 if family else 4)  # the rows ride, and the probes
    assert np.isfinite(out[0][1]).all() and np.abs(out[0][1]).max() > 0
    for a, w in zip(*out):
        assert_bits_equal(a, w)


@pytest.mark.parametrize("first", ["sgpu_advance_h", "sgpu_advance_hx", "sgpu_advance_hz", "sgpu_advance_magnetic_cpml"])
@pytest.mark.parametrize("n,layers", [((5, 6, 7), 1), ((61, 40, 37), 5)])
def test_a_context_that_begins_with_h(n, layers, first):
    """The first quad kernel of a context follows the kernel that makes its
    tables, and reads them before it waits; the register-marching kernels, which
    have no tables, are the reference."""
    pb, _ = _case(n, layers)
    out = []
    for family in (1, 0):
        rng = np.random.default_rng(3)
        with Solver(pb, kernel_family=family) as s:
            for c in range(6):
                s.upload_field(c, rng.standard_normal(s.field_shape(c)).astype(np.float32))
            call = getattr(s.lib, first)
            s._check(call(s.handle, 0) if first == "sgpu_advance_h" else call(s.handle), first)
            out.append([s.field(c) for c in range(6)])
    for c, (a, w) in enumerate(zip(*out)):
        assert_bits_equal(a, w, err_msg=f"component {c}")


def test_an_instance_without_room_for_its_tables():
    """The quad tables of a batch's instance come from the device's memory pool,
    not the arena: where the pool refuses them the ring serves the instance."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    from semba_fdtd_b200.batch import Batch

    def ok(r):
        assert int(r[0]) == 0, r
        return r[1] if len(r) == 2 else None

    pb, _ = _case((41, 26, 23), 3)
    o = oracle.Oracle(pb)
    want = o.step(pb.nsteps + 1)
    with Batch(64 << 20, 2) as b:
        full, taken = rt.cudaMemPoolProps(), []
        full.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
        full.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
        full.maxSize = 2 << 20
        default, full = ok(rt.cudaDeviceGetDefaultMemPool(0)), ok(rt.cudaMemPoolCreate(full))
        for size in (1 << 20, 1 << 12):
            while True:
                err, p = rt.cudaMallocFromPoolAsync(size, full, rt.cudaStream_t(0))
                if int(err):
                    break
                taken.append(p)
                assert len(taken) < 1 << 12, "the pool is not bounded"
        ok(rt.cudaDeviceSetMemPool(0, full))
        try:
            slot = b.add(pb)
        finally:
            ok(rt.cudaDeviceSetMemPool(0, default))
            for p in taken:
                ok(rt.cudaFreeAsync(p, rt.cudaStream_t(0)))
            ok(rt.cudaStreamSynchronize(rt.cudaStream_t(0)))
            ok(rt.cudaMemPoolDestroy(full))
        ctx, k = ctypes.c_void_p(), ctypes.c_int()
        b._check(b.lib.sgpu_batch_instance(b._h, slot, ctypes.byref(ctx)), "instance")
        assert b.lib.sgpu_kernels_per_step(ctx, ctypes.byref(k)) == 0
        assert k.value == 4  # E, H, sources and probes: with the quads the probes ride
        b.run_all()
        assert_bits_equal(b.probes(slot), want)
        for c in range(6):
            assert_bits_equal(b.field(slot, c), o.field(c), err_msg=f"component {c}")


@pytest.mark.parametrize("family", [1, 0])
def test_a_time_vector_set_between_captured_steps(family):
    """Captured steps read the vector set last; half steps called one by one, which
    are not captured, are the reference."""
    pb, _ = _case((41, 26, 23), 3, steps=140)
    out = []
    for mode in ("graph", "fused"):
        with Solver(pb, kernel_family=family) as s:
            s.step(64, mode=mode)
            t = np.ascontiguousarray(s.time_vector() * 1.25)
            s._check(s.lib.sgpu_set_time(s.handle, 0, len(t), t.ctypes.data_as(_lib.c_double_p)), "sgpu_set_time")
            s.step(64, mode=mode)
            out.append([s.probes()] + [s.field(c) for c in range(6)])
    for a, w in zip(*out):
        assert_bits_equal(a, w)


@pytest.mark.parametrize("family", [1, 0])
def test_probes_set_between_captured_steps(family):
    """Captured steps write the ring of the probes set last; half steps called one
    by one are the reference."""
    pb, _ = _case((41, 26, 23), 3, steps=140)
    cijk = np.array([[0, 20, 13, 11], [5, 19, 12, 12], [1, 21, 13, 11], [2, 20, 13, 12]], np.int32)
    out = []
    for mode in ("graph", "fused"):
        with Solver(pb, kernel_family=family) as s:
            s.step(64, mode=mode)
            first = s.probes()
            s._check(s.lib.sgpu_set_probes(s.handle, len(cijk), cijk.ctypes.data_as(_lib.c_int_p), 64), "sgpu_set_probes")
            s._probe_base, s._probe_rows, s.nprobes = s.n, [], len(cijk)
            s.step(64, mode=mode)
            out.append([first, s.probes()] + [s.field(c) for c in range(6)])
            assert out[-1][1].shape == (64, 4)
    for a, w in zip(*out):
        assert_bits_equal(a, w)


def test_a_batch_of_more_items_than_blocks():
    """Two instances of 715 items a side, more together than the 1184 resident
    blocks, which claim the rest; one of them finishes first, in mid-chunk, so that
    its items do nothing for the steps left."""
    from semba_fdtd_b200.batch import Batch
    pb, _ = _case((110, 100, 90), 6)
    pbs = [replace(pb, nsteps=3), replace(pb, nsteps=9)]
    want = oracle.Oracle(pb).step(10)
    with Batch(1 << 30, 2) as b:
        slots = [b.add(q) for q in pbs]
        b.advance(10)
        b.synchronize()
        assert_bits_equal(b.probes(slots[0]), want[:4])
        assert_bits_equal(b.probes(slots[1]), want)
