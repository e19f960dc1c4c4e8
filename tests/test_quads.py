"""The quad half-step kernels at the sizes where a quad can go wrong: widths
around multiples of four and of the 32-cell pitch, CPML slabs that begin and
end inside a quad, both sides of an axis in one quad, grids of one block and
a few planes, and both sides of the line to the TMA ring."""
import tempfile
from dataclasses import replace
from pathlib import Path

import numpy as np
import pytest

import oracle
from bits import assert_bits_equal
from semba_fdtd_b200 import Solver, casegen, read_case

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


@pytest.mark.parametrize("n", [(203, 187, 179), (301, 249, 197)])
def test_both_sides_of_the_line_equal_the_oracle(n):
    """Just below and just above 16 Mi padded cells, where the quads hand over
    to the TMA ring; four steps."""
    pb, _ = _case(n, 6)
    pb = replace(pb, nsteps=3)
    o = oracle.Oracle(pb)
    with Solver(pb) as s:
        assert_bits_equal(s.run(), o.step(4))
        for c in range(6):
            assert_bits_equal(s.field(c), o.field(c), err_msg=f"component {c}")

