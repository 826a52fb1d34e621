"""'TM' source boxes in, at, next to and a few cells past the z and x slabs, on
both sides: Ez's x-slab term and Ex's z-slab term read Hy - J there.  EXACT runs
of the vector and the ordered form equal the per-cell launches bit for bit.
FAST runs: an update has fewer than 16 roundings of 2^-24 (float32) or 2^-53
each and leapfrog keeps them from growing, so 30 steps stay below 30 * 16 of
them, 2.9e-5 and 5.4e-14 of the largest value; 1e-4 and 1e-12 are allowed.  J
is as large as the fields, so a term without it is off by far more."""
import numpy as np
import pytest

from oidt_b200 import workloads as W
from oidt_b200.engine import Engine
from oidt_b200.spec import PSI

pytestmark = pytest.mark.gpu

NX, NY, NZ, P = 24, 18, 41, 5
LO, HZ, HX = 2, NZ - 2, NX - 2  # updated cells: [2, n - 2)


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _spec(axis, box):
    s = W.strip3d(nx=NX, ny=NY, nz=NZ, P=P, src_gap=4, port_gap=4, steps=30, nf=3, core_x_nm=120, core_y_nm=160,
                  source="TM", seed=3)
    lo, hi = list(s.src_lo), list(s.src_hi)
    lo[axis], hi[axis] = box
    s.src_lo, s.src_hi = tuple(lo), tuple(hi)
    s.j_src = np.random.default_rng(2).standard_normal(30) * 1e-2
    return s


def _run(eng, spec, precision, arith, variant):
    job = eng.submit(spec, arith=arith, precision=precision, variant=variant, ring_steps=7)
    rng = np.random.default_rng(11)
    for f in job.fields():
        job.set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(precision))
    job.advance(30).sync(60000)
    got = dict(job.fields())
    got.update(("psi %s %d %d" % (f, ax, s), job.psi(f, ax, s)) for f, ax in PSI[spec.mode] for s in (0, 1))
    job.release()
    return got


Z = [(LO + 2, LO + 3), (LO + 4, LO + 5), (LO + 5, LO + 6), (LO + 6, LO + 7), (LO + 7, LO + 8), (LO + 3, LO + 9),
     (HZ - 2, HZ - 1), (HZ - 5, HZ - 4), (HZ - 6, HZ - 5), (HZ - 7, HZ - 6), (LO + 1, HZ)]
X = [(LO + 1, LO + 4), (LO + 4, LO + 6), (LO + 5, LO + 8), (LO + 6, LO + 9), (HX - 3, HX), (HX - 6, HX - 5),
     (HX - 7, HX - 6), (LO + 1, HX)]


@pytest.mark.parametrize("axis,box", [(2, b) for b in Z] + [(0, b) for b in X])
def test_source_at_the_slabs(eng, axis, box):
    spec = _spec(axis, box)
    for precision, tol in ((np.float64, 1e-12), (np.float32, 1e-4)):
        want = _run(eng, spec, precision, "exact", "cell")
        for variant in ("vec", "wave"):
            for k, v in _run(eng, spec, precision, "exact", variant).items():
                np.testing.assert_array_equal(v, want[k], err_msg="%s %s" % (variant, k))
            for k, v in _run(eng, spec, precision, "fast", variant).items():
                assert np.abs(v - want[k]).max() <= tol * np.abs(want[k]).max(), (variant, k)
