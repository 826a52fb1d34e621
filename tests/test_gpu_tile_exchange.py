"""The 2D tile form's exchange between tiles in float64 and EXACT arithmetic
(tile2d.cuh): long blocks and their remainders, sub-blocks of 1 to 8 steps,
psi of slabs that straddle tiles.  EXACT runs equal the per-cell launches bit
for bit; so do float64 fast runs, whose fusing is written out."""
import numpy as np
import pytest

from oidt_b200 import workloads as W
from oidt_b200.engine import Engine
from oidt_b200.spec import PSI

pytestmark = pytest.mark.gpu

STEPS = (141, 128, 33)  # a long block and a remainder, a long block alone, short blocks


def _te(**kw):
    from oidt_b200.refsetup import staggered_eps
    s = W.slab2d(**kw)
    s.mode = "te2"
    ex, ey = staggered_eps(s.meta["dt"] / s.cb["z"], np.float64, (0, 1))
    s.cb = {"x": s.meta["dt"] / ex, "y": s.meta["dt"] / ey}
    s.src_field = 5  # HZ
    lo, hi = s.src_lo[1], s.src_hi[1]
    s.src_lo, s.src_hi = (s.src_lo[0], lo + 1, 0), (s.src_lo[0] + 1, hi - 2, 1)
    return s


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _run(eng, spec, **choice):
    rng = np.random.default_rng(7)
    job = eng.submit(spec, **choice)
    for f in job.fields():
        job.set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(choice["precision"]))
    for n in STEPS:
        job.advance(n)
    job.sync(60000)
    got = dict(job.fields())
    got.update(("psi %s %d %d" % (f, ax, s), job.psi(f, ax, s)) for f, ax in PSI[spec.mode] for s in (0, 1))
    got.update(("dft %d %d" % (p, c), job.dft(p, c)) for p in (0, 1) for c in (0, 1))
    job.release()
    return got


@pytest.mark.parametrize("precision,arith", [(np.float64, "exact"), (np.float64, "fast"), (np.float32, "exact")])
@pytest.mark.parametrize("make", [W.slab2d, _te], ids=["tm2", "te2"])
@pytest.mark.parametrize("nx,ny,P,ports", [(66, 57, 4, (20, 46)), (40, 31, 1, (10, 30)), (203, 149, 10, (60, 61))])
def test_tiles_equal_per_cell_launches(eng, make, nx, ny, P, ports, precision, arith):
    spec = make(nx=nx, ny=ny, P=P, core_cells=9, src_x=8 + P // 2, ports=ports, steps=sum(STEPS), nf=3)
    kw = dict(precision=precision, arith=arith, ring_steps=16)
    want = _run(eng, spec, variant="cell", **kw)
    for choice in [dict()] + [dict(tile_steps=h) for h in (1, 3, 8)] + [dict(tile_coop=False)]:
        got = _run(eng, spec, variant="tile", **kw, **choice)
        for k, v in want.items():
            np.testing.assert_array_equal(got[k], v, err_msg="%s %r" % (k, choice))
