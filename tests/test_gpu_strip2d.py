"""The 2D tile form's float32 fast kernel (strip2d.cuh) against the per-cell
launches of the same arithmetic, where its split can go wrong: grids smaller
than a strip or a halo, strips with a ragged last one, one-cell CPML slabs,
ports on one strip, tiles at every halo, ring blocks shorter than a sub-block,
long blocks and their remainders.  Both forms run the same operations, so
fields, CPML state and DFTs are equal bit for bit."""
import numpy as np
import pytest

from oidt_b200 import workloads as W
from oidt_b200.engine import Engine
from oidt_b200.spec import PSI

pytestmark = pytest.mark.gpu

STEPS = (141, 128, 33)  # a long block and a remainder, a long block alone, short blocks


def _tm(**kw):
    return W.slab2d(steps=sum(STEPS), nf=3, precision=np.float32, **kw)


def _te(**kw):
    from oidt_b200.refsetup import staggered_eps
    s = _tm(**kw)
    s.mode = "te2"
    ex, ey = staggered_eps(s.meta["dt"] / s.cb["z"], np.float64, (0, 1))
    s.cb = {"x": (s.meta["dt"] / ex).astype(np.float32), "y": (s.meta["dt"] / ey).astype(np.float32)}
    s.src_field = 5  # HZ
    lo, hi = s.src_lo[1], s.src_hi[1]
    s.src_lo, s.src_hi = (s.src_lo[0], lo + 1, 0), (s.src_lo[0] + 1, hi - 2, 1)
    return s


GRIDS = {
    "narrow": dict(nx=14, ny=40, P=2, core_cells=7, src_x=4, ports=(6, 10)),
    "p1": dict(nx=40, ny=31, P=1, core_cells=7, src_x=6, ports=(10, 30), rough=True, sigma_nm=30, lc_nm=60, seed=4),
    "tall": dict(nx=37, ny=1100, P=3, core_cells=9, src_x=6, ports=(10, 28)),
    "near": dict(nx=67, ny=58, P=4, core_cells=9, src_x=12, ports=(31, 34)),
    "same": dict(nx=66, ny=57, P=4, core_cells=9, src_x=12, ports=(31, 31)),
    "next": dict(nx=131, ny=97, P=6, core_cells=9, src_x=12, ports=(60, 61)),
    "slab": dict(nx=253, ny=149, P=10, core_cells=9, src_x=30, ports=(50, 203)),
    "waves": dict(nx=905, ny=431, P=8, core_cells=9, src_x=30, ports=(50, 803)),
}


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _run(eng, spec, **choice):
    rng = np.random.default_rng(7)
    job = eng.submit(spec, arith="fast", precision=np.float32, **choice)
    for f in job.fields():
        job.set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(np.float32))
    for n in STEPS:
        job.advance(n)
    job.sync(60000)
    got = {f: v for f, v in job.fields().items()}
    got.update(("psi %s %d %d" % (f, ax, s), job.psi(f, ax, s)) for f, ax in PSI[spec.mode] for s in (0, 1))
    got.update(("dft %d %d" % (p, c), job.dft(p, c)) for p in (0, 1) for c in (0, 1))
    job.release()
    return got


@pytest.mark.parametrize("mode", [_tm, _te], ids=["tm2", "te2"])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_strips_equal_per_cell_launches(eng, grid, mode):
    spec = mode(**GRIDS[grid])
    for ring in (1, 7, 32):
        want = _run(eng, spec, variant="cell", ring_steps=ring)
        for choice in [dict()] + [dict(tile_steps=h) for h in (1, 2, 3, 8)] + [dict(tile_coop=False),
                                                                              dict(tile_steps=5, tile_coop=False)]:
            got = _run(eng, spec, variant="tile", ring_steps=ring, **choice)
            assert got.keys() == want.keys()
            for k, v in want.items():
                np.testing.assert_array_equal(got[k], v, err_msg="%s ring %d %r" % (k, ring, choice))
