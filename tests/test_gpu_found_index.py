"""The vector form's material index found in dt/eps grids: 1, 2, 256 different
(CBX, CBY, CBZ) triples (the index is used), 257 with the last one in the last
cell (it is not), signed zeros, z extents around the run length the search
takes at once.  The per-cell launches read the grids themselves; EXACT runs of
both are equal bit for bit, cells next to the source included."""
import numpy as np
import pytest

from oidt_b200 import workloads as W
from oidt_b200.engine import Engine
from oidt_b200.spec import PSI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _run(eng, spec, precision, variant):
    job = eng.submit(spec, arith="exact", precision=precision, variant=variant, ring_steps=7, material=False)
    rng = np.random.default_rng(5)
    for f in job.fields():
        job.set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(precision))
    job.advance(25).sync(60000)
    got = dict(job.fields())
    got.update(("psi %s %d %d" % (f, ax, s), job.psi(f, ax, s)) for f, ax in PSI[spec.mode] for s in (0, 1))
    job.release()
    return got


@pytest.mark.parametrize("source", ["TE", "TM"])
@pytest.mark.parametrize("nz", [31, 32, 45])
@pytest.mark.parametrize("triples", [1, 2, 256, 257])
@pytest.mark.parametrize("precision", [np.float64, np.float32])
def test_found_index_equals_grids(eng, precision, triples, nz, source):
    spec = W.strip3d(nx=20, ny=17, nz=nz, P=4, src_gap=2, port_gap=3, steps=30, nf=3, core_x_nm=120, core_y_nm=160,
                     source=source, seed=9)
    rng = np.random.default_rng(triples + nz)
    n = int(np.prod(spec.shape))
    pick = rng.integers(0, min(triples, 256), n)
    pick = np.repeat(pick[:: 3], 3)[:n]  # runs
    pick[: min(triples, 256)] = np.arange(min(triples, 256))
    if triples == 257:
        pick[-1] = 256
    for k, a in spec.cb.items():
        tab = float(a.flat[0]) * (1.0 + 0.01 * rng.random(257))
        if triples > 1:
            tab[1] = -0.0
        spec.cb[k] = tab[pick].reshape(spec.shape)
    spec.mat_idx = spec.mat_tab = None
    want = _run(eng, spec, precision, "cell")
    for k, v in _run(eng, spec, precision, "vec").items():
        np.testing.assert_array_equal(v, want[k], err_msg=k)
