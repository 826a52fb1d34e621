"""The vector form's group widths (four cells a thread in float32, two in
float64) where a group can go wrong: port planes on every cell of a group,
z extents that are no multiple of the group, CPML slabs that end inside one,
one range of cells out of the fast quotient's range.  EXACT runs equal the
per-cell launches bit for bit; FAST float64 runs stay within rounding of them:
an update has fewer than 16 roundings of 2^-53 each, leapfrog keeps them from
growing, so 40 steps stay below 40 * 16 * 2^-53 < 1e-13 of the largest value
by a wide margin (1e-12 allowed)."""
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


def _run(eng, spec, precision, arith, variant, init):
    job = eng.submit(spec, arith=arith, precision=precision, variant=variant, ring_steps=7)
    for f, v in init.items():
        job.set_field(f, v.astype(precision))
    job.advance(10).advance(30).sync(60000)
    got = dict(job.fields())
    got.update(("psi %s %d %d" % (f, ax, s), job.psi(f, ax, s)) for f, ax in PSI[spec.mode] for s in (0, 1))
    got.update(("dft %d %d" % (p, c), job.dft(p, c)) for p in (0, 1) for c in range(4))
    job.release()
    return got


@pytest.mark.parametrize("nz", [36, 37, 38, 39])
@pytest.mark.parametrize("P", [3, 4, 5])
@pytest.mark.parametrize("source", ["TE", "TM"])
def test_group_widths(eng, nz, P, source):
    spec = W.strip3d(nx=21, ny=18, nz=nz, P=P, src_gap=1 + P % 2, port_gap=2 + nz % 4, steps=40, nf=3, core_x_nm=120,
                     core_y_nm=160, source=source, seed=nz)
    rng = np.random.default_rng(nz * 10 + P)
    init = {f: rng.standard_normal(spec.shape) * 1e-2 for f in ("EX", "EY", "EZ", "HX", "HY", "HZ")}
    for precision in (np.float64, np.float32):
        want = _run(eng, spec, precision, "exact", "cell", init)
        for k, v in _run(eng, spec, precision, "exact", "vec", init).items():
            np.testing.assert_array_equal(v, want[k], err_msg=k)
        if precision == np.float64:
            for k, v in _run(eng, spec, precision, "fast", "vec", init).items():
                scale = np.abs(want[k]).max()
                assert np.abs(v - want[k]).max() <= 1e-12 * max(scale, 1e-300), k
    # a block of cells below and above the quotients' range: those groups divide directly
    for lo, f in ((1e-290, np.float64), (1e280, np.float64)):
        far = {k: v.copy() for k, v in init.items()}
        for v in far.values():
            v[8:12, 5:9, 13:22] *= lo
        want = _run(eng, spec, f, "exact", "cell", far)
        for k, v in _run(eng, spec, f, "exact", "vec", far).items():
            np.testing.assert_array_equal(v, want[k], err_msg=k)
