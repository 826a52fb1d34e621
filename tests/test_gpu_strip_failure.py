"""The exchange words of the 2D tile form's two kernels (float32 fast: strips;
float64: one cell a thread).  A bounded wait that runs out is reported, and the
job recovers by a reset with the default bound; a job that is reset part-way
through its blocks runs again as a new job does, although the numbers of its
sub-blocks repeat (the words are cleared with the counters)."""
import numpy as np
import pytest

from oidt_b200 import workloads as W
from oidt_b200.engine import Engine, TimeoutError_

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _state(job):
    got = {f: job.field(f) for f in ("EZ", "HX", "HY")}
    got.update(("dft %d %d" % (p, c), job.dft(p, c)) for p in (0, 1) for c in (0, 1))
    return got


def _fill(job, spec, precision, seed):
    rng = np.random.default_rng(seed)
    for f in ("EZ", "HX", "HY"):
        job.set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(precision))


@pytest.mark.parametrize("precision", [np.float32, np.float64])
def test_wait_expiry_is_reported_and_recoverable(eng, precision):
    """With a bound of one cycle the waits run out wherever a neighbour tile is
    still computing when a tile polls its words (144 tiles and more, tens of
    sub-blocks a launch); later waits of the launch give up at once and the
    launch ends."""
    spec = W.slab2d(steps=256)
    job = eng.submit(spec, variant="tile", precision=precision)
    _fill(job, spec, precision, 1)
    job.advance(200).sync(60000)
    want = _state(job)
    job.reset().set_wait_limit(1)
    job.advance(128)
    with pytest.raises(TimeoutError_, match="bounded wait"):
        job.sync(60000)
    other = eng.submit(spec, variant="tile", precision=precision)  # the context still works
    _fill(other, spec, precision, 1)
    other.advance(200).sync(60000)
    for k, v in _state(other).items():
        np.testing.assert_array_equal(v, want[k], err_msg=k)
    other.release()
    job.set_wait_limit(0).reset()
    _fill(job, spec, precision, 1)
    job.advance(200).sync(60000)
    for k, v in _state(job).items():
        np.testing.assert_array_equal(v, want[k], err_msg=k)
    job.release()


@pytest.mark.parametrize("precision", [np.float32, np.float64])
@pytest.mark.parametrize("first", [(128,), (141, 7), (32, 33, 64), (256,)])
def test_reset_job_runs_as_a_new_one(eng, precision, first):
    spec = W.slab2d(nx=253, ny=149, core_cells=9, src_x=30, ports=(50, 203), steps=256, nf=3)
    fresh = eng.submit(spec, variant="tile", precision=precision)
    _fill(fresh, spec, precision, 2)
    fresh.advance(141).advance(100).sync(60000)
    want = _state(fresh)
    fresh.release()
    job = eng.submit(spec, variant="tile", precision=precision)
    _fill(job, spec, precision, 3)
    for n in first:
        job.advance(n)
    job.reset()
    _fill(job, spec, precision, 2)
    job.advance(141).advance(100).sync(60000)
    for k, v in _state(job).items():
        np.testing.assert_array_equal(v, want[k], err_msg=k)
    job.release()
