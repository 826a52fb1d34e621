"""What a 2D tile-form job needs: two buffers of its state, the ring of
ring_steps steps it asks for and the accumulators.  Its long blocks' ring and
its exchange words are extra: not counted by oidt_job_bytes, and given back
when another job needs the room, so a budget holds the jobs that fit it by
what they need; results are the same without."""
import ctypes

import numpy as np
import pytest

from oidt_b200 import workloads as W
from oidt_b200.spec import to_desc


def _spec(nx=300, ny=150, steps=300):
    return W.slab2d(nx=nx, ny=ny, core_cells=9, src_x=30, ports=(50, nx - 50), steps=steps, nf=3)


@pytest.mark.parametrize("precision,arith", [(np.float32, "fast"), (np.float32, "exact"), (np.float64, "exact")])
def test_bytes_needed(precision, arith):
    from oidt_b200.engine import load_library
    lib = load_library()

    def need(**kw):
        d, keep = to_desc(_spec(), precision=precision, arith=arith, **kw)
        n = ctypes.c_uint64()
        assert lib.oidt_job_bytes(ctypes.byref(d), ctypes.byref(n)) == 0
        return n.value
    step = 2 * 3 * 150 * np.dtype(precision).itemsize  # two ports, three slots of a line of ny
    assert need() == need(tile_coop=False)
    for k in (8, 16, 64, 128):
        assert abs(need(ring_steps=k) - need() - (k - 32) * step) <= 256, k
    # fields twice, dt/eps, CPML psi twice, accumulators, source, twiddles, ring; 256-byte pieces and tables besides
    cells, esz, P = 300 * 150, np.dtype(precision).itemsize, 10
    state = (7 * cells + 2 * 2 * 2 * P * (300 + 150)) * esz + 2 * 2 * 3 * 150 * 16 + 300 * esz + 4 * 3 * 300 * 8 + 32 * step
    assert state <= need() <= state + 32768


def _finish(job, spec, precision, n):
    job.advance(n).sync(60000)
    got = {f: job.field(f) for f in ("EZ", "HX", "HY")}
    got.update(("psi %s %d %d" % (f, ax, s), job.psi(f, ax, s)) for f, ax in (("EZ", 0), ("HX", 1)) for s in (0, 1))
    got.update(("dft %d %d" % (p, c), job.dft(p, c)) for p in (0, 1) for c in (0, 1))
    return got


def _submit(eng, spec, precision, seed):
    job = eng.submit(spec, precision=precision)
    rng = np.random.default_rng(seed)
    for f in ("EZ", "HX", "HY"):
        job.set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(precision))
    return job


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [np.float32, np.float64])
def test_budget_holds_the_jobs_that_fit_it(precision):
    from oidt_b200.engine import BudgetError, Engine
    spec = _spec()
    with Engine(0) as eng:
        need = eng.job_bytes(spec, precision=precision)
        a = _submit(eng, spec, precision, 0)
        a.advance(141)
        want = [_finish(a, spec, precision, 150)]
        a.release()
        for seed in (1, 2, 3):
            a = _submit(eng, spec, precision, seed)
            want.append(_finish(a, spec, precision, 291))
            a.release()
    with Engine(0, hbm_budget=4 * need) as eng:
        jobs = [_submit(eng, spec, precision, 0)]
        jobs[0].advance(141)  # a long block and a remainder, in flight while the next jobs need the room
        jobs += [_submit(eng, spec, precision, seed) for seed in (1, 2, 3)]
        with pytest.raises(BudgetError):
            eng.submit(spec, precision=precision)
        assert eng.stats()["hbm_in_use"] == 4 * need
        got = [_finish(j, spec, precision, n) for j, n in zip(jobs, (150, 291, 291, 291))]
        for g, w in zip(got, want):
            for k, v in w.items():
                np.testing.assert_array_equal(g[k], v, err_msg=k)
        for j in jobs[1:]:
            j.release()
        jobs[0].reset()  # the job that gave its memory back, from step 0; a new one beside it takes some again
        rng = np.random.default_rng(0)
        for f in ("EZ", "HX", "HY"):
            jobs[0].set_field(f, (rng.standard_normal(spec.shape) * 1e-2).astype(precision))
        new = _submit(eng, spec, precision, 1)
        jobs[0].advance(141)
        for g, w in ((_finish(jobs[0], spec, precision, 150), want[0]), (_finish(new, spec, precision, 291), want[1])):
            for k, v in w.items():
                np.testing.assert_array_equal(g[k], v, err_msg=k)
        jobs[0].release()
        new.release()
        assert eng.stats()["hbm_in_use"] == 0
    with Engine(0, hbm_budget=4 * need) as eng:  # multi-job blocks, one job without its extra memory
        jobs = [_submit(eng, spec, precision, seed) for seed in (1, 2, 3, 1)]
        eng.batch_advance(jobs, 291)
        for j, w in zip(jobs, want[1:] + want[1:2]):
            for k, v in _finish(j, spec, precision, 0).items():
                np.testing.assert_array_equal(v, w[k], err_msg=k)
            j.release()
