"""Engines of different row counts that live at the same time.

A kernel's limit on dynamic shared memory holds for the process, not for an engine,
and the kernels' needs differ by engine: they grow with the rows (scan, preparation),
and the paired evaluation's drop where two record buffers give way to one (past 56
rows Rayleigh, 168 Love).  An engine must run after any other was made, and return
what it returns alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PERIODS = np.geomspace(.5, 40., 11)


def _stack(rows):
    rng = np.random.default_rng(rows)
    B = 12
    vs = np.sort(rng.uniform(.5, 4., (B, rows)), axis=1)
    vs[:, -1] = 4.2
    vp = vs * rng.uniform(1.7, 2., (B, rows))
    h = rng.uniform(20., 60., (B, rows)) / rows
    h[:, -1] = 0.
    return h, vp, vs, 1.74 * vp ** .25


def _engine(rows, single):
    from modisp_b200 import _native
    o = _native.default_options()
    o.single_precision, o.scan_mode = single, 2 if single else 0
    return _native.Engine(0, 12, rows, PERIODS.size, 3, o)


def _run(engine, rows, wave):
    return engine.run(*_stack(rows), PERIODS, None, 1e-10, 1., wave)


@pytest.mark.parametrize("wave,single,first,second", [
    (0, 1, 40, 60), (0, 1, 56, 57), (0, 1, 256, 12), (1, 1, 168, 172), (1, 1, 256, 12),
    (0, 0, 256, 12), (1, 0, 256, 12), (0, 0, 12, 256)])
def test_an_engine_runs_after_another_was_made(wave, single, first, second):
    alone = _engine(first, single)
    try:
        expected = _run(alone, first, wave)
        other = _engine(second, single)
        try:
            _run(other, second, wave)
            again = _run(alone, first, wave)
        finally:
            other.close()
    finally:
        alone.close()
    for key in ("velocity", "flags", "counts"):
        np.testing.assert_array_equal(again[key], expected[key], err_msg=key)
