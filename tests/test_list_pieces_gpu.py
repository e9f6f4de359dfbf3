"""Model-order lists in pieces of eight ranks and sixty-four periods: whole, started and left pieces.

A run large enough for the lists equals the same models in runs below the line, bit
for bit, whatever pieces its ranks and periods make; ragged models may have more
periods than the pieces of the batch's geometry cover at once.
"""
import numpy as np
import pytest

from test_model_lists_gpu import _models, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wave,single", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("B,T,nmodes", [(65, 64, 6), (64, 65, 7), (34, 128, 8), (33, 129, 9), (70, 60, 256), (9, 500, 17)])
def test_large_run_equals_small_runs(B, T, nmodes, wave, single):
    b = _models(B, B + T)
    periods = np.geomspace(.1, 20., T)
    whole = _solve(b, periods, nmodes, wave, single, B)
    parts = _solve(b, periods, nmodes, wave, single, max(1, 4000 // T))
    for k, v in whole.items():
        assert np.array_equal(v, parts[k], equal_nan=v.dtype.kind == "f"), k


def test_ragged_models_longer_than_the_geometry():
    """period_offsets may give one model more periods than the engine's count."""
    from modisp_b200 import _native
    b = _models(60, 3)
    arrays = [b[k] for k in ("thickness", "vp", "vs", "rho")]
    counts = np.full(60, 70)
    counts[7], counts[8:20] = 70 + 12 * 60, 10
    offsets = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    periods = np.concatenate([np.geomspace(.2, 20., n) for n in counts])
    modes = np.full(60, 5, np.int32)
    o = _native.default_options()
    o.group_velocity = 1
    assert offsets[-1] == 60 * 70 and offsets[-1] >= 4096

    def run(keep):
        e = _native.Engine(0, len(keep), arrays[0].shape[1], int(counts[keep].max()) if len(keep) < 60 else 70, 5, o)
        try:
            off = np.concatenate([[0], np.cumsum(counts[keep])]).astype(np.int32)
            per = np.concatenate([periods[offsets[i]:offsets[i + 1]] for i in keep])
            return e.run_ragged(*(np.ascontiguousarray(a[keep]) for a in arrays), off, per, modes[keep], 1e-10, 1., 0,
                                group=True)
        finally:
            e.close()

    whole = run(np.arange(60))
    for i in (0, 7, 8, 59):
        part = run(np.array([i]))
        for key in ("velocity", "group_velocity", "group_velocity_flags"):
            cells = slice(5 * offsets[i], 5 * offsets[i + 1])
            assert np.array_equal(whole[key][cells], part[key], equal_nan=key != "group_velocity_flags"), (i, key)
        assert np.array_equal(whole["flags"][offsets[i]:offsets[i + 1]], part["flags"])
