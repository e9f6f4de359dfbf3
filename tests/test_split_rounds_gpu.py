"""Rounds of the split scan: more modes ask for more of them, but only as many as the run fills."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launches(B, T, nmodes, mode, rows=21):
    from modisp_b200 import _native
    rng = np.random.default_rng(1)
    vs = np.sort(rng.uniform(.5, 4., (B, rows)), axis=1)
    vp = 1.8 * vs
    h = np.full((B, rows), .5)
    h[:, -1] = 0.
    o = _native.default_options()
    o.single_precision, o.scan_mode = 1, mode
    e = _native.Engine(0, B, rows, T, nmodes, o)
    try:
        out = e.run(h, vp, vs, 1.74 * vp ** .25, np.geomspace(1., 40., T), None, 1e-6, 1., 0)
        return e.kernel_launches(), out
    finally:
        e.close()


# (a round is seven launches, the hand-over two instead of the fused scan's one)
@pytest.mark.parametrize("B,T,nmodes,rounds", [
    (1024, 16, 5, 4), (1024, 16, 100, 4), (1024, 16, 256, 4), (1100, 40, 100, 9), (3000, 20, 10, 5), (4000, 40, 5, 4)])
def test_rounds_follow_traces_and_modes(B, T, nmodes, rounds):
    fused, a = _launches(B, T, nmodes, 1)
    split, b = _launches(B, T, nmodes, 2)
    assert (split - fused - 1) / 7 == rounds
    for key in ("velocity", "flags", "counts", "levels"):
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)
