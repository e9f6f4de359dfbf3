"""The automatic scan form on either side of its lines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AUTO, FUSED, SPLIT = 0, 1, 2


def _run(B, periods, wave, mode):
    from modisp_b200 import _native
    rng = np.random.default_rng(4)
    vs = np.sort(rng.uniform(.5, 4., (B, 2)), axis=1)
    vs[:, -1] = 4.2
    vp = vs * rng.uniform(1.7, 2., (B, 2))
    h = rng.uniform(10., 30., (B, 2))
    h[:, -1] = 0.
    o = _native.default_options()
    o.single_precision, o.group_velocity, o.scan_mode = 1, 1, mode
    e = _native.Engine(0, B, 2, periods.size, 1, o)
    try:
        out = e.run(h, vp, vs, 1.74 * vp ** .25, periods, None, 1e-10, 1., wave, group=True)
        return e.kernel_launches(), out
    finally:
        e.close()


@pytest.mark.parametrize("wave,models", [(0, 1024), (1, 12288)])
def test_the_automatic_form_changes_at_its_line(wave, models):
    """16 periods: 16,384 Rayleigh and 196,608 Love traces (in one chunk of the host-array run)."""
    periods = np.geomspace(2., 20., 16)
    for B, form in ((models - 1, FUSED), (models, SPLIT)):
        launches, auto = _run(B, periods, wave, AUTO)
        forced = {m: _run(B, periods, wave, m) for m in (FUSED, SPLIT)}
        assert forced[FUSED][0] != forced[SPLIT][0] and launches == forced[form][0], B
        for _, out in forced.values():
            for key in ("velocity", "group_velocity", "flags", "levels", "counts", "group_velocity_flags"):
                np.testing.assert_array_equal(auto[key].view(np.uint8), out[key].view(np.uint8), err_msg=key)
