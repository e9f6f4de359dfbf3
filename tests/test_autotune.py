"""The autotuner's choice between the automatic scan form and a forced one."""
import numpy as np
import pytest


def _best(monkeypatch, tmp_path, times):
    from modisp_b200 import autotune
    monkeypatch.setenv("MODISP_B200_CACHE", str(tmp_path))
    sample = {k: np.ones((4, 6)) for k in ("thickness", "vp", "vs", "rho")}
    return autotune.autotune(sample, [1., 2.], 3, 1, True, candidates=tuple(times),
                             timer=lambda shape, *a: (times[shape], None))


@pytest.mark.parametrize("forced,expected", [(1.99, (4, 0, 0)), (1.95, (4, 0, 0)), (1.9, (4, 0, 1))])
def test_a_forced_form_needs_a_clear_gain(monkeypatch, tmp_path, forced, expected):
    """On a small sample the automatic form is one of the forced ones: noise must not pin it for
    the large runs, where it is the other."""
    times = {(4, 0, 0): 2., (4, 0, 1): forced, (4, 0, 2): 2.4, (2, 0, 0): 2.2}
    assert _best(monkeypatch, tmp_path, times) == expected


@pytest.mark.parametrize("other,expected", [(1.99, (4, 0)), (1.9, (2, 0))])
def test_the_engine_default_needs_a_clear_loss(monkeypatch, tmp_path, other, expected):
    assert _best(monkeypatch, tmp_path, {(4, 0): 2., (2, 0): other, (1, 0): 3.}) == expected
