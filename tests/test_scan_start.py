"""The scan leaves out velocities below a bound on the slowest root.

Love: the slowest shear velocity.  Rayleigh, solid stacks: the Rayleigh speed of a
half-space with the smallest bulk and shear moduli and the largest density of the
layers.  CPU: the oracle's secular function keeps one sign below the bound.  GPU:
the root that lies on the bound (a stack of equal layers) is found.
"""
import numpy as np
import pytest


def _rayleigh_speed(vp, vs):
    ratio = (vs / vp) ** 2
    a, b = 0., 1.
    for _ in range(60):
        x = .5 * (a + b)
        if ((x - 8.) * x + 24. - 16. * ratio) * x - 16. * (1. - ratio) < 0.:
            a = x
        else:
            b = x
    return vs * np.sqrt(.5 * (a + b))


def _bound(h, vp, vs, rho, wave):
    if wave:
        return vs.min()
    mu, bulk, heavy = (rho * vs ** 2).min(), (rho * (vp ** 2 - 4. / 3. * vs ** 2)).min(), rho.max()
    return _rayleigh_speed(np.sqrt((bulk + 4. / 3. * mu) / heavy), np.sqrt(mu / heavy))


@pytest.mark.parametrize("wave", [0, 1])
@pytest.mark.parametrize("trial", range(60))
def test_no_root_below_the_bound(trial, wave, oracle_lib):
    rng = np.random.default_rng(trial)
    L = int(rng.integers(2, 12))
    vs = rng.uniform(.4, 4., L)  # any order: low-velocity layers, stiff lids
    vs[-1] = 1.05 * vs.max()
    vp = vs * rng.uniform(1.3, 4., L)
    rho = rng.uniform(1., 4., L)
    h = np.append(rng.uniform(.05, 4., L - 1), 0.)
    c = np.geomspace(.125 * _bound(h, vp, vs, rho, wave), _bound(h, vp, vs, rho, wave) * (1. - 1e-9), 120)
    for period in (.2, 1., 5., 60.):
        # the bound is exact; a value at rounding distance from zero has no sign to hold
        F, g = oracle_lib.secular(h, vp, vs, rho, period, c, wave, True)
        F = F[np.abs(g) > 1e-9]
        assert np.all(F > 0.) or np.all(F < 0.)


@pytest.mark.gpu
@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("L", [2, 7])
def test_root_on_the_bound_is_found(L, single):
    from modisp_b200 import _native
    periods = np.geomspace(.1, 50., 40)
    h = np.full((1, L), .5)
    h[:, -1] = 0.
    vp, vs, rho = np.full((1, L), 2.), np.full((1, L), 1.1), np.full((1, L), 2.1)
    o = _native.default_options()
    o.single_precision = single
    e = _native.Engine(0, 1, L, periods.size, 2, o)
    try:
        out = e.run(h, vp, vs, rho, periods, None, 1e-10, 1., 0)
    finally:
        e.close()
    assert np.all(out["counts"] == 1)
    assert np.allclose(out["velocity"][0, 0], _rayleigh_speed(2., 1.1), rtol=1e-9, atol=0.)
