"""The derivative-carrying Rayleigh layer step (propagation of the potentials' minors) against the oracle.

Group velocities at the oracle's roots take the step's value and both of its
derivatives through every layer.  The stacks sit where the step could go wrong:
one and many layers, thin layers at long periods, stiff layers far above the
phase velocity, velocities close to a layer's, a fluid top.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUP_RTOL = 1e-9  # the parity bound of the group velocities


def _stack(kind, L, rng):
    vs = np.sort(rng.uniform(.6, 4., L))
    h = rng.uniform(.2, 2., L)
    if kind == "thin":
        h = rng.uniform(1e-3, 2e-2, L)
    elif kind == "stiff":  # a stiff lid on soft rows
        vs[0], vs[-1] = 6., 6.5
    elif kind == "close":  # neighbours a hair apart
        vs[: L // 2] = vs[0] * (1. + 1e-7 * np.arange(L // 2))
    vp = vs * rng.uniform(1.5, 2.5, L)
    rho = rng.uniform(1.5, 3.5, L)
    if kind == "water":
        vs[0], vp[0], rho[0] = 0., 1.5, 1.03
    h[-1] = 0.
    return h, vp, vs, rho


@pytest.mark.parametrize("kind", ["plain", "thin", "stiff", "close", "water"])
@pytest.mark.parametrize("L", [2, 3, 17, 60])
def test_group_velocity_through_the_layer_step(kind, L, oracle_lib):
    from modisp_b200 import _native
    rng = np.random.default_rng(L)
    checked = 0
    for _ in range(4):
        h, vp, vs, rho = _stack(kind, L, rng)
        lo, hi = oracle_lib.bounds(h, vp, vs, rho)[0]
        for period in (.3, 2., 30.):
            n, roots = oracle_lib.dense_roots(h, vp, vs, rho, period, lo, hi, 3)
            roots = roots[:min(n, 3)]
            if not roots.size:
                continue
            group, flags = _native.group_roots(h, vp, vs, rho, 0, period, roots, roots.size)
            for q in np.flatnonzero(flags == 0):
                want = oracle_lib.group(h, vp, vs, rho, period, roots[q], roots[q] * (1. - 1e-6),
                                        roots[q] * (1. + 1e-6))
                if np.isfinite(want) and want > 0.:
                    assert abs(group[q] - want) <= GROUP_RTOL * want
                    checked += 1
    assert checked >= 4
