"""Refinement and group-velocity lists in model order (runs of 4096 traces or more).

A run's results do not depend on the order its brackets are refined in: a batch
large enough for the model-order lists equals the same models in batches below
the line, bit for bit -- at the line, above it, with one mode (two of three
brackets are guards), with more modes than a warp has lanes, with models that have
no window of their own (Love without a guide) and in ragged form.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _models(B, seed):
    from modisp_b200 import workloads
    b = workloads.crustal_batch(B, seed, nmin=1, nmax=9, lvz_fraction=.3)
    b["vs"][::7] = 1.5  # no layer slower than the half-space
    b["vp"][::7] = 2.9
    return b


def _solve(b, periods, nmodes, wave, single, cut):
    from modisp_b200 import _native
    o = _native.default_options()
    o.single_precision, o.group_velocity = single, 1
    B, L = b["thickness"].shape
    parts = []
    for s in range(0, B, cut):
        part = [np.ascontiguousarray(b[k][s:s + cut]) for k in ("thickness", "vp", "vs", "rho")]
        e = _native.Engine(0, part[0].shape[0], L, periods.size, nmodes, o)
        try:
            parts.append(e.run(*part, periods, None, 1e-10, 1., wave, group=True))
        finally:
            e.close()
    return {k: np.concatenate([p[k] for p in parts]) for k in parts[0] if k not in ("stats", "bounds")}


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("wave", [0, 1])
@pytest.mark.parametrize("B,T,nmodes", [(128, 32, 5), (129, 33, 1), (140, 31, 40), (4200, 1, 3)])
def test_large_run_equals_small_runs(B, T, nmodes, wave, single):
    b = _models(B, 11 + T)
    periods = np.geomspace(.1, 20., T)
    whole = _solve(b, periods, nmodes, wave, single, B)
    parts = _solve(b, periods, nmodes, wave, single, max(1, 2000 // T))
    for k, v in whole.items():
        assert np.array_equal(v, parts[k], equal_nan=v.dtype.kind == "f"), k


@pytest.mark.parametrize("wave", ["rayleigh", "love"])
def test_ragged_run_equals_its_parts(wave):
    from modisp_b200.ragged import dispersion_ragged
    b = _models(150, 5)
    rng = np.random.default_rng(3)
    periods = [np.geomspace(.2, 20., int(n)) for n in rng.integers(1, 70, 150)]
    modes = rng.integers(1, 9, 150)
    assert sum(p.size for p in periods) > 4096
    r = dispersion_ragged(**b, periods=periods, nmodes=modes, wave=wave)
    for s in range(0, 150, 30):
        q = dispersion_ragged(**{k: v[s:s + 30] for k, v in b.items()}, periods=periods[s:s + 30],
                              nmodes=modes[s:s + 30], wave=wave)
        for i in range(30):
            assert np.array_equal(r.phase_velocity_of(s + i), q.phase_velocity_of(i), equal_nan=True)
            assert np.array_equal(r.group_velocity_of(s + i), q.group_velocity_of(i), equal_nan=True)
            assert np.array_equal(r.trace_flags_of(s + i), q.trace_flags_of(i))
