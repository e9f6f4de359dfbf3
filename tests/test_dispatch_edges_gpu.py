"""Edges of the engine's dispatch that the larger tests pass by.

The paired Love evaluation where two record buffers give way to one, an engine made
for device pointers that is given host arrays, search windows narrower than the scan's
grid and around the bound the scan starts from, stacks of any order against the
oracle's dense search, and the group-velocity flags of the derivative layer step.
"""
import numpy as np
import pytest

from test_layer_step_gpu import _stack

pytestmark = pytest.mark.gpu

FUSED, SPLIT = 1, 2
TOL = 1e-10  # c_tol_rel: refinement stops at an eighth of it, so two searches of a root agree within it


def _run(batch, periods, nmodes, wave, single=1, bounds=None, staging=True, **opts):
    from modisp_b200 import _native
    h = batch["thickness"]
    o = _native.default_options()
    o.single_precision, o.group_velocity = single, 1
    for k, v in opts.items():
        setattr(o, k, v)
    e = _native.Engine(0, h.shape[0], h.shape[1], periods.size, nmodes, o, staging=staging)
    try:
        return e.run(h, batch["vp"], batch["vs"], batch["rho"], periods, bounds, TOL, 1., wave, group=True)
    finally:
        e.close()


def _same(a, b):
    for key in ("velocity", "group_velocity", "flags", "levels", "counts", "group_velocity_flags"):
        np.testing.assert_array_equal(a[key].view(np.uint8), b[key].view(np.uint8), err_msg=key)


def _increasing(B, rows, seed):
    rng = np.random.default_rng(seed)
    vs = np.sort(rng.uniform(.5, 4., (B, rows)), axis=1)
    vs[:, -1] = 4.2
    vp = vs * rng.uniform(1.7, 2., (B, rows))
    h = rng.uniform(20., 60., (B, rows)) / rows
    h[:, -1] = 0.
    return dict(thickness=h, vp=vp, vs=vs, rho=1.74 * vp ** .25)


@pytest.mark.parametrize("rows", [2, 165, 168, 169, 172, 256])
def test_split_love_over_row_counts(rows):
    b = _increasing(24, rows, rows)
    if rows > 2:
        b["thickness"][::3, rows // 2:-1] = 0.  # shorter stacks in the same batch
    periods = np.geomspace(.5, 40., 23)
    _same(_run(b, periods, 4, 1, scan_mode=SPLIT), _run(b, periods, 4, 1, scan_mode=FUSED))


@pytest.mark.parametrize("single", [0, 1])
def test_host_arrays_through_an_engine_made_for_device_pointers(single):
    b = _increasing(17, 9, 1)
    periods = np.geomspace(.5, 40., 23)
    _same(_run(b, periods, 4, 0, single, staging=False), _run(b, periods, 4, 0, single))


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("wave", [0, 1])
@pytest.mark.parametrize("width", [1e-3, 1e-6, 2e-9, 5e-10, 1e-11, 1e-12])
def test_a_narrow_window_holds_its_root(width, wave, single):
    """From 1e-9 on the scan's start leaves samples out; below, log points could coincide."""
    b = _increasing(40, 8, 7)
    periods = np.array([3.])
    c = _run(b, periods, 2, wave, 0)["velocity"][:, 0, 0]
    assert np.isfinite(c).all()
    bounds = np.stack([c * (1. - .4 * width), c * (1. + .6 * width)], axis=1)
    out = _run(b, periods, 2, wave, single, bounds)
    np.testing.assert_array_equal(out["counts"][:, 0], 1)
    np.testing.assert_allclose(out["velocity"][:, 0, 0], c, rtol=TOL, atol=0.)


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("wave", [0, 1])
def test_windows_around_the_start_of_the_scan(wave, single):
    """The slowest shear velocity is Love's bound and lies above Rayleigh's."""
    b = _increasing(60, 9, 12)
    periods = np.geomspace(.5, 20., 9)
    slow = b["vs"].min(axis=1)
    auto = _run(b, periods, 4, wave, single)

    def window(lo, hi):
        return _run(b, periods, 4, wave, single, np.stack([slow * lo, slow * hi], axis=1))

    for lo in (1e-2, 1e-4, 1e-9):  # far below: the samples without a root are left out
        np.testing.assert_allclose(window(lo, 99.)["velocity"], auto["velocity"], rtol=TOL, atol=0.)
    assert not window(1e-3, .05)["counts"].any()  # ends below the bound
    above = window(1.3, 99.)  # starts above it
    lowest = 1.3 * slow[:, None]
    for i in range(60):
        for f in range(9):
            # modes 0 and 1 count from the first root above the window's start
            v = auto["velocity"][i, :, f]
            v = v[v > lowest[i] * (1. + 1e-6)]
            got = above["velocity"][i, :v.size, f]
            np.testing.assert_allclose(got, v, rtol=TOL, atol=0.)


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("wave", [0, 1])
def test_stacks_of_any_order_against_the_dense_search(wave, single, oracle_lib):
    from modisp_b200 import _native
    periods = np.array([.2, 1., 5., 60.])
    roots = 0
    for trial in range(40):
        rng = np.random.default_rng(1000 + trial)
        L = int(rng.integers(2, 12))
        vs = rng.uniform(.8, 4., L)  # any order: low-velocity layers, stiff lids
        vs[-1] = 1.05 * vs.max()
        vp = vs * rng.uniform(1.5, 2.5, L)
        rho = rng.uniform(1.5, 3.5, L)
        h = np.append(rng.uniform(.05, 1., L - 1), 0.)
        b = dict(zip(("thickness", "vp", "vs", "rho"), (x[None] for x in (h, vp, vs, rho))))
        out = _run(b, periods, 3, wave, single)
        lo, hi = out["bounds"][0]
        for f, period in enumerate(periods):
            n, want = oracle_lib.dense_roots(h, vp, vs, rho, period, lo, hi, 5, 1e-13, wave)
            if n < 0:  # (the dense search declined)
                continue
            assert out["counts"][0, f] == n, (trial, period)
            want = want[:min(n, 3)]
            np.testing.assert_allclose(out["velocity"][0, :want.size, f], want, rtol=1e-9, atol=0.)
            roots += want.size
    assert roots > 100


@pytest.mark.parametrize("kind", ["plain", "thin", "stiff", "close", "water"])
@pytest.mark.parametrize("L", [2, 3, 17, 60])
def test_the_layer_step_flags_no_good_group_velocity(kind, L, oracle_lib):
    """Where the oracle's group velocity is a number and positive, the engine's is not flagged
    (but for roots closer than the close-root distance) and agrees."""
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
            close = np.diff(roots) <= .005 * roots[1:]
            near = np.append(close, False) | np.append(False, close)
            group, flags = _native.group_roots(h, vp, vs, rho, 0, period, roots, roots.size)
            for q in range(roots.size):
                want = oracle_lib.group(h, vp, vs, rho, period, roots[q], roots[q] * (1. - 1e-6),
                                        roots[q] * (1. + 1e-6))
                if near[q] or not (np.isfinite(want) and want > 0.):
                    continue
                assert flags[q] == 0 and abs(group[q] - want) <= 1e-9 * want, (period, q, flags[q], group[q], want)
                checked += 1
    assert checked >= 8
