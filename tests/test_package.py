"""The masks of a result: md200_package equals the numpy form of the same rules."""
import numpy as np
import pytest


def _result(B, K, T, dtype, seed):
    rng = np.random.default_rng(seed)
    v = np.sort(rng.uniform(1., 1.2, (B, K, T)), axis=1)  # many gaps near the close-root distance
    v[rng.random(v.shape) < .2] = np.nan
    v[rng.random(v.shape) < .01] = np.inf
    if K > 1:
        v[::3, 1] = v[::3, 0] * (1. + .005)  # on the distance
    flags = rng.choice(np.array([0, 1, 4, 128, 129, 2048, 4096, 65536, 32768], np.uint32), (B, T))
    counts = rng.integers(-1, K + 2, (B, T)).astype(np.int32)
    group = rng.uniform(.5, 2., v.shape)
    group[rng.random(v.shape) < .2] = np.nan
    return v.astype(dtype), flags, counts, group, rng.integers(0, 2, v.shape).astype(np.uint32)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("B,K,T", [(1, 1, 1), (1, 2, 1), (3, 1, 7), (5, 7, 33), (2600, 3, 61)])
def test_package_equals_numpy(B, K, T, dtype):
    from modisp_b200 import _native, api
    _native.lib()
    v, flags, counts, group, gflags = _result(B, K, T, dtype, B + K + T)
    for extra in ((None, None), (group, gflags)):
        got = _native.package(v, flags, counts, .005, *extra)
        want = api._masks(v, flags, counts, .005, *extra)
        for g, w in zip(got, want):
            assert (g is None) == (w is None)
            if w is not None:
                assert g.dtype == w.dtype and np.array_equal(g, w)


def test_other_layouts_take_the_numpy_form():
    from modisp_b200 import _native
    _native.lib()
    v, flags, counts, _, _ = _result(4, 3, 5, np.float64, 1)
    assert _native.package(v[:, :, ::2], flags[:, ::2], counts[:, ::2], .005) is None
    assert _native.package(v, flags.astype(np.int64), counts, .005) is None
    assert _native.package(v, flags[:, :4], counts, .005) is None
