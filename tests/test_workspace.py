"""The workspace an engine reserves, and the chunks a memory budget leaves."""
import numpy as np
import pytest


def _options(single=0, continuation=0, continuity=1):
    from modisp_b200 import _native
    o = _native.default_options()
    o.single_precision, o.continuation, o.continuity_check = single, continuation, continuity
    return o


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("L,T,nmodes", [(2, 1, 1), (21, 60, 5), (256, 1, 5), (100, 20, 256)])
def test_workspace_counts_the_large_arrays(L, T, nmodes, single):
    from modisp_b200 import _native
    B, rows = 500, (L + 3) // 4 * 4
    n = _native.workspace_bytes(B, L, T, nmodes, _options(single))
    least = B * 9 * rows * 12 + B * T * ((nmodes + 2) * (5 * 8 + 2 * 4) + nmodes * (8 + 8 + 4 + 4))
    if single:  # paired records; a round's samples and their re-evaluation list
        least += B * rows * 96 + B * T * (64 * (8 + 4 * 4 + 8) + 64 * 4)
    assert least < n < 1.5 * least + B * ((129 + 2 * L) * 32 + (6 * L + 32) * 8 + 4 * L * 8 + T * 512) + 65536
    assert n < _native.workspace_bytes(B, L, T, nmodes, _options(single, continuation=1))


def test_invalid_geometry_has_no_workspace():
    from modisp_b200 import _native
    with pytest.raises(RuntimeError, match="invalid engine geometry"):
        _native.workspace_bytes(0, 3, 2, 1, _options())


@pytest.mark.parametrize("precision", ["float64", "mixed"])
@pytest.mark.parametrize("continuation", [False, True])
@pytest.mark.parametrize("budget", [300_000, 5_000_000, 123_456_789])
def test_chunks_stay_within_the_budget(budget, continuation, precision):
    from modisp_b200 import _native, api
    B, L, T, nmodes = 3000, 21, 60, 5
    s = api.Solver(precision=precision, workspace_bytes=budget)
    o = _options(int(precision != "float64"), int(continuation))
    n = s._capacity(B, L, T, nmodes, continuation)
    assert 1 <= n <= B
    assert _native.workspace_bytes(n, L, T, nmodes, o) <= budget
    assert n == B or _native.workspace_bytes(n + 1, L, T, nmodes, o) > budget
    assert api.Solver(precision=precision, workspace_bytes=budget, chunk_size=1)._capacity(B, L, T, nmodes) == 1


@pytest.mark.parametrize("precision", ["float64", "mixed"])
def test_the_smallest_budget_is_that_of_one_model(precision):
    from modisp_b200 import _native, api
    one = _native.workspace_bytes(1, 21, 60, 5, _options(int(precision != "float64")))
    assert api.Solver(precision=precision, workspace_bytes=one)._capacity(9, 21, 60, 5) == 1
    with pytest.raises(MemoryError, match="too small for one model"):
        api.Solver(precision=precision, workspace_bytes=one - 1)._capacity(9, 21, 60, 5)


def test_without_a_budget_the_free_memory_decides(monkeypatch):
    from modisp_b200 import _native, api
    s = api.Solver(precision="mixed")
    monkeypatch.setattr(_native, "memory_info", lambda: (170 << 30, 180 << 30))
    assert s._capacity(100_000, 21, 60, 5) == 100_000
    monkeypatch.setattr(_native, "memory_info", lambda: (64 << 20, 180 << 30))
    n = s._capacity(100_000, 21, 60, 5)
    assert _native.workspace_bytes(n, 21, 60, 5, _options(1)) <= 16 << 20
    monkeypatch.setattr(_native, "memory_info", lambda: (0, 180 << 30))
    assert s._capacity(100_000, 21, 60, 5) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("single", [0, 1])
def test_an_engine_takes_its_workspace(single):
    from modisp_b200 import _native
    o = _options(single)
    _native.Engine(0, 4, 21, 60, 5, o, staging=False).close()  # context and modules
    n = _native.workspace_bytes(5000, 21, 60, 5, o)
    before = _native.memory_info()[0]
    engine = _native.Engine(0, 5000, 21, 60, 5, o, staging=False)
    try:
        taken = before - _native.memory_info()[0]
    finally:
        engine.close()
    assert n <= taken <= n + (8 << 20)  # whole pages


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["float64", "mixed"])
def test_a_budgeted_solver_returns_the_same_result(precision):
    from modisp_b200 import api, workloads
    b = workloads.crustal_batch(64, 5)
    periods = np.geomspace(1., 40., 20)
    whole = api.Solver(precision=precision)(**b, periods=periods)
    parts = api.Solver(precision=precision, workspace_bytes=1_000_000)(**b, periods=periods)
    np.testing.assert_array_equal(whole.phase_velocity, parts.phase_velocity)
    np.testing.assert_array_equal(whole.trace_flags, parts.trace_flags)
