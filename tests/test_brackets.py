"""Rules on bracket slots (modisp_b200/csrc/brackets.cuh), built for the host.

A guard root that its bracket settles is not refined, so its slot holds the
bracket's midpoint.  That midpoint must never reach a reported rank.
"""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SOURCE = """
#include "brackets.cuh"
extern "C" int clear_of(const double *slots, int n, int i, double rtol) {
  return md200::guard_is_clear(slots, n, i, rtol);
}
extern "C" int confirm(double fa, double fb) { return md200::ends_confirm(fa, fb); }
"""
RTOL = .005


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    folder = tmp_path_factory.mktemp("brackets")
    (folder / "rules.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{ROOT / 'modisp_b200' / 'csrc'}",
                    "-o", str(folder / "rules.so"), str(folder / "rules.cpp")], check=True)
    lib = ctypes.CDLL(str(folder / "rules.so"))
    lib.clear_of.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_double]
    lib.confirm.argtypes = [ctypes.c_double, ctypes.c_double]
    return lib


def _slots(brackets):
    s = np.full((len(brackets), 5), np.nan)
    s[:, :2] = brackets
    return s


def _clear(rules, brackets, i):
    s = _slots(brackets)
    return bool(rules.clear_of(s.ctypes.data, len(s), i, RTOL))


def test_separate_guards_are_settled(rules):
    b = [(1., 1.1), (1.2, 1.3), (1.5, 1.6), (2., 2.1)]
    assert _clear(rules, b, 2) and _clear(rules, b, 3)


@pytest.mark.parametrize("pair", [(0, 1), (1, 2), (0, 2)])
def test_guards_after_brackets_that_may_share_a_zero_are_refined(rules, pair):
    # (neg, +0, neg): both brackets end on the zero, whose root counts once, so the
    # guards' ranks move down by one
    b = [(1., 1.1), (1.2, 1.3), (1.4, 1.5), (2., 2.1), (2.5, 2.6)]
    j, k = pair
    if k == j + 1:
        b[k] = (b[j][1], b[k][1])
    else:  # out of order
        b[0], b[2] = b[2], b[0]
    assert not _clear(rules, b, 3) and not _clear(rules, b, 4)


@pytest.mark.parametrize("side", ["left", "right"])
def test_the_close_root_distance_itself_is_not_clear(rules, side):
    """Roots at a gap of exactly the distance are close (gap <= rtol * upper root)."""
    guard = (2., 2.1)
    for gap, expected in ((RTOL * 2.1 if side == "left" else RTOL * 2.3, False), (.02, True), (1e-9, False)):
        if side == "left":
            b, i = [(1., 1.1), (1.5, guard[0] - gap), guard], 2
        else:
            upper = 2.3 if gap != .02 else 2.2
            b, i = [(1., 1.1), guard, (guard[1] + gap, upper)], 1
        assert _clear(rules, b, i) is expected, gap


def test_settled_guards_never_reach_a_reported_rank(rules):
    """Random bracket sets with touching and close neighbours: refining every bracket, or only
    those that are not settled, reports the same roots and counts."""
    rng = np.random.default_rng(3)
    settled = shared = 0
    for _ in range(4000):
        n = int(rng.integers(2, 9))
        modes = int(rng.integers(1, n))
        gaps = rng.choice([0., RTOL, .004, .05, .2], n)
        widths = rng.uniform(.001, .05, n)
        brackets, at = [], 1.
        for g, w in zip(gaps, widths):
            brackets.append((at + g * at, at + g * at + w))
            at = brackets[-1][1]
        roots = [rng.uniform(l, h) for l, h in brackets]
        for j in range(n - 1):
            if brackets[j][1] == brackets[j + 1][0] and rng.uniform() < .7:
                roots[j] = roots[j + 1] = brackets[j][1]  # an exact zero at the common end
                shared += 1
        clear = [j >= modes and _clear(rules, brackets, j) for j in range(n)]
        settled += sum(clear)
        kept = [.5 * (l + h) if c else r for c, r, (l, h) in zip(clear, roots, brackets)]

        def report(values):
            v = np.unique(values)  # ordered, exact duplicates once
            close = np.diff(v) <= RTOL * v[1:]
            near = [(bool(m and close[m - 1]), bool(m < close.size and close[m])) for m in range(min(modes, v.size))]
            return v[:modes].tolist(), v.size, near, bool(close.any())

        assert report(roots) == report(kept)
    assert settled > 500 and shared > 100


@pytest.mark.parametrize("fa,fb,expected", [
    (-1., 1., True), (1., -1e-300, True), (-1e-300, 1e-300, True), (-1e300, 1e300, True),
    (1., 1., False), (-1., -1., False), (0., 1., False), (-1., 0., False), (-0., 1., False),
    (-np.inf, 1., False), (1., -np.inf, False), (-np.inf, np.inf, False), (np.nan, 1., False), (-1., np.nan, False)])
def test_ends_that_settle_a_guard(rules, fa, fb, expected):
    """A guard is settled where refinement would end on a root: an infinite end fails there."""
    assert bool(rules.confirm(fa, fb)) is expected
