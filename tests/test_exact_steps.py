"""Where an exact truncated SVD looks at its residuals (exact_steps.hpp), on
residuals that fall by a given factor an iteration."""
import itertools
import math
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def solve(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    out = str(tmp_path_factory.mktemp("steps") / "exact_steps_host_check")
    subprocess.check_call([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "tenes_b200", "csrc"),
                           os.path.join(ROOT, "tests", "exact_steps_host_check.cpp"), "-o", out])

    def run(cases):
        text = "".join("%d %d %d %.17g %.17g %.17g\n" % c for c in cases)
        lines = subprocess.run([out], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
        assert len(lines) == len(cases)
        return [(int(a), int(b), float(c), int(d)) for a, b, c, d in (x.split() for x in lines)]

    return run


HINTS, RATIOS = [0, 1, 2, 7, 13, 20, 40], [1e2, 1e5, 1e9, 1e13]
DECAYS, EDGES = [0.01, 0.2, 0.5, 0.7, 0.8, 0.88], [0.0, 1e-20, 0.1, 0.45, 1.0]


def test_ends_where_the_decay_allows(solve):
    """No solve that needs at most 60 iterations is given up, whatever the
    hint and however much better a decay the spectrum promises, and none runs on
    for more than a gap of 16 beyond its hint and what it needs."""
    cases = [c for c in itertools.product([0], [0, 1], HINTS, RATIOS, DECAYS, EDGES)
             if math.log(c[3]) / -math.log(c[4]) <= 60]
    for c, (it, checks, ratio, hint) in zip(cases, solve(cases)):
        need = math.log(c[3]) / -math.log(c[4])
        assert it > 0 and ratio <= 1.0, c
        assert it <= max(c[2], 3, need) + 16, c
        assert hint >= 1 and 0 <= it - hint <= 2


def test_first_gap_has_an_iteration_in_hand(solve):
    """A solve without a hint that decays as its spectrum promises ends below
    the tolerance by an iteration's decay (or at its first check)."""
    cases = [(0, warm, 0, ratio0, decay, decay) for warm in (0, 1) for ratio0 in (1e2, 1e4) for decay in (0.2, 0.45)]
    for c, (it, checks, ratio, hint) in zip(cases, solve(cases)):
        assert checks == 1 or ratio <= c[4] * (1 + 1e-12), c
    assert max(checks for it, checks, ratio, hint in solve(cases)) > 1


def test_hints_settle_on_one_check(solve):
    """Solves that hand their hints on need one check each, no more than one
    iteration from the first that ends."""
    for ratio0, decay in itertools.product(RATIOS, [0.2, 0.5, 0.7]):
        hint = 40
        for _ in range(30):
            it, checks, ratio, hint = solve([(0, 1, hint, ratio0, decay, decay)])[0]
        need = math.ceil(math.log(ratio0) / -math.log(decay))
        assert checks == 1 and it - need <= 1, (ratio0, decay, it)


def test_hints_reach_one(solve):
    """Where one iteration is enough, the next solves look there."""
    for ratio0, decay in ((1e-3, 0.5), (0.5, 0.1), (5.0, 0.1)):
        hint = 7
        for _ in range(10):
            it, checks, ratio, hint = solve([(0, 1, hint, ratio0, decay, decay)])[0]
        assert (it, checks) == (1, 1)
    assert solve([(0, 1, 0, 0.5, 0.1, 0.1)])[0][:2] == (1, 1)


def test_flat_spectra_are_given_up(solve):
    for fixed, decay in itertools.product([0, 1], [0.95, 0.99, 1.0]):
        for it, checks, ratio, hint in solve([(fixed, 0, h, 1e13, decay, 1.0) for h in HINTS if not fixed or h == 0]):
            assert it == 0 and checks <= 12


def test_fixed_places(solve):
    """1 or 3, three later, then by the decay of the last two; above a ratio of
    one half between two of them, given up beyond iteration 12."""
    it, checks, ratio, _ = solve([(1, 0, 9, 1e5, 0.1, 0.3)])[0]
    assert (it, checks) == (6, 2)
    it, checks, ratio, _ = solve([(1, 1, 9, 1e7, 0.1, 0.3)])[0]
    r1, r4 = 1e7 * 0.1 ** 1, 1e7 * 0.1 ** 4
    assert (it, checks) == (4 + math.ceil(math.log(r4) / -math.log((r4 / r1) ** (1 / 3))), 3)
    assert solve([(1, 0, 0, 1e13, 0.97, 0.3)])[0][0] == 0
