"""The exact truncated SVD of the full-SVD projectors: which solves end in the
subspace iteration."""
import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200.env import CTMParams, Environment

pytestmark = pytest.mark.gpu


def site_tensors(dims, seed, falloff, is_complex=False, density=False):
    rng = np.random.default_rng(seed)
    out = []
    for d in dims:
        shape = tuple(d) + ((2, 2) if density else (2,))
        t = rng.normal(size=shape) + (1j * rng.normal(size=shape) if is_complex else 0)
        for leg, n in enumerate(d):
            t = t * np.exp(-falloff * np.arange(n)).reshape([-1 if a == leg else 1 for a in range(t.ndim)])
        out.append(t / np.abs(t).max())
    return out


def run(env, tensors):
    """One environment from scratch; the solver's counters it adds."""
    before = env.projector_svd_stats()
    for i, t in enumerate(tensors):
        env.set_site_tensor(i, t)
    env.calc_ctm_environment(True)
    after = env.projector_svd_stats()
    return {k: after[k] - before[k] for k in after}


@pytest.mark.parametrize("size,is_complex", [(1, False), (2, True)])
def test_slow_decay_is_no_stall(size, is_complex):
    """A flat spectrum at the block's edge, 30 iterations a solve: none of them
    is given up for the dense SVD."""
    dims = [[4] * 4] * size ** 2
    env = Environment(size, size, [2] * len(dims), dims,
                      CTMParams(chi=60, max_ctm_iteration=5, ctm_convergence_epsilon=1e-10), is_complex)
    tensors = site_tensors(dims, 3, 0.0, is_complex)
    for _ in range(2):
        counts = run(env, tensors)
        assert counts["solves"] == 20 * len(dims) and counts["dense"] == 0
    env.close()


@pytest.mark.parametrize("D,chi,is_complex,density", [(3, 24, False, False), (3, 20, True, False), (6, 24, False, True)])
def test_from_scratch_whatever_was_before(D, chi, is_complex, density):
    """A context that has computed another state's environment gives the same
    environment as a new one, bit for bit, with the same iterations and checks."""
    dims = [[D] * 4] * 4
    first, other = (site_tensors(dims, seed, 0.4, is_complex, density) for seed in (11, 12))
    got = []
    for before in ([], [other], [first, other]):
        env = Environment(2, 2, [2] * 4, dims, CTMParams(chi=chi, max_ctm_iteration=3, ctm_convergence_epsilon=1e-10,
                                                         density=density), is_complex)
        for tensors in before:
            run(env, tensors)
        counts = run(env, first)
        assert counts["solves"] == 48
        got.append((counts, [env.get_env(w, i) for w in range(8) for i in range(4)]))
        env.close()
    for counts, tensors in got[1:]:
        assert counts == got[0][0]
        for a, b in zip(tensors, got[0][1]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("falloff,is_complex", [(6.0, True), (6.0, False), (0.5, False)])
def test_rows_do_not_depend_on_each_other(falloff, is_complex):
    """Six rows whose solves take turns on four streams give what they give one
    after the other, as they run under the profiler, bit for bit and with the
    same iterations.  The steep tensors' panels are rank deficient: CholeskyQR
    meets a pivot that is not positive in some of the rows."""
    dims = [[3] * 4] * 12
    tensors = site_tensors(dims, 7, falloff, is_complex)
    got = []
    for one_by_one in (0, 1):
        _lib.load().tg_profile_enable(one_by_one)
        try:
            env = Environment(2, 6, [2] * 12, dims,
                              CTMParams(chi=16, max_ctm_iteration=2, ctm_convergence_epsilon=1e-10), is_complex)
            got.append((run(env, tensors), [env.get_env(w, i) for w in range(8) for i in range(12)]))
            env.close()
        finally:
            _lib.load().tg_profile_enable(0)
    assert got[0][0]["solves"] == 96 and got[0][0] == got[1][0]
    for a, b in zip(got[0][1], got[1][1]):
        assert np.array_equal(a, b)
