"""The exact truncated SVD of the full-SVD projectors: which solves end in the
subspace iteration."""
import numpy as np
import pytest

from tenes_b200.env import CTMParams, Environment

pytestmark = pytest.mark.gpu


def site_tensors(dims, seed, falloff, is_complex=False):
    rng = np.random.default_rng(seed)
    out = []
    for d in dims:
        shape = tuple(d) + (2,)
        t = rng.normal(size=shape) + (1j * rng.normal(size=shape) if is_complex else 0)
        for leg, n in enumerate(d):
            t = t * np.exp(-falloff * np.arange(n)).reshape([-1 if a == leg else 1 for a in range(5)])
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
