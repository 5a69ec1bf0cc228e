"""Sweeps replayed from a CUDA graph equal eagerly launched ones bit for bit, for
every kind of context whose sweep stays on the device: small full-SVD matrices,
randomised up/down projectors, and D = 1 legs beside randomised ones."""
import numpy as np
import pytest

from tenes_b200.env import CTMParams, Environment

pytestmark = pytest.mark.gpu

BRICK = [[3, 1, 2, 3], [2, 3, 3, 1], [2, 3, 3, 1], [3, 1, 2, 3]]  # (left, up, right, down), 2 x 2


@pytest.mark.parametrize("dims,chi,is_complex,kw", [
    ([[2] * 4] * 4, 6, False, {}),
    ([[2] * 4] * 4, 5, True, {}),
    ([[3] * 4] * 4, 8, False, dict(use_rsvd=True, rsvd_oversample_abs=4, projector_corner=False)),
    ([[3] * 4] * 4, 8, True, dict(use_rsvd=True, rsvd_oversample_abs=4, projector_corner=False)),
    (BRICK, 7, True, dict(use_rsvd=True, rsvd_oversample_abs=3)),
    (BRICK, 7, False, {}),
])
def test_replayed_equals_eager(dims, chi, is_complex, kw):
    rng = np.random.default_rng(chi)
    tensors = []
    for d in dims:
        t = rng.uniform(-1, 1, tuple(d) + (2,)) + (1j * rng.uniform(-1, 1, tuple(d) + (2,)) if is_complex else 0.0)
        for leg, n in enumerate(d):
            t = t * (0.5 ** np.arange(n)).reshape([-1 if a == leg else 1 for a in range(5)])
        tensors.append(t)
    got = []
    for graph in (True, False):
        env = Environment(2, 2, [2] * 4, dims, CTMParams(chi=chi, cuda_graph=graph, **kw), is_complex)
        for i, t in enumerate(tensors):
            env.set_site_tensor(i, t)
        env.init_env()
        for _ in range(5):
            env.sweep()
        got.append([env.get_env(w, i) for w in range(8) for i in range(4)])
        env.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
