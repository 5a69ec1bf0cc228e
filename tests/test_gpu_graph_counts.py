"""Which contexts replay their sweeps from a CUDA graph: every one whose sweep
stays on the device, from the second of a run without a limit on (or from the
seventh, where runs are shorter than six), and none that waits for the host."""
import numpy as np
import pytest

from tenes_b200.env import CTMParams, Environment

pytestmark = pytest.mark.gpu

BRICK = [[3, 1, 2, 3], [2, 3, 3, 1], [2, 3, 3, 1], [3, 1, 2, 3]]  # (left, up, right, down), 2 x 2


def context(dims, chi, is_complex, **kw):
    rng = np.random.default_rng(chi)
    env = Environment(2, 2, [2] * 4, dims, CTMParams(chi=chi, **kw), is_complex)
    for i, d in enumerate(dims):
        t = rng.uniform(-1, 1, tuple(d) + (2,)) + (1j * rng.uniform(-1, 1, tuple(d) + (2,)) if is_complex else 0.0)
        for leg, n in enumerate(d):
            t = t * (0.5 ** np.arange(n)).reshape([-1 if a == leg else 1 for a in range(5)])
        env.set_site_tensor(i, t)
    return env


ON_DEVICE = [
    ([[2] * 4] * 4, 6, False, {}),
    ([[2] * 4] * 4, 5, True, {}),
    ([[3] * 4] * 4, 8, False, dict(use_rsvd=True, rsvd_oversample_abs=4)),
    ([[3] * 4] * 4, 8, False, dict(use_rsvd=True, rsvd_oversample_abs=4, projector_corner=False)),
    ([[3] * 4] * 4, 8, True, dict(use_rsvd=True, rsvd_oversample_abs=4, projector_corner=False)),
    (BRICK, 7, True, dict(use_rsvd=True, rsvd_oversample_abs=3)),
    (BRICK, 7, False, {}),
]


@pytest.mark.parametrize("dims,chi,is_complex,kw", ON_DEVICE)
def test_replayed(dims, chi, is_complex, kw):
    for graph, replays in ((True, 4), (False, 0)):
        env = context(dims, chi, is_complex, cuda_graph=graph, **kw)
        env.init_env()
        for _ in range(5):
            env.sweep()
        assert env.graph_stats() == {"replays": replays, "captures": 1 if replays else 0}
        env.close()


def test_short_runs():
    env = context([[2] * 4] * 4, 6, False, max_ctm_iteration=4, ctm_convergence_epsilon=1e-15)
    counts = []
    for _ in range(3):
        env.calc_ctm_environment(True)
        counts.append(env.graph_stats()["replays"])
    assert counts == [0, 2, 6] and env.graph_stats()["captures"] == 1
    env.close()


@pytest.mark.parametrize("kw", [dict(chi=16), dict(chi=6, svd_solver=1), dict(chi=6, projector_corner=False)])
def test_waiting_for_the_host(kw):
    """The exact truncated SVD, gesvd, and full-SVD projectors from four corners."""
    env = context([[3] * 4] * 4, is_complex=False, **kw)
    env.init_env()
    for _ in range(4):
        env.sweep()
    assert env.graph_stats() == {"replays": 0, "captures": 0}
    env.close()
