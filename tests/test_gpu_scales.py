"""The factorisations of small matrices far from unit scale: results are those of
the same matrix at unit scale, times the scale."""
import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200._lib import check, dptr
from tenes_b200.env import CTMParams, Environment

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
SCALES = [1e-200, 1e-90, 1e-60, 1e60, 1e90, 1e140]


def matrix(n, is_complex, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if is_complex else 0.0)


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("n", [12, 40, 97])
def test_jacobi_svd(n, is_complex):
    if is_complex and n > 84:
        n = 84
    A = matrix(n, is_complex, n)
    ref = np.linalg.svd(A, compute_uv=False)
    for scale in SCALES:
        B = np.ascontiguousarray(A * scale)
        Uo, Wo, S = np.empty_like(B), np.empty_like(B), np.empty(n)
        check(_lib.load().tg_jacobi_host(n, int(is_complex), 0, dptr(B), dptr(Uo), dptr(S), dptr(Wo)))
        tol = 32 * n * U  # the bound at unit scale (test_gpu_jacobi.py)
        assert np.abs(S / scale - ref).max() <= tol * np.linalg.norm(A)
        assert np.linalg.norm(Uo * (S / scale) @ Wo.conj().T - A) <= tol * np.linalg.norm(A)


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("chi", [7, 33, 100])
def test_corner_spectrum(chi, is_complex):
    env = Environment(1, 1, [2], [[2] * 4], CTMParams(chi=chi), is_complex)
    A = matrix(chi, is_complex, chi)
    ref = np.linalg.svd(A, compute_uv=False)
    for scale in SCALES:
        env.set_env(0, 0, np.ascontiguousarray(A * scale))
        # normalised by its 2-norm; 32 n u as above
        assert np.abs(env.corner_spectrum(0, 0) - ref / np.linalg.norm(ref)).max() <= 32 * chi * U
    env.close()
