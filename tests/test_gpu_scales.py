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


def dense_svd(A):
    m, n = A.shape
    k = min(m, n)
    Uo, VT, S = np.empty((m, k), A.dtype), np.empty((k, n), A.dtype), np.empty(k)
    check(_lib.load().tg_svd_host(m, n, int(np.iscomplexobj(A)), dptr(A), dptr(Uo), dptr(S), dptr(VT)))
    return Uo, S, VT


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("m,n", [(1, 1), (12, 12), (33, 20), (40, 90), (201, 72)])  # 201 x 72 complex: all but 32 B of 227 KB
def test_dense_svd(m, n, is_complex):
    A = matrix(max(m, n), is_complex, m + n)[:m, :n]
    tol = 40 * min(m, n) * U * np.linalg.norm(A)  # the bound at unit scale (test_gpu_dense_svd.py)
    for scale in SCALES + [1e160, 1e300]:
        Uo, S, VT = dense_svd(np.ascontiguousarray(A * scale))
        assert np.abs(S / scale - np.linalg.svd(A, compute_uv=False)).max() <= tol
        assert np.linalg.norm(Uo * (S / scale) @ VT - A) <= tol


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("tiny", [1e-110, 1e-158, 1e-170, 1e-260, 1e-300])
def test_dense_svd_tiny_columns(tiny, is_complex):
    """Columns whose squares lose digits or vanish beside ordinary ones."""
    m, n, live = 24, 20, 14
    A = np.ascontiguousarray(matrix(m, is_complex, 3)[:, :n] * np.where(np.arange(n) < live, 1.0, tiny))
    Uo, S, VT = dense_svd(A)
    tol = 40 * n * U
    assert np.linalg.norm(Uo * S @ VT - A) <= tol * np.linalg.norm(A)
    assert np.abs(Uo[:, :live].conj().T @ Uo[:, :live] - np.eye(live)).max() <= tol
    assert np.abs(VT[:live] @ VT[:live].conj().T - np.eye(live)).max() <= tol
