"""The one-sided Jacobi SVD (jacobi.cu) against its definition, at the edges of
its lane layouts: A = U S W^H, orthonormal factors, and LAPACK's singular
values.  A column takes part in about 8 n rotations (8 sweeps), each adding at
most 4 u to it, which bounds the backward error by 32 n u ||A||; two columns
count as orthogonal at 2 n u."""
import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200._lib import check, dptr

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("circle", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 16, 17, 32, 33, 48, 49, 64, 65, 84, 96, 97, 119])
def test_jacobi_svd(n, circle, is_complex):
    if is_complex and n > 84:
        pytest.skip("complex matrices up to 84")
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if is_complex else 0.0)
    A = np.ascontiguousarray(np.linalg.qr(A)[1].conj().T * np.exp(-0.1 * np.arange(n)))  # graded, as a projector's core
    Uo, Wo, S = np.empty_like(A), np.empty_like(A), np.empty(n)
    check(_lib.load().tg_jacobi_host(n, int(is_complex), circle, dptr(A), dptr(Uo), dptr(S), dptr(Wo)))
    scale, tol = np.linalg.norm(A), 32 * max(n, 4) * U
    eye = np.eye(n)
    assert np.linalg.norm(Uo * S @ Wo.conj().T - A) <= tol * scale
    assert np.abs(Wo.conj().T @ Wo - eye).max() <= tol
    assert np.abs(Uo.conj().T @ Uo - eye).max() <= tol
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.abs(S - ref).max() <= tol * scale
