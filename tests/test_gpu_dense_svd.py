"""The dense SVD of small projector matrices (dense_svd.cu) against its
definition and LAPACK's singular values: tall, wide and square, graded over 16
decades, rank deficient, not finite.  k Householder reflectors and 8 Jacobi
sweeps bound the backward error by (8 + 32) k u ||A||."""
import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200._lib import TGError, check, dptr

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def svd(A):
    m, n = A.shape
    k = min(m, n)
    Uo, VT, S = np.empty((m, k), A.dtype), np.empty((k, n), A.dtype), np.empty(k)
    check(_lib.load().tg_svd_host(m, n, int(np.iscomplexobj(A)), dptr(A), dptr(Uo), dptr(S), dptr(VT)))
    return Uo, S, VT


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("kind", ["graded", "deficient"])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 1), (1, 7), (9, 9), (21, 24), (32, 32), (33, 33), (40, 40), (64, 65),
                                 (84, 84), (90, 60), (60, 150), (96, 96), (119, 119)])
def test_dense_svd(m, n, kind, is_complex):
    if is_complex and min(m, n) > 84:
        pytest.skip("complex matrices up to 84 on the short side")
    rng = np.random.default_rng(m * 131 + n)
    k = min(m, n)

    def basis(r):
        x = rng.standard_normal((r, k)) + (1j * rng.standard_normal((r, k)) if is_complex else 0.0)
        return np.linalg.qr(x)[0]

    s = 10.0 ** (-16.0 * np.arange(k) / max(k - 1, 1))
    if kind == "deficient":
        s[(k + 1) // 2:] = 0.0
    A = np.ascontiguousarray(basis(m) * s @ basis(n).conj().T)
    if kind == "deficient":
        A[:, n // 2] = 0.0
    Uo, S, VT = svd(A)
    scale, tol = np.linalg.norm(A), 40 * max(k, 4) * U
    assert np.linalg.norm(Uo * S @ VT - A) <= tol * scale
    assert np.abs(S - np.linalg.svd(A, compute_uv=False)).max() <= tol * scale
    live = S > 1e-12 * S[0]  # the triplets a truncation keeps
    eye = np.eye(int(live.sum()))
    assert np.abs(Uo[:, live].conj().T @ Uo[:, live] - eye).max(initial=0.0) <= tol
    assert np.abs(VT[live] @ VT[live].conj().T - eye).max(initial=0.0) <= tol


def test_not_finite():
    A = np.eye(12)
    A[3, 4] = np.inf
    with pytest.raises(TGError):
        svd(A)
