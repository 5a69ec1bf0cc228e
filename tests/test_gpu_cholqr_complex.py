"""The one-launch cluster CholeskyQR of complex panels against numpy, at edges of
its 8-column blocks, of the rows a CTA holds (48 staged at once) and of the
cluster's row ranges: orthonormality, the span, Householder's Q, rank deficiency."""
import ctypes as C

import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200._lib import check, dptr

pytestmark = pytest.mark.gpu


def cholqr(Y, passes):
    n, k = Y.shape
    flag = C.c_int(0)
    buf = np.ascontiguousarray(Y.T)  # column-major n x k = row-major k x n
    check(_lib.load().tg_cholqr_host_complex(n, k, dptr(buf), passes, C.byref(flag)))
    return buf.T.copy(), flag.value


def panel(n, k, cond, seed):
    rng = np.random.default_rng(seed)
    U, _ = np.linalg.qr(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k)))
    V, _ = np.linalg.qr(rng.standard_normal((k, k)) + 1j * rng.standard_normal((k, k)))
    s = np.logspace(0, -np.log10(cond), k) if k > 1 else np.ones(1)
    return (U * s) @ V.conj().T


@pytest.mark.parametrize("n,k", [(1, 1), (9, 1), (5, 3), (37, 8), (64, 64), (243, 43), (768, 88), (769, 17),
                                 (2600, 40)])
@pytest.mark.parametrize("passes", [2, 4])
def test_orthonormal_and_same_span(n, k, passes):
    # the bounds of the real kernel's test: two shifted passes leave a condition number of ~1e4 at most
    Y = panel(n, k, 1e6, n + k)
    Q, flag = cholqr(Y, passes)
    assert flag == 0
    orth = np.abs(Q.conj().T @ Q - np.eye(k)).max()
    assert orth <= (1e-2 if passes == 2 else 1e-13 * max(1, k / 32)), orth
    Qo, _ = np.linalg.qr(Q)
    resid = np.linalg.norm(Y - Qo @ (Qo.conj().T @ Y)) / np.linalg.norm(Y)
    assert resid <= 1e-12, resid


@pytest.mark.parametrize("n,k", [(1000, 40), (243, 43)])
def test_equals_householder_q(n, k):
    Y = panel(n, k, 1e3, 7 * n + k)
    Q, flag = cholqr(Y, 4)
    assert flag == 0
    Qh, R = np.linalg.qr(Y)
    d = np.diag(R)
    # the 1e-14 perturbation and rounding amplified by the condition number 1e3
    assert np.abs(Q - Qh * (d / np.abs(d))).max() <= 1e-10


def test_rank_deficient_panel():
    n, k = 1200, 60
    rng = np.random.default_rng(3)
    Y = panel(n, 40, 1e4, 11) @ (rng.standard_normal((40, k)) + 1j * rng.standard_normal((40, k)))
    Y[::3] = 0.0  # exactly-zero rows, as zero-padded environment legs give
    Q, flag = cholqr(Y, 4)
    assert flag == 0
    assert np.abs(Q.conj().T @ Q - np.eye(k)).max() <= 1e-12
    assert np.linalg.norm(Y - Q @ (Q.conj().T @ Y)) / np.linalg.norm(Y) <= 1e-12
