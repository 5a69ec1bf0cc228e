"""CholeskyQR panels on both sides of the width (48 columns) where a warp's share
of the Gram blocks changes, real and complex, one 8-column block fewer and more."""
import ctypes as C

import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200._lib import check, dptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("k", [40, 41, 47, 48, 49, 56])
def test_orthonormal_and_same_span(k, is_complex):
    n = 333
    rng = np.random.default_rng(k)
    rand = lambda *s: rng.standard_normal(s) + (1j * rng.standard_normal(s) if is_complex else 0.0)  # noqa: E731
    U, V = np.linalg.qr(rand(n, k))[0], np.linalg.qr(rand(k, k))[0]
    Y = (U * np.logspace(0, -6, k)) @ V.conj().T
    flag = C.c_int(0)
    buf = np.ascontiguousarray(Y.T)  # column-major n x k = row-major k x n
    f = _lib.load().tg_cholqr_host_complex if is_complex else _lib.load().tg_cholqr_host
    check(f(n, k, dptr(buf), 4, C.byref(flag)))
    Q = buf.T
    assert flag.value == 0
    # orthonormal to rounding; the span to the 1e-14 perturbation, both as in the panels' own tests
    assert np.abs(Q.conj().T @ Q - np.eye(k)).max() <= 1e-13 * k / 32
    assert np.linalg.norm(Y - Q @ (Q.conj().T @ Y)) / np.linalg.norm(Y) <= 1e-12
