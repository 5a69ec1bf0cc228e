"""The FP64 products on small tiles (tile_gemm.cu) against numpy: edges of
tiles and K stages, K split over a cluster or into partial buffers, every
layout, conjugation.  An FP64 sum of K products is within K u of its terms'
absolute sum."""
import numpy as np
import pytest

from tenes_b200 import _lib
from tenes_b200._lib import check, dptr

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (5, 3, 2), (16, 16, 32), (17, 25, 33), (33, 17, 31), (47, 31, 65), (40, 40, 40), (100, 50, 128),
          (243, 37, 243), (512, 42, 512), (64, 64, 4097), (7, 300, 1000), (48, 48, 1200), (17, 2000, 97),
          # one long side, the others at most 8: a row a thread (skinny.cu)
          (2048, 1, 1), (2500, 2, 2), (3, 5000, 8), (4097, 8, 5), (4, 70001, 3)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("is_complex", [False, True])
def test_products_match_numpy(M, N, K, is_complex):
    rng = np.random.default_rng(M + 3 * N + 7 * K)

    def matrix(r, c):
        x = rng.standard_normal((r, c))
        return x + 1j * rng.standard_normal((r, c)) if is_complex else x

    A, B = matrix(M, K), matrix(K, N)
    bound = (np.abs(A) @ np.abs(B)) * 4 * (K + 4) * 2.0 ** -53
    for q, (la, lb, lc) in enumerate((a, b, c) for a in "rc" for b in "rc" for c in "rc"):
        a, b = (x if l == "r" else np.ascontiguousarray(x.T) for x, l in ((A, la), (B, lb)))
        c = np.full((M, N) if lc == "r" else (N, M), np.nan, dtype=A.dtype)
        strides = [((K, 1) if la == "r" else (1, M)), ((N, 1) if lb == "r" else (1, K)), ((N, 1) if lc == "r" else (1, M))]
        args = (M, N, K, dptr(a), *strides[0], dptr(b), *strides[1], dptr(c), *strides[2])
        ca, cb = (q & 1, q >> 1 & 1) if is_complex else (0, 0)
        if is_complex:
            check(_lib.load().tg_gemm_host_complex(*args, ca, cb))
        else:
            check(_lib.load().tg_gemm_host(*args, 0))
        ref = (A.conj() if ca else A) @ (B.conj() if cb else B)
        assert np.all(np.abs((c if lc == "r" else c.T) - ref) <= bound), (la, lb, lc)
