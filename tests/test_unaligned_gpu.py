"""SGEMM on an A that TMA cannot address as it stands (odd leading dimensions,
shifted bases): the tensor-core form hml_sgemm_ex routes it to, against the
FP64 oracle (GPU).

Tolerance: the FP32 bound every FP32-accurate form is held to, componentwise
2 gamma_{K+2} and normwise 2e-6 (tests/test_tc_gpu.py).  The shapes lie above
the size from which the form is taken, or have it chosen by N > 16 and
M >= 1024, and cover: every residue of the leading dimension and of the base
modulo 4 floats, both orders of A, all tile widths and their remainders, a
last row tile of 1 row, a K of one block more or less than the 64-deep chunk,
split K, and more row tiles than SMs (the partial last wave).
"""
import numpy as np
import pytest

import hiperml_b200 as hml
import oracle
from hiperml_b200 import datagen as dg
from tests.gpu_util import gamma
from tests.test_sgemm_gpu import fetch, store

pytestmark = pytest.mark.gpu


def run(M, N, K, order, ta, pad, offset, alpha=0.5, beta=0.0, edit=None):
    import torch
    A = dg.matrix(K if ta else M, M if ta else K, 3, 0, dg.UNIFORM, order="C")
    B = dg.matrix(K, N, 3, 1, dg.UNIFORM, order="C")
    C = dg.matrix(M, N, 3, 2, dg.UNIFORM, order="C")
    if edit:
        edit(A, B)
    Ab, Ap, lda = store(A, order, pad, offset)
    Bb, Bp, ldb = store(B, order, 0, 0)
    Cb, Cp, ldc = store(C, order, 0, 0)
    hml.sgemm_ex(order, ta, 0, M, N, K, alpha, Ap, lda, Bp, ldb, beta, Cp, ldc)
    torch.cuda.synchronize()
    assert hml.device_error() == 0
    return fetch(Cb, 0, order, ldc, M, N), A, B, C


def check(got, A, B, C, ta, alpha, beta, what):
    K = B.shape[0]
    D, absD = oracle.dgemm(A, B, C, alpha, beta, transA=bool(ta), transB=False, with_abs=True)
    e = oracle.rel_errors(got, D, absD)
    assert e["normwise"] <= 2e-6 and e["compwise"] <= 2 * gamma(K + 2), (what, e)


@pytest.mark.parametrize("order,ta", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad", [0, 1, 2, 3])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_unaligned_residues(cuda, order, ta, pad, offset):
    for M, N, K in ((2177, 45, 385), (4225, 7, 1033)):
        got, A, B, C = run(M, N, K, order, ta, pad, offset, beta=-2.0)
        check(got, A, B, C, ta, 0.5, -2.0, (order, ta, pad, offset, M, N, K))


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("M,N,K", [
    (1025, 17, 511), (1025, 32, 513), (1151, 64, 575), (1153, 65, 577), (2049, 128, 641),
    (1500, 129, 321), (300, 20, 9001), (40001, 33, 259), (20011, 16, 1027)])
def test_unaligned_tiles(cuda, ta, M, N, K):
    got, A, B, C = run(M, N, K, 0, ta, 1 if (K if ta else M) % 4 == 0 else 0, 0)
    check(got, A, B, C, ta, 0.5, 0.0, (ta, M, N, K))


@pytest.mark.parametrize("ta", [0, 1])
# whole K, split K, several waves of tiles
@pytest.mark.parametrize("M,N,K", [(3001, 45, 701), (517, 20, 9001), (40001, 20, 301)])
def test_unaligned_not_finite(cuda, ta, M, N, K):
    """Infinities, NaN and the largest finite values give what plain FP32
    products give (their BF16 residuals alone would give NaN)."""
    big = np.finfo(np.float32).max

    def edit(A, B):
        At = A.T if ta else A
        At[5, 17] = np.inf
        At[131, 0] = -np.inf
        At[M - 1, K - 1] = np.nan
        At[260, 33] = big
        B[64, 3] = np.inf
        B[K - 1, N - 1] = big

    got, A, B, C = run(M, N, K, 0, ta, 1 if (K if ta else M) % 4 == 0 else 0, 0, alpha=1.0,
                       edit=edit)
    At = (A.T if ta else A).astype(np.float64)
    with np.errstate(invalid="ignore", over="ignore"):
        exact = At @ B.astype(np.float64)
    odd = ~np.isfinite(exact)
    assert odd[5].all() and odd[131].all() and odd[M - 1].all() and odd[:, 3].all()
    np.testing.assert_array_equal(np.isnan(got[odd]), np.isnan(exact[odd]))
    np.testing.assert_array_equal(got[odd & ~np.isnan(exact)], exact[odd & ~np.isnan(exact)])
    fine = ~odd
    bound = 2 * gamma(K + 2) * (np.abs(At[:, :]).clip(max=3.4e38) @ np.abs(B.astype(np.float64)))
    inside = fine & (np.abs(exact) < 0.5 * big)
    assert (np.abs(got - exact)[inside] <= bound[inside] + 1e-37).all()
