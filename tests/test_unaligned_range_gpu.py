"""SGEMM on an A that TMA cannot address, over FP32's whole range: elements down
to the subnormals and products near its ends, which the BF16 planes of the
tensor-core form hold only scaled (GPU).

Tolerance: the classical FP32 bound 2 gamma_{K+2} |A||B|, and per product and
sum the rounding of subnormal values, 2^-149, that FP32 arithmetic itself makes.
A is exact: whole range means nothing is flushed on the way in.
"""
import numpy as np
import pytest

import hiperml_b200 as hml
from tests.gpu_util import gamma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("M,N,K", [(2049, 20, 1501), (517, 45, 9001), (40001, 33, 259)])
@pytest.mark.parametrize("ea,eb", [(-118, 0), (0, -120), (-125, 60), (-140, 100), (-60, -62),
                                   (100, 10), (-110, 110), (120, -118), (59, 56)])
def test_unaligned_range(cuda, ta, M, N, K, ea, eb):
    import torch
    g = torch.Generator(device="cuda").manual_seed(K + ea)
    lda = (M + 1 if M % 4 == 0 else M) if ta else K

    def draw(r, c, e):
        x = torch.empty(r, c, device="cuda").uniform_(-1, 1, generator=g)
        return (x.double() * 2.0 ** e).float()

    A = draw(K, lda, ea)[:, :M] if ta else draw(M, K, ea)
    B = draw(K, N, eb)
    C = torch.empty(M, N, device="cuda")
    hml.sgemm_ex(hml.ROW_MAJOR, ta, 0, M, N, K, 1.0, A, lda, B, N, 0.0, C, N)
    assert hml.device_error() == 0
    a, b = (A.t() if ta else A).double(), B.double()
    exact, scale = a @ b, a.abs() @ b.abs()
    bound = 2 * gamma(K + 2) * scale + (K + 1) * 2.0 ** -149
    inside = scale < np.finfo(np.float32).max  # else partial sums may overflow in FP32 too
    err = (C.double() - exact).abs()
    assert inside.any() and (err <= bound)[inside].all(), (err / bound)[inside].max().item()
