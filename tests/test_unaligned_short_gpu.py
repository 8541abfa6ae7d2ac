"""SGEMM of a short, wide problem with an unaligned A, which the tensor-core form
takes in narrow tiles so that its grid fills the device: several column tiles,
their remainders, one wave and a little more of tiles, K below and above 256, whole
and split (GPU).  Against FP64 products, 2 gamma_{K+2} |A||B|."""
import pytest

import hiperml_b200 as hml
from tests.gpu_util import gamma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("M,N,K", [
    (1501, 300, 101), (3257, 104, 127), (1021, 130, 301), (1021, 256, 193), (3257, 300, 255),
    (18945, 65, 101), (18817, 130, 131), (1501, 40, 601), (131, 129, 2001)])
def test_unaligned_short(cuda, ta, M, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N)
    lda = (M + 1 if M % 4 == 0 else M) if ta else K
    A = torch.empty(K if ta else M, lda, device="cuda").uniform_(-1, 1, generator=g)
    B = torch.empty(K, N, device="cuda").uniform_(-1, 1, generator=g)
    C0 = torch.empty(M, N, device="cuda").uniform_(-1, 1, generator=g)
    C = C0.clone()
    hml.sgemm_ex(hml.ROW_MAJOR, ta, 0, M, N, K, 0.5, A, lda, B, N, -2.0, C, N)
    a = (A[:, :M].t() if ta else A).double()
    exact = 0.5 * a @ B.double() - 2.0 * C0.double()
    bound = 2 * gamma(K + 2) * (0.5 * a.abs() @ B.double().abs() + 2.0 * C0.double().abs())
    assert ((C.double() - exact).abs() <= bound).all()
    assert hml.device_error() == 0
