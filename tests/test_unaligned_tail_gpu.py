"""An unaligned A a few rows longer than whole waves of 128-row tiles: the last
wave is one tile of 1 to 5 rows, run split in K -- after one whole wave as a grid
of its own, whose four views of A have fewer lines than classes, after more as
the persistent form's tail (GPU).  Against the FP64 oracle on the last rows and
the rows at the tiles' edges (2 gamma_{K+2}, as tests/test_unaligned_gpu.py),
with A ending where its allocation is followed by NaN, and bit for bit equal on
a repeat.
"""
import pytest

import hiperml_b200 as hml
from tests.gpu_util import gamma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("waves", [1, 2, 3])
@pytest.mark.parametrize("rest", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,K", [(45, 513), (20, 1027), (8, 1501)])
def test_tail_of_few_rows(cuda, ta, waves, rest, N, K):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    M = waves * sms * 128 + rest
    lda = (M + 1 if M % 4 == 0 else M) if ta else K     # row-major; A^T is stored K x M
    g = torch.Generator(device="cuda").manual_seed(M + N)
    lines, length = (K, M) if ta else (M, K)
    buf = torch.full((lines * lda + 4 * lda,), float("nan"), device="cuda")
    A = buf[:lines * lda].view(lines, lda)[:, :length]
    A.uniform_(-1, 1, generator=g)
    B = torch.empty(K, N, device="cuda").uniform_(-1, 1, generator=g)
    C0 = torch.empty(M, N, device="cuda").uniform_(-1, 1, generator=g)

    def run():
        C = C0.clone()
        hml.sgemm_ex(hml.ROW_MAJOR, ta, 0, M, N, K, 0.5, buf, lda, B, N, -2.0, C, N)
        return C

    got = run()
    assert torch.equal(got, run()) and hml.device_error() == 0
    rows = torch.cat([torch.arange(0, 130), torch.arange(M - 140, M)]).cuda()
    a = (A[:, rows].t() if ta else A[rows]).double()
    b, c = B.double(), C0[rows].double()
    exact = 0.5 * a @ b - 2.0 * c
    scale = 0.5 * a.abs() @ b.abs() + 2.0 * c.abs()
    err = ((got[rows].double() - exact).abs() / scale).max().item()
    assert err <= 2 * gamma(K + 2), err
    assert torch.isfinite(got).all()
