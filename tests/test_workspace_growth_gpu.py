"""Workspaces of the tensor-core path and CUDA graphs (GPU): after one call of the
largest shape on a stream, no smaller one may move a buffer that a captured
graph uses or need an allocation inside a capture -- although a smaller problem
can have a split last wave where the larger one has none.  And a call on an A
that TMA cannot address, which the SIMT tiles serve without a workspace, can be
captured by a stream that made no call before.
"""
import pytest

import hiperml_b200 as hml
from hiperml_b200._lib import lib
from tests.gpu_util import gamma

pytestmark = pytest.mark.gpu
N, K = 32, 1024


def operands(M, N, K, order="col"):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.empty(*((K, M) if order == "col" else (M, K)), device="cuda").uniform_(-1, 1, generator=g)
    B = torch.empty(*((N, K) if order == "col" else (K, N)), device="cuda").uniform_(-1, 1, generator=g)
    return A, B


def call(M, A, B, C):
    hml.sgemm_ex(0, 0, 0, M, N, K, 1.0, A, M, B, K, 0.0, C, M)


@pytest.fixture
def sizes(cuda):
    """Rows of four whole waves, and of three and a tail that is split in K."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lib.hml_release_resources()
    yield 4 * sms * 128, (3 * sms + sms * 68 // 148) * 128
    lib.hml_release_resources()


def capture(stream, f, n=1):
    import torch
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        for _ in range(n):
            f()
    return g


def test_smaller_call_after_a_capture(sizes):
    import torch
    big, small = sizes
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        A, B = operands(big, N, K)
        a, b = operands(small, N, K)
        C, c = torch.zeros(N, big, device="cuda"), torch.zeros(N, small, device="cuda")
        call(big, A, B, C)
        want = C.clone()
        g = capture(s, lambda: call(big, A, B, C))
        held = torch.cuda.mem_get_info()[0]
        call(small, a, b, c)
        s.synchronize()
        assert torch.cuda.mem_get_info()[0] == held  # nothing moved
        C.zero_()
        g.replay()
        assert torch.equal(C, want)
        s.synchronize()
        del g
    assert hml.device_error() == 0


def test_smaller_call_in_a_capture(sizes):
    import torch
    big, small = sizes
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(other):
        a, b = operands(small, N, K)
        c = torch.zeros(N, small, device="cuda")
        call(small, a, b, c)
        want = c.clone()
        other.synchronize()
    with torch.cuda.stream(s):
        A, B = operands(big, N, K)
        C = torch.zeros(N, big, device="cuda")
        call(big, A, B, C)
        c.zero_()
        g = capture(s, lambda: call(small, a, b, c), 2)
        for _ in range(3):
            c.zero_()
            g.replay()
            assert torch.equal(c, want)
        s.synchronize()
        del g
    assert hml.device_error() == 0


def test_tail_without_its_buffer(sizes):
    """Planes held from an explicit call, no tail buffer: captured as grids, the
    same bits."""
    import torch
    _, small = sizes
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    a, b = operands(small, N, K)
    c = torch.zeros(N, small, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        call(small, a, b, c)
        want = c.clone()
        other.synchronize()
    with torch.cuda.stream(s):
        hml.sgemm_ex(0, 0, 0, small, N, K, 1.0, a, small, b, K, 0.0, c, small,
                     config=hml.SgemmConfig(hml.ALGO_BF16X6, 128, 32, 1, 6, 1))
        g = capture(s, lambda: call(small, a, b, c))
        c.zero_()
        g.replay()
        assert torch.equal(c, want)
        s.synchronize()
        del g
    assert hml.device_error() == 0


@pytest.mark.parametrize("M,N,K", [(2049, 20, 1501), (20011, 45, 701)])
def test_unaligned_call_captured_first(sizes, M, N, K):
    import torch
    A, B = operands(M, N, K, "row")
    C = torch.zeros(M, N, device="cuda")
    hml.sgemm(A, B)  # on another stream: the device's own set-up
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    lib.hml_release_resources()
    with torch.cuda.stream(s):
        g = capture(s, lambda: hml.sgemm_ex(1, 0, 0, M, N, K, 1.0, A, K, B, N, 0.0, C, N))
        g.replay()
        s.synchronize()
        del g
    exact = A.double() @ B.double()
    bound = 2 * gamma(K + 2) * (A.double().abs() @ B.double().abs())
    assert ((C.double() - exact).abs() <= bound).all()
    assert hml.device_error() == 0
