"""Which configuration hml_sgemm_ex runs a product with an unaligned A with (GPU):
a record that the program tuned or loaded for the shape stands, and one
selection -- one inference of the predictor at most -- settles whether the
tensor cores or the SIMT tiles take it.
"""
import os

import pytest

import hiperml_b200 as hml
from hiperml_b200 import predictor as pr
from hiperml_b200._lib import lib
from tests.test_fit_tile_gpu import SIMT8, X64, rig

pytestmark = pytest.mark.gpu


def operands(M, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M)
    A = torch.empty(M, K, device="cuda").uniform_(-1, 1, generator=g)
    B = torch.empty(K, N, device="cuda").uniform_(-1, 1, generator=g)
    return A, B, torch.empty(M, N, device="cuda")


def call(A, B, C, config=None):
    (M, K), N = A.shape, B.shape[1]
    hml.sgemm_ex(1, 0, 0, M, N, K, 1.0, A, K, B, N, 0.0, C, N, config=config)
    return C.clone()


@pytest.mark.parametrize("M,N,K", [(20011, 45, 1501), (2049, 20, 701)])
def test_own_record_stands(cuda, tmp_path, M, N, K):
    import torch
    A, B, C = operands(M, N, K)
    cfg = hml.SgemmConfig(hml.ALGO_SIMT, 128, 32, 2, 3, 2)
    want, other = call(A, B, C, cfg), call(A, B, C)
    assert not torch.equal(want, other)  # the tensor cores' without the record
    f = tmp_path / "tuned.txt"
    f.write_text("#HML-B200 tuning v2\n1 0 %d %d %d : %s 1.0\n"
                 % (M, N, K, " ".join(str(v) for v in cfg.as_tuple())))
    try:
        hml.tune_clear()
        assert hml.tune_load(str(f)) == 1
        assert torch.equal(call(A, B, C), want)
    finally:
        hml.tune_clear()
    assert torch.equal(call(A, B, C), other)
    assert hml.device_error() == 0


@pytest.mark.parametrize("want,M,N,K", [(SIMT8, 300, 15, 77), (SIMT8, 900, 9, 257), (X64, 901, 9, 257),
                                        (SIMT8, 20011, 45, 1501)])
def test_one_inference(cuda, tmp_path, want, M, N, K):
    """Kernels launched by the first call beyond those of the next: one
    inference's, as for an aligned A of a size near by."""
    import torch

    def extra(K):
        A, B, C = operands(M, N, K)
        n = [lib.hml_launch_count()]
        for _ in range(2):
            call(A, B, C)
            n.append(lib.hml_launch_count())
        return n[1] - n[0] - (n[2] - n[1])

    hml.tune_clear()
    try:
        rig(tmp_path / "m.txt", want)
        one = extra(K // 4 * 4)
        assert one > 0
        assert extra(K) == one
    finally:
        pr.clear()
