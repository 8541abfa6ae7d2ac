"""What hml_sgemm_ex runs where a predicted configuration is brought to the
tile that holds N (GPU): a rigged network that always prefers one
configuration stands in for a wrong prediction; the rule's edges are N at and
one past half of a tile, and row tiles at half a wave, one wave and two waves.
A SIMT choice stays as it is."""
import numpy as np
import pytest
import torch

import hiperml_b200 as hml
from hiperml_b200 import predictor as pr
from tests.gpu_util import assert_within_fp32_bound

pytestmark = pytest.mark.gpu

SIMT8, X64, X128, X64S2 = ((1, 128, 8), 4), ((3, 128, 64), 1), ((3, 128, 128), 1), ((3, 128, 64), 2)


def rig(path, want):
    """A network whose scores are its last biases: 0 for `want`, else 1."""
    (algo, tm, tn), split = want
    cfgs = hml.configs()
    n = pr.n_params(len(cfgs))
    params = np.zeros(n)
    pick = [i for i, c in enumerate(cfgs)
            if (c.algo, c.tile_m, c.tile_n, c.split_k) == (algo, tm, tn, split)]
    params[n - len(cfgs):] = 1.0
    params[[n - len(cfgs) + i for i in pick]] = 0.0
    with open(path, "w") as f:
        f.write("#HML-B200 predictor v1\ninputs 5 hidden 64 64 outputs %d\n" % len(cfgs))
        for c in cfgs:
            f.write("config " + " ".join(str(x) for x in c.as_tuple()) + "\n")
        f.write("params %d\n" % n + " ".join(f"{x:.9g}" for x in params) + "\n")
    pr.load(str(path))


# predicted, M in row tiles of the SM count's fractions, N, K, (algo, tile_n, split) run
CASES = [(X128, 0.3, 64, 300, (3, 64, 1)), (X128, 0.3, 65, 300, (3, 128, 1)),
         (X128, 3.4, 16, 300, (3, 16, 1)), (X64, 0.5, 80, 300, (3, 64, 1)),
         (X64, 0.51, 80, 300, (3, 128, 1)), (X64, 1.0, 128, 300, (3, 128, 1)),
         (X64, 1.01, 128, 300, (3, 64, 1)), (X64, 2.0, 100, 300, (3, 128, 1)),
         (X64S2, 1.5, 64, 640, (3, 64, 2)), (X64S2, 2.0, 64, 640, (3, 64, 1)),
         (SIMT8, 0.6, 9, 300, (1, 8, 4)), (SIMT8, 2.0, 64, 300, (1, 8, 4))]


@pytest.mark.parametrize("want,part,N,K,run", CASES,
                         ids=[f"{c[0][0][2]}-{c[1]}-{c[2]}-{c[3]}" for c in CASES])
def test_fit_tile(cuda, tmp_path, want, part, N, K, run):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = int(part * sms) + (0 if float(part * sms).is_integer() else 1)
    M = 128 * tiles - (0 if float(part).is_integer() or part == 0.5 else 4)
    hml.tune_clear()
    try:
        rig(tmp_path / "m.txt", want)
        c = hml.select(0, 0, 0, M, N, K)
        assert (c.algo, c.tile_n, c.split_k) == run
        g = torch.Generator(device="cuda").manual_seed(3)
        A = torch.randn(K, M, device="cuda", generator=g)
        B = torch.randn(N, K, device="cuda", generator=g)
        C = torch.full((N, M), float("nan"), device="cuda")
        hml.sgemm_ex(0, 0, 0, M, N, K, 1.0, A, M, B, K, 0.0, C, M)
        exact = (B.double() @ A.double()).cpu().numpy()
        bound = (B.double().abs() @ A.double().abs()).cpu().numpy()
        assert_within_fp32_bound(C.cpu().numpy(), exact, bound, K)
    finally:
        pr.clear()
