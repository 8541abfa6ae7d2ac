"""Batch plans made one after another at the same device addresses (GPU): a new
plan's tensor maps lie where an earlier plan's lay, with other operands, layouts
and tile widths, and its first launch must load with the new ones.  Each result
equals, bit for bit, the single-problem kernel's with the configuration that the
batch reports."""
import random

import pytest
import torch

import hiperml_b200 as hml

pytestmark = pytest.mark.gpu


def problems(r, pool, count):
    """Operands anywhere in `pool`, tile widths and layouts in a new order."""
    out = []
    for i in range(count):
        ta, tb = r.randrange(2), r.randrange(2)
        M, N, K = r.choice([130, 300, 700]), r.choice([9, 20, 33, 64, 65, 100, 128, 150]), r.choice([64, 100, 500])
        up = lambda v: (v + 3) // 4 * 4
        lda, ldb = up(K if ta else M), up(N if tb else K)
        a, b = r.randrange(0, 400000, 4), r.randrange(0, 400000, 4)
        C = torch.zeros(N, M, device="cuda")
        out.append((ta, tb, M, N, K, 1.0, pool[a:], lda, pool[b:], ldb, 0.0, C, M))
    return out


def test_plans_in_place_of_others(cuda):
    r = random.Random(5)
    g = torch.Generator(device="cuda").manual_seed(5)
    pool = torch.randn(1 << 20, device="cuda", generator=g)
    for turn in range(60):
        probs = problems(r, pool, 40)
        with hml.BatchPlan(0, probs) as plan:
            plan.graph_launch() if turn % 2 else plan.run()
            torch.cuda.synchronize()
        assert hml.device_error() == 0, turn
        if turn % 6 == 5:
            hml.sgemm_batched(0, problems(r, pool, 40))
        for p in probs:
            want = torch.zeros_like(p[11])
            hml.sgemm_ex(0, *p[:11], want, p[12], config=hml.batch_problem_config(0, p))
            assert torch.equal(p[11], want), (turn, p[:5])
    assert hml.device_error() == 0
