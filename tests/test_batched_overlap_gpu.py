"""Batches whose tile widths run at the same time (GPU): long tiles in the
wide class, short ones in the narrow, so that the later kernels finish first.
B changes on the stream before each run and C is copied on it right after, so
a run that ended before all of its kernels, or read B's planes before they
were complete, shows.  Each result equals, bit for bit, the single-problem
kernel's with the configuration that the batch reports."""
import pytest
import torch

import hiperml_b200 as hml

pytestmark = pytest.mark.gpu

# (M, N, K): a few tiles of K = 4096, many of K <= 130, the edges of a tile
WIDTHS = {128: [(300, 128, 4096), (1025, 65, 130)], 64: [(20000, 64, 100), (129, 33, 2000)],
          32: [(30000, 32, 64), (127, 9, 70)]}


@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("widths", [(128, 64, 32), (128, 32), (64, 32), (64,)],
                         ids=lambda w: "+".join(map(str, w)))
def test_widths_together(cuda, widths, beta):
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    probs, Bs, Cs, C0 = [], [], [], []
    for w in widths:
        for M, N, K in WIDTHS[w]:
            ld = (M + 3) // 4 * 4
            A, B, C = rnd(K, ld), rnd(N, K), rnd(N, M)
            probs.append((0, 0, M, N, K, 1.5, A, ld, B, K, beta, C, M))
            Bs.append(B)
            Cs.append(C)
            C0.append(C.clone())
    want = {}
    for sign in (1, -1):
        want[sign] = []
        for p, c0 in zip(probs, C0):
            out = c0.clone()
            hml.sgemm_ex(0, *p[:11], out, p[12], config=hml.batch_problem_config(0, p))
            want[sign].append(out)
        for B in Bs:
            B.neg_()
    snaps = []
    with hml.BatchPlan(0, probs) as plan:
        for i in range(12):
            for C, c0 in zip(Cs, C0):
                C.copy_(c0)
            plan.graph_launch() if i % 3 == 2 else plan.run()
            snaps.append([C.clone() for C in Cs])
            for B in Bs:
                B.neg_()
        torch.cuda.synchronize()
    for i, snap in enumerate(snaps):
        for got, w in zip(snap, want[1 if i % 2 == 0 else -1]):
            assert torch.equal(got, w)
    assert hml.device_error() == 0
