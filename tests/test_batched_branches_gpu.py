"""A batch plan with a SIMT and a tensor-core part, run in each of its ways:
eagerly, as the plan's graph, and inside a capture of the caller's, where both
parts are branches of one stream's capture (GPU).  Before each run the operands
change on the stream and after it C is read on it, so a branch that starts early
or is not waited for shows; results equal the single-problem kernels', bit for
bit.  Plans that live at the same time and one after another take their own
streams.
"""
import pytest
import torch

import hiperml_b200 as hml

pytestmark = pytest.mark.gpu

SHAPES = [(30000, 4, 700), (300, 128, 2000), (5000, 8, 900), (20000, 33, 130), (127, 1, 70)]


class Batch:
    def __init__(self, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
        self.A = [rnd(K, (M + 3) // 4 * 4) for M, N, K in SHAPES]
        self.B = [rnd(N, K) for M, N, K in SHAPES]
        self.B0 = [b.clone() for b in self.B]
        self.C = [torch.zeros(N, M, device="cuda") for M, N, K in SHAPES]
        self.out = [c.clone() for c in self.C]
        self.probs = [(0, 0, M, N, K, 1.5, a, a.shape[1], b, K, 0.0, c, M)
                      for (M, N, K), a, b, c in zip(SHAPES, self.A, self.B, self.C)]
        self.plan = hml.BatchPlan(0, self.probs)

    def step(self, scale, launch):
        for b, b0 in zip(self.B, self.B0):
            torch.mul(b0, scale, out=b)
        launch()
        for o, c in zip(self.out, self.C):
            o.copy_(c)
        for b in self.B:
            b.fill_(float("nan"))

    def check(self, scale):
        for (M, N, K), a, b0, o, prob in zip(SHAPES, self.A, self.B0, self.out, self.probs):
            want = torch.zeros(N, M, device="cuda")
            hml.sgemm_ex(0, 0, 0, M, N, K, 1.5, a, a.shape[1], b0 * scale, K, 0.0, want, M,
                         config=hml.batch_problem_config(0, prob))
            assert torch.equal(o, want), (M, N, K)
        assert hml.device_error() == 0


@pytest.mark.parametrize("way", ["run", "graph", "captured"])
def test_ways(cuda, way):
    b = Batch(1)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for scale in (1.0, -0.5, 2.0):
            if way == "captured":
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s):
                    b.step(scale, b.plan.run)
                for _ in range(3):
                    g.replay()
                s.synchronize()
                del g
            else:
                b.step(scale, b.plan.run if way == "run" else b.plan.graph_launch)
                s.synchronize()
            b.check(scale)
    b.plan.close()


def test_several_plans(cuda):
    """Alive together on streams of their own, and made anew in turn."""
    streams = [torch.cuda.Stream() for _ in range(3)]
    for rnd in range(3):
        bs = [Batch(10 * rnd + i) for i in range(3)]
        torch.cuda.synchronize()
        for scale in (1.0, 3.0):
            for b, s in zip(bs, streams):
                with torch.cuda.stream(s):
                    b.step(scale, b.plan.run)
            torch.cuda.synchronize()
            for b in bs:
                b.check(scale)
        for b in bs:
            b.plan.close()
