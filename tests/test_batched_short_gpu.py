"""Plans of short problems in wide tiles, launched many times (GPU): every role of
a tile kernel counts the chunks of the items its CTA takes from records in shared
memory, and with items of one chunk it uses a record as soon as it has read it.
No bounded wait may run out (a miscounted chunk shows as one, 2 s later), and the
results equal the single-problem kernel's, bit for bit.
"""
import random
import time

import pytest
import torch

import hiperml_b200 as hml

pytestmark = pytest.mark.gpu


# (transA, transB, M, N, K): problems of one to four chunks in 128-wide tiles
SHORT = [(0, 1, 7202, 79, 162), (1, 0, 73, 149, 83), (1, 1, 9399, 116, 47), (1, 0, 87, 132, 56),
         (1, 0, 8725, 80, 224), (1, 1, 588, 149, 131), (1, 1, 6401, 78, 253),
         (1, 0, 271, 117, 67), (0, 1, 185, 142, 164), (0, 0, 2335, 137, 41),
         (1, 0, 4662, 138, 144), (1, 0, 4076, 132, 220), (1, 0, 2143, 72, 122),
         (1, 0, 266, 108, 74), (0, 0, 15584, 131, 113)]


def drawn(seed, max_k):
    r = random.Random(100 * seed + max_k)
    return [(r.randrange(2), r.randrange(2), int(round(64 * 256 ** r.random())),
             r.randint(65, 160) if i % 4 else r.randint(9, 64), r.randint(32, max_k))
            for i in range(16)]


@pytest.mark.parametrize("shapes", [SHORT, drawn(1, 64), drawn(2, 256), drawn(3, 700)],
                         ids=["short", "64", "256", "700"])
def test_short_items(cuda, shapes):
    g = torch.Generator(device="cuda").manual_seed(1)
    pool = torch.randn(80 << 20, device="cuda", generator=g)
    up = lambda v: (v + 3) // 4 * 4
    for turn in range(4):
        probs = [(ta, tb, M, N, K, 1.0, pool, up(K if ta else M), pool[4 * i:],
                  up(N if tb else K), 0.0, torch.zeros(N, up(M), device="cuda"), up(M))
                 for i, (ta, tb, M, N, K) in enumerate(shapes)]
        with hml.BatchPlan(0, probs) as plan:
            for _ in range(8):
                t0 = time.time()
                for _ in range(8):
                    plan.run()
                torch.cuda.synchronize()
                assert hml.device_error() == 0 and time.time() - t0 < 1.5, turn
    for p in probs:
        want = torch.zeros_like(p[11])
        hml.sgemm_ex(0, *p[:11], want, p[12], config=hml.batch_problem_config(0, p))
        assert torch.equal(p[11][:, :p[2]], want[:, :p[2]])
