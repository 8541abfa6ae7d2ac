"""An explicitly given split-precision configuration runs with the ring depth it
names: its kernel's shared memory follows the depth, 16 KB a slot (GPU).  The
results of all depths are equal, bit for bit."""
import json

import pytest

import hiperml_b200 as hml

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [hml.ALGO_BF16X6, hml.ALGO_BF16X3, hml.ALGO_TF32X3,
                                  hml.ALGO_FP16X3])
@pytest.mark.parametrize("ta", [0, 1])
def test_depth_as_given(cuda, tmp_path, algo, ta):
    import torch
    from torch.profiler import ProfilerActivity, profile
    M, N, K = 3000, 32, 1000
    g = torch.Generator(device="cuda").manual_seed(algo)
    A = torch.empty(M * K, device="cuda").uniform_(-1, 1, generator=g)
    B = torch.empty(N * K, device="cuda").uniform_(-1, 1, generator=g)
    out = {}

    def run(stages):
        C = torch.zeros(N, M, device="cuda")
        hml.sgemm_ex(0, ta, 0, M, N, K, 1.0, A, K if ta else M, B, K, 0.0, C, M,
                     config=hml.SgemmConfig(algo, 128, N, 1, stages, 1))
        return C

    for stages in (2, 4, 6):
        out[stages] = run(stages)
        torch.cuda.synchronize()
    assert torch.equal(out[2], out[4]) and torch.equal(out[4], out[6])
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for stages in (2, 4, 6):
            run(stages)
        torch.cuda.synchronize()
    f = tmp_path / "trace.json"
    prof.export_chrome_trace(str(f))
    smem = [e["args"]["shared memory"] for e in json.loads(f.read_text())["traceEvents"]
            if e.get("cat") == "kernel" and "tc_kernel" in e["name"]]
    assert len(smem) == 3
    slot = 16 * 1024
    # (barriers, and alignment, beside the slots)
    assert 2 * slot <= smem[1] - smem[0] <= 2 * slot + 256
    assert 2 * slot <= smem[2] - smem[1] <= 2 * slot + 256
