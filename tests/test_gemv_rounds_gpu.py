"""The row GEMV's last, partial round of loads: row lengths around every
remainder of a thread's round (4 float4 groups when rows are 16-byte aligned,
6 elements when not), for each number of threads per row.  Elements past a
row's end are NaN (the padding of A, the elements after x), so a load that is
not masked shows.  The bound is the suite's FP32 dot-product bound against the
float64 oracle."""
import numpy as np
import pytest
import torch

import hiperml_b200 as hml
from hiperml_b200 import datagen as dg
from tests.gpu_util import assert_within_fp32_bound

pytestmark = pytest.mark.gpu


def lengths(tpr, vec):
    per = 4 if vec else 1            # elements of one load
    rnd = 4 if vec else 6            # loads of a whole round
    out = set()
    for whole in (0, 1, 2):
        for rest in range(rnd):
            n = (whole * rnd + rest) * tpr * per
            out |= {n + d * per for d in (-1, 0, 1)}
    return sorted(n for n in out if n > 0)


@pytest.mark.parametrize("vec", [True, False], ids=["vectors", "elements"])
@pytest.mark.parametrize("tpr", [4, 32, 64, 256])
def test_gemv_rows_last_round(cuda, tpr, vec):
    M = 2 * (256 // tpr) + 1
    for Q in lengths(tpr, vec):
        ld = Q + (4 if vec else 3 + Q % 2)
        A = dg.matrix(M, Q, 111, 0, dg.NORMAL, order="C")
        x = dg.fill(Q, 111, 1)
        buf = torch.full((M * ld + 8,), float("nan"), dtype=torch.float32, device="cuda")
        off = 0 if vec else 1
        buf[off:off + M * ld].view(M, ld)[:, :Q] = torch.from_numpy(np.ascontiguousarray(A)).cuda()
        xv = torch.full((Q + 300,), float("nan"), dtype=torch.float32, device="cuda")
        xv[:Q] = torch.from_numpy(x).cuda()
        y = torch.full((M,), float("nan"), dtype=torch.float32, device="cuda")
        hml.sgemv_ex(hml.ROW_MAJOR, hml.OP_N, M, Q, 1.0, buf.data_ptr() + 4 * off, ld,
                     xv, 0.0, y, variant=tpr)
        A64, x64 = A.astype(np.float64), x.astype(np.float64)
        assert_within_fp32_bound(y.cpu().numpy(), A64 @ x64, np.abs(A64) @ np.abs(x64), Q,
                                 what=f"tpr{tpr} Q{Q}")
