"""k-means assignment where ||x||^2, ||c||^2 or their products leave FP32's range
while the distances themselves do not: points at (or a few ulps from) centroids
of 1e18 to 3e38, beside small ones, every form, against the C restatement of the
reference kernel (GPU).  Indices must be equal.
"""
import numpy as np
import pytest

import hiperml_b200 as hml
import oracle
from tests.test_kmeans_gpu import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", [0, 1, 2, 3])
@pytest.mark.parametrize("d,k", [(1, 4), (4, 3), (32, 64), (7, 20), (64, 130), (100, 50)])
@pytest.mark.parametrize("scale", [1e17, 1.5e19, 1e20, 1e30, 1.2e38])
def test_large_coordinates(cuda, method, d, k, scale):
    if method == 3 and (d % 4 or d > 64):
        pytest.skip("not a shape method 3 takes")
    rng = np.random.default_rng(d * 1000 + k)
    C = rng.uniform(-1, 1, (k, d)).astype(np.float32)
    C[: (k + 1) // 2] *= np.float32(scale)
    which = rng.integers(0, k, 700)
    P = C[which].copy()
    P[200:400] *= np.float32(1 + 2.0 ** -22)
    P[400:500] = P[400:500] + rng.uniform(-1, 1, (100, d)).astype(np.float32)
    P[500:600] = -P[500:600]
    want = oracle.kmeans_assign(P, C)
    assert len(np.unique(want)) > 1
    got = hml.kmeans_assign(dev(P), dev(C), method=method)
    np.testing.assert_array_equal(got.cpu().numpy().astype(np.uint32), want)
    assert hml.device_error() == 0
