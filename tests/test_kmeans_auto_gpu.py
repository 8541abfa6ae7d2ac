"""The automatic k-means form over the shapes the tensor-core kernel takes:
every row alignment, dimensions around its 16- and 32-deep steps, centroid
counts around its accumulator widths (16, 32, 64, 128) and passes, point counts
around its 128-point tiles and the rows-modulo-4 classes, against the C
restatement of the reference kernel (GPU).  Indices must be equal: the screen's
products only decide which points are settled with the reference's own FP32
arithmetic.
"""
import numpy as np
import pytest

import hiperml_b200 as hml
import oracle
from tests.test_kmeans_gpu import clustered, dev

pytestmark = pytest.mark.gpu


def assign(P, C, offset=0):
    """Points stored `offset` floats past a 16-byte boundary."""
    import torch
    n, d = P.shape
    buf = torch.zeros(offset + n * d + 4, device="cuda")
    rows = buf[offset:offset + n * d].view(n, d)
    rows.copy_(dev(P))
    out, exact = hml.kmeans_assign(rows, dev(C), count_exact=True)
    assert hml.device_error() == 0
    return out.cpu().numpy().astype(np.uint32), exact


@pytest.mark.parametrize("d", [1, 2, 3, 15, 17, 30, 32, 33, 63, 65, 96, 99, 128, 129, 250, 256])
@pytest.mark.parametrize("k", [1, 16, 17, 33, 64, 65, 128, 129, 200, 256])
def test_shapes(cuda, d, k):
    rng = np.random.default_rng(1000 * d + k)
    P, C = clustered(rng, 1500 + d % 7, d, k)
    want = oracle.kmeans_assign(P, C)
    for offset in (0, d % 4):
        np.testing.assert_array_equal(assign(P, C, offset)[0], want)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 127, 128, 129, 131, 148 * 128 + 1, 148 * 512 + 77])
def test_point_counts(cuda, n):
    rng = np.random.default_rng(n)
    for d, k, offset in ((8, 20, 0), (8, 20, 1), (7, 70, 0), (100, 50, 0), (70, 90, 3)):
        P, C = clustered(rng, n, d, k)
        np.testing.assert_array_equal(assign(P, C, offset)[0], oracle.kmeans_assign(P, C))


@pytest.mark.parametrize("d,k", [(5, 12), (32, 64), (40, 130), (99, 40), (128, 256)])
def test_close_calls_and_not_finite(cuda, d, k):
    """Duplicated centroids (every point a close call), points far from the
    origin, on bisectors, at the ends of the FP32 range, infinite and NaN."""
    rng = np.random.default_rng(d + k)
    P, C = clustered(rng, 2000, d, k)
    C[k // 2] = C[0]
    C[k - 1] = C[1] * np.float32(1 + 2e-7)
    P[:300] = 0.5 * (C[rng.integers(0, k, 300)] + C[rng.integers(0, k, 300)])
    np.testing.assert_array_equal(assign(P, C)[0], oracle.kmeans_assign(P, C))
    both = assign(P, np.concatenate([C, C])[:256])
    np.testing.assert_array_equal(both[0], oracle.kmeans_assign(P, np.concatenate([C, C])[:256]))
    Q = P + np.float32(1000)
    np.testing.assert_array_equal(assign(Q, C + np.float32(1000))[0],
                                  oracle.kmeans_assign(Q, C + np.float32(1000)))
    R = P.copy()
    R[3] *= np.float32(1e18)
    R[4, 0] = np.inf
    R[5, d - 1] = np.nan
    R[6] = np.float32(3e38)
    R[7] *= np.float32(1e-38)
    R[8] = 0
    np.testing.assert_array_equal(assign(R, C)[0], oracle.kmeans_assign(R, C))
    C[2, 0] = np.nan
    C[3, 0] = np.inf
    C[4] *= np.float32(1e-30)
    np.testing.assert_array_equal(assign(R, C)[0], oracle.kmeans_assign(R, C))
