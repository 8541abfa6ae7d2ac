"""Host-pointer calls on pageable arrays (staged through pinned pieces of
1 MiB, 16 of them, from 2 MiB on) against the same call on pinned arrays,
which the DMA engine reads directly: equal bit for bit, since only the way of
A to the device differs.  Sizes at the edges of the threshold, of a piece, of
the ring of pieces and of the row chunks of a large A (64 MiB)."""
import threading

import numpy as np
import pytest
import torch

import hiperml_b200 as hml
from hiperml_b200 import datagen as dg
from hiperml_b200._lib import lib

pytestmark = pytest.mark.gpu

MIB = (1 << 20) // 4  # floats


def pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def pageable(a, offset):
    """A copy that starts `offset` floats into its allocation."""
    buf = np.empty(a.size + offset + 16, np.float32)
    out = buf[offset:offset + a.size].reshape(a.shape)
    out[...] = a
    return out


# (M, K) of A: one float below, at and above 2 MiB; a last piece of one row;
# the whole ring, the ring and one row; four chunks with a ragged last one
SHAPES = [(2 * MIB - 1, 1), (2048, 256), (2049, 256), (5 * 1024 + 1, 256), (16384, 256),
          (16385, 256), (16384, 1024), (16411, 1057)]


@pytest.mark.parametrize("offset", [0, 3])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_staged_sgemm_equals_pinned(cuda, shape, offset):
    M, K = shape
    N = 5
    A = dg.matrix(M, K, 121, 0, order="C")
    B = dg.matrix(K, N, 121, 1, order="C")
    C = dg.matrix(M, N, 121, 2, order="C")
    for beta in (0.0, 0.5):
        want, got = pinned(C), C.copy()
        hml.hmlSgemm(want, pinned(A), B, M, N, K, 1.0, beta)
        hml.hmlSgemm(got, pageable(A, offset), B, M, N, K, 1.0, beta)
        assert np.array_equal(got, want)


@pytest.mark.parametrize("shape", [(700, 1000), (4100, 1025)])
def test_staged_sgemv_equals_pinned(cuda, shape):
    M, N = shape
    A = dg.matrix(M, N, 122, 0, order="C")
    x = dg.fill(N, 122, 1)
    want, got = dg.fill(M, 122, 2), dg.fill(M, 122, 2)
    hml.hmlSgemv(want, pinned(A), x, M, N, 1.0, 0.25)
    hml.hmlSgemv(got, pageable(A, 1), x, M, N, 1.0, 0.25)
    assert np.array_equal(got, want)


def test_staged_calls_from_threads_and_after_release(cuda):
    M, N, K = 3000, 4, 700
    A = [dg.matrix(M, K, 123, i, order="C") for i in range(4)]
    B = dg.matrix(K, N, 123, 9, order="C")
    want = []
    for a in A:
        c = np.zeros((M, N), np.float32)
        hml.hmlSgemm(c, pinned(a), B, M, N, K, 1.0, 0.0)
        want.append(c)
    for _ in range(2):
        got = [np.zeros((M, N), np.float32) for _ in A]
        ts = [threading.Thread(target=hml.hmlSgemm, args=(got[i], A[i], B, M, N, K, 1.0, 0.0))
              for i in range(4)]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert all(np.array_equal(g, w) for g, w in zip(got, want))
        assert lib.hml_release_resources() == 0
