"""The walk of the splitting kernels over B's chunks (csrc/hml_walk.h), compiled
here by the host compiler: every chunk is visited once, also where there are
2^32 and more of them (16 columns of K near 2^31, 128 of K = 2^28)."""
import ctypes
import os
import subprocess

import pytest

import hiperml_b200

CSRC = os.path.join(os.path.dirname(hiperml_b200.__file__), "csrc")
SRC = """
#include "hml_walk.h"
using u64 = unsigned long long;
using Walk = hml::SplitWalk<uint64_t>;
extern "C" u64 chunks(long long sbk, long long sbn, int n_pad, int k_pad) {
  return Walk(sbk, sbn, n_pad, k_pad).chunks;
}
// in 32 bits
extern "C" void at32(long long sbk, long long sbn, int n_pad, int k_pad, unsigned c, int *out) {
  hml::SplitWalk<uint32_t>(sbk, sbn, n_pad, k_pad).at(c, out, out + 1);
}
extern "C" void at(long long sbk, long long sbn, int n_pad, int k_pad, u64 c, int *out) {
  Walk(sbk, sbn, n_pad, k_pad).at(c, out, out + 1);
}
// steps of a loop as the kernels write it, from `first`
extern "C" u64 steps(long long sbk, long long sbn, int n_pad, int k_pad, u64 first, unsigned step,
                     u64 most) {
  const Walk w(sbk, sbn, n_pad, k_pad);
  u64 n = 0;
  for (uint64_t c = first; c < w.chunks && n < most; c += step) ++n;
  return n;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk")
    (d / "w.cpp").write_text(SRC)
    so = str(d / "w.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "w.cpp"),
                    "-o", so], check=True)
    L = ctypes.CDLL(so)
    ll, i, u = ctypes.c_longlong, ctypes.c_int, ctypes.c_ulonglong
    L.chunks.argtypes, L.chunks.restype = [ll, ll, i, i], u
    L.at.argtypes = [ll, ll, i, i, u, ctypes.POINTER(i)]
    L.at32.argtypes = [ll, ll, i, i, ctypes.c_uint, ctypes.POINTER(i)]
    L.steps.argtypes, L.steps.restype = [ll, ll, i, i, u, ctypes.c_uint, u], u
    return L


@pytest.mark.parametrize("sbk,sbn", [(1, 5000), (40, 1), (1, 1), (3, 7)])
@pytest.mark.parametrize("n_pad,k_pad", [(16, 64), (48, 192), (128, 1088)])
def test_every_chunk_once(lib, sbk, sbn, n_pad, k_pad):
    out = (ctypes.c_int * 2)()
    seen = []
    for c in range(lib.chunks(sbk, sbn, n_pad, k_pad)):
        lib.at(sbk, sbn, n_pad, k_pad, c, out)
        seen.append((out[0], out[1]))
        lib.at32(sbk, sbn, n_pad, k_pad, c, out)
        assert seen[-1] == (out[0], out[1])
    assert sorted(seen) == [(n, k) for n in range(n_pad) for k in range(0, k_pad, 8)]
    if sbn == 1 and sbk != 1:  # consecutive chunks along n
        assert seen[1] == (1, 0)


@pytest.mark.parametrize("n_pad,k_pad", [(16, 2 ** 31 - 64), (128, 2 ** 28), (128, 2 ** 28 + 192)])
def test_many_chunks(lib, n_pad, k_pad):
    total = n_pad * (k_pad // 8)
    step = 4 * 148 * 256
    out = (ctypes.c_int * 2)()
    for sbk, sbn in ((1, 2 ** 28), (2, 1)):
        assert lib.chunks(sbk, sbn, n_pad, k_pad) == total
        for first in (0, step - 1):
            want = len(range(first, total, step))
            assert lib.steps(sbk, sbn, n_pad, k_pad, first, step, want + 5) == want
        for c in (0, 1, 2 ** 31, min(2 ** 32, total - 1), total - 1):
            lib.at(sbk, sbn, n_pad, k_pad, c, out)
            n, k = (c % n_pad, c // n_pad * 8) if sbn == 1 else (c // (k_pad // 8), c % (k_pad // 8) * 8)
            assert (out[0], out[1]) == (n, k)
