"""The four TMA views of a matrix whose lines are not 16-byte aligned
(csrc/hml_lines.h), compiled here by the host compiler: every view a kernel
loads from must lie inside the matrix (from the 16-byte granule of a line's
first float on) and start at a line of its class -- also when the matrix has
fewer lines than there are classes, as the split tail of a problem one to three
rows longer than whole waves of tiles has.
"""
import ctypes
import os
import subprocess

import pytest

import hiperml_b200

CSRC = os.path.join(os.path.dirname(hiperml_b200.__file__), "csrc")
SRC = """
#include "hml_lines.h"
extern "C" void view(unsigned long long A, long long ld, unsigned long long lines,
                     unsigned long long len, int r, long long *out) {
  const hml::LineClass c = hml::line_class(reinterpret_cast<const float *>(A), ld, lines, len, r);
  out[0] = reinterpret_cast<long long>(c.base); out[1] = c.skip;
  out[2] = c.lines; out[3] = c.len; out[4] = c.stride;
}
"""


@pytest.fixture(scope="module")
def view(tmp_path_factory):
    d = tmp_path_factory.mktemp("lines")
    (d / "v.cpp").write_text(SRC)
    so = str(d / "v.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "v.cpp"), "-o", so],
                   check=True)
    f = ctypes.CDLL(so).view
    f.argtypes = [ctypes.c_ulonglong, ctypes.c_longlong, ctypes.c_ulonglong, ctypes.c_ulonglong,
                  ctypes.c_int, ctypes.POINTER(ctypes.c_longlong)]

    def call(*a):
        out = (ctypes.c_longlong * 5)()
        f(*a, out)
        return list(out)
    return call


@pytest.mark.parametrize("lines", [1, 2, 3, 4, 5, 7, 8, 129])
@pytest.mark.parametrize("ld,length", [(1, 1), (5, 5), (7, 4), (1501, 1501), (1502, 1501)])
def test_views_stay_inside(view, lines, ld, length):
    for offset in range(4):
        A = (1 << 20) + 4 * offset
        end = A + 4 * ((lines - 1) * ld + length)
        for r in range(4):
            base, skip, n, ln, stride = view(A, ld, lines, length, r)
            first = r if r < lines else 0
            assert base % 16 == 0 and stride % 16 == 0 and 0 <= skip < 4
            assert base + 4 * skip == A + 4 * first * ld and ln == length + skip
            assert n == len(range(first, lines, 4)) >= 1
            assert base >= A // 16 * 16 and base + (n - 1) * stride + 4 * ln <= end
