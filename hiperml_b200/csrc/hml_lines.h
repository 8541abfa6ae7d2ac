// hml_lines.h -- how TMA reads a dense FP32 matrix whose lines (rows or
// columns, ld floats apart) do not start on 16-byte boundaries: lines 4 j + r
// lie 4 ld floats apart, a multiple of 16 bytes, so each class r = 0..3 is a
// view of its own from the 16-byte boundary at or before its first line.
#pragma once

#include <cstdint>

namespace hml {

struct LineClass {
  const float *base;  // 16-byte aligned
  int skip;           // floats from there to the line's first
  uint64_t lines, len;
  int64_t stride;  // bytes
};

// Class r of `lines` lines of `len` floats.  A class without a line (fewer
// than four lines in all) takes class 0's view: its loads, which the kernels
// issue all the same, then stay inside the matrix, and what they bring belongs
// to rows that are not stored.
inline LineClass line_class(const float *A, int64_t ld, uint64_t lines, uint64_t len, int r) {
  const uint64_t first = static_cast<uint64_t>(r) < lines ? r : 0;
  const float *p = A + static_cast<int64_t>(first) * ld;
  const int skip = static_cast<int>((reinterpret_cast<uintptr_t>(p) & 15u) / 4);
  return LineClass{p - skip, skip, (lines - first + 3) / 4, len + skip, ld * 16};
}

}  // namespace hml
