// hml_walk.h -- how the threads of a splitting kernel walk B's (n, 8-deep k)
// chunks.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HML_HD __host__ __device__ __forceinline__
#else
#define HML_HD inline
#endif

namespace hml {

// Consecutive threads along B's contiguous dimension, so that whole sectors are
// read.  (Along k always, an N-contiguous 4096 x 128 B took 5.3 us, 4.1 along
// n; the B of 56 uneven problems 22 us, now 16.)  Index: 32 bits where the
// planes of nearly 2^32 chunks are beyond the device's memory (three BF16 planes
// take 206 GB), so that an index and a step after it cannot wrap; 64 for two
// planes (137 GB), divided in 32 bits while they suffice.
template <typename Index>
struct SplitWalk {
  bool nfast;
  uint32_t inner;
  Index chunks;
  HML_HD SplitWalk(int64_t sbk, int64_t sbn, int n_pad, int k_pad)
      : nfast(sbn == 1 && sbk != 1), inner(static_cast<uint32_t>(nfast ? n_pad : k_pad / 8)),
        chunks(static_cast<Index>(n_pad) * static_cast<uint32_t>(k_pad / 8)) {}
  HML_HD void at(Index c, int *n, int *k0) const {
    uint32_t o, i;
    if (sizeof(Index) > 4 && static_cast<uint64_t>(c) >> 32) {
      o = static_cast<uint32_t>(c / inner);
      i = static_cast<uint32_t>(c % inner);
    } else {
      o = static_cast<uint32_t>(c) / inner;
      i = static_cast<uint32_t>(c) - o * inner;
    }
    *n = static_cast<int>(nfast ? i : o);
    *k0 = static_cast<int>(nfast ? o : i) * 8;
  }
};

}  // namespace hml
