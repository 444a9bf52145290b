// resident_shape.hpp -- how a resident solve of a node-block system is laid out over the
// SMs (plain C++: resident_pcg.cu, and a test on the host).
#pragma once
#include <stddef.h>

namespace tptfem {

constexpr int RP_THREADS = 512;
constexpr int RP_MAX_BLOCKS = 160;  // a multiple of 32
// Dynamic shared memory of a block: 227 KB less a kilobyte for what is static.
constexpr size_t RN_MAX_SMEM = 226 * 1024;

struct RnShape {
  int nc;      // chunks of 32 node groups per block
  int blocks;  // one per SM at most: they wait for one another
  int w;       // warps per chunk, a power of two: 16 warps over the chunks that a block has
  size_t smem;
};

// na, nm, nseg: aggregates, modes and segments of the coarse space (na 0: none).
inline RnShape rn_shape(int nchunks, int dpn, int sms, int na, int nm, int nseg) {
  const int most = sms < RP_MAX_BLOCKS ? sms : RP_MAX_BLOCKS;
  RnShape s{};
  s.nc = (nchunks + most - 1) / most;
  s.blocks = (nchunks + s.nc - 1) / s.nc;
  s.w = s.nc == 1 ? 16 : s.nc == 2 ? 8 : s.nc <= 4 ? 4 : s.nc <= 8 ? 2 : 1;
  const size_t rows = (size_t)s.nc * 32 * dpn;
  s.smem = (6 * rows + (size_t)s.nc * s.w * dpn * 32) * sizeof(double);
  if (na)
    s.smem += (((size_t)na + nseg) * nm + (size_t)RP_THREADS * nm) * sizeof(double) +
              ((size_t)na * 2 + nseg + (size_t)s.nc * 32) * sizeof(int);
  return s;
}

}  // namespace tptfem
