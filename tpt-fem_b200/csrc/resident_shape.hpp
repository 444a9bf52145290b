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
  int w;       // warps per chunk, a power of two (below)
  size_t smem;
};

// Warps per chunk: the block's 16 over its chunks, rounded down to a power of two.
// Microseconds an iteration with 1 / 2 / 4 / 8 / 16 of them (the choice in brackets):
// 2 chunks (9,840 rows, Jacobi) 5.0 / 4.1 / 3.7 / [3.8] / 4.6, (14,520, FSAI) 23.4 / 16.7 /
// 13.7 / [13.1] / 15.4; 3 chunks (37,800, FSAI) 26.9 / 19.5 / [16.0] / 17.8 / 21.0; 8 chunks
// (105,840, FSAI) 35.0 / [27.1] / 28.3 / 32.0 / 43.0; 14 chunks (187,500, Jacobi) [14.3] /
// 15.0 / 15.9 / 16.0 / 19.8; 22 chunks (103,823, Jacobi) [7.5] / 7.7 / 8.9 / 12.8 / 21.3.
//
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
