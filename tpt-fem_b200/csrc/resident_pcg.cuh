// resident_pcg.cuh -- exchanges between the blocks of a resident solve (one
// cooperative launch that runs a whole PCG): values that carry their own
// sequence number, and grid-wide sums built from them.
//
// A fence at gpu scope costs 500-700 cycles on B200 and empties the SM's L1,
// which holds the matrix of a small system.  So nothing here is ordered by
// fences: every exchanged double is stored together with a sequence number as
// one 16-byte access, and a reader repeats its load until it sees the number it
// expects.  A reader therefore never uses a value that is not there yet, in
// whatever order stores arrive, and waits for the values it needs only.
#pragma once
#include "common.cuh"
#include "resident_shape.hpp"

namespace tptfem {

// Repeats of one load before a kernel gives up (about a second): the launch is
// cooperative, so every block is resident and a wait ends in microseconds.
constexpr int RP_POLL_LIMIT = 1 << 21;

struct alignas(16) RpPair {
  double value;
  unsigned long long seq;
};

__device__ __forceinline__ void rp_put(RpPair* p, double value, unsigned long long seq) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
      "l"(__double_as_longlong(value)), "l"(seq));
}
__device__ __forceinline__ void rp_load(const RpPair* p, double& value, unsigned long long& seq) {
  long long v;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
               : "=l"(v), "=l"(seq)
               : "l"(p));
  value = __longlong_as_double(v);
}

// (no "memory" clobbers: pairs are touched by these accesses alone, and what
// surrounds them may move)

// The values p[k][0..N) (STRIDE pairs apart) of sequence seq, k < K, by every lane of a warp, all
// loads in flight together: a line that another SM has just written takes about
// 700 cycles.  (Loops whose lanes part ways are several times slower, so lanes
// without work of their own read valid addresses and drop the values.)  Sets
// `late` when the values do not arrive, and waits no more once it is set.
template <int K, int N, int STRIDE>
__device__ __forceinline__ void rp_get(const RpPair* const (&p)[K], unsigned long long seq, double (&v)[K][N],
                                       int& late) {
  int polls = 0;
  bool pending;
  do {
    pending = false;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        unsigned long long q;
        rp_load(p[k] + i * STRIDE, v[k][i], q);
        pending |= q != seq;
      }
    if (late || ++polls > RP_POLL_LIMIT) {
      late = 1;
      break;
    }
  } while (__any_sync(0xffffffffu, pending));
}

template <int NV>
__device__ __forceinline__ void rp_warp_sum(double (&v)[NV]) {
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
}

// Grid sums of three values.  Every block stores its partial sums to each of
// RP_COPIES tables: 32 bytes, two 16-byte accesses that carry a value, half of the
// third and a 32-bit sequence number each.  Every block's calling warp reads one
// whole table, a 16-byte access a lane so that a warp's are contiguous, and adds it
// in a fixed order (all blocks get the same bits).  One hop through L2, a block's
// values in one sector and a table shared by 37 readers: 2300 cycles for 148
// blocks, against 5200 with one table of 8-value lines and 3300 through a collecting
// block (with four values in 64 bytes a sum took as long as two of these).  Two
// tables by the parity of the sequence: a block stores sequence s + 2 only after it
// has read all of s + 1, which every block stores after reading s.  Tables are
// zeroed before the launch.
constexpr int RP_COPIES = 4, RP_VALUES = 3;
constexpr size_t RP_TABLE = 2 * (size_t)RP_COPIES * RP_MAX_BLOCKS * 2;  // pairs

struct RpGrid {
  RpPair* table;
  unsigned seq;
};

// Called by one warp per block; v: its lanes' parts, then the grid's sums in every lane.
__device__ __forceinline__ bool rp_allsum(RpGrid& g, double (&v)[RP_VALUES]) {
  const int lane = threadIdx.x & 31, nb = gridDim.x;
  rp_warp_sum(v);
  if (nb == 1) return true;
  ++g.seq;
  RpPair* set = g.table + (g.seq & 1) * (RP_TABLE / 2);
  const bool odd = lane & 1;
  if (lane < 2 * RP_COPIES) {
    const unsigned half = odd ? (unsigned)__double2loint(v[2]) : (unsigned)__double2hiint(v[2]);
    rp_put(set + ((size_t)(lane >> 1) * RP_MAX_BLOCKS + blockIdx.x) * 2 + odd, odd ? v[1] : v[0],
           (unsigned long long)half << 32 | g.seq);
  }
  const RpPair* from = set + (size_t)(blockIdx.x % RP_COPIES) * RP_MAX_BLOCKS * 2;
  constexpr int PER = RP_MAX_BLOCKS * 2 / 32;
  const int np = nb * 2;
  double t[PER];
  unsigned h[PER];
  int late = 0, polls = 0;
  bool pending;
  do {
    pending = false;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = k * 32 + lane;
      if (k * 32 < np) {  // uniform
        unsigned long long q;
        rp_load(from + (i < np ? i : odd), t[k], q);
        h[k] = (unsigned)(q >> 32);
        pending |= (unsigned)q != g.seq;
      }
    }
    if (++polls > RP_POLL_LIMIT) {
      late = 1;
      break;
    }
  } while (__any_sync(0xffffffffu, pending));
  double s = 0.0, s2 = 0.0;  // even lanes: values 0 and 2, odd ones: value 1
#pragma unroll
  for (int k = 0; k < PER; ++k)
    if (k * 32 < np) {
      const unsigned lo = __shfl_xor_sync(0xffffffffu, h[k], 1);
      if (k * 32 + lane < np) {
        s += t[k];
        if (!odd) s2 += __hiloint2double((int)h[k], (int)lo);
      }
    }
#pragma unroll
  for (int o = 2; o < 32; o <<= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  v[0] = __shfl_sync(0xffffffffu, s, 0);
  v[1] = __shfl_sync(0xffffffffu, s, 1);
  v[2] = __shfl_sync(0xffffffffu, s2, 0);
  return !__any_sync(0xffffffffu, late);
}

// What a resident solve reports.
struct RpResult {
  double rr;     // true ||b - A x||^2
  double bb;     // ||b||^2
  int iters;
  int outer;     // reliable updates
  int status;    // RP_*
  int pad;
};
enum { RP_CONVERGED = 0, RP_CAP = 1, RP_BREAKDOWN = 2, RP_BAD_DIAGONAL = 3, RP_LATE = 4 };

}  // namespace tptfem
