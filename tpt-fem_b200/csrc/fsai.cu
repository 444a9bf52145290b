// fsai.cu -- factorised sparse approximate inverse M^-1 = G^T G of the reduced
// SPD matrix A (Kolotilina-Yeremin FSAI), in the scaled form
//     G = diag(sigma) (I + L),   L strictly lower triangular,
// which is SPD by construction for any sigma > 0 and any L.  sigma^2 is kept in
// FP32 and L in FP16: the preconditioner is the low-precision part of the
// mixed-precision solver (the Krylov recurrences and the operator stay FP64).
//
// Pattern: the lower triangle of the NODE-BLOCK pattern of A -- row i may use
// every free dof j < i of every mesh node coupled to i's node in A (for
// scalar problems, one dof per node, this is tril(A) itself).  The same
// pattern carries the learned factor's values.
//
// Classic values: one thread per row i gathers A[P,P] for P = pattern(i) + {i}
// by merging sorted CSR rows, factors it by Cholesky (packed, local memory)
// and solves A[P,P] y = e_i; then sigma_i^2 = y_i and L_ij = y_j / y_i.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include <climits>

#include "objects.hpp"

namespace tptfem {

namespace {

constexpr int FSAI_MAXM = 48;  // longest pattern row (incl. the diagonal) handled
constexpr int FSAI_NARROW = 24;  // rows of up to this take the narrow form of the node kernel
constexpr int FSAI_NARROW_BLOCKS = 6;  // its blocks to an SM

// Strictly-lower node-block pattern of reduced row i (sorted), COUNT or FILL.
template <bool FILL>
__global__ void nb_lower_pattern(int n, int dpn, const int* __restrict__ rp, const int* __restrict__ ci,
                                 const int* __restrict__ free_map, const int* __restrict__ red_map,
                                 int* __restrict__ cnt, const int* __restrict__ lrp, int* __restrict__ lci,
                                 int* __restrict__ flag) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int node = free_map[i] / dpn;
  int g0 = i, g1 = i + 1;  // rows of the same node are consecutive
  while (g0 > 0 && free_map[g0 - 1] / dpn == node) --g0;
  while (g1 < n && free_map[g1] / dpn == node) ++g1;
  int list[FSAI_MAXM];
  int len = 0;
  bool over = false;
  for (int g = g0; g < g1 && !over; ++g)
    for (int k = rp[g]; k < rp[g + 1] && !over; ++k) {
      const int m = free_map[ci[k]] / dpn;
      for (int c = 0; c < dpn; ++c) {
        const int j = red_map[m * dpn + c];
        if (j < 0 || j >= i) continue;
        int lo = 0, hi = len;
        while (lo < hi) { int mid = (lo + hi) >> 1; if (list[mid] < j) lo = mid + 1; else hi = mid; }
        if (lo < len && list[lo] == j) continue;
        if (len == FSAI_MAXM - 1) { over = true; break; }
        for (int t = len; t > lo; --t) list[t] = list[t - 1];
        list[lo] = j;
        ++len;
      }
    }
  if (over) { atomicOr(flag, 1); len = 0; }
  if (!FILL) {
    cnt[i] = len;
  } else {
    const int o = lrp[i];
    for (int t = 0; t < len; ++t) lci[o + t] = list[t];
  }
}

// The same pattern from the node-group adjacency (sorted neighbour groups of
// each group, the union over its dofs' rows), valid when every free node has
// all its dofs free, so that reduced dof = group * dpn + component: row
// i = g dpn + a holds every component of the neighbour groups J < g, then the
// node's own components c < a.  Same rows, order and overflow rule as
// nb_lower_pattern.
template <bool FILL>
__global__ void nb_lower_from_groups(int n, int dpn, const int* __restrict__ gptr, const int* __restrict__ glist,
                                     int* __restrict__ cnt, const int* __restrict__ lrp, int* __restrict__ lci,
                                     int* __restrict__ flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int g = i / dpn, a = i - g * dpn;
  int nlow = 0;
  for (int k = gptr[g]; k < gptr[g + 1] && glist[k] < g; ++k) ++nlow;
  const int len = nlow * dpn + a;
  if (len >= FSAI_MAXM) {
    atomicOr(flag, 1);
    if (!FILL) cnt[i] = 0;
    return;
  }
  if (!FILL) {
    cnt[i] = len;
  } else {
    int* out = lci + lrp[i];
    for (int k = gptr[g]; k < gptr[g] + nlow; ++k)
      for (int c = 0; c < dpn; ++c) *out++ = glist[k] * dpn + c;
    for (int c = 0; c < a; ++c) *out++ = g * dpn + c;
  }
}

__global__ void col_counts(int64_t nnz, const int* __restrict__ gci, int* __restrict__ cnt) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nnz) atomicAdd(&cnt[gci[k]], 1);
}

// Scatter L's entries into the rows of L^T (unordered), recording L's index.
__global__ void transpose_fill(int n, const int* __restrict__ grp, const int* __restrict__ gci,
                               const int* __restrict__ trp, int* __restrict__ cursor, int* __restrict__ tci,
                               int* __restrict__ perm) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int k = grp[i]; k < grp[i + 1]; ++k) {
    int j = gci[k];
    int pos = trp[j] + atomicAdd(&cursor[j], 1);
    tci[pos] = i;
    perm[pos] = k;
  }
}

// Sort each L^T row by column -> deterministic.  One warp per row: rows of up
// to 64 entries are bitonic-sorted in registers (2 keys per lane); longer rows
// fall back to an insertion sort by one lane.
__global__ void transpose_sort(int n, const int* __restrict__ trp, int* __restrict__ tci, int* __restrict__ perm) {
  const int lane = threadIdx.x & 31;
  const int j = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (j >= n) return;
  const int b = trp[j], e = trp[j + 1], len = e - b;
  if (len <= 1) return;
  if (len > 64) {
    if (lane == 0)
      for (int a = b + 1; a < e; ++a) {
        int c = tci[a], p = perm[a];
        int q = a - 1;
        while (q >= b && tci[q] > c) { tci[q + 1] = tci[q]; perm[q + 1] = perm[q]; --q; }
        tci[q + 1] = c;
        perm[q + 1] = p;
      }
    return;
  }
  int key[2], val[2];
  for (int h = 0; h < 2; ++h) {
    const int t = 2 * lane + h;
    key[h] = t < len ? tci[b + t] : INT_MAX;
    val[h] = t < len ? perm[b + t] : 0;
  }
  for (int k = 2; k <= 64; k <<= 1)
    for (int d = k >> 1; d >= 1; d >>= 1) {
      if (d == 1) {
        const bool asc = ((2 * lane) & k) == 0;
        if (asc ? key[0] > key[1] : key[0] < key[1]) {
          int t = key[0]; key[0] = key[1]; key[1] = t;
          t = val[0]; val[0] = val[1]; val[1] = t;
        }
      } else {
        for (int h = 0; h < 2; ++h) {
          const int el = 2 * lane + h, pe = el ^ d;
          const int pk = __shfl_xor_sync(0xffffffffu, key[h], d >> 1);
          const int pv = __shfl_xor_sync(0xffffffffu, val[h], d >> 1);
          const bool asc = (el & k) == 0;
          const bool take_min = (el < pe) == asc;
          const bool swap = take_min ? pk < key[h] : pk > key[h];
          if (swap) { key[h] = pk; val[h] = pv; }
        }
      }
    }
  for (int h = 0; h < 2; ++h) {
    const int t = 2 * lane + h;
    if (t < len) { tci[b + t] = key[h]; perm[b + t] = val[h]; }
  }
}

// ---- classic FSAI rows, one warp per node -------------------------------------------
//
// Row i: B = A[P,P] with P = (L pattern of i, i), B = L D L^T with unit L, pivots D.
// B^-1 e_m = L^-T e_m / d_m, so sigma_i^2 = 1 / d_m and the row of the factor is
// z = L^-T e_m.  The D rows of a node usually have nested patterns (its lower
// neighbours' dofs, then its own lower dofs), so one factorisation of the last row's
// B, of which the others' are leading parts, serves all; otherwise the warp takes
// them one by one.
//
// A row of B per lane (rows lane and lane + 32 with RPL = 2), in registers.  Step k
// eliminates column k right-looking and moves the window of remaining columns down a
// register, so that the loop stays rolled; the window narrows by 8 columns every 8
// steps.  Column k goes round through shared memory, read two values at a time; the
// reciprocal of the pivot is the only division.  B's entries are found by the whole
// warp along a CSR row (coalesced, branch-free search in P), the next row's in
// flight, and the rows of L are left in shared memory for the back substitutions of
// the D rows together.
//
// A thread per row (one packed triangle of 2 to 9 KB in local memory each) was bound
// by that local memory: 5.2 ms at 806,880 rows of 22 entries; 1.9 now, bound by
// instruction issue (a Cholesky with square roots and divisions: 3.2; five blocks to
// an SM for six: 2.1).
template <int M>
struct FsaiWarp {
  static constexpr int LD = M + 1;  // odd: a lane per row meets no bank twice
  double c[M][LD];
  __align__(16) double col[2][M];
  int P[M];
};

// Steps k in [M - W, M - W + 8) and on to the next narrower window.
template <int M, int W, int RPL>
__device__ __forceinline__ bool fsai_eliminate(FsaiWarp<M>& sh, double (&r)[RPL][M], int m, int lane) {
  constexpr int K0 = M - W;
  const int kend = min(m, K0 + 8);
#pragma unroll 1
  for (int k = K0; k < kend; ++k) {
    double* col = sh.col[k & 1];
#pragma unroll
    for (int h = 0; h < RPL; ++h) {
      const int a = lane + 32 * h;
      if (a > k && a < M) col[a - k - 1] = r[h][0];
    }
    const double piv = RPL == 1 || k < 32 ? __shfl_sync(0xffffffffu, r[0][0], k)
                                          : __shfl_sync(0xffffffffu, r[RPL - 1][0], k - 32);
    if (!(piv > 0.0)) return false;
    const double inv = 1.0 / piv;
    double l[RPL];
#pragma unroll
    for (int h = 0; h < RPL; ++h) {
      const int a = lane + 32 * h;
      l[h] = r[h][0] * inv;
      if (a == k) sh.c[a][a] = inv;
      if (a > k && a < M) sh.c[a][k] = l[h];
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j + 1 < W; j += 2) {
      const double2 x = *reinterpret_cast<const double2*>(col + j);
#pragma unroll
      for (int h = 0; h < RPL; ++h) {
        r[h][j] = r[h][j + 1] - l[h] * x.x;
        if (j + 2 < W) r[h][j + 1] = r[h][j + 2] - l[h] * x.y;
      }
    }
  }
  if constexpr (W > 8) {
    if (kend < m) return fsai_eliminate<M, W - 8, RPL>(sh, r, m, lane);
  }
  return true;
}

// Rows last - NR + 1 .. last, whose patterns are nested (NR <= D).
template <int D, int M, int RPL>
__device__ __forceinline__ void fsai_group(FsaiWarp<M>& sh, int last, int NR, const int* __restrict__ rp,
                                           const int* __restrict__ ci, const double* __restrict__ va,
                                           const int* __restrict__ lrp, const int* __restrict__ lci,
                                           double* __restrict__ sig2, double* __restrict__ lva,
                                           int* __restrict__ flag) {
  constexpr int LD = FsaiWarp<M>::LD;
  const int lane = threadIdx.x & 31, l0 = lrp[last], m = lrp[last + 1] - l0 + 1;
  int r0[RPL], r1[RPL];  // the CSR rows of P
  __syncwarp();          // the previous rows of this warp are done with the shared memory
#pragma unroll
  for (int h = 0; h < RPL; ++h) {
    const int a = lane + 32 * h;
    r0[h] = r1[h] = 0;
    if (a < m) {
      const int v = a < m - 1 ? lci[l0 + a] : last;
      sh.P[a] = v;
      r0[h] = rp[v];
      r1[h] = rp[v + 1];
    }
  }
  for (int t = lane; t < m * LD; t += 32) (&sh.c[0][0])[t] = 0.0;
  for (int t = lane; t < 2 * M; t += 32) (&sh.col[0][0])[t] = 0.0;
  __syncwarp();
  auto range = [&](int a, int& b, int& e) {
    b = RPL == 1 || a < 32 ? __shfl_sync(0xffffffffu, r0[0], a & 31) : __shfl_sync(0xffffffffu, r0[RPL - 1], a & 31);
    e = RPL == 1 || a < 32 ? __shfl_sync(0xffffffffu, r1[0], a & 31) : __shfl_sync(0xffffffffu, r1[RPL - 1], a & 31);
  };
  int kb, ke;
  range(0, kb, ke);
  int c = kb + lane < ke ? ci[kb + lane] : INT_MAX;
  double v = kb + lane < ke ? va[kb + lane] : 0.0;
  for (int a = 0; a < m; ++a) {
    int nb = 0, ne = 0, cn = INT_MAX;
    double vn = 0.0;
    if (a + 1 < m) {  // the next row's first entries, in flight
      range(a + 1, nb, ne);
      if (nb + lane < ne) {
        cn = ci[nb + lane];
        vn = va[nb + lane];
      }
    }
    const int own = sh.P[a];
    for (int k = kb;;) {
      if (c <= own) {
        int lo = 0;  // the last position whose column is at most c
#pragma unroll
        for (int step = RPL == 1 ? 16 : 32; step > 0; step >>= 1)
          if (lo + step <= a && sh.P[lo + step] <= c) lo += step;
        if (sh.P[lo] == c) sh.c[a][lo] = v;
      }
      k += 32;
      // on while the row has more entries and may have more columns up to its own
      if (k >= ke || __shfl_sync(0xffffffffu, c, 31) > own) break;
      c = k + lane < ke ? ci[k + lane] : INT_MAX;
      v = k + lane < ke ? va[k + lane] : 0.0;
    }
    kb = nb;
    ke = ne;
    c = cn;
    v = vn;
  }
  __syncwarp();
  double r[RPL][M];
#pragma unroll
  for (int h = 0; h < RPL; ++h)
#pragma unroll
    for (int j = 0; j < M; ++j) {
      const int a = lane + 32 * h;
      r[h][j] = a < m && j <= a ? sh.c[a < M ? a : 0][j] : 0.0;
    }
  __syncwarp();
  if (!fsai_eliminate<M, M, RPL>(sh, r, m, lane)) {
    if (lane == 0) atomicOr(flag, 2);
    return;
  }
  __syncwarp();
  // z = L^-T e of row last - q: sigma^2 is the inverse of its last pivot, L its z
  double z[RPL][D];
#pragma unroll
  for (int h = 0; h < RPL; ++h)
#pragma unroll
    for (int q = 0; q < D; ++q) z[h][q] = lane + 32 * h == m - 1 - q ? 1.0 : 0.0;
  for (int t = m - 1; t > 0; --t) {
    double lt[RPL];
#pragma unroll
    for (int h = 0; h < RPL; ++h) lt[h] = lane + 32 * h < t ? sh.c[t][lane + 32 * h] : 0.0;
#pragma unroll
    for (int q = 0; q < D; ++q) {
      const double zt = RPL == 1 || t < 32 ? __shfl_sync(0xffffffffu, z[0][q], t & 31)
                                           : __shfl_sync(0xffffffffu, z[RPL - 1][q], t & 31);
#pragma unroll
      for (int h = 0; h < RPL; ++h) z[h][q] -= lt[h] * zt;
    }
  }
#pragma unroll
  for (int q = 0; q < D; ++q) {
    if (q >= NR) break;
    const int i = last - q, at = m - 1 - q, o = lrp[i];
    const double d = sh.c[at][at];
    if (!(d > 0.0) || !isfinite(d)) {
      if (lane == 0) atomicOr(flag, 2);
      continue;
    }
#pragma unroll
    for (int h = 0; h < RPL; ++h) {
      const int a = lane + 32 * h;
      if (a == at) sig2[i] = d;
      else if (a < at) lva[o + a] = z[h][q];
    }
  }
}

// The last row of every node, by the length of its B: up to 24 entries in the first
// list, longer ones in the second (each a count, then rows).
__global__ void fsai_last_rows(int n, int dpn, const int* __restrict__ free_map, const int* __restrict__ lrp,
                               int* __restrict__ narrow, int* __restrict__ wide) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < n && (i == n - 1 || free_map[i] / dpn != free_map[i + 1] / dpn);
  const int len = on ? lrp[i + 1] - lrp[i] + 1 : 0;
  const unsigned lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  const unsigned m = __ballot_sync(0xffffffffu, on && len <= FSAI_NARROW);
  int at = 0;
  if (lane == 0 && m) at = atomicAdd(narrow, __popc(m));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (on && len <= FSAI_NARROW) narrow[1 + at + __popc(m & below)] = i;
  if (on && len > FSAI_NARROW) wide[1 + atomicAdd(wide, 1)] = i;
}

template <int D, int M, int RPL>
__global__ void __launch_bounds__(128, M == FSAI_NARROW ? FSAI_NARROW_BLOCKS : 2) fsai_nodes(int dpn, const int* __restrict__ free_map, const int* __restrict__ rp,
                                                  const int* __restrict__ ci, const double* __restrict__ va,
                                                  const int* __restrict__ lrp, const int* __restrict__ lci,
                                                  double* __restrict__ sig2, double* __restrict__ lva,
                                                  int* __restrict__ flag, const int* __restrict__ rows) {
  extern __shared__ __align__(16) unsigned char fsai_smem[];
  FsaiWarp<M>& sh = reinterpret_cast<FsaiWarp<M>*>(fsai_smem)[threadIdx.x / 32];
  const int lane = threadIdx.x & 31, count = rows[0], stride = gridDim.x * (blockDim.x / 32);
  for (int w = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < count; w += stride) {
    const int last = rows[1 + w], ll = lrp[last], nl = lrp[last + 1] - ll;
    // the node's rows; nested: row last - q has the last row's first nl - q
    // entries, of which the rest are the node's rows from last - q on
    int nr = 1;
    while (nr < D && nr <= last && free_map[last - nr] / dpn == free_map[last] / dpn) ++nr;
    bool nested = nl >= nr - 1;
    for (int q = 1; q < nr; ++q) {
      const int o = lrp[last - q], len = lrp[last - q + 1] - o;
      nested = nested && len == nl - q;
      if (nested)
        for (int t = lane; t < len; t += 32) nested = nested && lci[o + t] == lci[ll + t];
      nested = nested && lci[ll + nl - q] == last - q;
      nested = __all_sync(0xffffffffu, nested);
    }
    for (int i = nested ? last : last - nr + 1; i <= last; ++i)
      fsai_group<D, M, RPL>(sh, i, nested ? nr : 1, rp, ci, va, lrp, lci, sig2, lva, flag);
  }
}

// The same with one thread per row, for short rows: Cholesky, y = B^-1 e_m.
__global__ void fsai_rows(int n, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ va,
                          const int* __restrict__ lrp, const int* __restrict__ lci, double* __restrict__ sig2,
                          double* __restrict__ lva, int* __restrict__ flag) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int l0 = lrp[i], m = lrp[i + 1] - l0 + 1;
  double B[FSAI_MAXM * (FSAI_MAXM + 1) / 2];  // packed lower triangle, row-major
  int P[FSAI_MAXM];
  for (int a = 0; a < m - 1; ++a) P[a] = lci[l0 + a];
  P[m - 1] = i;
  for (int a = 0; a < m; ++a) {
    const int r = P[a];
    int k = rp[r], b = 0;
    const int ke = rp[r + 1];
    double* row = B + a * (a + 1) / 2;
    for (int t = 0; t <= a; ++t) row[t] = 0.0;
    while (k < ke && b <= a) {
      const int c = ci[k];
      if (c == P[b]) { row[b] = va[k]; ++k; ++b; }
      else if (c < P[b]) ++k;
      else ++b;
    }
  }
  for (int a = 0; a < m; ++a) {
    double* ra = B + a * (a + 1) / 2;
    for (int b = 0; b <= a; ++b) {
      const double* rb = B + b * (b + 1) / 2;
      double s = ra[b];
      for (int t = 0; t < b; ++t) s -= ra[t] * rb[t];
      if (b == a) {
        if (!(s > 0.0)) { atomicOr(flag, 2); return; }
        ra[a] = sqrt(s);
      } else {
        ra[b] = s / rb[b];
      }
    }
  }
  double y[FSAI_MAXM];
  for (int a = 0; a < m; ++a) y[a] = 0.0;
  y[m - 1] = 1.0 / B[(m - 1) * m / 2 + (m - 1)];
  for (int a = m - 1; a >= 0; --a) {
    double s = y[a];
    for (int t = a + 1; t < m; ++t) s -= B[t * (t + 1) / 2 + a] * y[t];
    y[a] = s / B[a * (a + 1) / 2 + a];
  }
  const double d = y[m - 1];
  if (!(d > 0.0) || !isfinite(d)) { atomicOr(flag, 2); return; }
  sig2[i] = d;
  for (int a = 0; a < m - 1; ++a) lva[l0 + a] = y[a] / d;
}

__global__ void factor_to_lowp(int n, int64_t nnz, const double* __restrict__ sig2, const double* __restrict__ lva,
                               const int* __restrict__ perm, float* __restrict__ s32, __half* __restrict__ va16,
                               __half* __restrict__ tva16, int* __restrict__ flag) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) {
    const double s = sig2[k];
    if (!(s > 0.0) || !isfinite(s)) atomicOr(flag, 4);
    s32[k] = (float)s;
  }
  if (k < nnz) {
    const double v = lva[k];
    if (!isfinite(v) || fabs(v) > 6.0e4) atomicOr(flag, 4);  // outside FP16 range
    va16[k] = __double2half(v);
    if (perm) tva16[k] = __double2half(lva[perm[k]]);
  }
}

// Values of the explicit transpose from the FP16 factor: tva[k] = va[perm[k]].
__global__ void transpose_values(int64_t nnz, const int* __restrict__ perm, const __half* __restrict__ va,
                                 __half* __restrict__ tva) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nnz) tva[k] = va[perm[k]];
}

void launch_fsai_nodes(const SystemData& S, FsaiFactor& F, double* sig2, double* lva) {
  cudaStream_t s = S.ctx->stream;
  const int n = (int)F.n;
  if (!F.rows_listed) {  // once per pattern
    F.narrow.alloc((size_t)n + 1, s);
    F.wide.alloc((size_t)n + 1, s);
    TPT_CUDA(cudaMemsetAsync(F.narrow.p, 0, sizeof(int), s));
    TPT_CUDA(cudaMemsetAsync(F.wide.p, 0, sizeof(int), s));
    fsai_last_rows<<<ceil_div(n, 256), 256, 0, s>>>(n, S.dpn, S.free_map.p, F.rp.p, F.narrow.p, F.wide.p);
    TPT_CHECK_LAUNCH();
    F.rows_listed = true;
  }
  auto run = [&](auto kernel, size_t per_warp, int per_sm, const int* rows) {
    const size_t bytes = 4 * per_warp;
    allow_smem((const void*)kernel, bytes);  // (one size per kernel)
    kernel<<<std::min(ceil_div(n, 4), per_sm * sm_count()), 128, bytes, s>>>(
        S.dpn, S.free_map.p, S.row_ptr.p, S.col.p, S.val.p, F.rp.p, F.ci.p, sig2, lva, S.ctx->d_flag, rows);
    TPT_CHECK_LAUNCH();
  };
  run(fsai_nodes<3, FSAI_NARROW, 1>, sizeof(FsaiWarp<FSAI_NARROW>), FSAI_NARROW_BLOCKS, F.narrow.p);
  run(fsai_nodes<3, FSAI_MAXM, 2>, sizeof(FsaiWarp<FSAI_MAXM>), 2, F.wide.p);
}

}  // namespace

void fsai_build_pattern(const SystemData& S, FsaiFactor& F) {
  if (F.ready_pattern) return;
  cudaStream_t s = S.ctx->stream;
  const int n = (int)S.n_free;
  F.n = n;
  DevBuf<int> cnt;
  cnt.alloc(n + 1, s);
  TPT_CUDA(cudaMemsetAsync(S.ctx->d_flag, 0, sizeof(int), s));
  // from the node-group adjacency when the node-block operator exists (one pass
  // over each group's neighbour list instead of a sorted union per row)
  const bool groups = S.nb.state == 1 && S.nb.dpn == S.dpn;
  if (groups)
    nb_lower_from_groups<false><<<ceil_div(n, 256), 256, 0, s>>>(n, S.dpn, S.nb.gptr.p, S.nb.glist.p, cnt.p, nullptr,
                                                                 nullptr, S.ctx->d_flag);
  else
    nb_lower_pattern<false><<<ceil_div(n, 128), 128, 0, s>>>(n, S.dpn, S.row_ptr.p, S.col.p, S.free_map.p,
                                                              S.red_map.p, cnt.p, nullptr, nullptr, S.ctx->d_flag);
  TPT_CHECK_LAUNCH();
  F.rp.alloc(n + 1, s);
  F.nnz = exclusive_scan_i32(cnt.p, F.rp.p, n, s);
  int flag = 0;
  TPT_CUDA(cudaMemcpyAsync(&flag, S.ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, s));
  TPT_CUDA(cudaStreamSynchronize(s));
  F.overflow = flag != 0;
  F.ci.alloc(F.nnz, s);
  if (groups)
    nb_lower_from_groups<true><<<ceil_div(n, 256), 256, 0, s>>>(n, S.dpn, S.nb.gptr.p, S.nb.glist.p, nullptr, F.rp.p,
                                                                F.ci.p, S.ctx->d_flag);
  else
    nb_lower_pattern<true><<<ceil_div(n, 128), 128, 0, s>>>(n, S.dpn, S.row_ptr.p, S.col.p, S.free_map.p,
                                                             S.red_map.p, nullptr, F.rp.p, F.ci.p, S.ctx->d_flag);
  TPT_CHECK_LAUNCH();
  F.sigma2.alloc(n, s);
  F.va.alloc(F.nnz, s);
  F.ready_pattern = true;
}

void fsai_build_transpose(const SystemData& S, FsaiFactor& F) {
  if (F.transposed || !F.ready_pattern) return;
  cudaStream_t s = S.ctx->stream;
  const int n = (int)F.n;
  DevBuf<int> cnt;
  cnt.alloc(n + 1, s);
  cnt.zero();
  col_counts<<<ceil_div(std::max<int64_t>(F.nnz, 1), 256), 256, 0, s>>>(F.nnz, F.ci.p, cnt.p);
  TPT_CHECK_LAUNCH();
  F.trp.alloc(n + 1, s);
  exclusive_scan_i32(cnt.p, F.trp.p, n, s);
  F.tci.alloc(F.nnz, s);
  F.perm.alloc(F.nnz, s);
  cnt.zero();
  transpose_fill<<<ceil_div(n, 256), 256, 0, s>>>(n, F.rp.p, F.ci.p, F.trp.p, cnt.p, F.tci.p, F.perm.p);
  TPT_CHECK_LAUNCH();
  transpose_sort<<<ceil_div((int64_t)n * 32, 256), 256, 0, s>>>(n, F.trp.p, F.tci.p, F.perm.p);
  TPT_CHECK_LAUNCH();
  F.tva.alloc(F.nnz, s);
  if (F.values_set && F.nnz) {
    transpose_values<<<ceil_div(F.nnz, 256), 256, 0, s>>>(F.nnz, F.perm.p, F.va.p, F.tva.p);
    TPT_CHECK_LAUNCH();
  }
  F.transposed = true;
}

bool fsai_set_values(const SystemData& S, FsaiFactor& F, const double* d_sig2, const double* d_lva) {
  cudaStream_t s = S.ctx->stream;
  TPT_CUDA(cudaMemsetAsync(S.ctx->d_flag, 0, sizeof(int), s));
  const int64_t m = std::max<int64_t>(F.n, F.nnz);
  factor_to_lowp<<<ceil_div(std::max<int64_t>(m, 1), 256), 256, 0, s>>>(
      (int)F.n, F.nnz, d_sig2, d_lva, F.transposed ? F.perm.p : nullptr, F.sigma2.p, F.va.p,
      F.transposed ? F.tva.p : nullptr, S.ctx->d_flag);
  TPT_CHECK_LAUNCH();
  F.values_set = true;
  int flag = 0;
  TPT_CUDA(cudaMemcpyAsync(&flag, S.ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, s));
  TPT_CUDA(cudaStreamSynchronize(s));
  return flag == 0;
}

bool fsai_classic(const SystemData& S, FsaiFactor& F) {
  fsai_build_pattern(S, F);
  if (F.overflow) return false;
  cudaStream_t s = S.ctx->stream;
  DevBuf<double> sig2, lva;
  sig2.alloc(F.n, s);
  lva.alloc(std::max<int64_t>(F.nnz, 1), s);
  TPT_CUDA(cudaMemsetAsync(S.ctx->d_flag, 0, sizeof(int), s));
  // Rows of 22 entries and more (3 dofs per node) pay for a warp: one of 806,880 rows
  // 5.2 -> 1.9 ms, with rollers on one face 5.0 -> 2.0.  The short rows of 1 and 2 dofs
  // per node (4.5 and 9 entries) do not: 0.41 ms a thread each, 3.6 a warp each at
  // 2.1M rows of Poisson, 0.82 and 2.05 at 1M rows of plane stress.
  if (S.dpn == 3) {
    launch_fsai_nodes(S, F, sig2.p, lva.p);
  } else {
    fsai_rows<<<ceil_div(F.n, 128), 128, 0, s>>>((int)F.n, S.row_ptr.p, S.col.p, S.val.p, F.rp.p, F.ci.p, sig2.p,
                                                 lva.p, S.ctx->d_flag);
    TPT_CHECK_LAUNCH();
  }
  int flag = 0;
  TPT_CUDA(cudaMemcpyAsync(&flag, S.ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, s));
  TPT_CUDA(cudaStreamSynchronize(s));
  if (flag) return false;
  return fsai_set_values(S, F, sig2.p, lva.p);
}

}  // namespace tptfem
