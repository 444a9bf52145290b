// resident_pcg.cu -- PCG of small systems in one launch.
//
// The engine of solver.cu spends three to nine kernels an iteration; below a
// hundred thousand rows each of them lasts little longer than a launch and the
// whole system lies in L2, so an iteration is bound by launch gaps and by the
// serial chain of a row's loads.  Here one cooperative grid keeps the whole
// solve, the reliable updates (compensated true residual, see solver.cu)
// included: the host waits once and no graph is captured.  Same method, same
// stopping rules; every sum has a fixed order, so results repeat bit for bit.
//
// Microseconds an iteration on B200, engine -> here (whole solve / iterations):
//   Jacobi  343 rows 19 -> 3.6, 2-D Quad4 9,840 rows 15 -> 3.8,
//           13,872 rows (16^3 elasticity) 22 -> 4.4, 104,544 23 -> 9.2, 345,744 43 -> 27;
//           103,823 rows (48^3 Poisson) 17 -> 7.4, 250,047 22 -> 14
//   FSAI + coarse space  14,520 rows (40x10x10) 44 -> 12, 37,800 43 -> 15, 105,840 47 -> 26;
//           29,791 rows (32^3 Poisson) 33 -> 9.6, 103,823 37 -> 18
// An iteration is bound by its exchanges (a grid sum at about 2,300 cycles, and
// about 700 cycles for each vector that other SMs have just written), until the
// matrix outgrows what the SMs' L1 and then L2 hold; the size limits in
// objects.hpp lie where the engine, which streams it better, catches up (FSAI at
// 202,800 rows: 38 us there).
//
// A node-block iteration has one grid sum, not two: K is applied to z = M r instead
// of p, r.z, r.r and z.Kz are summed together, and K p = K z + beta K p' and
// p.Kp = z.Kz - beta^2 p'.Kp' follow (Chronopoulos and Gear's form of CG).  After a
// reliable update, where r is not the recurrence's, z.Kp' is summed as well, and
// where p.Kp comes out not positive K is applied to p itself before that counts as a
// breakdown (solves past FP64's accuracy otherwise ended in one).  With
// two sums: 9,840 rows 5.1 us, 104,544 rows 10.9, FSAI at 14,520 rows 14.3; the same
// iterations to the solution.
//
// A cooperative grid begins when all its SMs are free at once.  Beside another stream's
// ordinary kernels that costs little (103,823 rows beside 8192^3 GEMMs: 2.8 ms a solve,
// 38 with the engine's kernels), but a kernel that holds an SM for seconds holds up a
// solve of as many blocks as there are SMs; TPTFEM_SOLVE_FULL_OPERATOR selects the engine.
#include <algorithm>
#include <cmath>

#include "modes.cuh"
#include "nbblock.cuh"
#include "objects.hpp"
#include "resident_pcg.cuh"

namespace tptfem {

namespace {

constexpr int RN_WARPS = RP_THREADS / 32;

// b as the true residual of x = 0: an infinite entry is a NaN there (inf - inf in the
// compensated sum), which ends the solve as a breakdown, where the sums of squares would
// take infinity for converged.
__device__ __forceinline__ double residual_of_zero(double b) { return b + (b - b); }

// ---- Jacobi-PCG of a system that one block holds ----------------------------------------
// LANES lanes share a row of the CSR matrix (L1-resident), the vectors lie in
// shared memory: an iteration is three block barriers.
constexpr int RJ_THREADS = 512;
constexpr size_t RJ_MAX_SMEM = 6 * (RJ_MAX_LANES / 4) * sizeof(double);  // four lanes a row at least

struct RjArgs {
  int n;
  const int* rp;
  const int* ci;
  const double* va;
  const double* b;
  double* x;
  RpResult* res;
  double tol, delta;
  int max_it;
};

template <int NV>
__device__ __forceinline__ void rj_sum(double (&v)[NV], double (*sh)[RJ_THREADS / 32 + 1]) {
  constexpr int NW = RJ_THREADS / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  rp_warp_sum(v);
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NV; ++i) sh[i][wid] = v[i];
  __syncthreads();
  if (wid == 0) {  // one warp: shuffles of every warp would queue
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = lane < NW ? sh[i][lane] : 0.0;
    rp_warp_sum(v);
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < NV; ++i) sh[i][NW] = v[i];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = sh[i][NW];
}

template <int LANES>
__global__ void __launch_bounds__(RJ_THREADS, 1) resident_jacobi(RjArgs A) {
  extern __shared__ double dyn[];
  __shared__ double sh[3][RJ_THREADS / 32 + 1];
  const int n = A.n;
  double* xl = dyn;  // step since the last update, r, p, q, 1 / diagonal, x
  double* r = xl + n;
  double* p = r + n;
  double* q = p + n;
  double* dinv = q + n;
  double* x = dinv + n;
  const int t = threadIdx.x, sub = t / LANES, lane = t & (LANES - 1);
  constexpr int RPB = RJ_THREADS / LANES;
  RpResult out{};
  double v[3] = {0.0, 0.0, 0.0};
  for (int i = t; i < n; i += RJ_THREADS) {
    double d = 0.0;
    for (int k = A.rp[i]; k < A.rp[i + 1]; ++k)
      if (__ldg(A.ci + k) == i) d = __ldg(A.va + k);
    if (!(d > 0.0)) v[2] += 1.0;
    const double di = 1.0 / d, bi = residual_of_zero(A.b[i]);
    dinv[i] = di;
    r[i] = bi;
    p[i] = di * bi;
    xl[i] = 0.0;
    x[i] = 0.0;
    v[0] += bi * bi;
    v[1] += bi * (di * bi);
  }
  rj_sum(v, sh);
  double rr = v[0], rz = v[1], rz_old = 0.0;
  const double bnorm = sqrt(v[0]);
  const double target2 = A.tol * A.tol * bnorm * bnorm, final2 = 0.25 * target2;
  out.bb = v[0];
  out.status = v[2] != 0.0 ? RP_BAD_DIAGONAL : RP_CONVERGED;
  bool run = out.status == RP_CONVERGED && out.bb != 0.0 && !(rr <= target2);
  while (run) {
    const double upd2 = fmax(A.delta * A.delta * rr, final2);
    int done = 0;
    while (!done) {
      __syncthreads();  // p
      double w[1] = {0.0};
      for (int i0 = 0; i0 < n; i0 += RPB) {
        const int i = i0 + sub;
        double s = 0.0;
        if (i < n) {
          const int e = __ldg(A.rp + i + 1);
          for (int k = __ldg(A.rp + i) + lane; k < e; k += LANES) s += __ldg(A.va + k) * p[__ldg(A.ci + k)];
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
        if (i < n && lane == 0) {
          q[i] = s;
          w[0] += p[i] * s;
        }
      }
      rj_sum(w, sh);
      if (!(w[0] > 0.0)) { out.status = RP_BREAKDOWN; break; }
      const double alpha = rz / w[0];
      double u[2] = {0.0, 0.0};
      for (int i = t; i < n; i += RJ_THREADS) {
        xl[i] += alpha * p[i];
        const double ri = r[i] - alpha * q[i];
        r[i] = ri;
        u[0] += ri * (dinv[i] * ri);
        u[1] += ri * ri;
      }
      rj_sum(u, sh);
      rz_old = rz;
      const double beta = u[0] / rz;
      rz = u[0];
      out.iters += 1;
      if (!(u[1] == u[1]) || !(u[0] == u[0])) { out.status = RP_BREAKDOWN; break; }
      if (u[1] <= upd2) done = 4;
      else if (out.iters >= A.max_it) done = 3;
      else
        for (int i = t; i < n; i += RJ_THREADS) p[i] = dinv[i] * r[i] + beta * p[i];
    }
    if (!done) break;  // breakdown
    // reliable update: x += xl, r = b - A x (compensated)
    for (int i = t; i < n; i += RJ_THREADS) {
      x[i] += xl[i];
      xl[i] = 0.0;
    }
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += RPB) {
      const int i = i0 + sub;
      double hi = 0.0, lo = 0.0;
      if (i < n) {
        const int e = __ldg(A.rp + i + 1);
        for (int k = __ldg(A.rp + i) + lane; k < e; k += LANES) {
          double pr, pe, s, se;
          two_prod(__ldg(A.va + k), x[__ldg(A.ci + k)], pr, pe);
          two_sum(hi, pr, s, se);
          hi = s;
          lo += pe + se;
        }
      }
#pragma unroll
      for (int o = LANES / 2; o > 0; o >>= 1) {
        const double oh = __shfl_down_sync(0xffffffffu, hi, o, LANES);
        const double ol = __shfl_down_sync(0xffffffffu, lo, o, LANES);
        double s, se;
        two_sum(hi, oh, s, se);
        hi = s;
        lo += ol + se;
      }
      if (i < n && lane == 0) {
        double r1, e1;
        two_sum(A.b[i], -hi, r1, e1);
        r[i] = r1 + (e1 - lo);
      }
    }
    __syncthreads();
    double u[2] = {0.0, 0.0};
    for (int i = t; i < n; i += RJ_THREADS) {
      u[0] += r[i] * (dinv[i] * r[i]);
      u[1] += r[i] * r[i];
    }
    rj_sum(u, sh);
    rr = u[1];
    out.outer += 1;
    if (rr <= target2) break;
    if (done == 3) { out.status = RP_CAP; break; }
    const double beta = u[0] / rz_old;
    rz = u[0];
    for (int i = t; i < n; i += RJ_THREADS) p[i] = dinv[i] * r[i] + beta * p[i];
  }
  out.rr = rr;
  for (int i = t; i < n; i += RJ_THREADS) A.x[i] = x[i];
  if (t == 0) *A.res = out;
}

// ---- node-block systems: Jacobi or FSAI (with the coarse space) -----------------------
//
// A block owns NC chunks of 32 node groups; W warps share a chunk's slots
// (lower and transposed upper blocks of the symmetric storage, nbsell.cuh), so
// a row's load chain is short and every load is coalesced; their partial rows
// meet in shared memory and one thread per row finishes them.  The FSAI halves
// work the same way on the packed factor.  The vectors that other blocks gather
// (z; r and t = G r; the coarse restriction) are exchanged as pairs with their
// sequence numbers, laid out [chunk][component][lane] so that a warp's 16-byte
// accesses are contiguous; the only grid-wide wait of an iteration is its sum of
// r.z, r.r and z.Kz.  With the test on r.r beside z.Kz the preconditioner and K are
// applied once more than needed at the end of a segment.  The restriction
// moments of a segment of groups are summed by one block; every block then forms
// P^T r and applies its own aggregates' rows of A_c^-1 itself.  Nothing fences,
// so a block's part of the matrix stays in L1 while it fits.
constexpr int RN_MAX_COARSE = 256;
constexpr int RN_MAX_SEG = 512;
constexpr int RN_BATCH = 2;  // slots (or groups of an aggregate) whose vector entries are loaded together

struct RnArgs {
  int ngroups, nchunks, nc, w;  // nc: chunks per block, w: warps per chunk (a power of two)
  const int *lcptr, *lcol, *ucptr, *ucol, *ubase;
  const double *lval, *dval;
  const uint4 *lpack, *upack;
  const __half *ltail, *utail, *ldiag;
  const float* sigma2;
  const int *rp, *ci;  // CSR of K: true residuals
  const double *va, *b;
  double* x;
  RpPair *xp, *zp, *r, *t, *sm;  // zeroed before the launch, like the table
  // coarse space (na 0: none)
  int na, ld, nseg;
  const int *agg, *aseg, *sbeg, *send, *alist;
  const float *y, *Ainv;
  const double* T;
  double* M;  // per block: its aggregates' rows of T A_c^-1 T^T (at most na nm rows of na nm)
  RpPair* table;
  RpResult* res;
  double tol, delta;
  int max_it;
};

template <int DPN, bool FSAI>
__global__ void __launch_bounds__(RP_THREADS, 1) resident_nb(RnArgs A) {
  constexpr int D2 = DPN * DPN, NM = rigid_modes(DPN), CR = 32 * DPN;
  using Seq = unsigned long long;
  extern __shared__ double dyn[];
  __shared__ double sh[RP_VALUES][RN_WARPS];
  __shared__ double s_val[RP_VALUES];
  __shared__ int s_na;
  RpGrid g{A.table, 0};
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int c0 = blockIdx.x * A.nc, ncl = min(A.nchunks, c0 + A.nc) - c0;
  const int W = A.w, rows = A.nc * CR;
  const int g0 = c0 * 32, ngl = min(A.ngroups, (c0 + ncl) * 32) - g0;  // own groups
  const int mrows = ncl * CR;                                          // own rows, padded
  const int64_t o0 = (int64_t)c0 * CR;                                 // the first one's place in a pair vector
  // own rows i = (chunk DPN + component) 32 + lane
  double* xl = dyn;
  double* r = xl + rows;
  double* p = r + rows;
  double* z = p + rows;
  double* e = z + rows;     // 1 / diagonal (Jacobi) or the own part of t (FSAI)
  double* kp = e + rows;    // K p
  double* part = kp + rows;  // [chunk][w][component][lane]
  double* smo = part + A.nc * W * CR;
  double* cm = smo + A.nseg * NM;
  double* mom = cm + A.na * NM;                            // [mode][thread]
  int* aidx = reinterpret_cast<int*>(mom + RP_THREADS * NM);  // aggregate -> place in the block's list, or -1
  int* alst = aidx + A.na;
  int* sagg = alst + A.na;  // segment -> aggregate
  int* gidx = sagg + A.nseg;  // own group -> place of its aggregate
  RpResult out{};
  int late = 0;
  // place of component b of group J in a pair vector
  auto at = [](int J, int b) { return (int64_t)(J >> 5) * CR + b * 32 + (J & 31); };
  // the own row i: group within the block, component; false for padding
  auto row_of = [&](int i, int& gl, int& a) {
    gl = i / CR * 32 + lane;
    a = (i >> 5) % DPN;
    return gl < ngl;
  };
  // grid sums of every thread's values, for the whole block
  auto grid_sum = [&](double (&v)[RP_VALUES]) {
    if (wid * 32 < mrows) {
      rp_warp_sum(v);
#pragma unroll
      for (int k = 0; k < RP_VALUES; ++k)
        if (lane == 0) sh[k][wid] = v[k];
    }
    __syncthreads();
    if (wid == 0) {
      const bool on = lane < RN_WARPS && lane * 32 < mrows;
#pragma unroll
      for (int k = 0; k < RP_VALUES; ++k) v[k] = on ? sh[k][lane] : 0.0;
      if (!rp_allsum(g, v)) late = 1;
#pragma unroll
      for (int k = 0; k < RP_VALUES; ++k)
        if (lane == 0) s_val[k] = v[k];
    }
    late = __syncthreads_or(late);
#pragma unroll
    for (int k = 0; k < RP_VALUES; ++k) v[k] = s_val[k];
  };
  // sum of the W partial rows of own row i
  auto gathered = [&](int i) {
    const double* q = part + i / CR * W * CR + i % CR;
    if (W == 1) return q[0];
    double s0 = q[0], s1 = q[CR];
#pragma unroll 4
    for (int w = 2; w < W; w += 2) {
      s0 += q[w * CR];
      s1 += q[(w + 1) * CR];
    }
    return s0 + s1;
  };

  // aggregates of the own groups
  if (FSAI && A.na) {
    for (int i = t; i < A.na; i += RP_THREADS) aidx[i] = -1;
    __syncthreads();
    for (int i = t; i < ngl; i += RP_THREADS) aidx[A.agg[g0 + i]] = 0;
    __syncthreads();
    if (t == 0) {
      int k = 0;
      for (int i = 0; i < A.na; ++i)
        if (aidx[i] == 0) {
          aidx[i] = k;
          alst[k++] = i;
        }
      s_na = k;
    }
    __syncthreads();
    for (int i = t; i < ngl; i += RP_THREADS) gidx[i] = aidx[A.agg[g0 + i]];
    for (int I = t; I < A.na; I += RP_THREADS)
      for (int q = A.aseg[I]; q < A.aseg[I + 1]; ++q) sagg[q] = I;
    // the raw-mode coefficients of P A_c^-1 P^T r from the segments' raw moments:
    // rows T_I (A_c^-1)_IJ T_J^T of the own aggregates I, in FP64
    const int nc = A.na * NM;
    double* M = A.M + (int64_t)blockIdx.x * nc * nc;
    for (int i = t; i < s_na * NM * nc; i += RP_THREADS) {
      const int row = i / nc, col = i % nc, I = alst[row / NM], k = row % NM, J = col / NM, l = col % NM;
      const double* TI = A.T + (int64_t)I * NM * NM + k * NM;
      const double* TJ = A.T + (int64_t)J * NM * NM + l * NM;
      double s = 0.0;
#pragma unroll
      for (int a = 0; a < NM; ++a) {
        const float* inv = A.Ainv + (int64_t)(I * NM + a) * A.ld + J * NM;
        double u = 0.0;
#pragma unroll
        for (int b = 0; b < NM; ++b) u += (double)inv[b] * TJ[b];
        s += TI[a] * u;
      }
      M[i] = s;
    }
  }

  // Partial rows of L or L^T (packed blocks) times the exchanged vector vec.
  auto factor_part = [&](const int* cptr, const int* col, const uint4* pack, const __half* tail, const RpPair* vec,
                         Seq seq) {
    for (int task = wid; task < ncl * W; task += RN_WARPS) {
      const int cl = task / W, w = task % W, c = c0 + cl;
      const bool valid = c * 32 + lane < A.ngroups;
      double acc[DPN];
#pragma unroll
      for (int a = 0; a < DPN; ++a) acc[a] = 0.0;
      const int s1 = __ldg(cptr + c + 1);
      for (int s = __ldg(cptr + c) + w; s < s1; s += RN_BATCH * W) {
        const RpPair* from[RN_BATCH];
        double xj[RN_BATCH][DPN];
        float f[RN_BATCH][D2];
        bool use[RN_BATCH];
#pragma unroll
        for (int u = 0; u < RN_BATCH; ++u) {
          use[u] = valid && s + u * W < s1;
          const int64_t idx = (int64_t)(s + u * W) * 32 + lane;
          from[u] = vec + at(use[u] ? __ldg(col + idx) : g0, 0);
          if (use[u]) load_half_block<DPN>(pack, tail, idx, f[u]);
        }
        rp_get<RN_BATCH, DPN, 32>(from, seq, xj, late);
#pragma unroll
        for (int u = 0; u < RN_BATCH; ++u)
          if (use[u]) {
#pragma unroll
            for (int a = 0; a < DPN; ++a)
#pragma unroll
              for (int b = 0; b < DPN; ++b) acc[a] += (double)f[u][a * DPN + b] * xj[u][b];
          }
      }
#pragma unroll
      for (int a = 0; a < DPN; ++a) part[((cl * W + w) * DPN + a) * 32 + lane] = acc[a];
    }
  };

  // z = M r (own rows; r published with sequence seq); returns the thread's part
  // of r.z.  Every thread calls.
  auto precondition = [&](Seq seq) {
    factor_part(A.lcptr, A.lcol, A.lpack, A.ltail, A.r, seq);
    for (int I = blockIdx.x; I < A.nseg; I += gridDim.x) {  // raw moments of the segments this block sums
      double s[NM];
#pragma unroll
      for (int k = 0; k < NM; ++k) s[k] = 0.0;
      const int q1 = __ldg(A.send + I);
      for (int q0 = __ldg(A.sbeg + I) + wid * 32; q0 < q1; q0 += RN_BATCH * RP_THREADS) {
        const RpPair* from[RN_BATCH];
        double ra[RN_BATCH][DPN];
        int gr[RN_BATCH];
#pragma unroll
        for (int u = 0; u < RN_BATCH; ++u) {
          const int q = q0 + u * RP_THREADS + lane;
          gr[u] = q < q1 ? __ldg(A.alist + q) : -1;
          from[u] = A.r + at(gr[u] < 0 ? g0 : gr[u], 0);
        }
        rp_get<RN_BATCH, DPN, 32>(from, seq, ra, late);
#pragma unroll
        for (int u = 0; u < RN_BATCH; ++u) {
          if (gr[u] < 0) continue;
          double R[DPN][NM];
          mode_rows<DPN>(A.y + 3 * (int64_t)gr[u], R);
#pragma unroll
          for (int a = 0; a < DPN; ++a)
#pragma unroll
            for (int k = 0; k < NM; ++k) s[k] += R[a][k] * ra[u][a];
        }
      }
      // (through shared memory: shuffles of NM values in every warp would queue)
#pragma unroll
      for (int k = 0; k < NM; ++k) mom[k * RP_THREADS + t] = s[k];
      __syncthreads();
      if (wid < NM) {
        double sk[1] = {0.0};
#pragma unroll
        for (int w = 0; w < RN_WARPS; ++w) sk[0] += mom[wid * RP_THREADS + w * 32 + lane];
        rp_warp_sum(sk);
        if (lane == 0) rp_put(A.sm + I * NM + wid, sk[0], seq);
      }
      __syncthreads();
    }
    __syncthreads();
    for (int i = t; i < mrows; i += RP_THREADS) {  // t = sigma^2 (r + L r)
      int gl, a;
      if (!row_of(i, gl, a)) continue;
      double acc = r[i] + gathered(i);
      const int q = a * (a - 1) / 2;  // the diagonal block's strictly lower part
      for (int b = 0; b < a; ++b)
        acc += (double)__half2float(__ldg(A.ldiag + ((int64_t)(c0 + i / CR) * 3 + q + b) * 32 + lane)) *
               r[i + (b - a) * 32];
      const double ta = (double)__ldg(A.sigma2 + (int64_t)(g0 + gl) * DPN + a) * acc;
      e[i] = ta;
      rp_put(A.t + o0 + i, ta, seq);
    }
    if (A.na) {  // the own aggregates' coefficients of the prolongation
      const int nrow = s_na * NM, nc = A.na * NM, nsm = A.nseg * NM;
      for (int i0 = wid * 32; i0 < nsm; i0 += RP_THREADS) {
        const int i = min(i0 + lane, nsm - 1);
        const RpPair* const from[1] = {A.sm + i};
        double y[1][1];
        rp_get<1, 1, 32>(from, seq, y, late);
        smo[i] = y[0][0];
      }
      __syncthreads();
      constexpr int L = 8;  // lanes per row
      const double* M = A.M + (int64_t)blockIdx.x * nc * nc;
      for (int i0 = 0; i0 < nrow; i0 += RP_THREADS / L) {
        const int i = i0 + t / L;
        double s = 0.0;
        if (i < nrow)
#pragma unroll 4
          for (int j = t & (L - 1); j < nsm; j += L) s += M[i * nc + sagg[j / NM] * NM + j % NM] * smo[j];
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, L);
        if (i < nrow && (t & (L - 1)) == 0) cm[i] = s;
      }
    } else {
      __syncthreads();  // the partial rows have been read
    }
    factor_part(A.ucptr, A.ucol, A.upack, A.utail, A.t, seq);
    __syncthreads();
    double rzp = 0.0;
    for (int i = t; i < mrows; i += RP_THREADS) {  // z = t + L^T t + P uc
      int gl, a;
      if (!row_of(i, gl, a)) continue;
      double acc = e[i] + gathered(i);
      for (int b = a + 1; b < DPN; ++b)  // column a of the diagonal block's strictly lower part
        acc += (double)__half2float(__ldg(A.ldiag + ((int64_t)(c0 + i / CR) * 3 + b * (b - 1) / 2 + a) * 32 + lane)) *
               e[i + (b - a) * 32];
      if (A.na) {
        const double* cI = cm + gidx[gl] * NM;
        double R[DPN][NM];
        mode_rows<DPN>(A.y + 3 * (int64_t)(g0 + gl), R);
#pragma unroll
        for (int k = 0; k < NM; ++k) {
          double Ra = R[0][k];
#pragma unroll
          for (int b = 1; b < DPN; ++b) Ra = a == b ? R[b][k] : Ra;
          acc += Ra * cI[k];
        }
      }
      z[i] = acc;
      rzp += r[i] * acc;
    }
    return rzp;
  };

  // r = b
  Seq zt = 1, pt = 1;  // sequences of r (and t, the moments) and of z
  double rz_own = 0.0, rr_own = 0.0, bad = 0.0;  // this thread's parts of r.z and r.r, bad diagonals
  for (int i = t; i < mrows; i += RP_THREADS) {
    int gl, a;
    xl[i] = p[i] = kp[i] = r[i] = z[i] = e[i] = 0.0;  // (padding rows stay zero)
    if (!row_of(i, gl, a)) continue;
    const int64_t row = (int64_t)(g0 + gl) * DPN + a;
    const double bi = residual_of_zero(A.b[row]);
    if (!FSAI) {
      const double d = A.dval[((int64_t)(c0 + i / CR) * D2 + a * DPN + a) * 32 + lane];
      if (!(d > 0.0)) bad += 1.0;
      const double di = 1.0 / d, zi = di * bi;
      e[i] = di;
      z[i] = zi;
      rz_own += bi * zi;
    } else {
      rp_put(A.r + o0 + i, bi, zt);
    }
    r[i] = bi;
    A.x[row] = 0.0;
    rr_own += bi * bi;
  }
  double rr = 0.0, rz = 0.0, pap = 0.0;  // r.r of the last true residual; rz, pap: of the last direction
  double target2 = 0.0, final2 = 0.0, upd2 = 0.0;
  bool fresh = true, started = false;  // r is a true residual, not the recurrence's
  bool direct = false;                 // z holds the direction itself (below)
  int done = 0;
  // (one copy of the preconditioner, of K z and of the sums: the loop body has to stay
  // in the instruction cache and, but for 180 bytes that FSAI with 3 dofs reloads and 24
  // with 2, in registers)
  for (;;) {
    if (FSAI && !direct) {
      __syncthreads();
      rz_own = precondition(zt);
    }
    for (int i = t; i < mrows; i += RP_THREADS) rp_put(A.zp + o0 + i, z[i], pt);
    __syncthreads();
    for (int task = wid; task < ncl * W; task += RN_WARPS) {  // K z
      const int cl = task / W, w = task % W, c = c0 + cl;
      const bool valid = c * 32 + lane < A.ngroups;
      double acc[DPN];
#pragma unroll
      for (int a = 0; a < DPN; ++a) acc[a] = 0.0;
      const int l0 = __ldg(A.lcptr + c), nl = __ldg(A.lcptr + c + 1) - l0;
      const int u0 = __ldg(A.ucptr + c), nu = __ldg(A.ucptr + c + 1) - u0;
      if (w == W - 1 && valid) {  // the diagonal block
        double xi[DPN];
#pragma unroll
        for (int b = 0; b < DPN; ++b) xi[b] = z[cl * CR + b * 32 + lane];
#pragma unroll
        for (int a = 0; a < DPN; ++a)
#pragma unroll
          for (int b = 0; b < DPN; ++b)
            acc[a] += __ldg(A.dval + ((int64_t)c * D2 + a * DPN + b) * 32 + lane) * xi[b];
      }
      for (int it = w; it < nl + nu; it += RN_BATCH * W) {
        const RpPair* from[RN_BATCH];
        double xj[RN_BATCH][DPN];
        int base[RN_BATCH];
#pragma unroll
        for (int u = 0; u < RN_BATCH; ++u) {
          const int iu = it + u * W;
          const bool low = iu < nl, on = valid && iu < nl + nu;
          const int64_t idx = (int64_t)(low ? l0 + iu : u0 + iu - nl) * 32 + lane;
          base[u] = !on ? -1 : low ? (l0 + iu) * (D2 * 32) + lane : __ldg(A.ubase + idx);
          from[u] = A.zp + at(on ? __ldg((low ? A.lcol : A.ucol) + idx) : g0, 0);
        }
        rp_get<RN_BATCH, DPN, 32>(from, pt, xj, late);
#pragma unroll
        for (int u = 0; u < RN_BATCH; ++u) {
          if (base[u] < 0) continue;
          const bool low = it + u * W < nl;
          const double* bv = A.lval + base[u];
#pragma unroll
          for (int a = 0; a < DPN; ++a)
#pragma unroll
            for (int b = 0; b < DPN; ++b) acc[a] += __ldg(bv + (low ? a * DPN + b : b * DPN + a) * 32) * xj[u][b];
        }
      }
#pragma unroll
      for (int a = 0; a < DPN; ++a) part[((cl * W + w) * DPN + a) * 32 + lane] = acc[a];
    }
    __syncthreads();
    double w[RP_VALUES] = {rz_own, rr_own, 0.0};  // r.z, r.r, z.Kz
    double zkp[RP_VALUES] = {0.0, bad, 0.0};      // z.Kp
    for (int i = t; i < mrows; i += RP_THREADS) {
      const double q = gathered(i);
      part[i / CR * W * CR + i % CR] = q;  // (the row's own partial sums are read)
      w[2] += z[i] * q;
      if (fresh) zkp[0] += z[i] * kp[i];
    }
    for (int k = 0; k < (fresh && !direct ? 2 : 1); ++k) {
      double v[RP_VALUES];
#pragma unroll
      for (int j = 0; j < RP_VALUES; ++j) v[j] = k ? zkp[j] : w[j];
      grid_sum(v);
#pragma unroll
      for (int j = 0; j < RP_VALUES; ++j) (k ? zkp[j] : w[j]) = v[j];
    }
    ++pt;
    if (late) { out.status = RP_LATE; break; }
    if (direct) {
      // (tested before)
    } else if (fresh) {
      rr = w[1];
      if (!started) {
        started = true;
        out.bb = rr;
        const double bnorm = sqrt(out.bb);
        target2 = A.tol * A.tol * bnorm * bnorm;
        final2 = 0.25 * target2;
        if (zkp[1] != 0.0) { out.status = RP_BAD_DIAGONAL; break; }
        if (out.bb == 0.0 || rr <= target2) break;
        if (!(w[0] > 0.0)) { out.status = RP_BREAKDOWN; break; }
      } else {
        out.outer += 1;
        if (rr <= target2) break;
        if (done == 3) { out.status = RP_CAP; break; }
        if (FSAI && !(w[0] > 0.0)) { out.status = RP_BREAKDOWN; break; }
      }
      upd2 = fmax(A.delta * A.delta * rr, final2);
    } else {
      if (!(w[1] == w[1]) || !(w[0] == w[0])) { out.status = RP_BREAKDOWN; break; }
      done = w[1] <= upd2 ? 4 : out.iters >= A.max_it ? 3 : 0;
      if (!done && FSAI && !(w[0] > 0.0)) { out.status = RP_BREAKDOWN; break; }  // the preconditioner is not SPD
      if (done) {
        // reliable update: x += xl, r = b - A x (compensated)
        const Seq xt = (Seq)out.outer + 1;
        for (int i = t; i < mrows; i += RP_THREADS) {
          int gl, a;
          if (!row_of(i, gl, a)) continue;
          const int64_t row = (int64_t)(g0 + gl) * DPN + a;
          const double xi = A.x[row] + xl[i];
          A.x[row] = xi;
          rp_put(A.xp + o0 + i, xi, xt);
          xl[i] = 0.0;
        }
        __syncthreads();
        constexpr int LANES = 8;
        for (int i0 = 0; i0 < ngl * DPN; i0 += RP_THREADS / LANES) {
          const int i = i0 + t / LANES, row = g0 * DPN + min(i, ngl * DPN - 1);
          double hi = 0.0, lo = 0.0;
          const int k1 = __ldg(A.rp + row + 1);
          for (int k = __ldg(A.rp + row) + (t & (LANES - 1)); __any_sync(0xffffffffu, k < k1); k += LANES) {
            const bool in = k < k1;
            const int col = in ? __ldg(A.ci + k) : row;
            const RpPair* const from[1] = {A.xp + at(col / DPN, col % DPN)};
            double xj[1][1];
            rp_get<1, 1, 32>(from, xt, xj, late);
            if (in) {
              double pr, pe, s, se;
              two_prod(__ldg(A.va + k), xj[0][0], pr, pe);
              two_sum(hi, pr, s, se);
              hi = s;
              lo += pe + se;
            }
          }
#pragma unroll
          for (int o = LANES / 2; o > 0; o >>= 1) {
            const double oh = __shfl_down_sync(0xffffffffu, hi, o, LANES);
            const double ol = __shfl_down_sync(0xffffffffu, lo, o, LANES);
            double s, se;
            two_sum(hi, oh, s, se);
            hi = s;
            lo += ol + se;
          }
          if (i < ngl * DPN && (t & (LANES - 1)) == 0) {
            double r1, e1;
            two_sum(A.b[row], -hi, r1, e1);
            const int gl = i / DPN, a = i % DPN;
            r[(gl >> 5) * CR + a * 32 + (gl & 31)] = r1 + (e1 - lo);
          }
        }
        __syncthreads();
        rz_own = rr_own = 0.0;
        ++zt;
        for (int i = t; i < mrows; i += RP_THREADS) {
          int gl, a;
          if (!row_of(i, gl, a)) continue;
          const double ri = r[i];
          if (FSAI) {
            rp_put(A.r + o0 + i, ri, zt);
          } else {
            const double zi = e[i] * ri;
            z[i] = zi;
            rz_own += ri * zi;
          }
          rr_own += ri * ri;
        }
        fresh = true;
        continue;
      }
    }
    // p = z + beta p and p.Kp = z.Kz + 2 beta z.Kp + beta^2 (p.Kp of before), where
    // z.Kp = -beta (p.Kp of before) while r is the recurrence's residual
    const double beta = out.iters && !direct ? w[0] / rz : 0.0;
    const double pkp = direct  ? w[2]
                       : fresh ? w[2] + beta * (2.0 * zkp[0] + beta * pap)
                               : w[2] - beta * beta * pap;
    if (!(pkp > 0.0)) {
      // at the limit of accuracy K p's recurrence may have drifted: K is applied to
      // the direction itself, and that product decides
      if (direct) { out.status = RP_BREAKDOWN; break; }
      direct = true;
      for (int i = t; i < mrows; i += RP_THREADS) z[i] += beta * p[i];
      continue;
    }
    direct = false;
    pap = pkp;
    rz = w[0];
    const double alpha = rz / pap;
    rz_own = rr_own = 0.0;
    ++zt;
    for (int i = t; i < mrows; i += RP_THREADS) {
      int gl, a;
      if (!row_of(i, gl, a)) continue;
      const double pi = z[i] + beta * p[i], qi = part[i / CR * W * CR + i % CR] + beta * kp[i];
      p[i] = pi;
      kp[i] = qi;
      xl[i] += alpha * pi;
      const double ri = r[i] - alpha * qi;
      r[i] = ri;
      if (FSAI) {
        rp_put(A.r + o0 + i, ri, zt);
      } else {
        const double zi = e[i] * ri;
        z[i] = zi;
        rz_own += ri * zi;
      }
      rr_own += ri * ri;
    }
    out.iters += 1;
    fresh = false;
  }
  out.rr = rr;
  if (blockIdx.x == 0 && t == 0) *A.res = out;
}

// Lanes per row of the one-block solve, so that a row's entries take few passes.
// Microseconds an iteration with 4 / 8 / 16: 125 rows of 5.8 entries 2.8 / 2.9 / 3.9, 343 of
// 6.1 3.3 / 4.3; 81 rows of 20.8 2.1 / 2.4 / 2.7, 264 of 16.0 2.9 / 3.7, so up to 23 entries
// four lanes would do (rows of more than 24 have not been measured).
int rj_lanes(int64_t n, int64_t nnz) {
  const double avg = (double)nnz / (double)std::max<int64_t>(n, 1);
  return avg <= 12 ? 4 : avg <= 40 ? 8 : 16;
}

template <int DPN>
const void* rn_kernel(bool fsai) {
  return fsai ? (const void*)resident_nb<DPN, true> : (const void*)resident_nb<DPN, false>;
}

RnShape shape_of(const SystemData& S, bool coarse) {
  const CoarseSpace& C = S.coarse;
  return rn_shape(S.nb.nchunks, S.nb.dpn, sm_count(), coarse ? C.na : 0, coarse ? C.nm : 0, coarse ? C.nseg : 0);
}

RpOutcome outcome(const SystemData& S, const RpResult* d_res) {
  cudaStream_t s = S.ctx->stream;
  RpResult h{};
  TPT_CUDA(cudaMemcpyAsync(&h, d_res, sizeof(h), cudaMemcpyDeviceToHost, s));
  TPT_CUDA(cudaStreamSynchronize(s));
  TPT_REQUIRE(h.status != RP_LATE, TPTFEM_ERR_DEVICE, "resident PCG: an exchanged value did not arrive in time");
  TPT_REQUIRE(h.status != RP_BAD_DIAGONAL, TPTFEM_ERR_NUMERIC,
              "reduced matrix has a missing or non-positive diagonal entry (not SPD)");
  RpOutcome o;
  o.iterations = h.iters;
  o.outer_steps = h.outer;
  o.breakdown = h.status == RP_BREAKDOWN;
  o.rr = h.rr;
  o.bb = h.bb;
  return o;
}

}  // namespace

bool resident_jacobi_applies(const SystemData& S) {
  return S.n_free > 0 && S.n_free * rj_lanes(S.n_free, S.nnz) <= RJ_MAX_LANES;
}

bool resident_nb_applies(const SystemData& S, bool fsai, bool coarse) {
  const NbSell& N = S.nb;
  if (N.state != 1 || S.n_free <= 0 || S.n_free > (fsai ? RN_MAX_ROWS_FSAI : RN_MAX_ROWS_JACOBI)) return false;
  if (coarse && (S.coarse.nc > RN_MAX_COARSE || S.coarse.nseg > RN_MAX_SEG)) return false;
  return shape_of(S, coarse).smem <= RN_MAX_SMEM;  // (a part of a GPU has fewer SMs for the same rows)
}

RpOutcome resident_jacobi_solve(SystemData& S, ResidentWork& W, double tol, double delta, int64_t max_it) {
  cudaStream_t s = S.ctx->stream;
  if (!W.res.p) W.res.alloc(sizeof(RpResult), s);
  RjArgs A{};
  A.n = (int)S.n_free;
  A.rp = S.row_ptr.p;
  A.ci = S.col.p;
  A.va = S.val.p;
  A.b = S.fred.p;
  A.x = S.x.p;
  A.res = reinterpret_cast<RpResult*>(W.res.p);
  A.tol = tol;
  A.delta = delta;
  A.max_it = (int)std::min<int64_t>(max_it, 1 << 30);
  const int lanes = rj_lanes(S.n_free, S.nnz);
  auto* k = lanes == 4 ? resident_jacobi<4> : lanes == 8 ? resident_jacobi<8> : resident_jacobi<16>;
  const size_t smem = 6 * (size_t)A.n * sizeof(double);
  allow_smem((const void*)k, RJ_MAX_SMEM);
  k<<<1, RJ_THREADS, smem, s>>>(A);
  TPT_CHECK_LAUNCH();
  return outcome(S, A.res);
}

RpOutcome resident_nb_solve(SystemData& S, ResidentWork& W, const float* sigma2, bool coarse, double tol, double delta,
                            int64_t max_it) {
  cudaStream_t s = S.ctx->stream;
  const NbSell& N = S.nb;
  const bool fsai = sigma2 != nullptr;
  RnArgs A{};
  A.ngroups = N.ngroups;
  A.nchunks = N.nchunks;
  const RnShape shape = shape_of(S, coarse);
  const int blocks = shape.blocks;
  A.nc = shape.nc;
  A.w = shape.w;
  A.lcptr = N.l_cptr.p; A.lcol = N.l_col.p; A.ucptr = N.u_cptr.p; A.ucol = N.u_col.p; A.ubase = N.ku_base.p;
  A.lval = N.ks_lval.p; A.dval = N.ks_diag.p;
  A.lpack = N.l_pack.p; A.upack = N.u_pack.p; A.ltail = N.l_tail.p; A.utail = N.u_tail.p; A.ldiag = N.l_diag.p;
  A.sigma2 = sigma2;
  A.rp = S.row_ptr.p; A.ci = S.col.p; A.va = S.val.p; A.b = S.fred.p;
  A.x = S.x.p;
  if (coarse) {
    const CoarseSpace& C = S.coarse;
    A.na = C.na;
    A.ld = C.ld;
    A.nseg = C.nseg;
    A.agg = C.agg.p; A.aseg = C.aseg.p; A.sbeg = C.sbeg.p; A.send = C.send.p; A.alist = C.alist.p;
    A.y = C.y.p; A.Ainv = C.Ainv.p; A.T = C.T.p;
  }
  const size_t np = (size_t)N.nchunks * 32 * N.dpn;  // a pair vector, padded to whole chunks
  const size_t nsm = coarse ? (size_t)S.coarse.nseg * S.coarse.nm : 0;
  const size_t pairs = RP_TABLE + (fsai ? 4 : 2) * np + nsm;
  if (W.pairs.n < pairs * sizeof(RpPair)) W.pairs.alloc(pairs * sizeof(RpPair), s);
  if (!W.res.p) W.res.alloc(sizeof(RpResult), s);
  const size_t nM = coarse ? (size_t)blocks * S.coarse.nc * S.coarse.nc : 0;
  if (W.M.n < nM) W.M.alloc(nM, s);
  A.M = W.M.p;
  TPT_CUDA(cudaMemsetAsync(W.pairs.p, 0, pairs * sizeof(RpPair), s));
  A.table = reinterpret_cast<RpPair*>(W.pairs.p);
  A.xp = A.table + RP_TABLE;
  A.zp = A.xp + np;
  A.r = fsai ? A.zp + np : nullptr;
  A.t = fsai ? A.r + np : nullptr;
  A.sm = coarse ? A.t + np : nullptr;
  A.res = reinterpret_cast<RpResult*>(W.res.p);
  A.tol = tol;
  A.delta = delta;
  A.max_it = (int)std::min<int64_t>(max_it, 1 << 30);
  const void* k = N.dpn == 3 ? rn_kernel<3>(fsai) : N.dpn == 2 ? rn_kernel<2>(fsai) : rn_kernel<1>(fsai);
  allow_smem(k, RN_MAX_SMEM);
  void* args[] = {&A};
  TPT_CUDA(cudaLaunchCooperativeKernel(k, dim3(blocks), dim3(RP_THREADS), args, shape.smem, s));
  return outcome(S, A.res);
}

}  // namespace tptfem
