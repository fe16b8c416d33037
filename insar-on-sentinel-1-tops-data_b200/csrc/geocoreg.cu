// geocoreg.cu -- DEM-assisted geometric coregistration (sm_100a, FP64).
//
// Reference (GeoCoreg_warp_cuda, Geocoreg_cuda.cu:610-913): per DEM pixel
//   llh2xyz (:87-99) -> ECEF target; for master and slave a zero-Doppler
//   Newton solve (ell2lpGeo :211-323 with getPos/getVelo/getAcc :123-205
//   and SolveNewtonEq :101-112, <= 11 iterations, |step| < 1e-10 s) giving
//   (line, pixel); weight 1 if the DEM is valid and the master position is
//   inside the burst box (WeighthSet :548-574); A row [1, L, P, L^2, LP, P^2]
//   of the normalised master position (AMatrixSet :576-605); then
//   N = (WA)^T A, rhs = (WA)^T {slave line, slave pixel} by cuBLAS and a
//   Cholesky solve by cuSOLVER (:822-851).
//
// B200 design: one kernel per launch of up to 16 bursts.  The DEM is cut into
// tiles of GC_TR rows x GC_NT columns; the sine, cosine and prime-vertical
// radius of each tile row and the sine and cosine of each column are computed
// once per tile (the reference computes them per pixel; the values are the
// same), then each thread geocodes its column's pixels (master and slave share
// the target position) and accumulates the 21 distinct entries of N and the
// two right-hand sides (33 FP64 sums) in registers; warp shuffles and a fixed
// order of the warps reduce them to one partial per tile.  A one-block kernel
// per burst sums the partials in a fixed order and solves the 6x6 system with
// the reference's own Cholesky scheme (Func.cpp:959-1013).  No per-pixel
// buffers touch HBM; results are bit-for-bit reproducible run to run.  Orbit
// polynomials and their first two derivatives are evaluated with Horner's rule
// instead of pow(), and the Newton step folds the reference's velocity / 10 and
// acceleration / 100 scalings into one division; the root and the stopping rule
// are the reference's, the rounding of the iterates differs in the last bits.
// Down a column, each solve starts from the previous solutions extrapolated
// linearly, and its first Newton step takes the orbit state there from a Taylor
// shift of the previous solve's position, velocity and acceleration, so most
// solves need one polynomial evaluation.
//
// What bounds it: the serial FP64 chain of a column (32 rows of two solves, 66
// us at any size of one wave), then the FP64 pipe (a few hundred operations per
// pixel at 16 warps per SM).  Small launches therefore split a column's master
// and slave solves over a pair of warps.  Measured, in us, with the solve:
//   DEM  162 x 162   72 -> 48      670 x 670  81 -> 53
//   DEM 1232 x 1770  91 -> 86     1232 x 2970  143 -> 137   (unsplit; the solve)
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>
#include <vector>

#include "common.cuh"

namespace tops {

constexpr int GC_NT = 256;  // DEM columns of a tile
constexpr int GC_TR = 32;   // DEM rows per tile (each starts its columns' Newton chains afresh)
constexpr int GC_NWF = 8;   // warps of a CTA where one warp solves both
constexpr int GC_MAXJOBS = 16;
constexpr int GC_NSUM = 33;
constexpr double kEllA = 6378137.0;                              // cuConstants.cuh:5
constexpr double kEllB = 6356752.3142451794975639665996337;      // cuConstants.cuh:6

struct GcBatch {
  int njobs, total_blocks;
  int dem_is_int;
  GeoJob jobs[GC_MAXJOBS];
};

// Position and the first two derivatives with respect to the normalised time
// t of an orbit polynomial (getPos/getVelo/getAcc, Geocoreg_cuda.cu:123-205,
// return the derivatives divided by 10 and 100).
// The same with the coefficient count N known at compile time (fully
// unrolled; the orbit fit returns 6 coefficients for more than 6 state
// vectors, Func.cpp:1050-1126).
template <int N>
__device__ __forceinline__ void orbit_eval_n(const double (*c)[8], double t, double p[3],
                                             double v[3], double a[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double pp = c[k][N - 1], vv = 0.0, aa = 0.0;
#pragma unroll
    for (int i = N - 2; i >= 0; --i) {
      aa = fma(aa, t, 2.0 * vv);
      vv = fma(vv, t, pp);
      pp = fma(pp, t, c[k][i]);
    }
    p[k] = pp;
    v[k] = vv;
    a[k] = aa;
  }
}

__device__ __forceinline__ void orbit_eval(const double (*c)[8], int n, double t, double p[3],
                                           double v[3], double a[3]) {
  if (n == 6) {
    orbit_eval_n<6>(c, t, p, v, a);
    return;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double pp = c[k][n - 1], vv = 0.0, aa = 0.0;
    for (int i = n - 2; i >= 0; --i) {
      aa = fma(aa, t, 2.0 * vv);
      vv = fma(vv, t, pp);
      pp = fma(pp, t, c[k][i]);
    }
    p[k] = pp;
    v[k] = vv;
    a[k] = aa;
  }
}

__device__ __forceinline__ void orbit_pos(const double (*c)[8], int n, double t, double p[3]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double pp = c[k][n - 1];
    for (int i = n - 2; i >= 0; --i) pp = fma(pp, t, c[k][i]);
    p[k] = pp;
  }
}

// Zero-Doppler (line, pixel) of target T for image k of job J.
// 1/x: the hardware's approximate FP64 reciprocal refined by two
// Newton-Raphson steps r <- r + r (1 - x r) (each doubles the correct bits;
// a Newton step of the zero-Doppler solve needs no correctly rounded
// quotient, only its root does not move)
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  r = fma(r, e, r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}

// az: the Newton start on entry (the reference starts every pixel at the
// burst-centre time; here a thread starts from the solutions of the pixels
// above in its column, extrapolated linearly, which converges to the same
// root in fewer steps), the zero-Doppler azimuth time on return.  P, V, A: the
// orbit position, velocity and acceleration at the last solution of this
// column, valid when have is set, and delta = start - that solution.  The
// first Newton step then takes the orbit state at the start from a Taylor
// shift (a few FMAs) instead of a polynomial evaluation; on return they hold
// this solve's state.
template <int K>
__device__ __forceinline__ void ell2lp(const GeoJob &J, const double T[3], double &az,
                                       double delta, double &line, double &pixel, double (&P)[3],
                                       double (&V)[3], double (&A)[3], bool &have) {
  constexpr int k = K;
  const double (*c)[8] = J.coef[k];
  const int n = J.ncoef[k];
  double sol = 0.0;
  int it0 = 0;
  if (have) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      // shift by dt = delta / 10 in normalised time (third-order term: below
      // 1e-9 m for the millisecond steps between DEM rows)
      const double dt = 0.1 * delta;
      const double a = A[q], v = V[q];
      P[q] = fma(dt, fma(0.5 * dt, a, v), P[q]);
      V[q] = fma(dt, a, v);
    }
    const double dx = T[0] - P[0], dy = T[1] - P[1], dz = T[2] - P[2];
    sol = -10.0 * (V[0] * dx + V[1] * dy + V[2] * dz) *
          rcp_nr((A[0] * dx + A[1] * dy + A[2] * dz) - V[0] * V[0] - V[1] * V[1] - V[2] * V[2]);
    az += sol;
    it0 = 1;   // that step is the solve's first iteration
  }
  // at least one step from an exact orbit evaluation, also when the shifted
  // step is already below the bound: the zero-Doppler root is sensitive to
  // the velocity's direction, which the shift only approximates
  for (int it = it0; it <= 10 && !(it > it0 && fabs(sol) < 1e-010); it++) {
    const double t = (az - J.mid_time[k]) * 0.1;
    orbit_eval(c, n, t, P, V, A);
    const double dx = T[0] - P[0], dy = T[1] - P[1], dz = T[2] - P[2];
    // -(V/10 . d) / ((A/100 . d) - |V/10|^2) (SolveNewtonEq, :101-112)
    sol = -10.0 * (V[0] * dx + V[1] * dy + V[2] * dz) *
          rcp_nr((A[0] * dx + A[1] * dy + A[2] * dz) - V[0] * V[0] - V[1] * V[1] - V[2] * V[2]);
    az += sol;
    if (fabs(sol) < 1e-010) break;
  }
  // position at the final az: from the last evaluation and one Taylor term
  // when the last step was below the stopping bound (dP/daz = V / 10; the
  // next term is below 1e-19 m), else evaluated afresh
  if (fabs(sol) < 1e-010) {
#pragma unroll
    for (int q = 0; q < 3; q++) P[q] = fma(0.1 * sol, V[q], P[q]);
  } else {
    orbit_pos(c, n, (az - J.mid_time[k]) * 0.1, P);
  }
  line = J.line_offset[k] + (az - J.first_line_time[k]) * J.inv_dt[k];
  const double r = sqrt((T[0] - P[0]) * (T[0] - P[0]) + (T[1] - P[1]) * (T[1] - P[1]) +
                        (T[2] - P[2]) * (T[2] - P[2]));
  pixel = (r - J.slr_time[k] * kSol) * J.inv_range_spacing[k];
  have = true;
}

// Sum over the lanes in a fixed order.
__device__ __forceinline__ double gc_warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void gc_pair_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, 64;" ::: "memory");
}

// The two forms of the kernel; a tile is a cluster's work, and a warp (FUSED)
// or a pair of warps (PAIR) has 32 of its columns.
//   FUSED  each thread solves its column's master and slave positions in turn
//          and sums all 27 products; the orbit states wait in shared memory.
//   PAIR   a CTA's first warp solves the master and sums the monomials, the
//          second follows a row behind, solves the slave where the pixel
//          is inside the burst, and sums its products: half the serial chain
//          of a column, but idle warps where few pixels are inside.
// Both do the same arithmetic in the same order.
enum { GC_FUSED = 0, GC_PAIR = 1 };
template <int FORM>
struct GcShape {
  static constexpr int kWarps = FORM == GC_PAIR ? 1 : GC_NWF;   // of 32 columns
  static constexpr int kThreads = FORM == GC_PAIR ? 64 : 32 * GC_NWF;
  static constexpr int kCtas = GC_NT / 32 / kWarps;             // per tile
  // (for pairs a bound of 8 spilled: 52 us where none took 47)
  static constexpr int kMinCtas = FORM == GC_PAIR ? 0 : 2;
};

template <int FORM>
__global__ void __cluster_dims__(GcShape<FORM>::kCtas, 1, 1)
    __launch_bounds__(GcShape<FORM>::kThreads, GcShape<FORM>::kMinCtas)
        geocoreg_kernel(const __grid_constant__ GcBatch B, double *partials) {
  using S = GcShape<FORM>;
  constexpr bool PAIR = FORM == GC_PAIR;
  __shared__ double red[S::kWarps][GC_NSUM];
  __shared__ double row_s[GC_TR], row_c[GC_TR], row_n[GC_TR], col_s[32], col_c[32];
  __shared__ double2 pos[2][32];          // normalised master positions; x NaN: no pixel
  __shared__ double ostate[PAIR ? 1 : 2][9][PAIR ? 1 : S::kThreads];
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int blk = blockIdx.x / S::kCtas, part = blockIdx.x % S::kCtas;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool master = !PAIR || warp == 0, slave = !PAIR || warp == 1;
  int jb = 0;
  while (jb + 1 < B.njobs && B.jobs[jb + 1].block_begin <= blk) jb++;
  const GeoJob &J = B.jobs[jb];
  const int lblk = blk - J.block_begin;
  const double e2 = 1.0 - (kEllB * kEllB / kEllA / kEllA);
  const double d2r = kPi / 180.0;
  const int tiles_x = (J.pixels + GC_NT - 1) / GC_NT;
  const int tiles = tiles_x * ((J.lines + GC_TR - 1) / GC_TR);
  const double ymid = 0.5 * ((double)J.ymin + (double)J.ymax);
  const double xmid = 0.5 * ((double)J.xmin + (double)J.xmax);
  // sums of the monomials L^i P^j (i + j <= 4) of the design row a = (1, L,
  // P, L^2, LP, P^2) -- its 21 distinct products a_i a_j are 15 monomials --
  // and (from acs on) of a_i times the slave line and pixel: 27 accumulators,
  // expanded to the 33 normal-equation sums after the loop
  constexpr int NACC = PAIR ? 15 : 27, ACS = PAIR ? 0 : 15;
  double acc[NACC];
#pragma unroll
  for (int q = 0; q < NACC; q++) acc[q] = 0.0;

  for (int tile = lblk; tile < tiles; tile += J.blocks) {
    const int row0 = (tile / tiles_x) * GC_TR;
    const int cta0 = (tile % tiles_x) * GC_NT + 32 * S::kWarps * part;
    const int col = cta0 + (PAIR ? lane : threadIdx.x);
    if (cta0 >= J.pixels) continue;   // the whole CTA
    const bool have_col = col < J.pixels;
    // llh2xyz (Geocoreg_cuda.cu:87-99): the latitude terms per tile row, the
    // longitude terms per column
    __syncthreads();   // the previous tile's terms are no longer read
    double slam, clam;
    if (slave && (PAIR || warp == 0) && row0 + lane < J.lines) {
      double sphi, cphi;
      sincos((J.lat0 - J.dlat * (row0 + lane)) * d2r, &sphi, &cphi);
      row_s[lane] = sphi;
      row_c[lane] = cphi;
      row_n[lane] = kEllA / sqrt(1.0 - e2 * sphi * sphi);
    }
    if (master) {
      sincos((J.lon0 + J.dlon * col) * d2r, &slam, &clam);
      if (PAIR) {
        col_s[lane] = slam;
        col_c[lane] = clam;
      }
    }
    __syncthreads();
    if (PAIR) {
      slam = col_s[lane];
      clam = col_c[lane];
    }
    const int nr = min(GC_TR, J.lines - row0);
    // The state of an image's Newton chain down the column.
    struct Chain {
      double az;                 // the last solution: the next start
      double dz = 0.0;           // its change per row between the last two solved
                                 // rows (0 unless adjacent): extrapolates the start
      int last = -2;             // last row solved
      double P[3], V[3], A[3];   // orbit state there
      bool have = false;
    };
    // the DEM sample and target of row rr
    auto target = [&](int rr, double (&T)[3]) {
      const long off = (long)(row0 + rr) * J.dem_pitch + col;
      float h;
      if (B.dem_is_int)
        h = (float)reinterpret_cast<const int *>(J.dem)[off];
      else
        h = J.dem[off];
      const double sphi = row_s[rr], cphi = row_c[rr];
      const double nph = row_n[rr] + h;
      T[0] = nph * cphi * clam;
      T[1] = nph * cphi * slam;
      T[2] = (nph - e2 * (nph - h)) * sphi;
      return h != (float)J.nodata;
    };
    auto solve = [&](auto kk, Chain &c, int rr, const double (&T)[3], double &line,
                     double &pixel) {
      constexpr int k = decltype(kk)::value;
      const double d = c.last == rr - 1 ? c.dz : 0.0;
      double a = c.az + d;
      if (!PAIR && c.have) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
          c.P[q] = ostate[k][q][threadIdx.x];
          c.V[q] = ostate[k][3 + q][threadIdx.x];
          c.A[q] = ostate[k][6 + q][threadIdx.x];
        }
      }
      ell2lp<k>(J, T, a, d, line, pixel, c.P, c.V, c.A, c.have);
      if (!PAIR) {
#pragma unroll
        for (int q = 0; q < 3; q++) {
          ostate[k][q][threadIdx.x] = c.P[q];
          ostate[k][3 + q][threadIdx.x] = c.V[q];
          ostate[k][6 + q][threadIdx.x] = c.A[q];
        }
      }
      c.dz = (c.last == rr - 1) ? a - c.az : 0.0;
      c.az = a;
      c.last = rr;
    };
    // the normalised master position of a pixel inside the burst
    auto master_row = [&](Chain &c, int rr, const double (&T)[3], double2 &q) {
      double ml, mp;
      solve(std::integral_constant<int, 0>(), c, rr, T, ml, mp);
      if (!(ml >= J.ymin && ml <= J.ymax && mp >= J.xmin && mp <= J.xmax)) return false;
      q = make_double2((ml - ymid) * J.inv_yq, (mp - xmid) * J.inv_xq);
      return true;
    };
    auto sum_master = [&](double2 q) {
      const double L = q.x, P = q.y, L2 = L * L, LP = L * P, P2 = P * P;
      // monomials in the order M00 M10 M01 M20 M11 M02 M30 M21 M12 M03 M40
      // M31 M22 M13 M04
      const double m[15] = {1.0, L, P, L2, LP, P2, L2 * L, L2 * P, L * P2, P2 * P,
                            L2 * L2, L2 * LP, L2 * P2, LP * P2, P2 * P2};
#pragma unroll
      for (int i = 0; i < 15; i++) acc[i] += m[i];
    };
    auto sum_slave = [&](double2 q, double sl, double sp) {
      const double L = q.x, P = q.y;
      const double a[6] = {1.0, L, P, L * L, L * P, P * P};
#pragma unroll
      for (int i = 0; i < 6; i++) {
        acc[ACS + i] = fma(a[i], sl, acc[ACS + i]);
        acc[ACS + 6 + i] = fma(a[i], sp, acc[ACS + 6 + i]);
      }
    };
    if constexpr (!PAIR) {
      Chain cm, cs;
      cm.az = J.azi_init[0];
      cs.az = J.azi_init[1];
      if (have_col) {
        for (int rr = 0; rr < nr; rr++) {
          double T[3], sl, sp;
          double2 q;
          if (!target(rr, T) || !master_row(cm, rr, T, q)) continue;
          solve(std::integral_constant<int, 1>(), cs, rr, T, sl, sp);
          sum_master(q);
          sum_slave(q, sl, sp);
        }
      }
    } else if (!slave) {
      // row rr's positions are written before barrier rr, read after it, and
      // their half of the buffer is written again after barrier rr + 1
      Chain c;
      c.az = J.azi_init[0];
      for (int rr = 0; rr < nr; rr++) {
        double2 q = make_double2(__longlong_as_double(0x7ff8000000000000LL), 0.0);
        double T[3];
        if (have_col && target(rr, T) && master_row(c, rr, T, q)) sum_master(q);
        pos[rr & 1][lane] = q;
        gc_pair_sync();
      }
    } else {
      Chain c;
      c.az = J.azi_init[1];
      for (int rr = 0; rr < nr; rr++) {
        gc_pair_sync();
        const double2 q = pos[rr & 1][lane];
        if (!(q.x == q.x)) continue;
        double T[3], sl, sp;
        target(rr, T);
        solve(std::integral_constant<int, 1>(), c, rr, T, sl, sp);
        sum_slave(q, sl, sp);
      }
    }
  }
  // the 33 sums: a_i a_j (i <= j, row-major) from the monomials, then the
  // slave-line and slave-pixel sums; over the lanes, then over the cluster's
  // warps in order
  constexpr int kMono[21] = {0, 1, 2, 3, 4, 5,     // 1 x (1 L P L2 LP P2)
                             3, 4, 6, 7, 8,        // L x (L P L2 LP P2)
                             5, 7, 8, 9,           // P x (P L2 LP P2)
                             10, 11, 12,           // L2 x (L2 LP P2)
                             12, 13,               // LP x (LP P2)
                             14};                  // P2 x P2
#pragma unroll
  for (int q = 0; q < NACC; q++) acc[q] = gc_warp_sum(acc[q]);
  if (lane == 0) {
    double *r = red[PAIR ? 0 : warp];
    if (master) {
#pragma unroll
      for (int q = 0; q < 21; q++) r[q] = acc[kMono[q]];
    }
    if (slave) {
#pragma unroll
      for (int q = 0; q < 12; q++) r[21 + q] = acc[ACS + q];
    }
  }
  cluster.sync();
  if (part == 0 && threadIdx.x < GC_NSUM) {
    double v = 0.0;
    for (int w = 0; w < GC_NT / 32; w++)
      v += cluster.map_shared_rank(&red[w % S::kWarps][0], w / S::kWarps)[threadIdx.x];
    partials[(long)blk * GC_NSUM + threadIdx.x] = v;
  }
  cluster.sync();   // red stays until it has been read
}

// Cholesky solve of the 6x6 normal equations (choles/solvechol semantics,
// Func.cpp:959-1013); one block per job.  The partials of GC_SB blocks at a
// time come in by all threads, the next ones while a thread per sum adds them
// up in block order; then a thread per right-hand side factors and solves.
constexpr int GC_ST = 512, GC_SB = 128, GC_SL = (GC_SB * GC_NSUM + GC_ST - 1) / GC_ST;

__global__ void __launch_bounds__(GC_ST)
    geocoreg_solve_kernel(const __grid_constant__ GcBatch B, const double *partials) {
  __shared__ double in[GC_SB * GC_NSUM];
  __shared__ double tot[GC_NSUM];
  const GeoJob &J = B.jobs[blockIdx.x];
  const double *part = partials + (long)J.block_begin * GC_NSUM;
  const int n_in = J.blocks * GC_NSUM;
  double next[GC_SL];
  auto load = [&](int i0) {
#pragma unroll
    for (int k = 0; k < GC_SL; k++) {
      const int i = threadIdx.x + k * GC_ST;
      next[k] = i < GC_SB * GC_NSUM && i0 + i < n_in ? part[i0 + i] : 0.0;
    }
  };
  load(0);
  double v = 0.0;
  for (int b0 = 0; b0 < J.blocks; b0 += GC_SB) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GC_SL; k++) {
      const int i = threadIdx.x + k * GC_ST;
      if (i < GC_SB * GC_NSUM) in[i] = next[k];
    }
    __syncthreads();
    load((b0 + GC_SB) * GC_NSUM);
    if (threadIdx.x < GC_NSUM) {
      const int nb = min(GC_SB, J.blocks - b0);
#pragma unroll 8
      for (int b = 0; b < nb; b++) v += in[b * GC_NSUM + threadIdx.x];
    }
  }
  if (threadIdx.x < GC_NSUM) tot[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x >= 2) return;
  double n[6][6];
  {
    int q = 0;
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
      for (int j = i; j < 6; j++) {
        n[i][j] = tot[q];
        n[j][i] = tot[q];
        q++;
      }
  }
  int bad = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = i; j < 6; ++j) {
      double sum = n[i][j];
#pragma unroll
      for (int k = i - 1; k >= 0; --k) sum -= n[i][k] * n[j][k];
      if (i == j) {
        if (!(sum > 0.0)) bad = 1;
        n[i][i] = sqrt(sum);
      } else {
        n[j][i] = sum / n[i][i];
      }
    }
  const int r = threadIdx.x;
  if (bad) {
    if (r == 0) *J.status = TOPS_E_NOT_PD;
    return;
  }
  double b[6];
#pragma unroll
  for (int i = 0; i < 6; i++) b[i] = tot[21 + 6 * r + i];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    double sum = b[i];
#pragma unroll
    for (int j = i - 1; j >= 0; --j) sum -= n[i][j] * b[j];
    b[i] = sum / n[i][i];
  }
#pragma unroll
  for (int i = 5; i >= 0; --i) {
    double sum = b[i];
#pragma unroll
    for (int j = i + 1; j < 6; ++j) sum -= n[j][i] * b[j];
    b[i] = sum / n[i][i];
  }
#pragma unroll
  for (int i = 0; i < 6; i++) J.cpm[6 * r + i] = b[i];
  if (r == 0) *J.status = TOPS_OK;
}

static int gc_blocks_for(int lines, int pixels) {
  // one block per tile up to 4096 blocks (a tile is GC_TR rows x GC_NT columns)
  long t = (long)((pixels + GC_NT - 1) / GC_NT) * ((lines + GC_TR - 1) / GC_TR);
  if (t < 1) t = 1;
  if (t > 4096) t = 4096;
  return (int)t;
}

int fill_geo_job(const tops_geo_job &u, GeoJob &J) {
  if (!u.dem || !u.cpm_dev || !u.status_dev || u.dem_lines <= 0 || u.dem_pixels <= 0)
    return TOPS_E_INVALID;
  if (u.dem_pitch % sizeof(float)) return TOPS_E_INVALID;
  if (u.xmax <= u.xmin || u.ymax <= u.ymin) return TOPS_E_INVALID;
  for (int k = 0; k < 2; k++)
    if (u.ncoef[k] < 2 || u.ncoef[k] > 8 || u.dt[k] == 0.0 || u.range_spacing[k] == 0.0)
      return TOPS_E_INVALID;
  J.dem = u.dem;
  J.dem_pitch = (long)(u.dem_pitch / sizeof(float));
  if (J.dem_pitch < u.dem_pixels) return TOPS_E_INVALID;
  J.lines = u.dem_lines;
  J.pixels = u.dem_pixels;
  J.lat0 = u.lat0;
  J.lon0 = u.lon0;
  J.dlat = u.dlat;
  J.dlon = u.dlon;
  J.nodata = u.nodata;
  J.xmin = u.xmin;
  J.xmax = u.xmax;
  J.ymin = u.ymin;
  J.ymax = u.ymax;
  J.inv_yq = 1.0 / (0.25 * ((double)u.ymax - (double)u.ymin));
  J.inv_xq = 1.0 / (0.25 * ((double)u.xmax - (double)u.xmin));
  for (int k = 0; k < 2; k++) {
    J.dt[k] = u.dt[k];
    J.inv_dt[k] = 1.0 / u.dt[k];
    J.inv_range_spacing[k] = 1.0 / u.range_spacing[k];
    J.first_line_time[k] = u.first_line_time[k];
    J.slr_time[k] = u.slr_time[k];
    J.range_spacing[k] = u.range_spacing[k];
    J.mid_time[k] = u.mid_time[k];
    J.azi_init[k] = u.azi_init[k];
    J.line_offset[k] = u.line_offset[k];
    J.ncoef[k] = u.ncoef[k];
    for (int a = 0; a < 3; a++)
      for (int i = 0; i < 8; i++) J.coef[k][a][i] = u.coef[k][a][i];
  }
  J.cpm = u.cpm_dev;
  J.status = u.status_dev;
  J.blocks = gc_blocks_for(u.dem_lines, u.dem_pixels);
  return TOPS_OK;
}

size_t geocoreg_scratch(const GeoJob *J, int n) {
  size_t blocks = 0;
  for (int i = 0; i < n; i++) blocks += J[i].blocks;
  return blocks * GC_NSUM * sizeof(double);
}

int launch_geocoreg(const GeoJob *jobs, int njobs, bool dem_is_int, void *scratch,
                    size_t scratch_bytes, cudaStream_t st) {
  if (geocoreg_scratch(jobs, njobs) > scratch_bytes || (!scratch && njobs > 0))
    return TOPS_E_INVALID;
  int dev = 0;
  TOPS_CUDA_TRY(cudaGetDevice(&dev));
  static PerDeviceOnce setup;
  int sms = 0;
  const int s0 = once_per_device(
      setup, dev,
      [&](int &v) -> int {
        TOPS_CUDA_TRY(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
        return TOPS_OK;
      },
      &sms);
  if (s0 != TOPS_OK) return s0;
  double *part = static_cast<double *>(scratch);
  for (int j0 = 0; j0 < njobs; j0 += GC_MAXJOBS) {
    GcBatch B;
    B.njobs = 0;
    B.dem_is_int = dem_is_int ? 1 : 0;
    int blocks = 0;
    for (int j = j0; j < njobs && j < j0 + GC_MAXJOBS; j++) {
      B.jobs[B.njobs] = jobs[j];
      B.jobs[B.njobs].block_begin = blocks;
      blocks += jobs[j].blocks;
      B.njobs++;
    }
    B.total_blocks = blocks;
    // Pairs of warps while all of them (8 per tile, 8 per SM) fit at once; with
    // more waves the fused form, whose warps are never idle, is faster: 124
    // tiles 70 us against 80, 195 tiles 91 against 76.
    if (blocks <= sms)
      geocoreg_kernel<GC_PAIR>
          <<<blocks * GcShape<GC_PAIR>::kCtas, GcShape<GC_PAIR>::kThreads, 0, st>>>(B, part);
    else
      geocoreg_kernel<GC_FUSED>
          <<<blocks * GcShape<GC_FUSED>::kCtas, GcShape<GC_FUSED>::kThreads, 0, st>>>(B, part);
    TOPS_CUDA_TRY(cudaGetLastError());
    geocoreg_solve_kernel<<<B.njobs, GC_ST, 0, st>>>(B, part);
    TOPS_CUDA_TRY(cudaGetLastError());
    part += (size_t)blocks * GC_NSUM;
  }
  return TOPS_OK;
}

}  // namespace tops

using namespace tops;

extern "C" size_t tops_geocoreg_scratch_bytes(const tops_geo_job *jobs, int njobs) {
  std::vector<GeoJob> J(njobs > 0 ? njobs : 0);
  for (int i = 0; i < njobs; i++)
    if (fill_geo_job(jobs[i], J[i]) != TOPS_OK) return 0;
  return geocoreg_scratch(J.data(), njobs);
}

extern "C" int tops_geocoreg(const tops_geo_job *jobs, int njobs, void *scratch_dev,
                             size_t scratch_bytes, void *stream) {
  if ((!jobs && njobs > 0) || njobs < 0) return TOPS_E_INVALID;
  std::vector<GeoJob> J(njobs);
  for (int i = 0; i < njobs; i++) {
    int s = fill_geo_job(jobs[i], J[i]);
    if (s != TOPS_OK) return s;
  }
  return launch_geocoreg(J.data(), njobs, false, scratch_dev, scratch_bytes,
                         static_cast<cudaStream_t>(stream));
}
