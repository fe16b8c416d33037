// resample.cu -- TOPS deramp + demodulation + 12-point LUT sinc resampling
// + reramp of slave bursts onto the master grid (sm_100a).
//
// Computes the reference algorithm of DerampDemod_Shared
// (DerampAndResample.cu:117-183) followed by Interpolation_12p
// (DerampAndResample.cu:349-520), GetIndexes (:108-112) and my_polyval /
// normalizeWarp (cuConstants.cuh:53-65):
//   position  y = polyAz(L^, P^) + shift,  x = polyRg(L^, P^)
//   index     L0 = trunc(y), bin = int(frac * 2047 + 0.5)  (same for x)
//   regions   outside the slave box -> 0; within 5/7 samples of its edge ->
//             the nearest sample; interior -> separable 12x12 LUT sinc of the
//             deramped slave d = s exp(i phi), reramped with the LUT-weighted
//             sum of the deramp phase phi.
//
// B200 design (no textures, no phase array in HBM).  A CTA of 64 threads
// owns a strip of RS_TW = 112 output columns with a ring of 128 slave columns
// (two per thread) and a segment of up to 252 output rows (a work item).  The rows are prepared in chunks and computed in
// halves of 6 rows:
//
// Chunk prologue.  Row keys: per row, the runs of equal azimuth key
// (L0, bin) along the strip, found by bisection of the exact per-pixel key on
// monotone pieces; each run is an "entry" (its columns, its reramp terms).
// Nearly parallel orbits give one entry per row, crossing orbits a few.
// Column keys: thread per column pair, the runs of the range key over the
// chunk's rows, each with its residual phase terms.  A chunk is as many rows
// (up to 96) as the entry and run tables hold; where a run table is full before
// 12 rows (kKeyedRows), the columns' rows behind it are keyed: [C] finds each
// pixel's key and terms anew.
//
// Half of 6 rows.
//   [A] azimuth pass, thread = 2 adjacent ring columns: six new slave lines
//       (staged with cp.async while earlier halves ran) are deramped in
//       registers and pushed into a 12-line register window whose slots
//       rotate statically; after each push the entries whose line is the
//       window's are summed, v = sum_j kAz[j] d(L0-5+j), with FP32x2 FMAs
//       over the two columns, into the tile: 16-byte units (re, re', im, im')
//       of two columns.  An entry covers only the ring columns its output
//       columns need, so a row of several entries costs little more than one.
//   [B] range pass, thread = 2 adjacent output columns: 7 tile units; one
//       column's 12 taps start at a unit boundary, the other's one sample
//       later, so it takes 7 units with taps shifted by one (0, w0 .. w11, 0).
//       An FP32x2 FMA multiplies two taps with the two samples of a unit.
// Halves 2k and 2k + 1 share one tile and one [B] when their entries fit.
//
// The phase.  The reference reramps with the 144-tap FP64 sum
// Phi = sum_j sum_i kAz[j] kRg[i] phi(y_j, x_i).  With phi = phi_ref(y) +
// G(y, x), phi_ref the deramp phase of the strip's reference column and G
// exactly quadratic in the burst-local time tc (G = g2 tc^2 + g1 tc + g0 per
// column), Phi = (1 + sp) Psi + G2 R2 + G1 R1 + G0 R0, with
//   Psi = sum_j kAz[j] phi_ref(y_j)                   (entry, FP64, reduced)
//   sp  = sum_i kRg[i] - 1, Gk = sum_i kRg[i] gk(x_i)  (column key run)
//   R2 = M0 tc0^2 + 2 tc0 dt M1 + dt^2 M2, R1 = M0 tc0 + dt M1, R0 = M0
//        (entry; M0..M2 the azimuth taps' moments, tc0 = tc(L0)),
// equal to the reference's sum in exact arithmetic.
//
// What bounds it: the latency of each warp's instruction stream (about 7 cycles
// per instruction) with 12 warps per SM: the window, the taps of two columns and
// a row's samples need 168 registers.  Two columns per thread share a line's
// terms, a row's taps and the bookkeeping, and fill the FP32x2 lanes: 110
// thread instructions per pixel, the uniform ones included, where one column
// per thread took 158.  A burst of 1500 x 21000 (one entry per row) 0.462 ->
// 0.292 ms (818 -> 1295 GB/s of 12 bytes per pixel); a burst of 300 x 512 70 ->
// 23 us (short segments: a row costs a lone CTA 0.7 us).  Rows whose strip
// spans several azimuth keys took a per-pixel path from HBM before, columns
// with many range keys a keyed one: a burst of 1539 x 10867 of crossing orbits
// 3.89 -> 0.58 ms.
//
// Which path a pixel takes, and the order of its sums, depend on its row, its
// column and its strip only, never on the work item, so a job that produces a
// subset of the rows gives those rows bit for bit.  The per-pixel path from HBM
// takes rows with more than RS_MAXKEY azimuth runs in the strip or whose entries
// need more than RS_ROWU tile units (a full strip: 56 and about 8 for each run,
// so 9 runs fit), and pixels whose range support leaves the ring.
//
// Precision modes: TOPS_PREC_SPLIT (default) forms each sample's deramp
// phase in FP32 as rho(y) + G(y, x), rho the FP64 reference phase reduced
// once per slave line and G the FP32 quadratic about the burst's centre
// time, both in turns (cycles), so that the sum is reduced exactly by
// t - rint(t) before the sine and cosine.  TOPS_PREC_FP64 evaluates every
// sample's deramp phase and its reduction in FP64.  The reramp phase is
// formed in turns in both modes.  Positions, LUT bins and Psi are FP64 in
// both.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "launch.h"

namespace tops {

constexpr int RS_NT = 64;                  // threads per CTA
constexpr int RS_TW = 112;                 // output columns per strip
constexpr int RS_FW = 128;                 // ring (slave) columns of a strip
constexpr int RS_UN = RS_FW / 2;           // 2-column units of a ring
constexpr int RS_DT = RS_TW / 2;           // range-pass threads per strip
constexpr int RS_H = 6;                    // rows (and pushed lines) per half
constexpr int RS_MAXSEG = 252;             // longest work item
constexpr int RS_CH = 96;                  // rows per chunk
constexpr int RS_NH = RS_CH / RS_H;        // halves per chunk
constexpr int RS_ECAP = 112;               // entries per chunk and strip
constexpr int RS_TU = 2 * RS_H * RS_UN;    // tile units
constexpr int RS_ROWU = RS_TU / RS_H;      // most tile units of a row
constexpr int RS_MAXKEY = 12;              // most entries of a row
constexpr int RS_MAXJOBS = 32;
static_assert(RS_UN == RS_NT, "one unit per thread in the azimuth pass");
static_assert(RS_DT <= RS_NT && RS_CH <= 2 * RS_NT && RS_CH % (2 * RS_H) == 0 &&
                  RS_MAXKEY <= RS_ECAP && RS_TW < 128 && RS_NH <= RS_NT &&
                  RS_CH * RS_MAXKEY * 8 <= RS_TU * 16,
              "thread mappings and table fields assume these sizes");

// A chunk whose run tables end before this many rows is not cut there: columns
// with a full table are keyed behind it.  A shorter chunk prepares and refills
// for each tile what it needs only once per 96 rows; at the line both cost the
// same (300 x 6000, 0.34 keys per row: split chunks of 12 rows 83 us, keyed 86;
// FP64, 4 runs per table, chunks of 9 rows 111 us, keyed 87), and beyond it the
// chunks lose (310 x 25000, 0.55 keys per row: split 417 and 304, FP64 519 and
// 304 us; the kernel before the run tables of a chunk took 333 and 341).  The
// last rows of an item are cut where two chunks hold them: short items pay
// one more prologue for it (300 x 300, 0.55 keys per row, items of 12 rows: 46
// us, keyed 50).
constexpr int kKeyedRows = 2 * RS_H;

enum : int { REG_OUT = 0, REG_EDGE = 1, REG_IN = 2 };
// A half: has interior entries; fills its window anew; has entries off its
// window; shares its tile with the next half; has per-pixel rows; every row is
// one interior entry; and, besides, 6 rows with the window's lines and one bin;
// has keyed rows.
enum : int { HG_ON = 1, HG_FILL = 2, HG_DIRECT = 4, HG_JOIN = 8, HG_PIX = 16, HG_ONE = 32,
             HG_PLAIN = 64, HG_KEY = 128 };
constexpr int E_DIRECT = 4;                // entry flag beside its region

using RsLut = LutPtrs;

struct RsBatch {
  int njobs;
  int total_items;
  int *counter;            // persistent launch: work-item queue (else null)
  ResampleJob jobs[RS_MAXJOBS];
};

// One half of a strip: 6 rows and the 6 lines its window pushes.
struct __align__(16) RsHalf {
  int lb;                  // line of the first row's window
  int flags;
  int tbase;               // first tile unit
  int units;
  short pos[8];            // entries of window position q - 1: [pos[q], pos[q + 1])
};

// Deramp terms of one slave line: the burst-local azimuth time (FP64
// mode), or the reference-column phase in turns and ta - tm (split mode).
union RsSlaveRow {
  double ta;
  struct {
    float rho, tc;
  } f;
};

// Deramp coefficients of the ring columns: G's by unit and, in FP64 mode, the
// FP64 quadratics.
template <bool kSplit>
struct RsRing {
  float2 g2[RS_UN], g1[RS_UN], g0[RS_UN];
  double2 a21[RS_FW];
  double a0[RS_FW];
};
template <>
struct RsRing<true> {
  float2 g2[RS_UN], g1[RS_UN], g0[RS_UN];
};

template <bool kSplit>
struct __align__(16) RsStrip {
  // range-key runs per column and chunk: what 37 KB per CTA leave room for
  static constexpr int kRuns = kSplit ? 5 : 4;
  float4 tile[RS_TU];                 // azimuth-interpolated units
  float run_g[kRuns][3][RS_TW];       // per run: G2, G1, G0
  int2 run_rk[kRuns][RS_TW];          // (chunk row of the next run, key = p0 * 4096 + bin)
  float4 eA[RS_ECAP];                 // entries: reramp terms (rho, psif, R2, R1)
  int4 eM[RS_ECAP];                   // (L0, bin | region << 12 | c_lo << 16 | c_hi << 24, R0,
                                      //  (tile offset & 0xffff) | first unit << 16 | last unit << 24)
  RsHalf half[RS_NH];
  RsSlaveRow srow[RS_NH * RS_H];      // the lines the halves push
  int rowe[RS_CH];                    // first entry | entries << 16 (0 entries: per-pixel row)
  unsigned gen[2 * RS_H][4];          // pixels of the tile's rows left to the per-pixel path
  unsigned missb[RS_NT / 32];         // pairs with rows the pair path left, and the rows
  unsigned short miss[RS_NT];
  int scan[RS_NT / 32];
  RsRing<kSplit> ring;
  double ref_a0, ref_a1, ref_a2, tm;  // reference column's phase, burst centre time
  int xo, dlo, dhi;                   // ring origin, bounds of (ring column - strip column)
  int nfit, cov, gen_any, prev_line;
  int kfrom;                          // first keyed row of the chunk
  int n_border;                       // border columns of the chunk
  unsigned char border[RS_TW];
};

template <bool kSplit>
struct __align__(16) RsShared {
  RsStrip<kSplit> strip;
  uint2 stage[2 * RS_H][RS_NT];       // raw slave lines of the next two halves
  double caz[6], crg[6], shift;
  int next_item;
};

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// Asynchronous global -> shared copies; src_bytes 0 fills zeros.
__device__ __forceinline__ void cp_async_4(unsigned d, const void *src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src),
               "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_8(unsigned d, const void *src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src),
               "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Deramp + demodulation phase (DerampAndResample.cu:151-158), FP64, as the
// quadratic a2 ta^2 + a1 ta + a0 of the burst-local azimuth time ta:
//   -pi kt (ta - tref)^2 - 2 pi fdc ta.
struct DerampQuad {
  double a0, a1, a2;
};
__device__ __forceinline__ DerampQuad deramp_quad(double kt, double tref, double fdc) {
  DerampQuad q;
  q.a2 = -kPi * kt;
  q.a1 = 2.0 * kPi * kt * tref - 2.0 * kPi * fdc;
  q.a0 = -kPi * kt * tref * tref;
  return q;
}
__device__ __forceinline__ double quad_eval(const DerampQuad &q, double ta) {
  return fma(fma(q.a2, ta, q.a1), ta, q.a0);
}
// G = phi - phi_ref about the centre time tm, in turns: (g2, g1, g0).
__device__ __forceinline__ float3 residual_phase(const DerampQuad &q, const DerampQuad &ref,
                                                 double tm) {
  const double d2 = q.a2 - ref.a2, d1 = q.a1 - ref.a1, d0 = q.a0 - ref.a0;
  return make_float3((float)(d2 * kInvTwoPi), (float)((2.0 * d2 * tm + d1) * kInvTwoPi),
                     (float)(((d2 * tm + d1) * tm + d0) * kInvTwoPi));
}
__device__ __forceinline__ double deramp_phase(double ta, double kt, double tref, double fdc) {
  const double e = ta - tref;
  return -kPi * kt * (e * e) - 2.0 * kPi * fdc * ta;
}

// Phases of the split arithmetic are carried in turns (cycles): a turn is
// reduced to [-1/2, 1/2] by t - rint(t), exact for |t| < 2^22, and scaled
// by 2 pi once for the sine and cosine.
constexpr float kTwoPiF = 6.28318530717958647692f;
__device__ __forceinline__ float turns_reduce(float t) { return t - rintf(t); }
// An FP64 phase in radians as turns reduced to [-1/2, 1/2].
__device__ __forceinline__ float to_turns(double phi) {
  const double u = phi * kInvTwoPi;
  return (float)(u - rint(u));
}
// Two phases in turns as reduced phases in radians; t - rint(t) by packed
// adds of 3 2^22, which rounds |t| < 2^22 to the nearest integer as rint does.
__device__ __forceinline__ float2 turns_to_rad2(float2 t) {
  const float2 big = make_float2(12582912.f, 12582912.f);
  const float2 nbig = make_float2(-12582912.f, -12582912.f);
  const float2 m1 = make_float2(-1.f, -1.f);
  const float2 r = __fadd2_rn(__fadd2_rn(t, big), nbig);
  return __fmul2_rn(__ffma2_rn(r, m1, t), make_float2(kTwoPiF, kTwoPiF));
}
// a exp(-i f)
__device__ __forceinline__ float2 cmul_conj(float2 a, float f) {
  float s, c;
  __sincosf(f, &s, &c);
  return make_float2(a.x * c + a.y * s, a.y * c - a.x * s);
}
// a * exp(-i 2 pi t), t in turns
__device__ __forceinline__ float2 cmul_conj_turns(float2 a, float t) {
  return cmul_conj(a, turns_reduce(t) * kTwoPiF);
}

// Integer index and LUT bin of a position (GetIndexes, DerampAndResample.cu:
// 108-112): trunc, then int(frac * 2047 + 0.5) without FMA contraction; the
// bin is clamped as the reference's texture fetch clamps.
__device__ __forceinline__ void split_pos(double v, int &i0, int &bin) {
  i0 = __double2int_rz(v);
  const int b = __double2int_rz(__dadd_rn(__dmul_rn(v - (double)i0, (double)kInterval), 0.5));
  bin = min(max(b, 0), kLutBins - 1);
}

__device__ __forceinline__ int region_1d(int v, int lo, int hi) {
  if (v > hi || v < lo) return REG_OUT;
  return (v > hi - 7 || v < lo + 5) ? REG_EDGE : REG_IN;
}

// my_polyval grouped by row: position = fma(B(row), P^, A(row) + c5 P^2)
// with A = c0 + c1 L^ + c3 L^2 and B = c2 + c4 L^.  Every path of the kernel
// evaluates positions with these functions, so their keys agree bit for bit.
__device__ __forceinline__ double row_L(const ResampleJob &J, int r) {
  return ((double)(r + J.my0) - J.midL) * J.invL;
}
__device__ __forceinline__ double col_P(const ResampleJob &J, int c) {
  return ((double)c - J.midP) * J.invP;
}
__device__ __forceinline__ double row_a(const double *c, double L) {
  return fma(fma(c[3], L, c[1]), L, c[0]);
}
__device__ __forceinline__ double row_b(const double *c, double L) { return fma(c[4], L, c[2]); }
__device__ __forceinline__ double pix_pos(double A, double B, double c5, double P) {
  return fma(B, P, __dadd_rn(A, __dmul_rn(__dmul_rn(c5, P), P)));
}

// Range [lo, hi] of the position over P in [p0, p1]: the ends and, when
// inside, the vertex.  Widened by 1e-9 so that rounding of the per-pixel
// evaluation cannot leave it.
__device__ __forceinline__ void quad_span(double a, double b, double c, double p0, double p1,
                                          double &lo, double &hi) {
  const double f0 = pix_pos(a, b, c, p0), f1 = pix_pos(a, b, c, p1);
  lo = fmin(f0, f1);
  hi = fmax(f0, f1);
  // the vertex lies inside only if the slope changes sign over [p0, p1]
  const double s0 = fma(2.0 * c, p0, b), s1 = fma(2.0 * c, p1, b);
  if ((s0 < 0.0) != (s1 < 0.0)) {
    const double fv = pix_pos(a, b, c, -b / (2.0 * c));
    lo = fmin(lo, fv);
    hi = fmax(hi, fv);
  }
  lo -= 1e-9;
  hi += 1e-9;
}

// Range key (p0 * 4096 + bin) of a row's terms (A, B) and a column's P, and of
// pixel (box row r, P).
__device__ __forceinline__ int rg_key_at(double A, double B, double c5, double P) {
  int p0, b;
  split_pos(pix_pos(A, B, c5, P), p0, b);
  return min(max(p0, -(1 << 19)), (1 << 19) - 1) * 4096 + b;
}
__device__ __forceinline__ int rg_key(const double *crg, const ResampleJob &J, int r, double P) {
  const double L = row_L(J, r);
  return rg_key_at(row_a(crg, L), row_b(crg, L), crg[5], P);
}

// ---------------------------------------------------- HBM slow path
// Per-pixel interior resample straight from the CInt16 slave in HBM (rows
// and pixels the shared passes do not cover).
__device__ __forceinline__ float2 interior_from_global(const ResampleJob &J, int L0, int bL, int P0,
                                                    int bP) {
  const float *kl = J.lut.kaz + bL * kTaps;
  const float *kp = J.lut.krg + bP * kTaps;
  float sre = 0.f, sim = 0.f;
  double ph = 0.0;
#pragma unroll 1
  for (int j = 0; j < kTaps; j++) {
    int y = L0 - 5 + j;
    double ta = (double)(y - J.s_first_line) * J.dt;
    float tre = 0.f, tim = 0.f;
    double tph = 0.0;
#pragma unroll 1
    for (int i = 0; i < kTaps; i++) {
      int x = P0 - 5 + i;
      short2 s = J.slave[(long)(y - J.sy0) * J.slave_pitch + (x - J.sx0)];
      double phi = deramp_phase(ta, J.kt[x], J.tref[x], J.fdc[x]);
      float sn, cs;
      __sincosf(reduce_2pi(phi), &sn, &cs);
      float dre = (float)s.x * cs - (float)s.y * sn;
      float dim = (float)s.x * sn + (float)s.y * cs;
      tre = fmaf(kp[i], dre, tre);
      tim = fmaf(kp[i], dim, tim);
      tph = fma((double)kp[i], phi, tph);
    }
    sre = fmaf(kl[j], tre, sre);
    sim = fmaf(kl[j], tim, sim);
    ph = fma((double)kl[j], tph, ph);
  }
  float s, c;
  __sincosf(reduce_2pi(ph), &s, &c);
  return make_float2(sre * c + sim * s, sim * c - sre * s);
}

// Any pixel (box row r, box column c) by the per-pixel definition.
template <bool kSplit>
__device__ __forceinline__ float2 pixel_generic(const RsShared<kSplit> &S, const ResampleJob &J,
                                                int r, int c) {
  const double L = row_L(J, r), P = col_P(J, c);
  int l0, bl, p0, bp;
  split_pos(pix_pos(row_a(S.caz, L) + S.shift, row_b(S.caz, L), S.caz[5], P), l0, bl);
  split_pos(pix_pos(row_a(S.crg, L), row_b(S.crg, L), S.crg[5], P), p0, bp);
  const int reg = min(region_1d(l0, J.sy0, J.sy1), region_1d(p0, J.sx0, J.sx1));
  if (reg == REG_OUT) return make_float2(0.f, 0.f);
  if (reg == REG_EDGE) {
    const short2 sv = J.slave[(long)(l0 - J.sy0) * J.slave_pitch + (p0 - J.sx0)];
    return make_float2((float)sv.x, (float)sv.y);
  }
  return interior_from_global(J, l0, bl, p0, bp);
}

// The per-pixel rows and the listed pixels of nrows tile rows (chunk rows from
// cr0, box rows from r0 on), all threads; the rows end to end, so that no lane
// idles at the end of each (1000 x 6000, all rows of more than 12 azimuth runs:
// 4670 -> 4270 us).  Out of line: rare, and the other chunks run faster with less
// text (a 9-burst pair 6.92 -> 6.77 ms).
template <bool kSplit>
__device__ __noinline__ void pixel_pass(const RsShared<kSplit> &S, const RsStrip<kSplit> &Q,
                                           const ResampleJob &J, int u, int cr0, int r0, int nrows,
                                           int c0, int cN) {
  int k = 0;
  for (int c = u;; c += RS_NT) {
    for (; c >= cN; c -= cN) k++;
    if (k >= nrows) break;
    const int r = r0 + k;
    if ((Q.rowe[cr0 + k] >> 16) == 0 || ((Q.gen[k][c >> 5] >> (c & 31)) & 1u))
      J.out[(long)(r - J.row0) * J.out_pitch + c0 + c] = pixel_generic(S, J, r, c0 + c);
  }
}

// ---------------------------------------------------- azimuth pass
// Deramp coefficients of a thread's two ring columns.
template <bool kSplit>
struct RingPhase;
template <>
struct RingPhase<true> {
  float2 g2, g1, g0;
};
template <>
struct RingPhase<false> {
  DerampQuad x, y;
};
template <bool kSplit>
__device__ __forceinline__ RingPhase<kSplit> ring_load(const RsStrip<kSplit> &Q, int u) {
  if constexpr (kSplit) {
    return {Q.ring.g2[u], Q.ring.g1[u], Q.ring.g0[u]};
  } else {
    const double2 a = Q.ring.a21[2 * u], b = Q.ring.a21[2 * u + 1];
    return {DerampQuad{Q.ring.a0[2 * u], a.y, a.x}, DerampQuad{Q.ring.a0[2 * u + 1], b.y, b.x}};
  }
}
// Deramp terms of line y.
template <bool kSplit>
__device__ __forceinline__ RsSlaveRow line_terms(const RsStrip<kSplit> &Q, const ResampleJob &J,
                                                 int y) {
  const double ta = (double)(y - J.s_first_line) * J.dt;
  RsSlaveRow sr;
  if (kSplit) {
    const DerampQuad refq = {Q.ref_a0, Q.ref_a1, Q.ref_a2};
    sr.f.rho = to_turns(quad_eval(refq, ta));
    sr.f.tc = (float)(ta - Q.tm);
  } else {
    sr.ta = ta;
  }
  return sr;
}

// Two deramped samples: (re, re') and (im, im').
struct Dpair {
  float2 re, im;
};
template <bool kSplit>
__device__ __forceinline__ Dpair deramp_pair(uint2 raw, RsSlaveRow sr,
                                             const RingPhase<kSplit> &R) {
  const short2 a = *reinterpret_cast<const short2 *>(&raw.x);
  const short2 b = *reinterpret_cast<const short2 *>(&raw.y);
  const float2 sx = make_float2((float)a.x, (float)b.x), sy = make_float2((float)a.y, (float)b.y);
  float2 f;
  if constexpr (kSplit) {
    const float2 tc = make_float2(sr.f.tc, sr.f.tc);
    const float2 G = __ffma2_rn(__ffma2_rn(R.g2, tc, R.g1), tc, R.g0);
    f = turns_to_rad2(__fadd2_rn(make_float2(sr.f.rho, sr.f.rho), G));
  } else {
    f.x = reduce_2pi(quad_eval(R.x, sr.ta));
    f.y = reduce_2pi(quad_eval(R.y, sr.ta));
  }
  float2 sn, cs;
  __sincosf(f.x, &sn.x, &cs.x);
  __sincosf(f.y, &sn.y, &cs.y);
  Dpair d;
  d.re = __ffma2_rn(sx, cs, __fmul2_rn(sy, make_float2(-sn.x, -sn.y)));
  d.im = __ffma2_rn(sx, sn, __fmul2_rn(sy, cs));
  return d;
}

// Raw samples of line y in the ring columns xa, xa + 1 (zeros outside the box).
__device__ __forceinline__ uint2 raw_pair(const ResampleJob &J, int xa, int y) {
  uint2 v = make_uint2(0u, 0u);
  if (y < J.sy0 || y > J.sy1) return v;
  const short2 *p = J.slave + (long)(y - J.sy0) * J.slave_pitch + (xa - J.sx0);
  if (xa >= J.sx0 && xa <= J.sx1) v.x = *reinterpret_cast<const unsigned *>(p);
  if (xa + 1 >= J.sx0 && xa + 1 <= J.sx1) v.y = *reinterpret_cast<const unsigned *>(p + 1);
  return v;
}

// Stages lines y0 .. y0 + 5 into `slot` .. `slot + 5` (zeros outside the box).
template <bool kSplit>
__device__ __forceinline__ void stage_half(RsShared<kSplit> &S, const ResampleJob &J, int u,
                                           int xa, int slot, int y0) {
  const unsigned d = smem_u32(&S.stage[slot][u]);
  constexpr unsigned kRow = RS_NT * sizeof(uint2);
  const bool in0 = xa >= J.sx0 && xa <= J.sx1, in1 = xa + 1 >= J.sx0 && xa + 1 <= J.sx1;
  const long off = (long)(y0 - J.sy0) * J.slave_pitch + (xa - J.sx0);
  if (J.slave_al8 && in0 && in1 && y0 >= J.sy0 && y0 + RS_H - 1 <= J.sy1) {
    const short2 *src = J.slave + off;
#pragma unroll
    for (int k = 0; k < RS_H; k++, src += J.slave_pitch) cp_async_8(d + k * kRow, src, 8);
  } else {
#pragma unroll 1
    for (int k = 0; k < RS_H; k++) {
      const bool yin = y0 + k >= J.sy0 && y0 + k <= J.sy1;
      const long o = off + (long)k * J.slave_pitch;
      const bool i0 = yin && in0, i1 = yin && in1;
      cp_async_4(d + k * kRow, J.slave + (i0 ? o : 0), i0 ? 4 : 0);
      cp_async_4(d + k * kRow + 4, J.slave + (i1 ? o + 1 : 0), i1 ? 4 : 0);
    }
  }
}

// v = sum_j w[j] d[j] of both columns over the window slots (rot + j) % 12;
// even and odd taps in two partial sums.
template <int ROT>
__device__ __forceinline__ float4 az_sum(const float4 (&wz)[6], const Dpair (&w)[12]) {
  float2 ar = make_float2(0.f, 0.f), ai = ar, br = ar, bi = ar;
#pragma unroll
  for (int j = 0; j < kTaps; j += 2) {
    const float2 w0 = make_float2(wz[j >> 1].x, wz[j >> 1].y);
    const float2 w1 = make_float2(wz[j >> 1].z, wz[j >> 1].w);
    const Dpair &d0 = w[(ROT + j) % 12], &d1 = w[(ROT + j + 1) % 12];
    ar = __ffma2_rn(w0, d0.re, ar);
    ai = __ffma2_rn(w0, d0.im, ai);
    br = __ffma2_rn(w1, d1.re, br);
    bi = __ffma2_rn(w1, d1.im, bi);
  }
  const float2 r = __fadd2_rn(ar, br), i = __fadd2_rn(ai, bi);
  return make_float4(r.x, r.y, i.x, i.y);
}

__device__ __forceinline__ void az_taps(float4 (&w)[6], const RsLut &lut, int bin) {
  const float4 *p = lut.kaz2 + bin * (kTaps / 2);
#pragma unroll
  for (int q = 0; q < kTaps / 2; q++) w[q] = __ldg(p + q);
}

// The entries [e0, e1) of one window position.
template <int ROT, bool kSplit>
__device__ __forceinline__ void az_entries(RsStrip<kSplit> &Q, const RsLut &lut, int u, int e0,
                                           int e1, int tbase, const Dpair (&w)[12]) {
#pragma unroll 1
  for (int e = e0; e < e1; e++) {
    const int4 M = Q.eM[e];
    if (((M.y >> 12) & 15) != REG_IN) continue;   // edge, outside, or summed directly
    const int off = (short)(M.w & 0xffff), ulo = (M.w >> 16) & 0xff, uhi = (M.w >> 24) & 0xff;
    if (uhi < (u & ~31) || ulo > (u | 31)) continue;   // none of the warp's columns
    float4 wz[6];
    az_taps(wz, lut, M.y & 0xfff);
    if (u >= ulo && u <= uhi) Q.tile[tbase + off + u] = az_sum<ROT>(wz, w);
  }
}

// The window before the first push of a half anew: lines lb - 6 .. lb + 5.
template <int HALF, bool kSplit>
__device__ __forceinline__ void az_fill(const RsStrip<kSplit> &Q, const ResampleJob &J, int xa,
                                        int lb, const RingPhase<kSplit> &R, Dpair (&w)[12]) {
  uint2 raw[12];
#pragma unroll
  for (int j = 0; j < 12; j++) raw[j] = raw_pair(J, xa, lb - 6 + j);
#pragma unroll
  for (int j = 0; j < 12; j++)
    w[(RS_H * HALF + j + 11) % 12] =
        deramp_pair<kSplit>(raw[j], line_terms<kSplit>(Q, J, lb - 6 + j), R);
}

// One half (number h of the chunk): the window of row k is slots
// (6 HALF + k + j) % 12.  A plain half takes its taps once and one sum per push.
template <int HALF, bool kSplit>
__device__ __forceinline__ void az_half(RsShared<kSplit> &S, RsStrip<kSplit> &Q,
                                        const ResampleJob &J, int u, int xa, int h,
                                        const RsHalf &H, Dpair (&w)[12]) {
  constexpr int R0 = RS_H * HALF;
  const RingPhase<kSplit> R = ring_load<kSplit>(Q, u);
  const RsLut &lut = J.lut;
  const RsSlaveRow *sr = &Q.srow[h * RS_H];
  if (H.flags & HG_FILL) az_fill<HALF, kSplit>(Q, J, xa, H.lb, R, w);
  cp_async_wait<1>();                    // this thread's staged lines of the half
  if (H.flags & HG_PLAIN) {
    float4 wz[6];
    az_taps(wz, lut, Q.eM[H.pos[0]].y & 0xfff);
    float4 *o = &Q.tile[H.tbase + u];
#define RS_PUSH(k)                                                              \
  w[(R0 + (k) + 11) % 12] = deramp_pair<kSplit>(S.stage[R0 + (k)][u], sr[k], R); \
  o[(k) * RS_UN] = az_sum<(R0 + (k)) % 12>(wz, w);
    RS_PUSH(0)
    RS_PUSH(1)
    RS_PUSH(2)
    RS_PUSH(3)
    RS_PUSH(4)
    RS_PUSH(5)
#undef RS_PUSH
    return;
  }
  az_entries<(R0 + 11) % 12, kSplit>(Q, lut, u, H.pos[0], H.pos[1], H.tbase, w);
#define RS_PUSH(k)                                                              \
  w[(R0 + (k) + 11) % 12] = deramp_pair<kSplit>(S.stage[R0 + (k)][u], sr[k], R); \
  az_entries<(R0 + (k)) % 12, kSplit>(Q, lut, u, H.pos[(k) + 1], H.pos[(k) + 2], H.tbase, w);
  RS_PUSH(0)
  RS_PUSH(1)
  RS_PUSH(2)
  RS_PUSH(3)
  RS_PUSH(4)
  RS_PUSH(5)
#undef RS_PUSH
}

// Entries whose line is no window position of their half (the row-to-line
// map skipped or repeated a line): the same sum, in the same order, over
// lines deramped anew.
template <bool kSplit>
__device__ __forceinline__ void az_direct(RsStrip<kSplit> &Q, const ResampleJob &J, int u, int xa,
                                          int tbase, int e0, int e1) {
  const RingPhase<kSplit> R = ring_load<kSplit>(Q, u);
#pragma unroll 1
  for (int e = e0; e < e1; e++) {
    const int4 M = Q.eM[e];
    if (((M.y >> 12) & 15) != (REG_IN | E_DIRECT)) continue;
    const int off = (short)(M.w & 0xffff), ulo = (M.w >> 16) & 0xff, uhi = (M.w >> 24) & 0xff;
    if (u < ulo || u > uhi) continue;
    const float4 *p = J.lut.kaz2 + (M.y & 0xfff) * (kTaps / 2);
    float2 ar = make_float2(0.f, 0.f), ai = ar, br = ar, bi = ar;
#pragma unroll 1
    for (int j = 0; j < kTaps; j += 2) {
      const float4 q = __ldg(p + (j >> 1));
      const int y = M.x - 5 + j;
      const Dpair d0 = deramp_pair<kSplit>(raw_pair(J, xa, y), line_terms<kSplit>(Q, J, y), R);
      const Dpair d1 =
          deramp_pair<kSplit>(raw_pair(J, xa, y + 1), line_terms<kSplit>(Q, J, y + 1), R);
      ar = __ffma2_rn(make_float2(q.x, q.y), d0.re, ar);
      ai = __ffma2_rn(make_float2(q.x, q.y), d0.im, ai);
      br = __ffma2_rn(make_float2(q.z, q.w), d1.re, br);
      bi = __ffma2_rn(make_float2(q.z, q.w), d1.im, bi);
    }
    const float2 r = __fadd2_rn(ar, br), i = __fadd2_rn(ai, bi);
    Q.tile[tbase + off + u] = make_float4(r.x, r.y, i.x, i.y);
  }
}

// ---------------------------------------------------- range pass
// Taps from unit boundaries: samples of units U[0..5], weights w[0..11].
template <int N>
__device__ __forceinline__ float2 rg_sum(const float4 (&w)[(N + 1) / 2], const float4 *U) {
  float2 re = make_float2(0.f, 0.f), im = re;
#pragma unroll
  for (int m = 0; m < N; m++) {
    const float2 ww = (m & 1) ? make_float2(w[m >> 1].z, w[m >> 1].w)
                              : make_float2(w[m >> 1].x, w[m >> 1].y);
    re = __ffma2_rn(ww, make_float2(U[m].x, U[m].y), re);
    im = __ffma2_rn(ww, make_float2(U[m].z, U[m].w), im);
  }
  return make_float2(re.x + re.y, im.x + im.y);
}

__device__ __forceinline__ void taps_even(float4 (&w)[3], const RsLut &lut, int bin) {
  const float4 *p = reinterpret_cast<const float4 *>(lut.krg) + bin * 3;
#pragma unroll
  for (int q = 0; q < 3; q++) w[q] = __ldg(p + q);
}
__device__ __forceinline__ void taps_odd(float4 (&w)[4], const RsLut &lut, int bin) {
  const float4 *p = lut.krgo + bin * 4;
#pragma unroll
  for (int q = 0; q < 4; q++) w[q] = __ldg(p + q);
}

// Reramp phase of a pixel in turns: (1 + sp) Psi + G2 R2 + G1 R1 + G0 R0, with
// Psi as its reduced value plus sp times its float value.  A: (rho, psif, R2,
// R1), g: (sp, G2, G1, G0).
__device__ __forceinline__ float run_phase(float4 A, float R0, float4 g) {
  return fmaf(g.x, A.y, A.x) + fmaf(g.y, A.z, fmaf(g.z, A.w, g.w * R0));
}

// The current runs of a thread's two output columns, kept over a chunk's tiles.
struct PairRuns {
  float4 gx, gy;         // pair: the columns' terms
  float4 we[3], wo[4];   // pair: taps of the even-aligned and of the odd column
  int next;              // chunk row of either column's next run
  int unit;              // first tile unit of the 14 samples; -1: no pair (the
                         // columns' samples are not adjacent or leave the ring)
  int m;                 // run numbers, first | second << 8
  bool odd;              // the first column is the odd-aligned one
  bool vec;              // both columns range-interior, outputs 16-byte aligned
  int in;                // range-interior columns: 1 the first, 2 the second
};

// The key of a column's last run where its table is full: the rows from there on
// are keyed, each pixel by its own key (the bin is no LUT bin).
constexpr int kKeyed = -(1 << 19) * 4096 + 4095;

// Ring column of a key's first tap when its 14 samples are inside the ring,
// else -1.
__device__ __forceinline__ int ring_col(int xo, int key) {
  const unsigned xb = (unsigned)(key >> 12) - 5u - (unsigned)xo;
  return xb < RS_FW - 13 ? (int)xb : -1;
}
__device__ __forceinline__ bool range_in(const ResampleJob &J, int key) {
  const int p0 = key >> 12;
  return p0 >= J.sx0 + 5 && p0 <= J.sx1 - 7;
}

// A run's terms with sp = sum_i kRg[i] - 1: (sp, G2, G1, G0).
template <bool kSplit>
__device__ __forceinline__ float4 run_load(const RsStrip<kSplit> &Q, const RsLut &lut, int m,
                                           int c, int key) {
  return make_float4(__ldg(lut.sp1 + (key & 4095)), Q.run_g[m][0][c], Q.run_g[m][1][c],
                     Q.run_g[m][2][c]);
}

// Residual-phase terms (G2, G1, G0), Gk = sum_i kRg[i] gk(x_i), of the taps that
// start at element OFF of w and ring column xb.
template <int OFF, bool kSplit, int N>
__device__ __forceinline__ float3 taps_terms(const RsStrip<kSplit> &Q, const float4 (&w)[N],
                                             int xb) {
  const float *g2 = reinterpret_cast<const float *>(Q.ring.g2) + xb;
  const float *g1 = reinterpret_cast<const float *>(Q.ring.g1) + xb;
  const float *g0 = reinterpret_cast<const float *>(Q.ring.g0) + xb;
  float3 G = make_float3(0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kTaps; i++) {
    const int j = i + OFF;
    const float4 q = w[j >> 2];
    const float t = (j & 3) == 0 ? q.x : (j & 3) == 1 ? q.y : (j & 3) == 2 ? q.z : q.w;
    G.x = fmaf(t, g2[i], G.x);
    G.y = fmaf(t, g1[i], G.y);
    G.z = fmaf(t, g0[i], G.z);
  }
  return G;
}
// Those of a range key (0 when its taps leave the ring).
template <bool kSplit>
__device__ __forceinline__ float3 key_terms(const RsStrip<kSplit> &Q, const RsLut &lut, int key) {
  const unsigned xb = (unsigned)(key >> 12) - 5u - (unsigned)Q.xo;
  if (xb > RS_FW - kTaps) return make_float3(0.f, 0.f, 0.f);
  float4 w[3];
  taps_even(w, lut, key & 4095);
  return taps_terms<0, kSplit>(Q, w, xb);
}

// Moves the runs on to chunk row `row`.
template <bool kSplit>
__device__ __forceinline__ void next_runs(PairRuns &P, const RsStrip<kSplit> &Q,
                                          const ResampleJob &J, int c, bool two, int row) {
  int mx = P.m & 0xff, my = P.m >> 8;
  int2 rx = Q.run_rk[mx][c];
  int2 ry = two ? Q.run_rk[my][c + 1] : make_int2(INT32_MAX, 0);
  while (row >= rx.x) rx = Q.run_rk[++mx][c];
  while (row >= ry.x) ry = Q.run_rk[++my][c + 1];
  P.m = mx | my << 8;
  P.next = min(rx.x, ry.x);
  const int xb = ring_col(Q.xo, rx.y);
  P.in = (range_in(J, rx.y) ? 1 : 0) | (two && range_in(J, ry.y) ? 2 : 0);
  P.vec = P.in == 3 && J.out_al16;
  P.unit = -1;
  if (two && xb >= 0 && ring_col(Q.xo, ry.y) == xb + 1) {
    const bool odd = (xb & 1) != 0;
    P.odd = odd;
    P.unit = xb >> 1;
    taps_even(P.we, J.lut, (odd ? ry.y : rx.y) & 4095);
    taps_odd(P.wo, J.lut, (odd ? rx.y : ry.y) & 4095);
    P.gx = run_load(Q, J.lut, mx, c, rx.y);
    P.gy = run_load(Q, J.lut, my, c + 1, ry.y);
  }
}

// Both columns of a pair in one row: U the units of its 14 samples, A and R0
// the entry's reramp terms.  Border columns are not stored.
__device__ __forceinline__ void pair_row(const PairRuns &P, const float4 *U, float4 A, float R0,
                                         float2 *o) {
  float4 V[7];
#pragma unroll
  for (int m = 0; m < 7; m++) V[m] = U[m];
  const float2 f = turns_to_rad2(make_float2(run_phase(A, R0, P.gx), run_phase(A, R0, P.gy)));
  float2 vx, vy;
  if (P.odd) {
    vx = rg_sum<7>(P.wo, V);
    vy = rg_sum<6>(P.we, V + 1);
  } else {
    vx = rg_sum<6>(P.we, V);
    vy = rg_sum<7>(P.wo, V);
  }
  vx = cmul_conj(vx, f.x);
  vy = cmul_conj(vy, f.y);
  if (P.vec) {
    *reinterpret_cast<float4 *>(o) = make_float4(vx.x, vx.y, vy.x, vy.y);
  } else {
    if (P.in & 1) o[0] = vx;
    if (P.in & 2) o[1] = vy;
  }
}

// A pixel off the slave box's interior: 0 outside, the nearest sample at the
// edge.
__device__ __forceinline__ float2 border_pixel(const ResampleJob &J, int reg, int L0, int p0) {
  reg = min(reg, region_1d(p0, J.sx0, J.sx1));
  if (reg == REG_OUT) return make_float2(0.f, 0.f);
  const short2 sv = J.slave[(long)(L0 - J.sy0) * J.slave_pitch + (p0 - J.sx0)];
  return make_float2((float)sv.x, (float)sv.y);
}

// One pixel (chunk row k, strip column c; its range key and the key's terms) of a
// shared row outside the pair path.
template <bool kSplit>
__device__ __forceinline__ void pixel_shared(RsStrip<kSplit> &Q, const ResampleJob &J, int k,
                                             int tbase, int kt, int c, int key, float4 g,
                                             float2 *out) {
  const int re = Q.rowe[k], ne = re >> 16;
  int e = re & 0xffff;
  for (int q = 1; q < ne; q++, e++) {
    const int z = Q.eM[e].y;
    if (c >= ((z >> 16) & 0xff) && c < ((z >> 24) & 0xff)) break;
  }
  const int4 M = Q.eM[e];
  const int p0 = key >> 12;
  const int reg = (M.y >> 12) & 3;
  if (min(reg, region_1d(p0, J.sx0, J.sx1)) != REG_IN) {
    *out = border_pixel(J, reg, M.x, p0);
    return;
  }
  const int xb = ring_col(Q.xo, key);
  const int ulo = (M.w >> 16) & 0xff, uhi = (M.w >> 24) & 0xff;
  if (xb < 0 || (xb >> 1) < ulo || ((xb + 12) >> 1) > uhi) {
    atomicOr(&Q.gen[kt][c >> 5], 1u << (c & 31));
    Q.gen_any = 1;
    return;
  }
  const float4 *U = &Q.tile[tbase + (short)(M.w & 0xffff) + (xb >> 1)];
  float2 v;
  if (xb & 1) {
    float4 w[4];
    taps_odd(w, J.lut, key & 4095);
    v = rg_sum<7>(w, U);
  } else {
    float4 w[3];
    taps_even(w, J.lut, key & 4095);
    v = rg_sum<6>(w, U);
  }
  *out = cmul_conj_turns(v, run_phase(Q.eA[e], __int_as_float(M.z), g));
}

// A pair of columns (strip columns c, c + 1) in chunk row k with range keys kx, ky.
template <bool kSplit>
__device__ __forceinline__ void keyed_pair(RsStrip<kSplit> &Q, const ResampleJob &J, int k, int c,
                                           int cN, int kx, int ky, int tbase, int kt, float2 *o) {
  const bool two = c + 1 < cN;
  const int re = Q.rowe[k], ne = re >> 16;
  if (ne == 0) return;                   // a per-pixel row
  int e = re & 0xffff;
  int4 M = Q.eM[e];
  for (int q = 1; q < ne && !(c >= ((M.y >> 16) & 0xff) && c < ((M.y >> 24) & 0xff)); q++)
    M = Q.eM[++e];
  const int xb = ring_col(Q.xo, kx), unit = xb >> 1;
  PairRuns P;
  P.in = (range_in(J, kx) ? 1 : 0) | (two && range_in(J, ky) ? 2 : 0);
  if (P.in == 3 && ((M.y >> 12) & 3) == REG_IN && c + 1 < ((M.y >> 24) & 0xff) && xb >= 0 &&
      ring_col(Q.xo, ky) == xb + 1 && unit >= ((M.w >> 16) & 0xff) &&
      unit + 6 <= ((M.w >> 24) & 0xff)) {
    P.vec = J.out_al16;
    P.odd = (xb & 1) != 0;
    taps_even(P.we, J.lut, (P.odd ? ky : kx) & 4095);
    taps_odd(P.wo, J.lut, (P.odd ? kx : ky) & 4095);
    const float3 ge = taps_terms<0, kSplit>(Q, P.we, P.odd ? xb + 1 : xb);
    const float3 go = taps_terms<1, kSplit>(Q, P.wo, P.odd ? xb : xb + 1);
    const float3 gx = P.odd ? go : ge, gy = P.odd ? ge : go;
    P.gx = make_float4(__ldg(J.lut.sp1 + (kx & 4095)), gx.x, gx.y, gx.z);
    P.gy = make_float4(__ldg(J.lut.sp1 + (ky & 4095)), gy.x, gy.y, gy.z);
    pair_row(P, &Q.tile[tbase + (short)(M.w & 0xffff) + unit], Q.eA[e], __int_as_float(M.z), o);
    return;
  }
#pragma unroll 1
  for (int q = 0; q < (two ? 2 : 1); q++) {
    const int key = q ? ky : kx;
    const float3 g = key_terms<kSplit>(Q, J.lut, key);
    pixel_shared(Q, J, k, tbase, kt, c + q, key,
                 make_float4(__ldg(J.lut.sp1 + (key & 4095)), g.x, g.y, g.z), o + q);
  }
}

// The range pass of chunk rows [ka, k1) of the tile that starts at row k0 with
// each pixel's key found anew, all threads.  From row ks on the entries' tile
// starts at tb1.
template <bool kSplit>
__device__ __forceinline__ void keyed_pairs(const ResampleJob &J, int rb, int k0, int ka, int k1,
                                         int ks, int tb1, int c0, int cN) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RsShared<kSplit> &S = *reinterpret_cast<RsShared<kSplit> *>(smem_raw);
  RsStrip<kSplit> &Q = S.strip;
  const int np = (cN + 1) / 2;
  int k = ka, c = 2 * (int)threadIdx.x;
  auto in_row = [&]() {                  // (k, c) of the pairs end to end
    for (; c >= 2 * np; c -= 2 * np) k++;
  };
  auto keys = [&]() {
    const double L = row_L(J, rb + k);
    const double A = row_a(S.crg, L), B = row_b(S.crg, L);
    return make_int2(rg_key_at(A, B, S.crg[5], col_P(J, c0 + c)),
                     rg_key_at(A, B, S.crg[5], col_P(J, c0 + c + 1)));
  };
  in_row();
  int2 next = keys();
  while (k < k1) {
    const int kx = next.x, ky = next.y, kr = k, cc = c;
    c += 2 * RS_NT;
    in_row();
    next = keys();                       // the next pair's, while this one's loads run
    keyed_pair<kSplit>(Q, J, kr, cc, cN, kx, ky, kr >= ks ? tb1 : 0, kr - k0,
                       J.out + (long)(rb + kr - J.row0) * J.out_pitch + c0 + cc);
  }
}

// The border pixels of a chunk's columns listed in Q.border (those off the
// range interior in some row): all rows at once, so that their loads overlap.
template <bool kSplit>
__device__ __forceinline__ void border_columns(const RsStrip<kSplit> &Q, const ResampleJob &J,
                                               int u, int n, float2 *obase) {
  const int nb = Q.n_border;
#pragma unroll 4
  for (int v = u; v < nb * n; v += RS_NT) {
    const int k = v / nb, c = Q.border[v - k * nb];
    const int re = Q.rowe[k], ne = re >> 16;
    if (ne == 0) continue;               // a per-pixel row
    int e = re & 0xffff;
    for (int q = 1; q < ne; q++, e++) {
      const int z = Q.eM[e].y;
      if (c >= ((z >> 16) & 0xff) && c < ((z >> 24) & 0xff)) break;
    }
    int m = 0;
    while (k >= Q.run_rk[m][c].x) m++;
    const int key = Q.run_rk[m][c].y;
    if (range_in(J, key) || key == kKeyed) continue;
    const int4 M = Q.eM[e];
    obase[(long)k * J.out_pitch + c] = border_pixel(J, (M.y >> 12) & 3, M.x, key >> 12);
  }
}

// The pixels the pair path left, all threads: pairs with a row in
// Q.miss, nrows tile rows from chunk row k0 on; from row ks on the entries'
// tile starts at tb1.  obase: the output at chunk row k0, strip column 0.
template <bool kSplit>
__device__ __forceinline__ void slow_pixels(RsStrip<kSplit> &Q, const ResampleJob &J, int u0,
                                            int k0, int nrows, int ks, int tb1, int cN,
                                            float2 *obase) {
  const int n0 = __popc(Q.missb[0]), np = n0 + __popc(Q.missb[1]);
  const int per = 2 * nrows;
  for (int v = u0; v < np * per; v += RS_NT) {
    int i = v / per;
    const int w = v - i * per, q = w >> 1;
    const int wq = i >= n0 ? 1 : 0;
    if (wq) i -= n0;
    unsigned m = Q.missb[wq];
    while (i-- > 0) m &= m - 1;
    const int uu = wq * 32 + __ffs(m) - 1;   // the pair's thread
    const int c = 2 * uu + (w & 1);
    if (c < cN && ((Q.miss[uu] >> q) & 1)) {
      int m = 0;
      while (k0 + q >= Q.run_rk[m][c].x) m++;
      const int key = Q.run_rk[m][c].y;
      if (key == kKeyed) continue;
      pixel_shared(Q, J, k0 + q, k0 + q >= ks ? tb1 : 0, q, c, key, run_load(Q, J.lut, m, c, key),
                   obase + (long)q * J.out_pitch + c);
    }
  }
}

// ---------------------------------------------------- chunk prologue
// Walks the azimuth-key runs of a row along the strip's columns, in the
// direction of ascending lines: emit(region, line, bin, c_lo, c_hi), until it
// returns false.
template <bool kSplit, class Emit>
__device__ __forceinline__ void walk_row(const RsShared<kSplit> &S, const ResampleJob &J, int r,
                                         int c0, int cN, Emit emit) {
  const double L = row_L(J, r);
  const double A = row_a(S.caz, L) + S.shift, B = row_b(S.caz, L), C = S.caz[5];
  const double pa = col_P(J, c0), pb = col_P(J, c0 + cN - 1);
  int base;                              // the row's lowest line inside the box
  {
    // the whole strip in one run?
    double ylo, yhi;
    quad_span(A, B, C, pa, pb, ylo, yhi);
    int l0, b0, l1, b1;
    split_pos(ylo, l0, b0);
    split_pos(yhi, l1, b1);
    const int g0 = region_1d(l0, J.sy0, J.sy1), g1 = region_1d(l1, J.sy0, J.sy1);
    if (g0 == g1 && ((l0 == l1 && (b0 == b1 || g0 == REG_EDGE)) ||
                     (g0 == REG_OUT && (l0 > J.sy1 || l1 < J.sy0)))) {
      emit(g0, l0, b0, 0, cN);
      return;
    }
    base = max(l0, J.sy0);
    if ((long)min(l1, J.sy1) - base >= 1 << 18) {   // more than a key holds: a per-pixel row
      while (emit(REG_OUT, 0, 0, 0, cN)) {
      }
      return;
    }
  }
  // key of column c, ascending with the position: before the box -1, edge
  // (line, 4095), interior (line, bin), past the box INT32_MAX; lines relative
  // to the row's lowest, since a box may have more than 2^19
  auto key = [&](int c) -> int {
    int l, b;
    split_pos(pix_pos(A, B, C, col_P(J, c0 + c)), l, b);
    const int g = region_1d(l, J.sy0, J.sy1);
    if (g == REG_OUT) return l < J.sy0 ? -1 : INT32_MAX;
    return (l - base) * 4096 + (g == REG_EDGE ? 4095 : b);
  };
  // monotone pieces: split at the vertex
  const double s0 = fma(2.0 * C, pa, B), s1 = fma(2.0 * C, pb, B);
  int vert = cN - 1;
  if ((s0 < 0.0) != (s1 < 0.0)) {
    const double v = (-B / (2.0 * C)) / J.invP + J.midP - (double)c0;
    if (v >= 0.0 && v < (double)(cN - 1)) vert = (int)v;
  }
  const bool rev = pix_pos(A, B, C, pb) < pix_pos(A, B, C, pa);
  auto at = [&](int i) { return key(rev ? cN - 1 - i : i); };
  int cur = -2, from = 0;
  auto put = [&](int k, int i0, int i1) -> bool {   // run [i0, i1) of key k
    const int c_lo = rev ? cN - i1 : i0, c_hi = rev ? cN - i0 : i1;
    if (k == -1 || k == INT32_MAX) return emit(REG_OUT, 0, 0, c_lo, c_hi);
    return emit((k & 4095) == 4095 ? REG_EDGE : REG_IN, base + (k >> 12), k & 4095, c_lo, c_hi);
  };
  const int split = rev ? cN - 2 - vert : vert;   // last index of the first piece
  int i = 0;
#pragma unroll 1
  for (int piece = 0; piece < 2; piece++) {
    const int end = (piece == 0 && split >= 0) ? split : cN - 1;
    if (i > end) continue;
    int k = at(i);
    const int kb = at(end);
    for (;;) {
      if (k != cur) {
        if (cur != -2 && !put(cur, from, i)) return;
        cur = k;
        from = i;
      }
      if (k == kb) break;   // monotone: the rest of the piece has this key
      int lo = i, hi = end, khi = kb;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        const int km = at(mid);
        if (km == k) {
          lo = mid;
        } else {
          hi = mid;
          khi = km;
        }
      }
      i = hi;
      k = khi;
    }
    i = end + 1;
  }
  put(cur, from, cN);
}

// Ring units of output columns [c_lo, c_hi), from the strip's bounds of
// (ring column - strip column); at least one, whatever the bounds are (those of
// positions that spread over 2^31 samples overflow), so that the tile offsets of
// a half's entries ascend from 0.
template <bool kSplit>
__device__ __forceinline__ void entry_units(const RsStrip<kSplit> &Q, int c_lo, int c_hi, int &ulo,
                                            int &uhi) {
  ulo = min(max(c_lo + Q.dlo, 0), RS_FW - 1) >> 1;
  uhi = max(min(max(c_hi - 1 + Q.dhi + 13, 0), RS_FW - 1) >> 1, ulo);
}

// [P4] A row's entries, to `out` (at most RS_MAXKEY): (line, bin | region << 12 |
// c_lo << 16 | c_hi << 24).  Returns their number, 0 for a per-pixel row.
template <bool kSplit>
__device__ __forceinline__ int find_entries(const RsShared<kSplit> &S, const RsStrip<kSplit> &Q,
                                            const ResampleJob &J, int r, int c0, int cN,
                                            int2 *out) {
  int m = 0, units = 0;
  walk_row(S, J, r, c0, cN, [&](int reg, int L0, int bin, int c_lo, int c_hi) -> bool {
    if (m < RS_MAXKEY) out[m] = make_int2(L0, bin | reg << 12 | c_lo << 16 | c_hi << 24);
    m++;
    if (reg == REG_IN) {
      int ulo, uhi;
      entry_units(Q, c_lo, c_hi, ulo, uhi);
      units += uhi - ulo + 1;
    }
    return m <= RS_MAXKEY;
  });
  return (m > RS_MAXKEY || (m > 1 && units > RS_ROWU)) ? 0 : m;
}

// Reramp terms of the azimuth key (L0, bin): Psi = sum_j kAz[j]
// phi_ref(L0 - 5 + j) (FP64) and the taps' moments about the burst centre
// time, as (rho, psif, R2, R1) and R0.
template <bool kSplit>
__device__ __forceinline__ float4 row_terms(const RsStrip<kSplit> &Q, const ResampleJob &J, int L0,
                                            int bin, float &R0) {
  const DerampQuad refq = {Q.ref_a0, Q.ref_a1, Q.ref_a2};
  const float *kl = J.lut.kaz + bin * kTaps;
  double psi = 0.0, m0 = 0.0, m1 = 0.0, m2 = 0.0;
  const double n0 = (double)(L0 - 5 - J.s_first_line);
#pragma unroll
  for (int j = 0; j < kTaps; j++) {
    const double w = (double)__ldg(kl + j), u = (double)(j - 5);
    const double ta = (n0 + (double)j) * J.dt;
    psi = fma(w, quad_eval(refq, ta), psi);
    m0 += w;
    m1 = fma(w, u, m1);
    m2 = fma(w, u * u, m2);
  }
  const double tc0 = (double)(L0 - J.s_first_line) * J.dt - Q.tm;
  const double dt = J.dt;
  R0 = (float)m0;
  return make_float4(to_turns(psi), (float)(psi * kInvTwoPi),
                     (float)(m0 * tc0 * tc0 + 2.0 * tc0 * dt * m1 + dt * dt * m2),
                     (float)(m0 * tc0 + dt * m1));
}

// [P5] An entry, with the reramp terms of its key.
template <bool kSplit>
__device__ __forceinline__ void write_entry(RsStrip<kSplit> &Q, const ResampleJob &J, int2 E,
                                            int cN, int e) {
  const int c_lo = (E.y >> 16) & 0xff, c_hi = (E.y >> 24) & 0xff;
  int ulo = 0, uhi = RS_UN - 1;
  if (c_hi - c_lo < cN) entry_units(Q, c_lo, c_hi, ulo, uhi);
  float R0 = 0.f;
  if (((E.y >> 12) & 15) == REG_IN) Q.eA[e] = row_terms(Q, J, E.x, E.y & 0xfff, R0);
  Q.eM[e] = make_int4(E.x, E.y, __float_as_int(R0), ulo << 16 | uhi << 24);
}

// The terms of a column's run.
template <bool kSplit>
__device__ __forceinline__ void run_terms(RsStrip<kSplit> &Q, const RsLut &lut, int m, int c,
                                          int key) {
  const float3 G = key_terms<kSplit>(Q, lut, key);
  Q.run_g[m][0][c] = G.x;
  Q.run_g[m][1][c] = G.y;
  Q.run_g[m][2][c] = G.z;
}
// [P6] The runs of column c's range key over chunk rows [0, n) (box rows rb
// ...).  Most columns hold one key: when the position is monotone over the
// rows and both ends agree (k0, k1 from the caller).  Else by bisection of the
// exact per-pixel key on the pieces where the position is monotone in the row;
// rows from the first change that does not fit the table on are left to the
// next chunk (Q.cov).
template <bool kSplit>
__device__ __forceinline__ bool build_runs(const RsShared<kSplit> &S, RsStrip<kSplit> &Q,
                                           const ResampleJob &J, int rb, int n, int c0, int c,
                                           bool mono, int ka, int kz) {
  run_terms(Q, J.lut, 0, c, ka);
  if (mono && ka == kz) {
    Q.run_rk[0][c] = make_int2(INT32_MAX, ka);
    return false;
  }
  const double P = col_P(J, c0 + c);
  auto keyat = [&](int ri) { return rg_key(S.crg, J, rb + ri, P); };
  int split = n - 1;                     // last row of the first piece
  if (!mono) {
    // x(L) = g0 + g2 P + g5 P^2 + (g1 + g4 P) L + g3 L^2: vertex in L
    const double *g = S.crg;
    const double Lv = -(g[1] + g[4] * P) / (2.0 * g[3]);
    const double rv = Lv / J.invL + J.midL - (double)J.my0 - (double)rb;
    if (rv > 0.0 && rv < (double)(n - 1)) split = (int)rv;
  }
  int m = 0, key = ka, from = 0;
  for (int pc = 0; pc < 2; pc++) {
    const int bend = pc == 0 ? split : n - 1;
    if (from > bend) continue;
    int r = from, k = pc == 0 ? ka : keyat(r);
    const int kb = bend == n - 1 ? kz : keyat(bend);
    for (;;) {
      if (k != key) {
        // run m ends here; is there room for the next?
        Q.run_rk[m][c] = make_int2(r, key);
        m++;
        if (m == RsStrip<kSplit>::kRuns) {
          atomicMin(&Q.cov, r);
          return true;
        }
        run_terms(Q, J.lut, m, c, k);
        key = k;
      }
      if (k == kb) break;   // monotone: the rest of the piece has this key
      int lo = r, hi = bend, khi = kb;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        const int km = keyat(mid);
        if (km == k) {
          lo = mid;
        } else {
          hi = mid;
          khi = km;
        }
      }
      r = hi;
      k = khi;
    }
    from = bend + 1;
  }
  Q.run_rk[m][c] = make_int2(INT32_MAX, key);
  return false;
}

// [P7] Half h of a chunk of n rows: its window's lines, the entries of each
// window position, tile offsets.
template <bool kSplit>
__device__ __forceinline__ void plan_half(RsStrip<kSplit> &Q, int h, int n) {
  RsHalf H;
  H.flags = 0;
  H.lb = 0;
  H.tbase = 0;
  H.units = 0;
  const int r0 = h * RS_H, r1 = min(r0 + RS_H, n);
  if (r1 - r0 == RS_H) {
    // the usual half: one interior entry per row, consecutive lines, one bin
    int re[RS_H];
    int2 M[RS_H];
    bool plain = true;
#pragma unroll
    for (int k = 0; k < RS_H; k++) re[k] = Q.rowe[r0 + k];
    const int e0 = re[0] & 0xffff;
#pragma unroll
    for (int k = 0; k < RS_H; k++) {
      plain = plain && re[k] >> 16 == 1;
      M[k] = *reinterpret_cast<const int2 *>(&Q.eM[min(e0 + k, RS_ECAP - 1)]);
    }
#pragma unroll
    for (int k = 0; k < RS_H; k++)
      plain = plain && ((M[k].y >> 12) & 15) == REG_IN && M[k].x == M[0].x + k &&
              (M[k].y & 0xfff) == (M[0].y & 0xfff);
    if (plain) {
      H.flags = HG_ON | HG_ONE | HG_PLAIN;
      H.lb = M[0].x;
      H.units = RS_H * RS_UN;
#pragma unroll
      for (int k = 0; k < 8; k++) H.pos[k] = (short)(e0 + min(max(k - 1, 0), RS_H));
#pragma unroll
      for (int k = 0; k < RS_H; k++) Q.eM[e0 + k].w = k * RS_UN | (RS_UN - 1) << 24;
      Q.half[h] = H;
      return;
    }
  }
  for (int r = r0; r < r1 && !(H.flags & HG_ON); r++) {
    const int re = Q.rowe[r], e0 = re & 0xffff, ne = re >> 16;
    for (int e = e0; e < e0 + ne; e++)
      if (((Q.eM[e].y >> 12) & 15) == REG_IN) {
        H.flags |= HG_ON;
        H.lb = Q.eM[e].x - (r - r0);   // the row's last (highest) line
      }
  }
  int cur = -1, end = Q.rowe[r0] & 0xffff;
  bool one = true;
  H.pos[0] = (short)end;
  for (int r = r0; r < r1; r++) {
    const int re = Q.rowe[r], e0 = re & 0xffff, ne = re >> 16;
    if (ne == 0) H.flags |= HG_PIX;
    one = one && ne == 1 && ((Q.eM[e0].y >> 12) & 15) == REG_IN;
    for (int e = e0; e < e0 + ne; e++) {
      int4 M = Q.eM[e];
      if (((M.y >> 12) & 15) == REG_IN) {
        const int ulo = (M.w >> 16) & 0xff, uhi = (M.w >> 24) & 0xff;
        const int p = M.x - H.lb;
        if (p < cur || p >= RS_H) {
          M.y |= E_DIRECT << 12;
          H.flags |= HG_DIRECT;
        } else {
          for (; cur < p; cur++) H.pos[cur + 2] = (short)e;
        }
        M.w = (M.w & ~0xffff) | ((H.units - ulo) & 0xffff);
        H.units += uhi - ulo + 1;
        Q.eM[e] = M;
      }
      end = e + 1;
    }
  }
  for (; cur < RS_H; cur++) H.pos[cur + 2] = (short)end;
  if (one) H.flags |= HG_ONE;
  Q.half[h] = H;
}

// One work item (strip x segment of one job); all threads of the CTA call it
// with the same item.
template <bool kSplit>
__device__ __forceinline__ void resample_item(RsShared<kSplit> &S, const RsBatch &B, int item) {
  const int u = threadIdx.x;
  RsStrip<kSplit> &Q = S.strip;
  constexpr int kRuns = RsStrip<kSplit>::kRuns;

  // ---- locate the work item (job, strip, segment)
  int jb = 0;
  while (jb + 1 < B.njobs && B.jobs[jb + 1].item_begin <= item) jb++;
  const ResampleJob &J = B.jobs[jb];
  const int local = item - J.item_begin;
  const int seg = local / J.strips;
  const int c0 = (local - seg * J.strips) * RS_TW;
  const int cN = min(RS_TW, J.mx1 - J.mx0 + 1 - c0);
  const int r_begin = J.row0 + seg * J.seg_rows;
  const int nr = min(J.seg_rows, J.row0 + J.nrows - r_begin);

  // ---- [P1] polynomials and shift
  if (u < 12) {
    const double v = J.cpm_dev ? J.cpm_dev[u] : (u < 6 ? J.caz[u] : J.crg[u - 6]);
    if (u < 6)
      S.caz[u] = v;
    else
      S.crg[u - 6] = v;
  }
  if (u == 12) {
    double sh = J.az_shift;
    if (J.az_shift_dev) {
      // a device-provided ESD shift above 100 px is invalid and reset to 0,
      // as the reference driver does (Func.cpp:2612-2621)
      sh = *J.az_shift_dev;
      if (!(fabs(sh) <= 100.0)) sh = 0.0;
    }
    S.shift = sh;
  }
  if (u < 2 * RS_H * 4) (&Q.gen[0][0])[u] = 0u;
  __syncthreads();

  // ---- [P2] the ring's origin, the bounds of (ring column - strip column)
  // and the reference column, from the range position at the corners and edge
  // midpoints of the strip over the whole master box: they depend on the strip
  // only, so a job that produces a subset of the rows gives those rows bit for
  // bit as the whole job does.
  if (u == 0) {
    double pmin = 1e300, dmin = 1e300, dmax = -1e300;
    const int box_rows = J.my1 - J.my0 + 1;
    for (int a = 0; a < 3; a++) {
      const int rr = (a == 0) ? 0 : (a == 1 ? (box_rows - 1) / 2 : box_rows - 1);
      const double L = row_L(J, rr);
      for (int b = 0; b < 3; b++) {
        const int cc = (b == 0) ? 0 : (b == 1 ? (cN - 1) / 2 : cN - 1);
        const double P = col_P(J, c0 + cc);
        const double *c = S.crg;
        const double x = c[0] + c[1] * L + c[2] * P + c[3] * L * L + c[4] * L * P + c[5] * P * P;
        pmin = fmin(pmin, x);
        dmin = fmin(dmin, x - (double)cc);
        dmax = fmax(dmax, x - (double)cc);
      }
    }
    // the range pass reads ring columns [p0 - 5, p0 + 8] of a column pair; one
    // column of margin for the position's variation inside the strip, and the
    // ring starts on a sample pair of the slave box's rows
    const int xw = (int)floor(pmin) - 6;
    const int xr = min(max(xw + RS_FW / 2, J.sx0), J.sx1);
    const DerampQuad q = deramp_quad(J.kt[xr], J.tref[xr], J.fdc[xr]);
    Q.ref_a0 = q.a0;
    Q.ref_a1 = q.a1;
    Q.ref_a2 = q.a2;
    Q.tm = 0.5 * (double)(J.sy0 + J.sy1 - 2 * J.s_first_line) * J.dt;
    const int xo = xw - ((xw - J.sx0) & 1);
    Q.xo = xo;
    Q.dlo = max((int)floor(dmin) - 6 - xo, -RS_FW);
    Q.dhi = min((int)floor(dmax) - 4 - xo, RS_FW);
    Q.gen_any = 0;
    Q.prev_line = INT32_MIN;
    Q.missb[0] = Q.missb[1] = 0u;
  }
  __syncthreads();

  // ---- [P3] this thread's two ring columns: G = phi - phi_ref about tm
  // (g2 tc^2 + g1 tc + g0)
  const int xa = Q.xo + 2 * u;           // absolute slave column
  {
    const DerampQuad refq = {Q.ref_a0, Q.ref_a1, Q.ref_a2};
    float3 g[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int x = xa + q;
      DerampQuad cq = refq;
      if (x >= J.sx0 && x <= J.sx1) cq = deramp_quad(J.kt[x], J.tref[x], J.fdc[x]);
      g[q] = residual_phase(cq, refq, Q.tm);
      if constexpr (!kSplit) {
        Q.ring.a21[2 * u + q] = make_double2(cq.a2, cq.a1);
        Q.ring.a0[2 * u + q] = cq.a0;
      }
    }
    Q.ring.g2[u] = make_float2(g[0].x, g[1].x);
    Q.ring.g1[u] = make_float2(g[0].y, g[1].y);
    Q.ring.g0[u] = make_float2(g[0].z, g[1].z);
  }

  // range-pass columns
  const int dc = 2 * u;
  const bool dval = u < RS_DT && dc < cN, dtwo = dval && dc + 1 < cN;

  // the 12-line window of the two ring columns
  Dpair w[12];
#pragma unroll
  for (int j = 0; j < 12; j++) w[j].re = w[j].im = make_float2(0.f, 0.f);

  int want = RS_CH;                      // rows to try for a chunk
  // the tile is free while a chunk is prepared: the rows' entries as found
  int2 *const found = reinterpret_cast<int2 *>(&Q.tile[0]);
  for (int ch0 = 0; ch0 < nr;) {
    // ---- [P4] the azimuth entries of the chunk's rows (thread u: rows u and
    // u + 64): counts, and a scan of both packed in one word
    const int nrc = min(min(want, RS_CH), nr - ch0);
    const int rb = r_begin + ch0;        // box row of the chunk's first row
    if (u == 0) {
      Q.nfit = nrc;
      Q.cov = nrc;
      Q.kfrom = INT32_MAX;
      Q.n_border = 0;
    }
    __syncthreads();                     // also: the ring's terms are written
    {
      int mm = 0;
#pragma unroll 1
      for (int i = 0; i < 2; i++) {
        const int r = u + RS_NT * i;
        if (r < nrc)
          mm |= find_entries(S, Q, J, rb + r, c0, cN, found + r * RS_MAXKEY) << (16 * i);
      }
      int v = mm;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v, o);
        if ((u & 31) >= o) v += x;
      }
      if ((u & 31) == 31) Q.scan[u >> 5] = v;
      __syncthreads();
      if (u >= 32) v += Q.scan[0];
      const int total0 = (Q.scan[0] + Q.scan[1]) & 0xffff;
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int r = u + RS_NT * i, m = (mm >> (16 * i)) & 0xffff;
        const int end = ((v >> (16 * i)) & 0xffff) + (i ? total0 : 0);
        if (r < nrc) {
          Q.rowe[r] = (end - m) | m << 16;
          if (end > RS_ECAP) atomicMin(&Q.nfit, r);
        }
      }
    }
    __syncthreads();
    const int nfit = Q.nfit;
    // ---- [P5] the entries, [P6] the range-key runs
#pragma unroll 1
    for (int r = u; r < nfit; r += RS_NT) {
      const int re = Q.rowe[r], e = re & 0xffff;
      for (int i = 0; i < re >> 16; i++)
        write_entry(Q, J, found[r * RS_MAXKEY + i], cN, e + i);
    }
    int full = 0;                        // columns whose run table is full: 1 the first, 2 the second
    if (dval) {
      const double La = row_L(J, rb), Lz = row_L(J, rb + nfit - 1), c5 = S.crg[5];
      const double Aa = row_a(S.crg, La), Ba = row_b(S.crg, La);
      const double Az = row_a(S.crg, Lz), Bz = row_b(S.crg, Lz);
      int ka[2], kz[2];
      bool mono[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const double Pc = col_P(J, c0 + dc + i);
        ka[i] = rg_key_at(Aa, Ba, c5, Pc);
        kz[i] = rg_key_at(Az, Bz, c5, Pc);
        // slope in the row: (g1 + g4 P) + 2 g3 L, of one sign over the rows
        const double s1 = fma(S.crg[4], Pc, S.crg[1]), s2 = 2.0 * S.crg[3];
        mono[i] = (fma(s2, La, s1) < 0.0) == (fma(s2, Lz, s1) < 0.0);
      }
#pragma unroll 1
      for (int i = 0; i < (dtwo ? 2 : 1); i++)
        full |= (int)build_runs(S, Q, J, rb, nfit, c0, dc + i, i ? mono[1] : mono[0],
                                i ? ka[1] : ka[0], i ? kz[1] : kz[0])
                << i;
    }
    __syncthreads();
    // ---- [P7] the halves; a chunk that does not end the item ends with a
    // pair of halves, so that the window carries over
    int n = Q.cov >= min(kKeyedRows, (nr - ch0 + 1) / 2) ? min(nfit, Q.cov) : nfit;
    if (n < nr - ch0 && n >= 2 * RS_H) n -= n % (2 * RS_H);
    const int nh = (n + RS_H - 1) / RS_H;
    if (dval) {
      if (Q.cov < n) {
#pragma unroll
        for (int i = 0; i < 2; i++)
          if ((full >> i) & 1) {
            Q.run_rk[kRuns - 1][dc + i] = make_int2(INT32_MAX, kKeyed);
            atomicMin(&Q.kfrom, Q.run_rk[kRuns - 2][dc + i].x);
          }
      }
      for (int c = dc; c < min(dc + 2, cN); c++) {
        bool out = false;
        for (int m = 0;; m++) {
          const int2 rk = Q.run_rk[m][c];
          out = out || !(range_in(J, rk.y) || rk.y == kKeyed);
          if (rk.x >= n) break;
        }
        if (out) Q.border[atomicAdd(&Q.n_border, 1)] = (unsigned char)c;
      }
    }
    if (u < nh) plan_half(Q, u, n);
    __syncthreads();
    int fl = 0, tb = 0;
    if (u < nh) {
      const RsHalf &H = Q.half[u];
      fl = H.flags;
      const int expect = u == 0 ? Q.prev_line
                         : (Q.half[u - 1].flags & HG_ON) ? Q.half[u - 1].lb + RS_H : INT32_MIN;
      if ((fl & HG_ON) && H.lb != expect) fl |= HG_FILL;
      if (min((u + 1) * RS_H, n) > Q.kfrom) fl |= HG_KEY;
      const int h0 = u & ~1;
      if (h0 + 1 < nh && Q.half[h0].units + Q.half[h0 + 1].units <= RS_TU) {
        if (u & 1)
          tb = Q.half[h0].units;
        else
          fl |= HG_JOIN;
      }
    }
    // deramp terms of the lines the halves push
    for (int i = u; i < nh * RS_H; i += RS_NT)
      Q.srow[i] = line_terms<kSplit>(Q, J, Q.half[i / RS_H].lb + RS_H + i % RS_H);
    __syncthreads();
    if (u < nh) {
      Q.half[u].flags = fl;
      Q.half[u].tbase = tb;
      if (u == nh - 1)
        Q.prev_line = (fl & HG_ON) && !(nh & 1) ? Q.half[u].lb + RS_H : INT32_MIN;
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (h < nh && (Q.half[h].flags & HG_ON))
        stage_half(S, J, u, xa, h * RS_H, Q.half[h].lb + RS_H);
      cp_async_commit();
    }

    if (Q.n_border)
      border_columns(Q, J, u, n, J.out + (long)(rb - J.row0) * J.out_pitch + c0);
    PairRuns P;
    P.m = 0;
    P.next = INT32_MIN;
    P.unit = -1;
    P.in = 0;
    for (int h = 0; h < nh; h++) {
      const RsHalf H = Q.half[h];
      const int flags = H.flags;
      // ---- [A]
      if (flags & HG_ON) {
        if (h & 1)
          az_half<1, kSplit>(S, Q, J, u, xa, h, H, w);
        else
          az_half<0, kSplit>(S, Q, J, u, xa, h, H, w);
        if (flags & HG_DIRECT) az_direct<kSplit>(Q, J, u, xa, H.tbase, H.pos[0], H.pos[7]);
      } else {
        cp_async_wait<1>();
      }
      if (h + 2 < nh && (Q.half[h + 2].flags & HG_ON))
        stage_half(S, J, u, xa, (h & 1) * RS_H, Q.half[h + 2].lb + RS_H);
      cp_async_commit();
      if (flags & HG_JOIN) continue;
      // ---- [B] range pass, reramp, store: 2 columns x the tile's rows
      const int h0 = (h & 1) && (Q.half[h - 1].flags & HG_JOIN) ? h - 1 : h;
      const int k0 = h0 * RS_H, k1 = min((h + 1) * RS_H, n);
      const int both = Q.half[h0].flags & flags, any = Q.half[h0].flags | flags;
      if (dval && k0 >= P.next) next_runs(P, Q, J, dc, dtwo, k0);
      __syncthreads();
      unsigned miss = 0;                 // rows the pair path leaves
      if (dval) {
        float2 *orow = J.out + (long)(rb + k0 - J.row0) * J.out_pitch + c0 + dc;
        const long pitch = J.out_pitch;
        int k = k0;
        if (both & HG_ONE) {
          // one interior entry per row: consecutive entries and tile rows
          const int e0 = (Q.rowe[k0] & 0xffff) - k0;
          const float4 *U = &Q.tile[0], *A = &Q.eA[e0 + k];
          const int *R = &Q.eM[e0 + k].z;
#pragma unroll 1
          for (; k < k1; k++, orow += pitch, U += RS_UN, A++, R += 4) {
            if (k >= P.next) next_runs(P, Q, J, dc, dtwo, k);
            if (P.unit >= 0) {
              pair_row(P, U + P.unit, *A, __int_as_float(*R), orow);
            } else if (P.in) {
              miss |= 1u << (k - k0);
            }
          }
        }
#pragma unroll 1
        for (; k < k1; k++, orow += pitch) {
          if (k >= P.next) next_runs(P, Q, J, dc, dtwo, k);
          const int re = Q.rowe[k], ne = re >> 16;
          if (ne == 0) continue;         // a per-pixel row
          int e = re & 0xffff;
          int4 M = Q.eM[e];
          for (int q = 1; q < ne && !(dc >= ((M.y >> 16) & 0xff) && dc < ((M.y >> 24) & 0xff));
               q++)
            M = Q.eM[++e];
          const bool same = dtwo && dc + 1 < ((M.y >> 24) & 0xff);
          const int reg = (M.y >> 12) & 3;
          if (reg != REG_IN && same) {
            orow[0] = border_pixel(J, reg, M.x, Q.run_rk[P.m & 0xff][dc].y >> 12);
            orow[1] = border_pixel(J, reg, M.x, Q.run_rk[P.m >> 8][dc + 1].y >> 12);
          } else if (P.unit >= 0 && same && P.unit >= ((M.w >> 16) & 0xff) &&
                     P.unit + 6 <= ((M.w >> 24) & 0xff)) {
            pair_row(P, &Q.tile[(k >= h * RS_H ? H.tbase : 0) + (short)(M.w & 0xffff) + P.unit],
                     Q.eA[e], __int_as_float(M.z), orow);
          } else if (P.in) {
            miss |= 1u << (k - k0);
          }
        }
      }
      {
        const unsigned b = __ballot_sync(0xffffffffu, miss != 0);
        if (miss) Q.miss[u] = (unsigned short)miss;
        if ((u & 31) == 0) Q.missb[u >> 5] = b;
      }
      __syncthreads();

      // ---- [C] the pixels the pair path left and the keyed rows, then
      // per-pixel rows and the pixels left to the per-pixel path
      if (Q.missb[0] | Q.missb[1]) {
        slow_pixels(Q, J, u, k0, k1 - k0, h * RS_H, H.tbase, cN,
                    J.out + (long)(rb + k0 - J.row0) * J.out_pitch + c0);
        __syncthreads();
      }
      if (Q.gen_any || (any & (HG_PIX | HG_KEY))) {
        if (any & HG_KEY) {
          keyed_pairs<kSplit>(J, rb, k0, max(k0, Q.kfrom), k1, h * RS_H, H.tbase, c0, cN);
          __syncthreads();
        }
        if (Q.gen_any || (any & HG_PIX)) pixel_pass(S, Q, J, u, k0, rb + k0, k1 - k0, c0, cN);
      }
      if (Q.gen_any) {
        __syncthreads();
        if (u < 2 * RS_H * 4) (&Q.gen[0][0])[u] = 0u;
        if (u == 0) Q.gen_any = 0;
      }
    }
    cp_async_wait<0>();
    ch0 += n;
    want = max(2 * RS_H, n + n);         // shrink to what the tables held, then grow
    want = (want + 2 * RS_H - 1) / (2 * RS_H) * (2 * RS_H);
    __syncthreads();   // the next chunk's (or item's) prologue rewrites the tables and the tile
  }
}

static_assert(6 * (sizeof(RsShared<true>) + 1024) <= 228 * 1024 &&
                  6 * (sizeof(RsShared<false>) + 1024) <= 228 * 1024,
              "6 CTAs per SM");

template <bool kSplit>
__global__ void __launch_bounds__(RS_NT, 6)
    resample_kernel(const __grid_constant__ RsBatch B) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RsShared<kSplit> &S = *reinterpret_cast<RsShared<kSplit> *>(smem_raw);
  // one work item per CTA, or (persistent) items from the queue until it
  // is empty; a single call site keeps one inlined copy of the item code
  int item = blockIdx.x;
  if (B.counter) {
    if (threadIdx.x == 0) S.next_item = atomicAdd(B.counter, 1);
    __syncthreads();
    item = S.next_item;
    __syncthreads();
  }
  while (item < B.total_items) {
    resample_item<kSplit>(S, B, item);
    if (!B.counter) break;
    if (threadIdx.x == 0) S.next_item = atomicAdd(B.counter, 1);
    __syncthreads();
    item = S.next_item;
    __syncthreads();
  }
}

// ---------------------------------------------------------------- host
// All tables of one LUT in one device allocation.
struct LutDev {
  void *mem = nullptr;
  LutPtrs p{};
};

}  // namespace tops

struct tops_lut_dev {
  tops::LutDev d;
};

using namespace tops;

extern "C" int tops_lut_create(const float *kaz, const float *krg, tops_lut_dev **out) {
  if (!kaz || !krg || !out) return TOPS_E_INVALID;
  // device layout: kaz2 [2048][24] | krgo [2048][16] | kaz [2048][12] |
  // krg [2048][12] | sp1 [2048]
  const size_t nb = kLutBins;
  const size_t o_krgo = nb * 24, o_kaz = o_krgo + nb * 16, o_krg = o_kaz + nb * kTaps,
               o_sp1 = o_krg + nb * kTaps, total = (o_sp1 + nb) * sizeof(float);
  std::vector<float> h(o_sp1 + nb, 0.f);
  float *kaz2 = h.data(), *krgo = kaz2 + o_krgo, *sp1 = kaz2 + o_sp1;
  std::copy(kaz, kaz + nb * kTaps, kaz2 + o_kaz);
  std::copy(krg, krg + nb * kTaps, kaz2 + o_krg);
  for (size_t b = 0; b < nb; b++) {
    double s = 0.0;
    for (int i = 0; i < kTaps; i++) {
      s += (double)krg[b * kTaps + i];
      kaz2[b * 24 + 2 * i] = kaz2[b * 24 + 2 * i + 1] = kaz[b * kTaps + i];
      krgo[b * 16 + 1 + i] = krg[b * kTaps + i];
    }
    sp1[b] = (float)(s - 1.0);
  }
  tops_lut_dev *L = new tops_lut_dev();
  cudaError_t e = cudaMalloc(&L->d.mem, total);
  if (e == cudaSuccess) e = cudaMemcpy(L->d.mem, h.data(), total, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    set_cuda_error(e);
    (void)cudaGetLastError();
    cudaFree(L->d.mem);
    delete L;
    return e == cudaErrorMemoryAllocation ? TOPS_E_NOMEM : TOPS_E_CUDA;
  }
  const float *m = static_cast<const float *>(L->d.mem);
  L->d.p.kaz2 = reinterpret_cast<const float4 *>(m);
  L->d.p.krgo = reinterpret_cast<const float4 *>(m + o_krgo);
  L->d.p.kaz = m + o_kaz;
  L->d.p.krg = m + o_krg;
  L->d.p.sp1 = m + o_sp1;
  *out = L;
  return TOPS_OK;
}

extern "C" int tops_lut_destroy(tops_lut_dev *L) {
  if (!L) return TOPS_OK;
  cudaFree(L->d.mem);
  delete L;
  return TOPS_OK;
}

namespace tops {

static int check_box(const int b[4]) { return b[1] >= b[0] && b[3] >= b[2]; }

int fill_resample_job(const tops_resample_job &u, ResampleJob &J) {
  if (!u.slave || !u.out || !u.kt || !u.tref || !u.fdc) return TOPS_E_INVALID;
  if (!check_box(u.mbox) || !check_box(u.sbox)) return TOPS_E_INVALID;
  if ((u.slave_pitch % sizeof(short2)) || (u.out_pitch % sizeof(float2))) return TOPS_E_INVALID;
  const int mlines = u.mbox[3] - u.mbox[2] + 1;
  J.slave = static_cast<const short2 *>(u.slave);
  J.slave_pitch = (long)(u.slave_pitch / sizeof(short2));
  J.out = static_cast<float2 *>(u.out);
  J.out_pitch = (long)(u.out_pitch / sizeof(float2));
  if (J.slave_pitch < u.sbox[1] - u.sbox[0] + 1 || J.out_pitch < u.mbox[1] - u.mbox[0] + 1)
    return TOPS_E_INVALID;
  // vector access needs aligned bases and pitches: 8-byte slave pairs and
  // 16-byte output pairs (scalar access otherwise)
  J.slave_al8 = ((reinterpret_cast<uintptr_t>(u.slave) & 7) == 0) && (u.slave_pitch % 8 == 0);
  J.out_al16 = ((reinterpret_cast<uintptr_t>(u.out) & 15) == 0) && (u.out_pitch % 16 == 0);
  J.kt = u.kt;
  J.tref = u.tref;
  J.fdc = u.fdc;
  J.mx0 = u.mbox[0];
  J.mx1 = u.mbox[1];
  J.my0 = u.mbox[2];
  J.my1 = u.mbox[3];
  J.sx0 = u.sbox[0];
  J.sx1 = u.sbox[1];
  J.sy0 = u.sbox[2];
  J.sy1 = u.sbox[3];
  for (int i = 0; i < 6; i++) {
    J.caz[i] = u.cpm_az[i];
    J.crg[i] = u.cpm_rg[i];
  }
  J.az_shift = u.az_shift;
  J.az_shift_dev = u.az_shift_dev;
  J.cpm_dev = u.cpm_dev;
  J.s_first_line = u.s_first_line;
  J.dt = u.dt;
  J.row0 = u.out_rows < 0 ? 0 : u.out_row0;
  J.nrows = u.out_rows < 0 ? mlines : u.out_rows;
  if (J.row0 < 0 || J.nrows < 0 || J.row0 + J.nrows > mlines) return TOPS_E_INVALID;
  // normalizeWarp(v, lo, hi) = (v - 0.5*(lo+hi)) / (0.25*(hi-lo))
  J.midP = 0.5 * ((double)u.mbox[0] + (double)u.mbox[1]);
  J.invP = 1.0 / (0.25 * ((double)u.mbox[1] - (double)u.mbox[0]));
  J.midL = 0.5 * ((double)u.mbox[2] + (double)u.mbox[3]);
  J.invL = 1.0 / (0.25 * ((double)u.mbox[3] - (double)u.mbox[2]));
  const int mpix = u.mbox[1] - u.mbox[0] + 1;
  J.strips = (mpix + RS_TW - 1) / RS_TW;
  J.seg_rows = RS_MAXSEG;
  J.segs = (J.nrows + RS_MAXSEG - 1) / RS_MAXSEG;
  return TOPS_OK;
}

template <bool kSplit>
static int launch_resample_t(const ResampleJob *jobs, int njobs, const TileCfg &cfg,
                             cudaStream_t st) {
  // the shared-memory opt-in is a per-device function attribute; the
  // persistent grid is the number of CTAs resident at once
  static PerDeviceOnce setup;
  int dev = 0, resident = 0;
  TOPS_CUDA_TRY(cudaGetDevice(&dev));
  const int s0 = once_per_device(
      setup, dev,
      [&](int &v) -> int {
        TOPS_CUDA_TRY(cudaFuncSetAttribute(
            resample_kernel<kSplit>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RsShared<kSplit>)));
        int per_sm = 0, sms = 0;
        TOPS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, resample_kernel<kSplit>, RS_NT,
                                                                    sizeof(RsShared<kSplit>)));
        TOPS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        v = per_sm * sms;
        return TOPS_OK;
      },
      &resident);
  if (s0 != TOPS_OK) return s0;
  if (cfg.seg_rows < 0 || cfg.seg_rows > RS_MAXSEG || (cfg.seg_rows && cfg.seg_rows < 2 * RS_H))
    return TOPS_E_INVALID;
  // segment rows: the fewest row times of the last CTA to finish, waves x (rows
  // + the prologue and the window's fill, worth about 24 rows), up to the
  // caller's limit; 8 waves and more at the limit take it as it is, since their
  // CTAs are out of step (27 bursts of three sub-swaths: limit 252 8.47 ms,
  // the choice up to it 8.83).  Outputs do not depend on it.
  const int most = cfg.seg_rows ? cfg.seg_rows : RS_MAXSEG;
  int seg_rows = 0;
  {
    const int kSegs[] = {most, 252, 204, 168, 144, 120, 96, 84, 72, 60, 48, 36, 24, 12};
    long best = 0;
    for (int sr : kSegs) {
      if (sr > most) continue;
      long items = 0;
      for (int j = 0; j < njobs; j++)
        items += (long)jobs[j].strips * ((jobs[j].nrows + sr - 1) / sr);
      const long cost = (items + resident - 1) / resident * (sr + 24);
      if (!seg_rows || cost < best) {
        best = cost;
        seg_rows = sr;
      }
      if (cfg.seg_rows && sr == most && items >= 8L * resident) break;
    }
  }
  for (int j0 = 0, k = 0; j0 < njobs; j0 += RS_MAXJOBS, k++) {
    RsBatch B;
    B.njobs = 0;
    B.counter = cfg.counters ? cfg.counters + k : nullptr;
    int items = 0;
    for (int j = j0; j < njobs && j < j0 + RS_MAXJOBS; j++) {
      ResampleJob &J = B.jobs[B.njobs];
      J = jobs[j];
      J.seg_rows = seg_rows;
      J.segs = (J.nrows + seg_rows - 1) / seg_rows;
      J.item_begin = items;
      items += J.strips * J.segs;
      B.njobs++;
    }
    B.total_items = items;
    if (items == 0) continue;
    int grid = items;
    if (B.counter) {
      TOPS_CUDA_TRY(cudaMemsetAsync(B.counter, 0, sizeof(int), st));
      grid = min(items, cfg.grid > 0 ? cfg.grid : resident);
    }
    resample_kernel<kSplit><<<grid, RS_NT, sizeof(RsShared<kSplit>), st>>>(B);
    TOPS_CUDA_TRY(cudaGetLastError());
  }
  return TOPS_OK;
}

static int launch_resample(const ResampleJob *jobs, int njobs, int precision, const TileCfg &cfg,
                           cudaStream_t st) {
  if (precision == TOPS_PREC_FP64) return launch_resample_t<false>(jobs, njobs, cfg, st);
  if (precision == TOPS_PREC_SPLIT) return launch_resample_t<true>(jobs, njobs, cfg, st);
  return TOPS_E_INVALID;
}

int resample_launch_multi(const tops_lut_dev *const *luts, const tops_resample_job *jobs,
                          int njobs, int precision, const TileCfg &cfg, cudaStream_t st) {
  if (!luts || (!jobs && njobs > 0) || njobs < 0) return TOPS_E_INVALID;
  std::vector<ResampleJob> J(njobs);
  for (int j = 0; j < njobs; j++) {
    if (!luts[j]) return TOPS_E_INVALID;
    int s = fill_resample_job(jobs[j], J[j]);
    if (s != TOPS_OK) return s;
    J[j].lut = luts[j]->d.p;
  }
  return launch_resample(J.data(), njobs, precision, cfg, st);
}

int resample_launch(const tops_lut_dev *lut, const tops_resample_job *jobs, int njobs,
                    int precision, const TileCfg &cfg, cudaStream_t st) {
  if (!lut || (!jobs && njobs > 0) || njobs < 0) return TOPS_E_INVALID;
  std::vector<const tops_lut_dev *> luts(njobs, lut);
  return resample_launch_multi(luts.data(), jobs, njobs, precision, cfg, st);
}

}  // namespace tops

extern "C" int tops_resample_ex(const tops_lut_dev *lut, const tops_resample_job *jobs,
                                int njobs, int precision, void *stream) {
  return resample_launch(lut, jobs, njobs, precision, TileCfg(),
                         static_cast<cudaStream_t>(stream));
}

extern "C" int tops_resample(const tops_lut_dev *lut, const tops_resample_job *jobs, int njobs,
                             void *stream) {
  return tops_resample_ex(lut, jobs, njobs, TOPS_PREC_SPLIT, stream);
}
