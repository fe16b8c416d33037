// coherence.cu -- windowed interferometric coherence (sm_100a).
//
// Reference: CohMatSet (EstCoh.cu:101-139) builds m*conj(s) and
// (|s|^2, |m|^2) in padded arrays; Cohbasic (EstCoh.cu:413-456) and the
// prefix-sum chain of CoherenceEst_ESD (EstCoh.cu:152-411) sum them over the
// box rows r-dy..r-dy+winAz-1, cols c-dx..c-dx+winRg-1 and output
//   gamma = |sum m s*| / sqrt(sum|s|^2 * sum|m|^2)   (0 if the product is 0)
// with gamma = 0 where |s(r,c)| < 0.001.  The reference leaves the pad
// uninitialised (EstCoh.cu:581-583); here it is zero.
//
// B200 design: no block barriers.  A warp owns a strip of 128 loaded columns,
// four per lane, and marches down a segment of rows.  Its rows come through a
// private ring of 4 slots in shared memory filled by asynchronous copies (three
// 16-byte ones per lane and row, or single samples where rows do not start on
// 16-byte boundaries; both zero-fill outside the image).  The products (m s*,
// |s|^2, |m|^2) of the last winAz - 1 rows stay in registers, so every input
// row is read once; output rows go in pairs whose common rows are summed once.
// The horizontal sums come from prefix, suffix and whole sums of the lanes' four
// columns that the lanes exchange with shuffles.  No sum is updated by
// subtraction, so the rounding error does not grow along a row, and a sample
// that is not finite spoils its own windows only.  For heights of up to 6 the
// sums are trees, whose error hardly grows with the window (7.8e-8 relative RMS
// at 10 x 3, 8.0e-8 at 24 x 6); taller windows add the rows that 4 output rows
// share one after another, an error of up to win_az roundings.
//
// What bounds it: instruction issue (10 x 3: 64 per output pixel, 11 of them
// packed adds and 9 shuffles; two thirds of the issue slots) and the L1 data pipe
// (the shuffles) at 16 warps per SM by registers, then the 16 bytes per pixel of
// memory traffic.  Measured, in us, against a kernel that staged the products of
// a block in shared memory and summed windows by sliding updates behind block
// barriers (a single burst with a cold L2 takes a few more than these, which
// found part of it there: 10 x 3 104 to 108, 4.7 to 4.8 TB/s):
//   1500 x 21000, 10 x 3   154 -> 97                 24 x 6   243 -> 156
//   1523 x 8193, 5 x 5     147 -> 48                 1200 x 7000, 30 x 9  180 -> 133
//   1200 x 7000, 17 x 2    129 -> 47                 300 x 512, 10 x 3    66 -> 9
//   800 x 9000, 2 x 1      111 -> 24                 33 x 7               152 -> 78
// Rows prefetched into registers instead of the ring took 121 us (10 x 3) and
// 229 us (24 x 6); a ring of 7 slots 109 us; 18 warps per SM, by spilling, 149.
#include <cuda_runtime.h>

#include <type_traits>
#include <vector>

#include "common.cuh"
#include "launch.h"

namespace tops {

constexpr int CO_CPL = 4;          // columns per lane
constexpr int CO_NW = 2;           // warps (adjacent strips) per CTA
constexpr int CO_NT = 32 * CO_NW;
constexpr int CO_D = 4;            // slots per warp: the row read last and 3 in flight
constexpr int CO_ROW = 2048;       // bytes of a slot: 128 columns of 4 and of 8, and a gap
constexpr int CO_ODD = 512 + 36 * 16;   // the slave's odd pieces in a slot
constexpr int CO_MAXJOBS = 32;
constexpr int CO_MAX_WIN_RG = 33;

struct CoBatch {
  int njobs, total_items, win_rg, win_az;
  int nl, nr;              // lanes whose columns only feed the windows: left, right
  int compensated;         // 1: both reciprocal square roots refined by a Newton step
  int *counter;            // persistent launch: work-item queue (else null)
  CohJob jobs[CO_MAXJOBS];
};

__device__ __forceinline__ float4 coh_product(short2 m, float2 s) {
  const float mr = m.x, mi = m.y;
  return make_float4(mr * s.x + mi * s.y,   // m * conj(s)
                     mi * s.x - mr * s.y, s.x * s.x + s.y * s.y, mr * mr + mi * mi);
}

// a + b with packed FP32x2 adds
__device__ __forceinline__ float4 add4(const float4 &a, const float4 &b) {
  const float2 c = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
  const float2 p = __fadd2_rn(make_float2(a.z, a.w), make_float2(b.z, b.w));
  return make_float4(c.x, c.y, p.x, p.y);
}
// the value of lane + off
__device__ __forceinline__ float4 lane4(const float4 &v, int off) {
  const int src = (int)(threadIdx.x & 31) + off;
  return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                     __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}
template <int OFF>
__device__ __forceinline__ float4 lane4(const float4 &v) {
  constexpr int n = OFF < 0 ? -OFF : OFF;
  auto s = [](float x) {
    return OFF < 0 ? __shfl_up_sync(0xffffffffu, x, n) : __shfl_down_sync(0xffffffffu, x, n);
  };
  return make_float4(s(v.x), s(v.y), s(v.z), s(v.w));
}

// Asynchronous global -> shared copies of B bytes: n from src, then zeros.
template <int B>
__device__ __forceinline__ void co_copy(unsigned d, const void *src, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(B),
               "r"(n)
               : "memory");
}

// A lane's column sums: the single columns, the whole, first two, first three,
// last two and last three of them.
struct CoSums {
  float4 v[CO_CPL], f, p2, p3, s2, s3;
  // the sum of the first / last N columns
  template <int N>
  __device__ __forceinline__ const float4 &first() const {
    return N == 1 ? v[0] : N == 2 ? p2 : N == 3 ? p3 : f;
  }
  template <int N>
  __device__ __forceinline__ const float4 &last() const {
    return N == 1 ? v[3] : N == 2 ? s2 : N == 3 ? s3 : f;
  }
};

// Windows of W <= 6 columns, W at compile time: column a of the window is in
// lane a >> 2, and at most one lane is whole.
template <int W>
__device__ __forceinline__ void box_small(const CoSums &c, float4 (&o)[CO_CPL]) {
  auto out = [&](auto uu) {
    constexpr int u = decltype(uu)::value;
    constexpr int a = u - (W - 1) / 2, b = a + W - 1;
    constexpr int lo = (a + 64) / 4 - 16, hi = (b + 64) / 4 - 16;
    constexpr int ka = a - 4 * lo, kb = b - 4 * hi;
    if constexpr (lo == hi) {
      float4 t = ka == 0 ? c.template first<kb + 1>() : c.v[ka];
      if constexpr (ka == 1 && kb == 3) t = c.s3;
      if constexpr (ka == 2 && kb == 3) t = c.s2;
      if constexpr (ka == 1 && kb == 2) t = add4(c.v[1], c.v[2]);
      o[u] = lo == 0 ? t : lane4<lo>(t);
    } else {
      const float4 &e0 = c.template last<4 - ka>(), &e1 = c.template first<kb + 1>();
      float4 t = lo == 0 ? e0 : lane4<lo>(e0);
      if constexpr (hi > lo + 1) t = add4(t, lo + 1 == 0 ? c.f : lane4<lo + 1>(c.f));
      o[u] = add4(t, hi == 0 ? e1 : lane4<hi>(e1));
    }
  };
  out(std::integral_constant<int, 0>());
  out(std::integral_constant<int, 1>());
  out(std::integral_constant<int, 2>());
  out(std::integral_constant<int, 3>());
}

// Windows of 7 columns or more: some lanes are whole in the windows of all four
// columns; before them column u's window holds another Q + 3 - u columns (Q 0
// to 3), after them Q + u.
template <int Q>
__device__ __forceinline__ void box_left(const CoSums &c, int l, float4 (&o)[CO_CPL]) {
  if constexpr (Q == 0) {                   // 3 2 1 0
    o[0] = lane4(c.s3, l);
    o[1] = lane4(c.s2, l);
    o[2] = lane4(c.v[3], l);
    o[3] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else if constexpr (Q == 1) {            // 4 3 2 1
    o[0] = lane4(c.f, l);
    o[1] = lane4(c.s3, l);
    o[2] = lane4(c.s2, l);
    o[3] = lane4(c.v[3], l);
  } else if constexpr (Q == 2) {            // 5 4 3 2
    const float4 w = lane4(c.f, l);
    o[0] = add4(lane4(c.v[3], l - 1), w);
    o[1] = w;
    o[2] = lane4(c.s3, l);
    o[3] = lane4(c.s2, l);
  } else {                                  // 6 5 4 3
    const float4 w = lane4(c.f, l);
    o[0] = add4(lane4(c.s2, l - 1), w);
    o[1] = add4(lane4(c.v[3], l - 1), w);
    o[2] = w;
    o[3] = lane4(c.s3, l);
  }
}
template <int Q>
__device__ __forceinline__ void box_right(const CoSums &c, int l, float4 (&o)[CO_CPL]) {
  if constexpr (Q == 0) {                   // 0 1 2 3
    o[1] = add4(o[1], lane4(c.v[0], l));
    o[2] = add4(o[2], lane4(c.p2, l));
    o[3] = add4(o[3], lane4(c.p3, l));
  } else if constexpr (Q == 1) {            // 1 2 3 4
    o[0] = add4(o[0], lane4(c.v[0], l));
    o[1] = add4(o[1], lane4(c.p2, l));
    o[2] = add4(o[2], lane4(c.p3, l));
    o[3] = add4(o[3], lane4(c.f, l));
  } else if constexpr (Q == 2) {            // 2 3 4 5
    const float4 w = lane4(c.f, l);
    o[0] = add4(o[0], lane4(c.p2, l));
    o[1] = add4(o[1], lane4(c.p3, l));
    o[2] = add4(o[2], w);
    o[3] = add4(o[3], add4(w, lane4(c.v[0], l + 1)));
  } else {                                  // 3 4 5 6
    const float4 w = lane4(c.f, l);
    o[0] = add4(o[0], lane4(c.p3, l));
    o[1] = add4(o[1], w);
    o[2] = add4(o[2], add4(w, lane4(c.v[0], l + 1)));
    o[3] = add4(o[3], add4(w, lane4(c.p2, l + 1)));
  }
}
template <int WRG>
__device__ __forceinline__ void box_large(const CoSums &c, int win, int dx,
                                          float4 (&o)[CO_CPL]) {
  const int ql = (dx + 1) & 3, qr = (win - dx) & 3;
  const int l0 = (ql + 3 - dx) / 4, l1 = (win - dx - qr) / 4;   // the whole lanes l0 .. l1 - 1
  // 1 to 7 whole lanes, from the sums of 1, 2 and 4 lanes from each lane on
  const int n = l1 - l0;
  int l = l0;
  bool any = false;
  float4 g = c.f, m = g;
  auto piece = [&](int lanes) {
    const float4 y = WRG > 0 && l == 0 ? g : lane4(g, l);
    m = any ? add4(m, y) : y;
    any = true;
    l += lanes;
  };
  if (n & 1) piece(1);
  if (n >= 2) g = add4(g, lane4<1>(g));
  if (n & 2) piece(2);
  if (n >= 4) {
    g = add4(g, lane4<2>(g));
    piece(4);
  }
  switch (ql) {
    case 0: box_left<0>(c, l0 - 1, o); break;
    case 1: box_left<1>(c, l0 - 1, o); break;
    case 2: box_left<2>(c, l0 - 1, o); break;
    default: box_left<3>(c, l0 - 1, o);
  }
  switch (qr) {
    case 0: box_right<0>(c, l1, o); break;
    case 1: box_right<1>(c, l1, o); break;
    case 2: box_right<2>(c, l1, o); break;
    default: box_right<3>(c, l1, o);
  }
  // the ends first: one rounding at the size of the whole sum
#pragma unroll
  for (int u = 0; u < CO_CPL; u++) o[u] = add4(m, o[u]);
}

// Horizontal sums o[u] of columns x + u - dx .. x + u - dx + win - 1 (x the
// lane's first column) from the lanes' vertical sums v.  WRG > 0: the window
// at compile time; CO_SMALL, CO_LARGE: any of up to 6, of 7 or more columns.
constexpr int CO_SMALL = 0, CO_LARGE = -1;
template <int WRG>
__device__ __forceinline__ void coh_box(const float4 (&v)[CO_CPL], int win, int dx,
                                        float4 (&o)[CO_CPL]) {
  CoSums c;
#pragma unroll
  for (int i = 0; i < CO_CPL; i++) c.v[i] = v[i];
  c.p2 = add4(v[0], v[1]);
  c.s2 = add4(v[2], v[3]);
  c.p3 = add4(c.p2, v[2]);
  c.s3 = add4(v[1], c.s2);
  c.f = add4(c.p2, c.s2);
  if constexpr (WRG == CO_SMALL) {
    switch (win) {
      case 1: box_small<1>(c, o); break;
      case 2: box_small<2>(c, o); break;
      case 3: box_small<3>(c, o); break;
      case 4: box_small<4>(c, o); break;
      case 5: box_small<5>(c, o); break;
      default: box_small<6>(c, o);
    }
  } else if constexpr (WRG == CO_LARGE) {
    box_large<0>(c, win, dx, o);
  } else {
    box_large<WRG>(c, WRG, (WRG - 1) / 2, o);
  }
}

// 1 / sqrt(x); FINE: with a Newton step
template <bool FINE>
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  if (FINE && x <= 3.4e38f) r = fmaf(0.5f * r, fmaf(-x * r, r, 1.f), r);
  return r;
}
// |sum m s*| / sqrt(sum |s|^2 sum |m|^2) as num rsqrt(num) rsqrt(p): two MUFU
// reciprocal square roots instead of an IEEE square root (relative error a few
// 1e-7); the amplitude mask |s| < 0.001 of the reference (EstCoh.cu:393, 446)
// is evaluated as |s|^2 < 1e-6.  A num below FLT_MIN is a coherence below
// 1e-15 and taken for 0; above it some |m|^2, a whole number, is not 0, so p
// is at least 1e-6 where the mask passes.
template <bool FINE>
__device__ __forceinline__ float coh_gamma(const float4 &w, float spow) {
  const float p = w.z * w.w;
  const float num = fmaf(w.x, w.x, w.y * w.y);
  const bool ok = num >= 1.17549435e-38f && spow >= 1e-6f;
  if (FINE && !ok) return 0.f;
  const float g = num * rsqrt_ftz<FINE>(num) * rsqrt_ftz<FINE>(p);
  return ok ? g : 0.f;
}

// One work item: the warp's strip of one segment; no thread synchronises with
// another warp.  WAZ > 0: the window height at compile time; AL: the input rows
// start on 16-byte boundaries.
template <int WAZ, int WRG, bool AL>
__device__ __forceinline__ void coherence_item(const CoBatch &B, int item,
                                               unsigned char *stage) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int jb = 0;
  while (jb + 1 < B.njobs && B.jobs[jb + 1].item_begin <= item) jb++;
  const CohJob &J = B.jobs[jb];
  const int local = item - J.item_begin;
  const int seg = local / J.strips;
  constexpr int DY = WAZ > 0 ? (WAZ - 1) / 2 : 0;
  constexpr int R = WAZ > 0 ? WAZ - 1 : 0; // rows of products kept
  const int win = WRG > 0 ? WRG : B.win_rg, dx = (win - 1) / 2;
  const int nl = WRG == 10 ? 1 : WRG == 24 ? 3 : B.nl, nr = WRG == 10 ? 2 : WRG == 24 ? 3 : B.nr;
  const int tw = CO_CPL * (32 - nl - nr);  // output columns of a warp
  const int x = ((local - seg * J.strips) * CO_NW + warp) * tw + CO_CPL * (lane - nl);
  if (x - CO_CPL * (lane - nl) >= J.pixels) return;   // the whole warp
  const int r_begin = seg * J.seg_rows, r_end = min(r_begin + J.seg_rows, J.lines);
  const bool out_lane = lane >= nl && lane < 32 - nr && x < J.pixels;
  const bool vec_out = out_lane && x + CO_CPL <= J.pixels && J.out_al16;
  // rows from here on are not needed
  const int y_end = WAZ > 0 ? min(r_end - DY + R, J.lines) : J.lines;
  // The warp's copies of a row: 128 columns from xw on.  AL: 16-byte pieces,
  // one of the master (columns c0 .. c0 + 3) and two of the slave (c1, c1 + 1
  // and c1 + 64, c1 + 65) per lane; a piece is cut off at the end of the row
  // (xw is a multiple of 4, so none reaches across column 0) and the copy puts
  // zeros behind.  Else single columns, xw + lane + 32 k.
  const int xw = x - CO_CPL * lane;
  const int c0 = AL ? x : xw + lane, c1 = xw + 2 * lane;
  auto bytes = [&](int c, int esz) {
    return c < 0 ? 0 : min(max(J.pixels - c, 0) * esz, 16);
  };
  auto clip = [&](int c) { return min(max(c, 0), J.pixels - 1); };
  const int nb0 = AL ? bytes(c0, 4) : 0, nb1 = AL ? bytes(c1, 8) : 0,
            nb2 = AL ? bytes(c1 + 64, 8) : 0;
  const short2 *const m0 = J.master + (AL ? clip(c0) & ~3 : 0);
  const float2 *const s1 = J.slave + (AL ? clip(c1) & ~1 : 0);
  const int s2 = AL ? (clip(c1 + 64) & ~1) - (clip(c1) & ~1) : 0;
  // Slave pieces of two columns: the even ones from 512 on, the odd ones from
  // CO_ODD on, 4 bank groups further, so that neither the copies nor the reads
  // of a lane's pieces 2 lane and 2 lane + 1 conflict (10 x 3 burst: 103 us with
  // the pieces in order, 97 so).
  const unsigned sd = AL ? 16 * (lane >> 1) + (lane & 1 ? CO_ODD : 512)
                         : 16 * (lane >> 2) + (lane & 2 ? CO_ODD : 512) + 8 * (lane & 1);
  unsigned char *const mine = stage + warp * (CO_D * CO_ROW);
  const unsigned base = (unsigned)__cvta_generic_to_shared(mine);
  // The copies issued ahead of the last row, which nothing reads, end before the
  // item does: the next item's are then the only ones on a slot, and none is in
  // flight when a warp leaves the kernel.
  auto drain = [&]() {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
  };
  unsigned wr = 0;                         // the slot to write next (byte offset)
  auto after = [](unsigned slot) { return (slot + CO_ROW) & (CO_D * CO_ROW - 1); };
  int y = 0;                               // the next row to copy, and where it is
  const short2 *mp = m0;
  const float2 *sp = s1;
  auto seek = [&](int row) {
    y = row;
    const long yc = min(max(row, 0), J.lines - 1);
    mp = m0 + yc * J.master_pitch;
    sp = s1 + yc * J.slave_pitch;
  };
  // copies row y's columns into the next slot; zeros outside the image
  auto issue = [&]() {
    const bool row = (unsigned)y < (unsigned)y_end;
    const unsigned d = base + wr;
    if (AL) {
      co_copy<16>(d + 16 * lane, mp, row ? nb0 : 0);
      co_copy<16>(d + sd, sp, row ? nb1 : 0);
      co_copy<16>(d + sd + 256, sp + s2, row ? nb2 : 0);
    } else {
#pragma unroll
      for (int k = 0; k < CO_CPL; k++) {
        const int c = c0 + 32 * k, o = clip(c);
        const bool ok = row && c == o;
        co_copy<4>(d + 4 * (lane + 32 * k), mp + o, ok ? 4 : 0);
        co_copy<8>(d + sd + 128 * k, sp + o, ok ? 8 : 0);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    wr = after(wr);
    if ((unsigned)y < (unsigned)(y_end - 1)) {
      mp += J.master_pitch;
      sp += J.slave_pitch;
    }
    y++;
  };
  // the oldest row in flight: its products.  The barrier shows every lane's
  // copies to the warp, and lets the slot read last be written again.
  auto take = [&](float4 (&p)[CO_CPL]) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(CO_D - 2) : "memory");
    __syncwarp();
    const unsigned char *q = mine + after(wr);
    const int4 a = *reinterpret_cast<const int4 *>(q + 16 * lane);
    const float4 b = *reinterpret_cast<const float4 *>(q + 512 + 16 * lane);
    const float4 c = *reinterpret_cast<const float4 *>(q + CO_ODD + 16 * lane);
    const int m[CO_CPL] = {a.x, a.y, a.z, a.w};
    const float2 sv[CO_CPL] = {make_float2(b.x, b.y), make_float2(b.z, b.w),
                               make_float2(c.x, c.y), make_float2(c.z, c.w)};
#pragma unroll
    for (int i = 0; i < CO_CPL; i++)
      p[i] = coh_product(*reinterpret_cast<const short2 *>(&m[i]), sv[i]);
  };
  float *orow = J.coh + (long)r_begin * J.coh_pitch + x;
  // the next output row
  auto store = [&](const float4 (&o)[CO_CPL], const float (&c)[CO_CPL]) {
    float g[CO_CPL];
#pragma unroll
    for (int u = 0; u < CO_CPL; u++) g[u] = coh_gamma<false>(o[u], c[u]);
    if (B.compensated) {
#pragma unroll
      for (int u = 0; u < CO_CPL; u++) g[u] = coh_gamma<true>(o[u], c[u]);
    }
    if (vec_out) {
      *reinterpret_cast<float4 *>(orow) = make_float4(g[0], g[1], g[2], g[3]);
    } else if (out_lane) {
#pragma unroll
      for (int u = 0; u < CO_CPL; u++)
        if (x + u < J.pixels) orow[u] = g[u];
    }
    orow += J.coh_pitch;
  };

  if constexpr (WAZ == 0) {
    // taller windows: 4 output rows at a time over their common input rows
    constexpr int GR = 4;
    const int win_az = B.win_az, dy = (win_az - 1) / 2;
    int rows = 0;                          // copied of the group; groups overlap
    auto next = [&]() {
      issue();
      if (++rows == win_az + GR - 1) {
        rows = 0;
        seek(y + 1 - win_az);
      }
    };
    seek(r_begin - dy);
#pragma unroll 1
    for (int j = 0; j < CO_D - 1; j++) next();
    auto add_to = [&](float4 (&a)[CO_CPL], const float4 (&b)[CO_CPL]) {
#pragma unroll
      for (int i = 0; i < CO_CPL; i++) a[i] = add4(a[i], b[i]);
    };
    for (int r = r_begin; r < r_end; r += GR) {
      float4 a[GR][CO_CPL], pn[CO_CPL];
      float c[GR][CO_CPL];
      // the rows of the first windows only: a[k] = rows k .. GR - 2
#pragma unroll
      for (int k = 0; k < GR - 1; k++) {
        take(a[k]);
        next();
#pragma unroll
        for (int q = 0; q < k; q++) add_to(a[q], a[k]);
      }
      // the rows of all windows, the centre rows among them (win_az >= 7)
      take(a[GR - 1]);
      next();
#pragma unroll
      for (int k = 0; k < GR; k++)
#pragma unroll
        for (int i = 0; i < CO_CPL; i++) c[k][i] = a[GR - 1][i].z;
#pragma unroll 1
      for (int j = GR; j < win_az; j++) {
        take(pn);
        next();
        add_to(a[GR - 1], pn);
#pragma unroll
        for (int k = 0; k < GR; k++)
#pragma unroll
          for (int i = 0; i < CO_CPL; i++) c[k][i] = j <= dy + k ? pn[i].z : c[k][i];
      }
#pragma unroll
      for (int k = 0; k < GR - 1; k++) add_to(a[k], a[GR - 1]);
      // the rows of the last windows only
      float4 o[CO_CPL], e[CO_CPL];
      coh_box<WRG>(a[0], win, dx, o);
      store(o, c[0]);
#pragma unroll
      for (int k = 1; k < GR; k++) {
        take(pn);
        next();
#pragma unroll
        for (int i = 0; i < CO_CPL; i++) {
          e[i] = k == 1 ? pn[i] : add4(e[i], pn[i]);
          a[k][i] = add4(a[k][i], e[i]);
        }
        coh_box<WRG>(a[k], win, dx, o);
        if (r + k < r_end) store(o, c[k]);
      }
    }
    drain();
    return;
  }

  // products of the last R rows in a ring: at a step with phase f, row j (0
  // the oldest) is p[(f + j) % R]
  constexpr int RR = R > 0 ? R : 1;
  float4 p[RR][CO_CPL];
  seek(r_begin - DY);
#pragma unroll 1
  for (int j = 0; j < CO_D - 1; j++) issue();
#pragma unroll
  for (int j = 0; j < R; j++) {
    take(p[j]);
    issue();
  }
  // Output rows in pairs: the R rows that both windows hold are summed once.
  constexpr int UN = R & 1 ? 2 * R : R > 0 ? R : 1;
  for (int r = r_begin; r < r_end; r += UN) {
    float4 t[CO_CPL];                      // the sum of a pair's common rows
#pragma unroll
    for (int f = 0; f < UN; f++) {
      if (r + f < r_end) {
        float4 pn[CO_CPL], v[CO_CPL], o[CO_CPL];
        take(pn);
        issue();
        float sp_c[CO_CPL];
#pragma unroll
        for (int i = 0; i < CO_CPL; i++) {
          // vertical sums; the centre row is row DY of the window
          if (R == 0) {
            v[i] = pn[i];
          } else if (f & 1) {
            v[i] = add4(t[i], pn[i]);
          } else {
            // (the newest row last: it comes from memory)
            t[i] = p[(f + 1) % RR][i];
            if (R == 3) t[i] = add4(t[i], p[(f + 2) % RR][i]);
            if (R > 3) t[i] = add4(t[i], p[(f + 2) % RR][i]);
            if (R == 4) t[i] = add4(t[i], p[(f + 3) % RR][i]);
            if (R == 5) t[i] = add4(t[i], add4(p[(f + 3) % RR][i], p[(f + 4) % RR][i]));
            t[i] = R > 1 ? add4(t[i], pn[i]) : pn[i];
            v[i] = add4(p[f % RR][i], t[i]);
          }
          sp_c[i] = DY < R ? p[(f + DY) % RR][i].z : pn[i].z;
          if (R > 0) p[f % RR][i] = pn[i];
        }
        coh_box<WRG>(v, win, dx, o);
        store(o, sp_c);
      }
    }
  }
  drain();
}

// Warps per SM: 16 where up to two rows of products are kept, 12 for three and
// four rows; 8 for the five rows of a height of 6 (24 x 6: 157 us, 179 with 12
// warps and spills) and for the four window sums of the taller ones (30 x 9:
// 137 and 142).
template <int WAZ, int WRG, bool AL>
__global__ void __launch_bounds__(CO_NT, WAZ == 0 || WAZ == 6 ? 4 : WAZ <= 3 ? 8 : 6)
    coherence_kernel(const __grid_constant__ CoBatch B) {
  __shared__ __align__(16) unsigned char stage[CO_NW * CO_D * CO_ROW];
  __shared__ int next_item;
  // one work item per CTA, or (persistent) items from the queue until it is
  // empty; a single call site keeps one inlined copy of the item code
  int item = blockIdx.x;
  if (B.counter) {
    if (threadIdx.x == 0) next_item = atomicAdd(B.counter, 1);
    __syncthreads();
    item = next_item;
    __syncthreads();
  }
  while (item < B.total_items) {
    coherence_item<WAZ, WRG, AL>(B, item, stage);
    if (!B.counter) break;
    __syncthreads();
    if (threadIdx.x == 0) next_item = atomicAdd(B.counter, 1);
    __syncthreads();
    item = next_item;
  }
}


// Lanes whose columns only feed the windows, left and right of the outputs.
static void window_lanes(int win_rg, int &nl, int &nr) {
  const int dx = (win_rg - 1) / 2;
  nl = (dx + CO_CPL - 1) / CO_CPL;
  nr = (CO_CPL - 1 - dx + win_rg - 1) / CO_CPL;
}

template <int WAZ, int WRG, bool AL>
static int launch_al(const CohJob *jobs, int njobs, int win_rg, int win_az, const TileCfg &cfg,
                    int dev, cudaStream_t st) {
  static PerDeviceOnce setup;
  int resident = 0;
  const int s0 = once_per_device(
      setup, dev,
      [&](int &v) -> int {
        int per_sm = 0, sms = 0;
        TOPS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, coherence_kernel<WAZ, WRG, AL>, CO_NT, 0));
        TOPS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        v = per_sm * sms;
        return TOPS_OK;
      },
      &resident);
  if (s0 != TOPS_OK) return s0;
  int nl, nr;
  window_lanes(win_rg, nl, nr);
  const int tw = CO_NW * CO_CPL * (32 - nl - nr);   // output columns of a CTA
  // segment rows: the fewest row times of the last CTA to finish, waves x (rows
  // + the window's halo and the first loads, worth about 8 rows), up to the
  // caller's limit, which 8 waves and more take as it is; whole groups, so that
  // a row's sums do not depend on the cut
  const int most = cfg.seg_rows ? (cfg.seg_rows + 3) & ~3 : 256;
  int seg_rows = 0;
  {
    const int kSegs[] = {most, 256, 192, 128, 96, 64, 48, 32, 24, 16, 8};
    long best = 0;
    for (int sr : kSegs) {
      if (sr > most) continue;
      long items = 0;
      for (int j = 0; j < njobs; j++)
        items += (long)((jobs[j].pixels + tw - 1) / tw) * ((jobs[j].lines + sr - 1) / sr);
      const long cost = (items + resident - 1) / resident * (sr + 8 + win_az);
      if (!seg_rows || cost < best) {
        best = cost;
        seg_rows = sr;
      }
      if (cfg.seg_rows && sr == most && items >= 8L * resident) break;
    }
  }
  for (int j0 = 0, k = 0; j0 < njobs; j0 += CO_MAXJOBS, k++) {
    CoBatch B;
    B.njobs = 0;
    B.win_rg = win_rg;
    B.win_az = win_az;
    B.compensated = cfg.compensated;
    B.nl = nl;
    B.nr = nr;
    B.counter = cfg.counters ? cfg.counters + k : nullptr;
    int items = 0;
    for (int j = j0; j < njobs && j < j0 + CO_MAXJOBS; j++) {
      CohJob &J = B.jobs[B.njobs];
      J = jobs[j];
      J.seg_rows = seg_rows;
      J.segs = (J.lines + seg_rows - 1) / seg_rows;
      J.strips = (J.pixels + tw - 1) / tw;
      J.item_begin = items;
      items += J.strips * J.segs;
      B.njobs++;
    }
    B.total_items = items;
    if (!items) continue;
    int grid = items;
    if (B.counter) {
      TOPS_CUDA_TRY(cudaMemsetAsync(B.counter, 0, sizeof(int), st));
      grid = min(items, cfg.grid > 0 ? cfg.grid : resident);
    }
    coherence_kernel<WAZ, WRG, AL><<<grid, CO_NT, 0, st>>>(B);
    TOPS_CUDA_TRY(cudaGetLastError());
  }
  return TOPS_OK;
}

template <int WAZ, int WRG>
static int launch_t(const CohJob *jobs, int njobs, int win_rg, int win_az, const TileCfg &cfg,
                    int dev, cudaStream_t st) {
  bool al = true;
  for (int j = 0; j < njobs; j++) al = al && jobs[j].al16;
  return al ? launch_al<WAZ, WRG, true>(jobs, njobs, win_rg, win_az, cfg, dev, st)
            : launch_al<WAZ, WRG, false>(jobs, njobs, win_rg, win_az, cfg, dev, st);
}

// Compiled windows: 10 and the reference driver's 24 samples
// (Func.cpp:2583-2584), with 3 and 6 rows (1500 x 21000, us, as any window of 7
// or more and so: 10 x 3 125 and 104, 10 x 6 209 and 144, 24 x 3 143 and 119,
// 24 x 6 238 and 162), and every height up to 6 rows with range windows of up to
// 6 samples (one compiled case each) and of 7 or more (5 x 5 took 133 us with
// the lane sums picked at run time, 49 this way).
// Taller windows sum the rows that 4 output rows share once.
int launch_coherence(const CohJob *jobs, int njobs, int win_rg, int win_az, const TileCfg &cfg,
                     cudaStream_t st) {
  if (win_rg < 1 || win_az < 1 || win_rg > CO_MAX_WIN_RG) return TOPS_E_INVALID;
  if (cfg.seg_rows < 0 || cfg.seg_rows > 512 || (cfg.seg_rows && cfg.seg_rows < 8))
    return TOPS_E_INVALID;
  int dev = 0;
  TOPS_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return TOPS_E_INVALID;
#define CO_LAUNCH(az, rg) return launch_t<az, rg>(jobs, njobs, win_rg, win_az, cfg, dev, st)
  if (win_rg == 10 && win_az == 3) CO_LAUNCH(3, 10);
  if (win_rg == 10 && win_az == 6) CO_LAUNCH(6, 10);
  if (win_rg == 24 && win_az == 3) CO_LAUNCH(3, 24);
  if (win_rg == 24 && win_az == 6) CO_LAUNCH(6, 24);
  if (win_rg <= 6) {
    switch (win_az) {
      case 1: CO_LAUNCH(1, CO_SMALL);
      case 2: CO_LAUNCH(2, CO_SMALL);
      case 3: CO_LAUNCH(3, CO_SMALL);
      case 4: CO_LAUNCH(4, CO_SMALL);
      case 5: CO_LAUNCH(5, CO_SMALL);
      case 6: CO_LAUNCH(6, CO_SMALL);
      default: CO_LAUNCH(0, CO_SMALL);
    }
  }
  switch (win_az) {
    case 1: CO_LAUNCH(1, CO_LARGE);
    case 2: CO_LAUNCH(2, CO_LARGE);
    case 3: CO_LAUNCH(3, CO_LARGE);
    case 4: CO_LAUNCH(4, CO_LARGE);
    case 5: CO_LAUNCH(5, CO_LARGE);
    case 6: CO_LAUNCH(6, CO_LARGE);
    default: CO_LAUNCH(0, CO_LARGE);
  }
#undef CO_LAUNCH
}

int fill_coh_job(const tops_coh_job &u, CohJob &J) {
  if (!u.master || !u.slave || !u.coh || u.lines <= 0 || u.pixels <= 0) return TOPS_E_INVALID;
  if ((u.master_pitch % sizeof(short2)) || (u.slave_pitch % sizeof(float2)) ||
      (u.coh_pitch % sizeof(float)))
    return TOPS_E_INVALID;
  J.master = static_cast<const short2 *>(u.master);
  J.master_pitch = (long)(u.master_pitch / sizeof(short2));
  J.slave = static_cast<const float2 *>(u.slave);
  J.slave_pitch = (long)(u.slave_pitch / sizeof(float2));
  J.coh = u.coh;
  J.coh_pitch = (long)(u.coh_pitch / sizeof(float));
  if (J.master_pitch < u.pixels || J.slave_pitch < u.pixels || J.coh_pitch < u.pixels)
    return TOPS_E_INVALID;
  J.lines = u.lines;
  J.pixels = u.pixels;
  // vector access: four columns of a row start on a 16-byte boundary
  const uintptr_t m = reinterpret_cast<uintptr_t>(u.master);
  const uintptr_t s = reinterpret_cast<uintptr_t>(u.slave);
  J.al16 = ((m | s | u.master_pitch | u.slave_pitch) & 15) == 0;
  J.out_al16 = ((reinterpret_cast<uintptr_t>(u.coh) | u.coh_pitch) & 15) == 0;
  return TOPS_OK;
}

}  // namespace tops

using namespace tops;

extern "C" int tops_coherence(const tops_coh_job *jobs, int njobs, int win_rg, int win_az,
                              void *stream) {
  if ((!jobs && njobs > 0) || njobs < 0) return TOPS_E_INVALID;
  std::vector<CohJob> J(njobs);
  for (int j = 0; j < njobs; j++) {
    int s = fill_coh_job(jobs[j], J[j]);
    if (s != TOPS_OK) return s;
  }
  return launch_coherence(J.data(), njobs, win_rg, win_az, TileCfg(),
                          static_cast<cudaStream_t>(stream));
}

namespace tops {

int coherence_launch(const tops_coh_job *jobs, int njobs, int win_rg, int win_az,
                     const TileCfg &cfg, cudaStream_t st) {
  if ((!jobs && njobs > 0) || njobs < 0) return TOPS_E_INVALID;
  std::vector<CohJob> J(njobs);
  for (int j = 0; j < njobs; j++) {
    int s = fill_coh_job(jobs[j], J[j]);
    if (s != TOPS_OK) return s;
  }
  return launch_coherence(J.data(), njobs, win_rg, win_az, cfg, st);
}

}  // namespace tops
