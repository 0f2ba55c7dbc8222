// Strip walk: the FP64 quadtree walk (TreeQuadParticles::walkTree_recur,
// include/quadTree.h:990-1128) for the 32 rays of a warp.
//
// The preorder node array is read 32 consecutive nodes (a strip) at a time,
// one node per lane, and each lane classifies its node against the bounding
// box of the warp's rays:
//   * A, accepted by all: the nearest point of the box is outside the node's
//     opening radius;
//   * O, opened by all: the farthest point is inside;
//   * M, mixed: the box straddles the radius; the rays take their own test.
// A node is visited only when no A node before it covers it (its index lies in
// that node's subtree), which one reduction over the strip's lanes gives.  So
// the opening test, the index arithmetic and the vote that a node-at-a-time
// walk repeats for every ray and node are done once per 32 nodes; far-field
// terms and leaf particles are then evaluated without tests.  The box tests
// are FP32 on FP64 differences from the box's centre, with a relative margin
// of 4e-6 (over ten times their rounding); inside it a node is M, so every ray
// interacts with exactly the nodes that its own walk would.
//
// Far-field rows are queued in shared memory (with the mask of the rays that
// take them) and summed from there; a leaf's particles are converted to double
// once per warp and read from shared memory.  The reciprocal is a seed from
// the PTX approximation and one third-order Newton-Raphson step, the screening
// exponential a table and a short polynomial: 38 FP64 instructions a far-field
// term and 25 a particle, where divisions and exp() took about three times as
// many.
//
// A ray's terms are added in node order, in the steps in which the
// node-at-a-time walk (walk_f64) adds them, so its sums do not depend on the
// other rays and stay within a few roundings of that walk's.
//
// Bound by FP64 latency and issue: 512^2 rays on 2^18 particles take 12.9 ms with
// walk_f64, 7.9 with one ray per lane (96 registers, 18 warps per SM), 7.0 with two
// (128 registers, 14 warps; FP64 pipe and issue 57 %).  Of the 7.9, 2.6 are far-field
// terms (76 % of the FP64 pipe's rate), 2.4 particles, 1.8 the exponentials of both,
// 2.1 strips and staging; 80 or 128 registers and loops unrolled by 2 are within 3 %
// of it, unrolled by 4 13.3 ms (the instruction cache).  Where most nodes of a strip
// are mixed (few rays in a large tree, small leaves, wide opening angles) walk_f64
// is the faster one: force_rule, host_force_rule and plane_parts_max draw the line.
#pragma once
#include "walk.cuh"

namespace glb {

// One warp's shared memory: the far-field queue (rows {cx, cy},
// {mass, q0}, {q2, mask}) and the particles of the leaf being evaluated.
struct StripWarp {
  double2 far[64 * 3];
  double2 part[32 * 2];
};

// 1/a: the PTX seed (a relative error of about 2^-20) and one Newton-Raphson step
// of third order, x (1 + e + e^2) with e = 1 - a x: 0.507 ulp measured, 3 in 10^4
// results differ from the division's.
__device__ __forceinline__ double strip_rcp(double a) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  const double e = __fma_rn(-a, x, 1.0);
  return __fma_rn(x, __fma_rn(e, e, e), x);
}

// exp(-t), t >= 0, by the table-driven method of P. T. P. Tang (ACM TOMS 15, 1989)
// with 512 table entries: t = n ln2/512 + r with |r| <= 6.8e-4 (ln2/512 in two parts,
// so that r is good to its last bit), exp(-t) = 2^(-n/512) (1 + p) with p = exp(-r) - 1
// by its Taylor polynomial of degree 4 (r^5/120 is below 1.3e-18).  The table holds
// 2^(-j/512) rounded (its high word plus 2048 j, so that 2048 n off it gives
// 2^(-n/512)) and what the rounding lost, relative; the latter joins p in the last
// product at no cost, and the error stays near half a unit in the last place (0.62
// measured up to t = 50, exp() 0.86; means 0.251 and 0.258).  1,024 entries, 16 KB,
// leave the L1 cache 60 KB beside five blocks in place of 92: 4,097 rays through ten
// planes 4.43 ms, with 512 entries 4.33.  The reciprocal of the step, the step's first
// part and the two highest terms of the polynomial have a zero low word, so that they
// are immediates; full double constants cost two instructions each per use.  t is
// held at 700 (by its high word), where exp(-t) is below 1e-304.  The table index is
// masked, whatever a NaN makes of n; the result is NaN by r.
constexpr double kC3 = -0x1.55555p-3, kC4 = 0x1.55555p-5;
constexpr double kStepInv = 0x1.71547p+9, kStep1 = 0x1.62e43p-10, kStep2 = -0x1.05c610ca86c39p-38;
__device__ __forceinline__ double strip_exp_neg(double t, const ExpTab &E) {
  constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52
  t = __hiloint2double(min(__double2hiint(t), 0x4085e000), __double2loint(t));
  const double s = __fma_rn(t, kStepInv, kShift);
  const int n = __double2loint(s);
  const double m = s - kShift;
  const double r = __fma_rn(m, -kStep2, __fma_rn(m, -kStep1, t));
  double p = __fma_rn(r, kC4, kC3);
  p = __fma_rn(p, r, 0.5);
  p = __fma_rn(p, r, -1.0);
  const double2 T = E.t[n & 511];
  const double h = __hiloint2double(__double2hiint(T.x) - n * 2048, __double2loint(T.x));
  return __fma_rn(h, __fma_rn(r, p, T.y), h);
}

// A block's copy of the table.
__device__ __forceinline__ void strip_exp_table(ExpTab &E, const ExpTab *src) {
  if (!src) return;  // no tree with nodes: the table is not read
  const double2 *f = reinterpret_cast<const double2 *>(src);
  double2 *t = reinterpret_cast<double2 *>(&E);
  for (int i = threadIdx.x; i < (int)(sizeof(ExpTab) / sizeof(double2)); i += blockDim.x) t[i] = __ldg(f + i);
}

// The tree as a walk reads it, by value: fields of a descriptor in global
// memory would be loaded again after every store to shared memory.
struct StripTree {
  const TNode *tnodes;
  const FNode *fnodes;
  const GNode *nodes;
  const float4 *parts;
  double s2, pia;  // screening scale squared, pi * inv_area
  const TreeDev *dev;
  __device__ __forceinline__ explicit StripTree(const TreeDev &T)
      : tnodes(T.tnodes), fnodes(T.fnodes), nodes(T.nodes), parts(T.parts), s2(T.screen2), pia(kPi * T.inv_area),
        dev(&T) {}
};

// One ray's sums: alpha, kappa, gamma (g1 halved), potential.
struct StripAcc {
  double a0 = 0, a1 = 0, k = 0, g0 = 0, g1 = 0, p = 0;
};

struct StripVec6 {
  double v[6];
};
// The B-spline correction of one particle, out of line (a few per ray).
template <bool PHI>
__device__ __noinline__ StripVec6 strip_bspline(double x0, double x1, double rr, float4 Q, double phic) {
  StripVec6 o = {{0, 0, 0, 0, 0, 0}};
  bspline_f64<PHI>(x0, x1, sqrt(rr), (double)Q.z, (double)Q.w, phic, o.v);
  return o;
}
template <bool PHI>
__device__ __forceinline__ void strip_soften(const TreeDev *T, double x0, double x1, double rr, float4 Q, StripAcc &L) {
  const StripVec6 o = strip_bspline<PHI>(x0, x1, rr, Q, PHI ? T->phiintconst : 0.0);
  L.a0 += o.v[0];
  L.a1 += o.v[1];
  L.k += o.v[2];
  L.g0 += o.v[3];
  L.g1 += 0.5 * o.v[4];
  if (PHI) L.p += o.v[5];
}

// The warp's constants of one walk.  R: rays per lane.
template <int R>
struct StripWalk {
  double rx[R], ry[R];  // this lane's rays
  double bx, by;        // centre of the box of the warp's valid rays
  float hx, hy;         // its half extents, rounded up
  unsigned vmask[R];    // lanes whose r-th ray is valid
  int lane;
  __device__ __forceinline__ bool has(const unsigned *m, int r) const { return m[r] >> lane & 1u; }
};

// One mask of lanes per ray of a lane.
template <int R>
struct StripMask {
  unsigned m[R];
  __device__ __forceinline__ bool any() const {
    unsigned a = m[0];
#pragma unroll
    for (int r = 1; r < R; ++r) a |= m[r];
    return a != 0u;
  }
  __device__ __forceinline__ bool is(const unsigned *v) const {
    bool e = true;
#pragma unroll
    for (int r = 0; r < R; ++r) e = e && m[r] == v[r];
    return e;
  }
};

// FP32 keys in the order of their values, for the integer warp reductions.
__device__ __forceinline__ int f_key(float f) {
  const int b = __float_as_int(f);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float key_f(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// The box is that of the rays rounded outwards to FP32 (a warp's rays spread
// far wider than that); rays that are not finite stay out of it (whatever their
// nodes' classes, their sums are not finite).
template <int R>
__device__ __forceinline__ StripWalk<R> strip_begin(const double *rx, const double *ry, const bool *valid) {
  StripWalk<R> w;
  w.lane = threadIdx.x & 31;
  constexpr float kBig = 1e30f;
  float a = kBig, b = -kBig, c = kBig, d = -kBig;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    w.rx[r] = rx[r];
    w.ry[r] = ry[r];
    w.vmask[r] = __ballot_sync(kFull, valid[r]);
    if (valid[r] && isfinite(rx[r]) && isfinite(ry[r])) {
      a = fminf(a, __double2float_rd(rx[r]));
      b = fmaxf(b, __double2float_ru(rx[r]));
      c = fminf(c, __double2float_rd(ry[r]));
      d = fmaxf(d, __double2float_ru(ry[r]));
    }
  }
  const float x0 = key_f(__reduce_min_sync(kFull, f_key(a))), x1 = key_f(__reduce_max_sync(kFull, f_key(b)));
  const float y0 = key_f(__reduce_min_sync(kFull, f_key(c))), y1 = key_f(__reduce_max_sync(kFull, f_key(d)));
  w.bx = 0.5 * ((double)x0 + (double)x1);
  w.by = 0.5 * ((double)y0 + (double)y1);
  w.hx = __double2float_ru(0.5 * ((double)x1 - (double)x0)) * 1.000001f;
  w.hy = __double2float_ru(0.5 * ((double)y1 - (double)y0)) * 1.000001f;
  return w;
}

// 1: accepted by all, 2: opened by all, 0: mixed.  olo, ohi: the squared
// opening radius less and plus the margin.  The half extents are rounded up
// by 1e-6, which covers the rounding of dx - hx where the two are close.
template <int R>
__device__ __forceinline__ int strip_class(const StripWalk<R> &w, double cx, double cy, float olo, float ohi) {
  const float dx = fabsf((float)(cx - w.bx)), dy = fabsf((float)(cy - w.by));
  const float nx = fmaxf(dx - w.hx, 0.f), ny = fmaxf(dy - w.hy, 0.f), fx = dx + w.hx, fy = dy + w.hy;
  return nx * nx + ny * ny >= ohi ? 1 : (fx * fx + fy * fy < olo ? 2 : 0);
}

// The cnt queued far-field rows for every valid lane, or with MASKED for the
// lanes of each row's mask.
template <bool PHI, bool SCREEN, bool SHEET, bool MASKED, int R>
__device__ __forceinline__ void strip_far_rows(const StripTree &T, const StripWalk<R> &w, const StripWarp &W, int cnt,
                                               const ExpTab &tab, StripAcc *LL) {
  const double s2 = T.s2, pia = T.pia;
  const double2 *row = W.far;
#pragma unroll 1
  for (int j = 0; j < cnt; ++j, row += 3) {
    const double2 c = row[0], mq = row[1], qm = row[2];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      StripAcc &L = LL[r];
      const double dx = c.x - w.rx[r], dy = c.y - w.ry[r];
      const double xx = __dmul_rn(dx, dx), r2 = __fma_rn(dy, dy, xx);
      const double ir2 = strip_rcp(r2);
      const double si = SCREEN ? __dmul_rn(strip_exp_neg(__dmul_rn(r2, s2), tab), ir2) : ir2;
      const double a = __dmul_rn(mq.x, si), s4 = __dmul_rn(si, ir2);  // mass/pi scr/r^2, scr/r^4
      const double qx = __fma_rn(mq.y, dx, __dmul_rn(qm.x, dy)), qy = __fma_rn(qm.x, dx, -__dmul_rn(mq.y, dy));
      const double e = __dmul_rn(__dmul_rn(4.0, s4), __dmul_rn(__fma_rn(qx, dx, __dmul_rn(qy, dy)), ir2));
      const double t = SHEET ? __fma_rn(mq.x, pia, -a) : -a;
      const double gc = __dmul_rn(a, ir2), dd = __fma_rn(-dy, dy, xx), xy = __dmul_rn(dx, dy);
      if (!MASKED || ((unsigned)(r == 0 ? __double2loint(qm.y) : __double2hiint(qm.y)) >> w.lane & 1u)) {
        L.a0 = __fma_rn(e, dx, __fma_rn(-s4, qx, __fma_rn(t, dx, L.a0)));
        L.a1 = __fma_rn(e, dy, __fma_rn(-s4, qy, __fma_rn(t, dy, L.a1)));
        L.g0 = __fma_rn(-gc, dd, L.g0);
        L.g1 = __fma_rn(-gc, xy, L.g1);
        if (PHI) {
          const double scr = __dmul_rn(si, r2) * (1.0 / kPi);
          L.p += 0.5 * T.dev->phi_mass * log(r2) * scr -
                 0.5 * (T.dev->phi_q0 * xx + T.dev->phi_q1 * dy * dy + 2 * T.dev->phi_q2 * xy) * (1.0 / kPi) * s4 -
                 0.5 * pia * mq.x * r2;
        }
      }
    }
  }
}

// The far-field queue: rows waiting, whether one of them is not for every
// valid lane.
struct StripQueue {
  int n = 0;
  bool masked = false;
};

// Queues the far-field rows of the strip positions in `who` (r0, r1, q2: this
// lane's row; fm: the lanes that take it).
template <int R>
__device__ __forceinline__ void strip_push(const StripWalk<R> &w, StripWarp &W, StripQueue &q, unsigned who, double2 r0,
                                           double2 r1, double q2, const StripMask<R> &fm) {
  if (who >> w.lane & 1u) {
    double2 *row = W.far + 3 * (q.n + __popc(who & ((1u << w.lane) - 1u)));
    row[0] = r0;
    row[1] = r1;
    row[2] = make_double2(q2, __hiloint2double(R > 1 ? (int)fm.m[R - 1] : 0, (int)fm.m[0]));
  }
  q.n += __popc(who);
}

// A leaf opened by the rays of `om`: its particles as point masses, with their
// softening where the leaf applies it (quadTree.h:1017-1077).
template <bool PHI, bool SCREEN, bool SHEET, int R>
__device__ __forceinline__ void strip_leaf(const StripTree &T, const StripWalk<R> &w, StripWarp &W, int node, int p0,
                                           int n, const StripMask<R> &om, const ExpTab &tab, StripAcc *LL) {
  float4 Q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (w.lane < n) Q = __ldg(T.parts + p0 + w.lane);  // in flight with the node's row
  const GNode *nd = T.nodes + node;
  const double width = nd->width;
  unsigned nearc = 0;  // bit r: this lane's r-th ray is within the near radius
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double cx = nd->cx - w.rx[r], cy = nd->cy - w.ry[r];
    if (w.has(om.m, r) && cx * cx + cy * cy < nd->near2) nearc |= 1u << r;
  }
  const double s2 = T.s2, pia = T.pia;
  // A particle within the 1e-10 of the coincidence clamp lies in a leaf whose
  // near radius (2.41 widths) the ray is in, unless the leaf is narrower than
  // that; other leaves need neither the clamp nor the softening test.
  const bool plain = !__any_sync(kFull, nearc != 0u) && width > 1e-9 && om.is(w.vmask);
  for (int q0 = 0; q0 < n; q0 += 32) {
    const int m = min(32, n - q0);
    __syncwarp();
    if (w.lane < m) {
      if (q0) Q = __ldg(T.parts + p0 + q0 + w.lane);
      const double size = (double)Q.w;
      W.part[2 * w.lane] = make_double2((double)Q.x, (double)Q.y);
      // mass / pi, and the squared radius of the softening this leaf applies
      W.part[2 * w.lane + 1] = make_double2((double)Q.z * (1.0 / kPi), size < width ? 4 * size * size : 0.0);
    }
    __syncwarp();
    const double2 *row = W.part;
    if (plain) {
#pragma unroll 1
      for (int j = 0; j < m; ++j, row += 2) {
        const double2 c = row[0];
        const double mpi = row[1].x;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          StripAcc &L = LL[r];
          const double x0 = c.x - w.rx[r], x1 = c.y - w.ry[r];
          const double xx = __dmul_rn(x0, x0), rr = __fma_rn(x1, x1, xx);
          const double ir2 = strip_rcp(rr);
          double pre = __dmul_rn(mpi, ir2);
          if (SCREEN) pre = __dmul_rn(pre, strip_exp_neg(__dmul_rn(rr, s2), tab));  // mass scr / (pi r^2)
          const double gc = __dmul_rn(pre, ir2), t = SHEET ? __fma_rn(-pia, mpi, pre) : pre;
          L.a0 = __fma_rn(-t, x0, L.a0);
          L.a1 = __fma_rn(-t, x1, L.a1);
          L.g0 = __fma_rn(-gc, __fma_rn(-x1, x1, xx), L.g0);
          L.g1 = __fma_rn(-gc, __dmul_rn(x0, x1), L.g1);
          if (PHI) L.p += 0.5 * pre * rr * log(rr) - 0.5 * pia * mpi * rr;
        }
      }
    } else {
#pragma unroll 1
      for (int j = 0; j < m; ++j, row += 2) {
        const double2 c = row[0], ms = row[1];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          StripAcc &L = LL[r];
          const double x0 = c.x - w.rx[r], x1 = c.y - w.ry[r];
          const double xx = __dmul_rn(x0, x0);
          double rr = __fma_rn(x1, x1, xx);
          const double t2 = __dmul_rn(rr, s2);
          rr = rr < 1e-20 ? 1e-20 : rr;
          const double ir2 = strip_rcp(rr);
          double pre = __dmul_rn(ms.x, ir2);
          if (SCREEN) pre = __dmul_rn(pre, strip_exp_neg(t2, tab));
          const double gc = __dmul_rn(pre, ir2), t = SHEET ? __fma_rn(-pia, ms.x, pre) : pre;
          if (w.has(om.m, r)) {
            L.a0 = __fma_rn(-t, x0, L.a0);
            L.a1 = __fma_rn(-t, x1, L.a1);
            L.g0 = __fma_rn(-gc, __fma_rn(-x1, x1, xx), L.g0);
            L.g1 = __fma_rn(-gc, __dmul_rn(x0, x1), L.g1);
            if (PHI) L.p += 0.5 * pre * rr * log(rr) - 0.5 * pia * ms.x * rr;
          }
          if ((nearc >> r & 1u) && rr < ms.y) strip_soften<PHI>(T.dev, x0, x1, rr, __ldg(T.parts + p0 + q0 + j), L);
        }
      }
    }
  }
}

// Softened particles listed at an internal node (quadTree.h:1048-1077).
template <bool PHI, int R>
__device__ __forceinline__ void strip_bigs(const StripTree &T, const StripWalk<R> &w, int node, const StripMask<R> &om,
                                           StripAcc *LL) {
  const GNode *nd = T.nodes + node;
#pragma unroll 1
  for (int r = 0; r < R; ++r) {
    const double rx = r == 0 ? w.rx[0] : w.rx[R - 1], ry = r == 0 ? w.ry[0] : w.ry[R - 1];
    const double cx = nd->cx - rx, cy = nd->cy - ry;
    if (!((r == 0 ? om.m[0] : om.m[R - 1]) >> w.lane & 1u) || !(cx * cx + cy * cy < nd->near2)) continue;
#pragma unroll 1
    for (int b = nd->bstart, e = b + nd->bcount; b < e; ++b) {
      const float4 Q = __ldg(T.dev->bigs + b);
      const double x0 = (double)Q.x - rx, x1 = (double)Q.y - ry;
      double rr = x0 * x0 + x1 * x1;
      if (rr < 1e-20) rr = 1e-20;
      const double size = (double)Q.w;
      if (rr < 4 * size * size) {
        if (r == 0)
          strip_soften<PHI>(T.dev, x0, x1, rr, Q, LL[0]);
        else
          strip_soften<PHI>(T.dev, x0, x1, rr, Q, LL[R - 1]);
      }
    }
  }
}

// The walk's nodes in [base, end): base moves to the next node to visit (it
// may pass end), resume is this lane's next node (it sits out nodes before
// it).  The loop keeps one copy of each evaluation, for the instruction cache.
template <bool PHI, bool SCREEN, bool SHEET, int R>
__device__ __forceinline__ void strip_range(const StripTree &T, const StripWalk<R> &w, StripWarp &W, const ExpTab &tab,
                                            int &base, int end, int *resume, StripAcc *L) {
  StripQueue q;
  while (base < end) {
    const int sbase = base, i = base + w.lane;
    const bool in = i < end;
    int skip = 0, info = 0, cls = 3;
    double2 r0 = make_double2(0, 0);
    if (in) {
      const double2 *sp = reinterpret_cast<const double2 *>(T.tnodes + i);
      r0 = __ldg(sp);
      const float4 o = __ldg(reinterpret_cast<const float4 *>(sp + 1));
      skip = __float_as_int(o.z);
      info = __float_as_int(o.w);
      cls = strip_class(w, r0.x, r0.y, o.x, o.y);
    }
    const int pstart = skip;
    if (info < 0) skip = i + 1;
    // strip positions inside the subtree of an A node before them
    const int span = min(skip - base, 32);
    const unsigned cov =
        (cls == 1 && span > w.lane + 1) ? (span >= 32 ? 0u : 1u << span) - (2u << w.lane) : 0u;
    const unsigned covered = __reduce_or_sync(kFull, cov);
    const bool live = in && !(covered >> w.lane & 1u);
    const bool isA = live && cls == 1;
    // this lane's far-field row, unless the node is certain to be opened
    double2 r1 = make_double2(0, 0);
    double q2 = 0;
    if (live && (cls & 2) == 0) {
      const double2 *f = reinterpret_cast<const double2 *>(T.fnodes + i);
      r1 = __ldg(f);
      q2 = __ldg(f + 1).x;
    }
    const unsigned am = __ballot_sync(kFull, isA), mm = __ballot_sync(kFull, live && cls == 0);
    const unsigned ev = mm | __ballot_sync(kFull, live && cls == 2 && info != 0);
    int next = max(min(base + 32, end), (int)__reduce_max_sync(kFull, isA ? (unsigned)skip : 0u));
    // slow: node by node, some rays sit out part of the strip or take a test
    bool late = false;
#pragma unroll
    for (int r = 0; r < R; ++r) late = late || (w.has(w.vmask, r) && resume[r] > base);
    const bool slow = mm != 0u || __any_sync(kFull, late);
    unsigned todo = slow ? am | ev : ev, pend = slow ? 0u : am;
    StripMask<R> fm;
#pragma unroll
    for (int r = 0; r < R; ++r) fm.m[r] = w.vmask[r];
    for (;;) {
      // the next node with particles to evaluate, and the far-field rows before it
      int node = -1, inf = 0;
      unsigned push = pend;
      StripMask<R> om;
#pragma unroll
      for (int r = 0; r < R; ++r) om.m[r] = w.vmask[r];
      while (todo) {
        const int b = __ffs(todo) - 1;
        todo &= todo - 1;
        inf = __shfl_sync(kFull, info, b);
        if (slow) {
          StripMask<R> act;
#pragma unroll
          for (int r = 0; r < R; ++r) act.m[r] = __ballot_sync(kFull, base + b >= resume[r]) & w.vmask[r];
          if (am >> b & 1u) {
            if (w.lane == b) fm = act;
            if (act.any()) pend |= 1u << b;
            continue;
          }
          const int sk = __shfl_sync(kFull, skip, b);
          om = act;
          if (mm >> b & 1u) {
            const GNode *nd = T.nodes + base + b;
            StripMask<R> fa;
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const double cx = nd->cx - w.rx[r], cy = nd->cy - w.ry[r];
              om.m[r] = __ballot_sync(kFull, cx * cx + cy * cy < nd->open2) & act.m[r];
              fa.m[r] = act.m[r] & ~om.m[r];
              if (w.has(fa.m, r)) resume[r] = sk;
            }
            if (w.lane == b) fm = fa;
            if (fa.any()) pend |= 1u << b;
          }
          if (!om.any()) {  // nobody opens it: past its subtree
            todo &= sk - base >= 32 ? 0u : ~((1u << (sk - base)) - 1u);
            next = max(next, sk);
            continue;
          }
          if (inf == 0) continue;
        } else {
          push = pend & ((1u << b) - 1u);
        }
        node = base + b;
        break;
      }
      if (slow) {
        push = pend;
        q.masked = q.masked || __any_sync(kFull, (push >> w.lane & 1u) && !fm.is(w.vmask));
      }
      strip_push(w, W, q, push, r0, r1, q2, fm);
      pend &= ~push;
      bool flush = q.n > 0;
      if (node < 0) {
        base = next;
        if (slow) {
          unsigned first = 0x7fffffffu;
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (w.has(w.vmask, r)) first = min(first, (unsigned)resume[r]);
          base = max(base, (int)__reduce_min_sync(kFull, first));
        }
        flush = q.n >= 32 || (base >= end && q.n > 0);
      }
      if (flush) {
        __syncwarp();
        if (q.masked)
          strip_far_rows<PHI, SCREEN, SHEET, true, R>(T, w, W, q.n, tab, L);
        else
          strip_far_rows<PHI, SCREEN, SHEET, false, R>(T, w, W, q.n, tab, L);
        __syncwarp();
        q.n = 0;
        q.masked = false;
      }
      if (node < 0) break;
      if (inf < 0)
        strip_leaf<PHI, SCREEN, SHEET, R>(T, w, W, node, __shfl_sync(kFull, pstart, node - sbase), -inf, om, tab, L);
      else
        strip_bigs<PHI, R>(T, w, node, om, L);
    }
  }
}

template <bool PHI, int R>
__device__ __forceinline__ void strip_run(const StripTree &T, const StripWalk<R> &w, StripWarp &W, const ExpTab &tab,
                                          int base, int end, int *resume, StripAcc *L) {
  if (T.pia != 0.0)
    strip_range<PHI, true, true, R>(T, w, W, tab, base, end, resume, L);
  else if (T.s2 != 0.0)
    strip_range<PHI, true, false, R>(T, w, W, tab, base, end, resume, L);
  else
    strip_range<PHI, false, false, R>(T, w, W, tab, base, end, resume, L);
}

// One whole walk for the R rays (rx[r], ry[r]) of every lane, added to
// acc[(6 r + c) * A], c = 0..4 (and 5, PHI) = {alpha0, alpha1, kappa, gamma0,
// gamma1, phi}.
template <bool PHI, int R>
__device__ __forceinline__ void walk_strip(const TreeDev &D, const double *rx, const double *ry, const bool *valid,
                                           StripWarp &W, const ExpTab &tab, double *acc, int A) {
  const int nn = D.nnodes;
  if (nn == 0) return;
  const StripTree T(D);
  const StripWalk<R> w = strip_begin<R>(rx, ry, valid);
  StripAcc L[R];
  int resume[R];
#pragma unroll
  for (int r = 0; r < R; ++r) resume[r] = valid[r] ? 0 : 0x7fffffff;
  strip_run<PHI, R>(T, w, W, tab, 0, nn, resume, L);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    double *o = acc + 6 * r * A;
    o[0] += L[r].a0;
    o[A] += L[r].a1;
    o[2 * A] += L[r].k;
    o[3 * A] += L[r].g0;
    o[4 * A] += 2.0 * L[r].g1;
    if (PHI) o[5 * A] += L[r].p;
    if (D.inv_area != 0.0 && w.has(w.vmask, r)) o[2 * A] -= D.inv_area * D.root_mass;  // every mass enters a walk once
  }
}

// The part [s0, end) of a walk shared by several warps (s0 a multiple of
// kCutStep): this ray's terms of the part's nodes.  The decisions at the
// ancestors of node s0 are taken again (their far-field terms belong to
// earlier parts), which gives the node where each ray enters the part; false
// if none does.
template <bool PHI>
__device__ __forceinline__ bool walk_strip_part(const TreeDev &D, double rx, double ry, bool valid, StripWarp &W,
                                                    const ExpTab &tab, int s0, int end, StripAcc &L) {
  const StripTree T(D);
  const StripWalk<1> w = strip_begin<1>(&rx, &ry, &valid);
  int resume = valid ? s0 : 0x7fffffff;
  const int a = __ldg(D.cutanc + (size_t)kMaxDepth * (s0 / kCutStep) + w.lane);
  int skip = 0, cls = 2;
  if (a >= 0) {
    const double2 *sp = reinterpret_cast<const double2 *>(T.tnodes + a);
    const double2 c = __ldg(sp);
    const float4 o = __ldg(reinterpret_cast<const float4 *>(sp + 1));
    skip = __float_as_int(o.z);
    cls = strip_class(w, c.x, c.y, o.x, o.y);
  }
  unsigned todo = __ballot_sync(kFull, a >= 0 && cls != 2);
  while (todo) {
    const int b = __ffs(todo) - 1;
    todo &= todo - 1;
    const int node = __shfl_sync(kFull, a, b), sk = __shfl_sync(kFull, skip, b), c = __shfl_sync(kFull, cls, b);
    const GNode *nd = T.nodes + node;
    const double cx = nd->cx - rx, cy = nd->cy - ry;
    // every ancestor's subtree holds s0, so the outermost one not opened decides
    if (c == 1 || !(cx * cx + cy * cy < nd->open2)) resume = max(resume, sk);
  }
  const int base = (int)__reduce_min_sync(kFull, valid ? (unsigned)resume : 0x7fffffffu);
  if (base >= end) return false;
  strip_run<PHI, 1>(T, w, W, tab, base, end, &resume, &L);
  return true;
}

}  // namespace glb
