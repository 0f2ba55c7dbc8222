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
// Bound by FP64 latency and issue: 512^2 rays on 2^18 particles take 7.9 ms
// (12.9 with walk_f64), 2.6 of them in far-field terms (76 % of the FP64 pipe's
// rate), 2.4 in particles, 1.8 in the exponentials of both, 2.1 in strips and
// staging; FP64 pipe 48 %, issue 61 % at 18 warps per SM (96 registers; 80 or
// 128 registers and loops unrolled by 2 within 3 % of it, unrolled by 4 13.3
// ms: the instruction cache).
#pragma once
#include "walk.cuh"

namespace glb {

// One warp's shared memory: the far-field queue (rows {cx, cy},
// {mass, q0}, {q2, mask}) and the particles of the leaf being evaluated.
struct StripWarp {
  double2 far[64 * 3];
  double2 part[32 * 2];
};

// 1/a: the PTX seed (a relative error below 2^-20) and one Newton-Raphson step
// of third order, x (1 + e + e^2) with e = 1 - a x.
__device__ __forceinline__ double strip_rcp(double a) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  const double e = __fma_rn(-a, x, 1.0);
  return __fma_rn(x, __fma_rn(e, e, e), x);
}

// exp(-t), t >= 0, by a table-driven method (after P. T. P. Tang, ACM TOMS 15,
// 1989, with a step of 2^-10 in place of a fraction of ln 2): t = m + j/1024 + r
// with |r| <= 2^-11, exact in double; exp(-m) and exp(-j/1024) from tables,
// exp(-r) - 1 by its Taylor polynomial of degree 4 (r^5/120 is below 3e-19).
// The constants of the two highest terms have a zero low word (r^3/6 is below
// 2e-11 and the rounding of its constant 6e-7 of it), so that they are
// immediates; full double constants cost two instructions each per use.  t is
// held at 700 (by its high word), where exp(-t) is below 1e-304.
constexpr double kC3 = -0x1.55555p-3, kC4 = 0x1.55555p-5;
__device__ __forceinline__ double strip_exp_neg(double t, const ExpTab &E) {
  constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52
  t = __hiloint2double(min(__double2hiint(t), 0x4085e000), __double2loint(t));
  const double s = __fma_rn(t, 1024.0, kShift);
  const int k = __double2loint(s);
  const double r = __fma_rn(s - kShift, -0x1p-10, t);
  double p = __fma_rn(r, kC4, kC3);
  p = __fma_rn(p, r, 0.5);
  p = __fma_rn(p, r, -1.0);
  const double e = __dmul_rn(E.hi[k >> 10], E.lo[k & 1023]);
  return __fma_rn(e, __dmul_rn(r, p), e);
}

// A block's copy of the tables.
__device__ __forceinline__ void strip_exp_table(ExpTab &E, const ExpTab *src) {
  if (!src) return;  // no tree with nodes: the tables are not read
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

// The warp's constants of one walk.
struct StripWalk {
  double rx, ry;   // this lane's ray
  double bx, by;   // centre of the box of the warp's valid rays
  float hx, hy;    // its half extents, rounded up
  unsigned vmask;  // lanes with a valid ray
  int lane;
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
__device__ __forceinline__ StripWalk strip_begin(double rx, double ry, bool valid) {
  StripWalk w;
  w.rx = rx;
  w.ry = ry;
  w.lane = threadIdx.x & 31;
  w.vmask = __ballot_sync(kFull, valid);
  const bool in = valid && isfinite(rx) && isfinite(ry);
  constexpr float kBig = 1e30f;
  const float x0 = key_f(__reduce_min_sync(kFull, f_key(in ? __double2float_rd(rx) : kBig)));
  const float x1 = key_f(__reduce_max_sync(kFull, f_key(in ? __double2float_ru(rx) : -kBig)));
  const float y0 = key_f(__reduce_min_sync(kFull, f_key(in ? __double2float_rd(ry) : kBig)));
  const float y1 = key_f(__reduce_max_sync(kFull, f_key(in ? __double2float_ru(ry) : -kBig)));
  w.bx = 0.5 * ((double)x0 + (double)x1);
  w.by = 0.5 * ((double)y0 + (double)y1);
  w.hx = __double2float_ru(0.5 * ((double)x1 - (double)x0)) * 1.000001f;
  w.hy = __double2float_ru(0.5 * ((double)y1 - (double)y0)) * 1.000001f;
  return w;
}

// 1: accepted by all, 2: opened by all, 0: mixed.  olo, ohi: the squared
// opening radius less and plus the margin.  The half extents are rounded up
// by 1e-6, which covers the rounding of dx - hx where the two are close.
__device__ __forceinline__ int strip_class(const StripWalk &w, double cx, double cy, float olo, float ohi) {
  const float dx = fabsf((float)(cx - w.bx)), dy = fabsf((float)(cy - w.by));
  const float nx = fmaxf(dx - w.hx, 0.f), ny = fmaxf(dy - w.hy, 0.f), fx = dx + w.hx, fy = dy + w.hy;
  return nx * nx + ny * ny >= ohi ? 1 : (fx * fx + fy * fy < olo ? 2 : 0);
}

// The cnt queued far-field rows for every valid lane, or with MASKED for the
// lanes of each row's mask.
template <bool PHI, bool SCREEN, bool SHEET, bool MASKED>
__device__ __forceinline__ void strip_far_rows(const StripTree &T, const StripWalk &w, const StripWarp &W, int cnt,
                                               const ExpTab &tab, StripAcc &L) {
  const double s2 = T.s2, pia = T.pia;
  const double2 *row = W.far;
#pragma unroll 1
  for (int j = 0; j < cnt; ++j, row += 3) {
    const double2 c = row[0], mq = row[1], qm = row[2];
    const double dx = c.x - w.rx, dy = c.y - w.ry;
    const double xx = __dmul_rn(dx, dx), r2 = __fma_rn(dy, dy, xx);
    const double ir2 = strip_rcp(r2);
    const double si = SCREEN ? __dmul_rn(strip_exp_neg(__dmul_rn(r2, s2), tab), ir2) : ir2;
    const double a = __dmul_rn(mq.x, si), s4 = __dmul_rn(si, ir2);  // mass/pi scr/r^2, scr/r^4
    const double qx = __fma_rn(mq.y, dx, __dmul_rn(qm.x, dy)), qy = __fma_rn(qm.x, dx, -__dmul_rn(mq.y, dy));
    const double e = __dmul_rn(__dmul_rn(4.0, s4), __dmul_rn(__fma_rn(qx, dx, __dmul_rn(qy, dy)), ir2));
    const double t = SHEET ? __fma_rn(mq.x, pia, -a) : -a;
    const double gc = __dmul_rn(a, ir2), dd = __fma_rn(-dy, dy, xx), xy = __dmul_rn(dx, dy);
    if (!MASKED || ((unsigned)__double2loint(qm.y) >> w.lane & 1u)) {
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

// The far-field queue: rows waiting, whether one of them is not for every
// valid lane.
struct StripQueue {
  int n = 0;
  bool masked = false;
};

// Queues the far-field rows of the strip positions in `who` (r0, r1, r2: this
// lane's row; fm: the lanes that take it).
__device__ __forceinline__ void strip_push(const StripWalk &w, StripWarp &W, StripQueue &q, unsigned who, double2 r0,
                                           double2 r1, double q2, unsigned fm) {
  if (who >> w.lane & 1u) {
    double2 *row = W.far + 3 * (q.n + __popc(who & ((1u << w.lane) - 1u)));
    row[0] = r0;
    row[1] = r1;
    row[2] = make_double2(q2, __hiloint2double(0, (int)fm));
  }
  q.n += __popc(who);
}

// A leaf opened by the rays of `om`: its particles as point masses, with their
// softening where the leaf applies it (quadTree.h:1017-1077).
template <bool PHI, bool SCREEN, bool SHEET>
__device__ __forceinline__ void strip_leaf(const StripTree &T, const StripWalk &w, StripWarp &W, int node, int p0, int n,
                                           unsigned om, const ExpTab &tab, StripAcc &L) {
  float4 Q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (w.lane < n) Q = __ldg(T.parts + p0 + w.lane);  // in flight with the node's row
  const GNode *nd = T.nodes + node;
  const double width = nd->width;
  const bool mine = om >> w.lane & 1u;
  const double cx = nd->cx - w.rx, cy = nd->cy - w.ry;
  const bool nearc = mine && (cx * cx + cy * cy < nd->near2);
  const double s2 = T.s2, pia = T.pia;
  // A particle within the 1e-10 of the coincidence clamp lies in a leaf whose
  // near radius (2.41 widths) the ray is in, unless the leaf is narrower than
  // that; other leaves need neither the clamp nor the softening test.
  const bool plain = !__any_sync(kFull, nearc) && width > 1e-9 && om == w.vmask;
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
        const double x0 = c.x - w.rx, x1 = c.y - w.ry;
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
    } else {
#pragma unroll 1
      for (int j = 0; j < m; ++j, row += 2) {
        const double2 c = row[0], ms = row[1];
        const double x0 = c.x - w.rx, x1 = c.y - w.ry;
        const double xx = __dmul_rn(x0, x0);
        double rr = __fma_rn(x1, x1, xx);
        const double t2 = __dmul_rn(rr, s2);
        rr = rr < 1e-20 ? 1e-20 : rr;
        const double ir2 = strip_rcp(rr);
        double pre = __dmul_rn(ms.x, ir2);
        if (SCREEN) pre = __dmul_rn(pre, strip_exp_neg(t2, tab));
        const double gc = __dmul_rn(pre, ir2), t = SHEET ? __fma_rn(-pia, ms.x, pre) : pre;
        if (mine) {
          L.a0 = __fma_rn(-t, x0, L.a0);
          L.a1 = __fma_rn(-t, x1, L.a1);
          L.g0 = __fma_rn(-gc, __fma_rn(-x1, x1, xx), L.g0);
          L.g1 = __fma_rn(-gc, __dmul_rn(x0, x1), L.g1);
          if (PHI) L.p += 0.5 * pre * rr * log(rr) - 0.5 * pia * ms.x * rr;
        }
        if (nearc && rr < ms.y) strip_soften<PHI>(T.dev, x0, x1, rr, __ldg(T.parts + p0 + q0 + j), L);
      }
    }
  }
}

// Softened particles listed at an internal node (quadTree.h:1048-1077).
template <bool PHI>
__device__ __forceinline__ void strip_bigs(const StripTree &T, const StripWalk &w, int node, unsigned om, StripAcc &L) {
  const GNode *nd = T.nodes + node;
  const double cx = nd->cx - w.rx, cy = nd->cy - w.ry;
  if (!((om >> w.lane & 1u) && cx * cx + cy * cy < nd->near2)) return;
#pragma unroll 1
  for (int b = nd->bstart, e = b + nd->bcount; b < e; ++b) {
    const float4 Q = __ldg(T.dev->bigs + b);
    const double x0 = (double)Q.x - w.rx, x1 = (double)Q.y - w.ry;
    double rr = x0 * x0 + x1 * x1;
    if (rr < 1e-20) rr = 1e-20;
    const double size = (double)Q.w;
    if (rr < 4 * size * size) strip_soften<PHI>(T.dev, x0, x1, rr, Q, L);
  }
}

// The walk's nodes in [base, end): base moves to the next node to visit (it
// may pass end), resume is this lane's next node (it sits out nodes before
// it).  The loop keeps one copy of each evaluation, for the instruction cache.
template <bool PHI, bool SCREEN, bool SHEET>
__device__ __forceinline__ void strip_range(const StripTree &T, const StripWalk &w, StripWarp &W, const ExpTab &tab,
                                            int &base, int end, int &resume, StripAcc &L) {
  const bool mine = w.vmask >> w.lane & 1u;
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
    const bool slow = mm != 0u || __any_sync(kFull, mine && resume > base);
    unsigned todo = slow ? am | ev : ev, pend = slow ? 0u : am, fm = w.vmask;
    for (;;) {
      // the next node with particles to evaluate, and the far-field rows before it
      int node = -1, inf = 0;
      unsigned om = w.vmask, push = pend;
      while (todo) {
        const int b = __ffs(todo) - 1;
        todo &= todo - 1;
        inf = __shfl_sync(kFull, info, b);
        if (slow) {
          const unsigned act = __ballot_sync(kFull, mine && base + b >= resume);
          if (am >> b & 1u) {
            if (w.lane == b) fm = act;
            if (act) pend |= 1u << b;
            continue;
          }
          const int sk = __shfl_sync(kFull, skip, b);
          om = act;
          if (mm >> b & 1u) {
            const GNode *nd = T.nodes + base + b;
            const double cx = nd->cx - w.rx, cy = nd->cy - w.ry;
            om = __ballot_sync(kFull, cx * cx + cy * cy < nd->open2) & act;
            const unsigned fa = act & ~om;
            if (w.lane == b) fm = fa;
            if (fa) pend |= 1u << b;
            if (fa >> w.lane & 1u) resume = sk;
          }
          if (om == 0u) {  // nobody opens it: past its subtree
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
        q.masked = q.masked || __any_sync(kFull, (push >> w.lane & 1u) && fm != w.vmask);
      }
      strip_push(w, W, q, push, r0, r1, q2, fm);
      pend &= ~push;
      bool flush = q.n > 0;
      if (node < 0) {
        base = slow ? max(next, (int)__reduce_min_sync(kFull, mine ? (unsigned)resume : 0x7fffffffu)) : next;
        flush = q.n >= 32 || (base >= end && q.n > 0);
      }
      if (flush) {
        __syncwarp();
        if (q.masked)
          strip_far_rows<PHI, SCREEN, SHEET, true>(T, w, W, q.n, tab, L);
        else
          strip_far_rows<PHI, SCREEN, SHEET, false>(T, w, W, q.n, tab, L);
        __syncwarp();
        q.n = 0;
        q.masked = false;
      }
      if (node < 0) break;
      if (inf < 0)
        strip_leaf<PHI, SCREEN, SHEET>(T, w, W, node, __shfl_sync(kFull, pstart, node - sbase), -inf, om, tab, L);
      else
        strip_bigs<PHI>(T, w, node, om, L);
    }
  }
}

template <bool PHI>
__device__ __forceinline__ void strip_run(const StripTree &T, const StripWalk &w, StripWarp &W, const ExpTab &tab,
                                          int base, int end, int resume, StripAcc &L) {
  if (T.pia != 0.0)
    strip_range<PHI, true, true>(T, w, W, tab, base, end, resume, L);
  else if (T.s2 != 0.0)
    strip_range<PHI, true, false>(T, w, W, tab, base, end, resume, L);
  else
    strip_range<PHI, false, false>(T, w, W, tab, base, end, resume, L);
}

// One whole walk for the ray (rx, ry), added to acc[c * A], c = 0..4 (and 5,
// PHI) = {alpha0, alpha1, kappa, gamma0, gamma1, phi}.
template <bool PHI>
__device__ __forceinline__ void walk_strip(const TreeDev &D, double rx, double ry, bool valid, StripWarp &W,
                                           const ExpTab &tab, double *acc, int A) {
  const int nn = D.nnodes;
  if (nn == 0) return;
  const StripTree T(D);
  const StripWalk w = strip_begin(rx, ry, valid);
  StripAcc L;
  strip_run<PHI>(T, w, W, tab, 0, nn, valid ? 0 : 0x7fffffff, L);
  acc[0] += L.a0;
  acc[A] += L.a1;
  acc[2 * A] += L.k;
  acc[3 * A] += L.g0;
  acc[4 * A] += 2.0 * L.g1;
  if (PHI) acc[5 * A] += L.p;
  if (D.inv_area != 0.0 && valid) acc[2 * A] -= D.inv_area * D.root_mass;  // every mass enters a walk once
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
  const StripWalk w = strip_begin(rx, ry, valid);
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
    const double cx = nd->cx - w.rx, cy = nd->cy - w.ry;
    // every ancestor's subtree holds s0, so the outermost one not opened decides
    if (c == 1 || !(cx * cx + cy * cy < nd->open2)) resume = max(resume, sk);
  }
  const int base = (int)__reduce_min_sync(kFull, valid ? (unsigned)resume : 0x7fffffffu);
  if (base >= end) return false;
  strip_run<PHI>(T, w, W, tab, base, end, resume, L);
  return true;
}

}  // namespace glb
