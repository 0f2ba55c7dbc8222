// List walk of the split form for the 32 rays of a warp: cells classified
// against the box of the warp's rays as in the group walk (walk_group.cuh), 32
// at a time from a queue, but summed in the order of a node-at-a-time walk, so
// that every ray's result is that walk's and does not depend on the other rays.
//
// The tree's preorder array is taken in windows of kLW nodes.  In a window the
// cells that some ray reaches are classified breadth first (children beyond the
// window wait for theirs); the outcome is kept in three bitmaps: accepted by
// all, opened by all with particles to sum, mixed.  Reading the bitmaps from
// the start gives the window's cells in preorder; far-field rows are staged 32
// list entries at a time, opened leaves summed as they come, mixed subtrees
// walked per ray.  A node-at-a-time walk tests about 5,200 cells per ray here;
// this one about 4,300 cells in rounds of 32, and per ray only the nodes of
// mixed subtrees.  48 uneven lenses in one launch (2.8M rays): 89 ms with the
// node-at-a-time walk, 70 with this one; 16 served requests 57 and 41 ms.
#pragma once
#include "walk_group.cuh"
#include "walk_strip.cuh"

namespace glb {

// Nodes per window: one plane of 2^18 particles and 512^2 rays take 4.80 ms; with
// 2,048 nodes 4.95, with 8,192 (shared memory) 5.52.
constexpr int kLBits = 12, kLW = 1 << kLBits;
constexpr int kLQ = 1024;  // classification queue (power of two)
constexpr int kLD = 128;   // cells waiting for later windows: at most three siblings a level

struct ListWarp {
  unsigned far[kLW / 32], open[kLW / 32], mixed[kLW / 32];
  int wait[kLD];
  float4 rows[64];  // far-field rows of 32 list entries
  float4 part[32];  // a leaf's particles
  unsigned short q[kLQ];
  unsigned short list[1024];
};

// The walk's next window: classifies the cells in [w0, w1) that some ray
// reaches; nwait cells wait before and after.
__device__ __forceinline__ void list_classify(const TreeDev &T, const StripWalk<1> &w, ListWarp &L, int &nwait, int &w0,
                                              int &w1) {
  const unsigned lt = (1u << w.lane) - 1u;
  int v[kLD / 32];
  unsigned first = 0x7fffffffu;
#pragma unroll
  for (int k = 0; k < kLD / 32; ++k) {
    v[k] = w.lane + 32 * k < nwait ? L.wait[w.lane + 32 * k] : 0x7fffffff;
    first = min(first, (unsigned)v[k]);
  }
  w0 = (int)__reduce_min_sync(kFull, first);
  w1 = min(w0 + kLW, T.nnodes);
#pragma unroll
  for (int k = 0; k < kLW / 1024; ++k) L.far[w.lane + 32 * k] = L.open[w.lane + 32 * k] = L.mixed[w.lane + 32 * k] = 0u;
  __syncwarp();
  int head = 0, tail = 0;
  nwait = 0;
#pragma unroll
  for (int k = 0; k < kLD / 32; ++k) {
    const bool now = v[k] < w1, later = v[k] != 0x7fffffff && !now;
    const unsigned a = __ballot_sync(kFull, now), b = __ballot_sync(kFull, later);
    if (now) L.q[tail + __popc(a & lt)] = (unsigned short)(v[k] - w0);
    if (later) L.wait[nwait + __popc(b & lt)] = v[k];
    tail += __popc(a);
    nwait += __popc(b);
  }
  __syncwarp();
  while (head != tail) {
    const int cnt = min(32, tail - head);
    int off = 0, cat = 0, packed = 0, info = 0;  // cat: 1 accepted, 2 opened, 3 mixed
    int4 ch = make_int4(-1, -1, -1, -1);
    if (w.lane < cnt) {
      off = L.q[(head + w.lane) & (kLQ - 1)];
      const double2 *sp = reinterpret_cast<const double2 *>(T.tnodes + w0 + off);
      const double2 c = __ldg(sp);
      const float4 o = __ldg(reinterpret_cast<const float4 *>(sp + 1));
      ch = __ldg(reinterpret_cast<const int4 *>(T.cnodes + w0 + off) + 2);
      info = __float_as_int(o.w);
      const int cls = strip_class(w, c.x, c.y, o.x, o.y);
      cat = cls == 0 ? 3 : cls;
      if (cat == 2) {
        const int n = (ch.x >= 0) + (ch.y >= 0) + (ch.z >= 0) + (ch.w >= 0);  // a leaf has none
        const int in = (ch.x >= 0 && ch.x < w1) + (ch.y >= 0 && ch.y < w1) + (ch.z >= 0 && ch.z < w1) +
                       (ch.w >= 0 && ch.w < w1);
        packed = in | (n - in) << 16;
      }
    }
    head += cnt;
    int incl = packed;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, incl, o);
      if (w.lane >= o) incl += t;
    }
    const int total = __shfl_sync(kFull, incl, 31), nin = total & 0xffff, nout = total >> 16;
    if (tail - head + nin > kLQ || nwait + nout > kLD) {
      if (packed) cat = 3;  // no room: the rays walk these subtrees themselves
    } else {
      if (packed) {
        int a = tail + ((incl - packed) & 0xffff), b = nwait + ((incl - packed) >> 16);
        const int c4[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (c4[k] >= 0) {
            if (c4[k] < w1)
              L.q[(a++) & (kLQ - 1)] = (unsigned short)(c4[k] - w0);
            else
              L.wait[b++] = c4[k];
          }
      }
      tail += nin;
      nwait += nout;
    }
    const unsigned bit = 1u << (off & 31);
    if (cat == 1) atomicOr(&L.far[off >> 5], bit);
    if ((cat == 2 && info != 0) || cat == 3) atomicOr(&L.open[off >> 5], bit);
    if (cat == 3) atomicOr(&L.mixed[off >> 5], bit);
    __syncwarp();
  }
}

// One walk for the ray (rxy[0], rxy[1]), added to its FP64 totals acc[0..4].
__device__ __forceinline__ void walk_list(const TreeDev &T, double rx, double ry, bool valid, ListWarp &L,
                                          double *acc) {
  if (T.nnodes == 0) return;
  const StripWalk<1> w = strip_begin<1>(&rx, &ry, &valid);
  const bool screen = T.screen2 != 0.0;
  const float s2f = (float)T.screen2, ns2l = -s2f * kLog2e;
  const bool sheet = T.inv_area != 0.0 && !T.sheet_closed;
  const float piaf = sheet ? (float)(kPi * T.inv_area) : 0.f;
  const double rxy[2] = {rx, ry};
  const float rxh = (float)rx, ryh = (float)ry;
  const float2 nrh = make_float2(-rxh, -ryh);
  const float2 nrl = make_float2(-(float)(rx - (double)rxh), -(float)(ry - (double)ryh));
  F32Acc fa;
  fa.zero();
  int nwait = 1;
  if (w.lane == 0) L.wait[0] = 0;
  __syncwarp();
  while (nwait > 0) {
    int w0, w1;
    list_classify(T, w, L, nwait, w0, w1);
#pragma unroll 1
    for (int h = 0; h < kLW / 1024; ++h) {
      // a quarter window's cells in order: offset | category << kLBits
      const unsigned f = L.far[32 * h + w.lane], e = L.open[32 * h + w.lane], m = L.mixed[32 * h + w.lane];
      unsigned all = f | e;
      if (!__any_sync(kFull, all != 0u)) continue;
      int incl = __popc(all);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (w.lane >= o) incl += t;
      }
      const int total = __shfl_sync(kFull, incl, 31);
      int pos = incl - __popc(all);
      while (all) {
        const int b = __ffs(all) - 1;
        all &= all - 1;
        const int cat = (e >> b & 1u) ? ((m >> b & 1u) ? 2 : 1) : 0;
        L.list[pos++] = (unsigned short)(32 * (32 * h + w.lane) + b | cat << kLBits);
      }
      __syncwarp();
      for (int l0 = 0; l0 < total; l0 += 32) {
        const int cnt = min(32, total - l0);
        int cat = 1, node = 0;
        if (w.lane < cnt) {
          const int x = L.list[l0 + w.lane];
          cat = x >> kLBits;
          node = w0 + (x & (kLW - 1));
          if (cat == 0) {
            const float4 *sp = reinterpret_cast<const float4 *>(T.fsnodes + node);
            L.rows[2 * w.lane] = __ldg(sp);
            L.rows[2 * w.lane + 1] = __ldg(sp + 1);
          }
        }
        const unsigned ev = __ballot_sync(kFull, w.lane < cnt && cat != 0), mx = __ballot_sync(kFull, cat == 2);
        __syncwarp();
        int p = 0;
        while (p < cnt) {
          const unsigned rest = ev & ~((1u << p) - 1u);
          const int b = rest ? __ffs(rest) - 1 : cnt;
          // far-field rows [p, b): runs without a test up to the next flush of
          // any lane (a leaf can leave exactly 32 terms: the next one joins them)
          while (p < b) {
            const int k = min(b - p, max(1, 32 - (int)__reduce_max_sync(kFull, valid ? (unsigned)fa.cnt : 0u)));
            const float4 *row = L.rows + 2 * p;
#pragma unroll 4
            for (int j = 0; j < k; ++j, row += 2) {
              const float4 c0 = row[0];
              const float2 d =
                  __fadd2_rn(__fadd2_rn(make_float2(c0.x, c0.y), nrh), __fadd2_rn(make_float2(c0.z, c0.w), nrl));
              far_sum(row[1], d, screen, ns2l, piaf, fa);
            }
            p += k;
            if (valid) {
              fa.cnt += k;
              if (fa.cnt >= 32) fa.flush(acc);
            }
          }
          if (b >= cnt) break;
          p = b + 1;
          const int nd = __shfl_sync(kFull, node, b);
          const float4 *sp = reinterpret_cast<const float4 *>(T.snodes + nd);
          const int4 c3 = __ldg(reinterpret_cast<const int4 *>(sp + 3));
          if (mx >> b & 1u) {
            group_subtree(T, rxy, valid, nrh, nrl, nd, c3.x, screen, s2f, ns2l, piaf, sheet, fa, acc, L.part);
            continue;
          }
          const float4 c0 = __ldg(sp), c1 = __ldg(sp + 1);
          const float2 d = __fadd2_rn(__fadd2_rn(make_float2(c0.x, c0.y), nrh), __fadd2_rn(make_float2(c0.z, c0.w), nrl));
          const float2 dd = __fmul2_rn(d, d);
          const float r2f = dd.x + dd.y;
          bool nearc = false;
          if (valid) {
            const float g = r2f - c1.y;
            nearc = g < 0.f;
            if (fabsf(g) <= kAmbiguous * c1.y) nearc = node_test_f64(T.nodes + nd, rx, ry, 1);
          }
          if (c3.y) {  // leaf
            const int p0 = c3.z, p1 = p0 + c3.w;
            const float wu = __ldg(sp + 2).z;
            const bool clear = !__any_sync(kFull, valid && r2f < __int_as_float(c3.y));
            if (valid && (nearc ? fa.cnt > 0 : fa.cnt + min(c3.w, 32) > 32)) fa.flush(acc);
            for (int q0 = p0; q0 < p1; q0 += 32) {
              const int n = min(32, p1 - q0);
              if (w.lane < n) L.part[w.lane] = __ldg(T.prel + q0 + w.lane);
              __syncwarp();
              if (clear) {  // (lanes without a ray add garbage nobody reads)
#pragma unroll 4
                for (int j = 0; j < n; ++j) clear_term(L.part[j], d, screen, ns2l, piaf, sheet, fa);
              } else if (valid) {
                for (int j = 0; j < n; ++j)
                  leaf_term(T, L.part[j], q0 + j, d, rxy, nearc, screen, s2f, ns2l, piaf, sheet, wu, nd, fa, acc);
              }
              if (valid) {
                fa.cnt += n;
                if (nearc || q0 + n < p1) fa.flush(acc);
              }
              __syncwarp();
            }
          } else if (nearc) {  // softened particles listed at an internal cell
            for (int i = c3.z; i < c3.z + c3.w; ++i) {
              const float4 P = __ldg(T.bigs + i);
              const double x0 = (double)P.x - rx, x1 = (double)P.y - ry;
              double rcm2 = x0 * x0 + x1 * x1;
              if (rcm2 < 1e-20) rcm2 = 1e-20;
              const double size = (double)P.w;
              if (rcm2 < 4 * size * size) bspline_f64<false>(x0, x1, sqrt(rcm2), (double)P.z, size, 0.0, acc);
            }
          }
        }
        __syncwarp();
      }
    }
  }
  if (valid) {
    fa.flush(acc);
    // the sheet's kappa is -inv_area x (total mass) for every walk; its
    // deflection is closed-form for masses of one sign
    if (T.inv_area != 0.0) {
      const double s = T.inv_area * T.root_mass;
      acc[2] -= s;
      if (T.sheet_closed) {
        acc[0] += s * (T.root_cx - rx);
        acc[1] += s * (T.root_cy - ry);
      }
    }
  }
}

}  // namespace glb
