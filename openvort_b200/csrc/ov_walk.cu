// ov_walk.cu - Barnes-Hut velocity walk (octree_get_vs, src/octree.c:275-343)
// for every node and every boundary image (src/tangle.c:605-609,627-636).
//
// Warp-coherent, stackless traversal: the cells are in depth-first preorder,
// so each lane only keeps the index of the next cell it must visit (c + 1
// after opening c, c.skip otherwise).  The warp visits the smallest of its
// lanes' next cells; lanes whose next cell it is take their own decision, so
// every lane evaluates exactly the interactions the reference's recursion
// would, and the warp's 32 targets (consecutive in key order, hence close in
// space) share every cell load.
//
// Decision per cell (reference order): N == 1 or min side < BH_grain ->
// direct sum over the cell's nodes; |r - com|/(wrapped) passes the opening
// test -> monopole + the reference's second-order terms; otherwise descend.
// The opening test compares the squared distance, computed with the
// reference's exact operations, against a per-cell threshold equivalent to
// Lm / d < theta in FP64.
//
// FP64 form: everything in FP64.  Mixed form: the expansion and far direct
// segments in FP32 from FP64-formed relative vectors, FP64 sums; the opening
// test and near segments (|R| < 4 |ds|) in FP64.
#include <float.h>

#include <algorithm>
#include <cmath>

#include "ov_internal.h"
#include "ov_pair.cuh"

namespace {

struct TreeView {
  const Cell* cells;
  const double* cell_lm;   // max box side per cell (opening test at a user theta)
  const int2* cell_range;  // first sorted node and count per cell
  const double* nodes64;   // per sorted node: r1, wrapped r2
  const int2* nodeids;     // per sorted node: slot, forward slot
  int n_cells;
  int n_nodes;
};

// squared distance from r to the cell's centre of mass after the reference's
// one-box wrap of the centre (seg_pwrap + segment_len, src/octree.c:286-287),
// with exactly its FP64 operations
__device__ __forceinline__ double mac_dist2(const OvParams& P, d3 r, double cx, double cy, double cz) {
  double u[3];
  const double rr[3] = {r.x, r.y, r.z};
  const double cc[3] = {cx, cy, cz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double c = cc[a];
    if (P.periodic[a]) {
      double d = __dsub_rn(c, rr[a]);
      if (d > P.L[a] * 0.5) c = __dsub_rn(c, P.L[a]);
      else if (d < -P.L[a] * 0.5) c = __dadd_rn(c, P.L[a]);
    }
    u[a] = __dsub_rn(rr[a], c);
  }
  double s = __dmul_rn(u[0], u[0]);
  s = __dadd_rn(s, __dmul_rn(u[1], u[1]));
  s = __dadd_rn(s, __dmul_rn(u[2], u[2]));
  return s;
}

// The reference's expansion (src/octree.c:303-328), moments pre-scaled by
// kappa/4pi: gam x R / |R|^3 + (M21, 0, 0) / |R|^3 + (M.2 R_z) x R / |R|^5,
// where (M.2 R_z) = (M02 Rz, M12 Rz, M22 Rz) is what its mat3_vmul returns.
// Since (M.2 R_z) x R / |R|^5 = ((M.2) R_z / |R|^2) x R / |R|^3, the sum is
// ((gam + M.2 R_z / |R|^2) x R + (M21, 0, 0)) / |R|^3: one cross product.
// m = (M21, M02, M12, M22).
__device__ __forceinline__ d3 expansion64(const double* g, const double* m, d3 R) {
  const double R2 = dot3(R, R);
  const double inv = rsqrt_nr(R2);
  const double inv2 = inv * inv;
  const double i3 = inv2 * inv;
  const double w = R.z * inv2;
  const d3 G = mk3(fma(m[1], w, g[0]), fma(m[2], w, g[1]), fma(m[3], w, g[2]));
  const d3 c = cross3(G, R);
  return mk3((c.x + m[0]) * i3, c.y * i3, c.z * i3);
}

__device__ __forceinline__ void expansion32(float g0, float g1, float g2, float m21, float m02,
                                            float m12, float m22, float Rx, float Ry, float Rz,
                                            float& vx, float& vy, float& vz) {
  const float R2 = fmaf(Rx, Rx, fmaf(Ry, Ry, Rz * Rz));
  const float inv = rsqrtf(R2);
  const float inv2 = inv * inv;
  const float i3 = inv2 * inv;
  const float w = Rz * inv2;
  const float Gx = fmaf(m02, w, g0), Gy = fmaf(m12, w, g1), Gz = fmaf(m22, w, g2);
  vx = fmaf(Gy, Rz, fmaf(-Gz, Ry, m21)) * i3;
  vy = fmaf(Gz, Rx, -Gx * Rz) * i3;
  vz = fmaf(Gx, Ry, -Gy * Rx) * i3;
}

__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

enum { ACT_NONE = 0, ACT_P2P1 = 1, ACT_P2PN = 2, ACT_FAR = 3, ACT_OPEN = 4 };

// One segment at rp: FP64 with the reference's cut-offs, or (mixed, far
// segments |R| >= 4 |ds|) FP32 from FP64-formed R and ds.
template <bool kMixed>
__device__ __forceinline__ void p2p_one(const OvParams& P, d3 r1, d3 r2, d3 rp, double& ax,
                                        double& ay, double& az) {
  if (kMixed) {
    d3 R = r1 - rp;
    d3 ds = r2 - r1;
    double R2 = dot3(R, R), ds2 = dot3(ds, ds);
    float vx, vy, vz;
    if (R2 >= 16.0 * ds2 && ds2 > 0 &&
        seg_vel32((float)P.f4pi, (float)R.x, (float)R.y, (float)R.z, (float)ds.x, (float)ds.y,
                  (float)ds.z, vx, vy, vz)) {
      ax += vx; ay += vy; az += vz;
      return;
    }
  }
  const d3 v = seg_vel64_nr(P.f4pi, r1, r2, rp);
  ax += v.x; ay += v.y; az += v.z;
}

// One walk of one warp: lane target rp (valid if `live`), skip rule `skip`.
// Each visited cell is one 128-byte record, loaded once for the warp; both
// possible successors (first child q+1 and skip) are prefetched into L1.
template <bool kMixed>
__device__ d3 warp_walk(const OvParams& P, const TreeView& T, d3 rp, bool live, int skip,
                        bool use_thr, double theta, unsigned long long& n_p2p,
                        unsigned long long& n_far, unsigned long long& n_iter) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int next = live ? 0 : T.n_cells;
  double ax = 0, ay = 0, az = 0;
  for (;;) {
    const int q = (int)__reduce_min_sync(FULL, (unsigned)next);
    if (q >= T.n_cells) break;
    const Cell* cp = T.cells + q;
    if (lane == 0 && q + 1 < T.n_cells) prefetch_l1(cp + 1);
    const int4 h = *reinterpret_cast<const int4*>(cp);              // a, b, skip, meta
    const double2 t0 = *reinterpret_cast<const double2*>(&cp->thr);  // thr, x0
    const double2 t1 = *reinterpret_cast<const double2*>(&cp->x[1]); // x1, x2
    const int kind = cell_kind(h.w);
    const int skp = h.z;
    if (lane == 1 && skp < T.n_cells) prefetch_l1(T.cells + skp);
    int act = ACT_NONE;
    if (next == q) {
      if (kind == CELL_LEAF1) {
        act = ACT_P2P1;
      } else if (kind == CELL_LEAFN) {
        act = ACT_P2PN;
      } else {
        double s = mac_dist2(P, rp, t0.y, t1.x, t1.y);
        bool pass = use_thr ? (s >= t0.x)
                            : (s > 0 && __ddiv_rn(T.cell_lm[q], __dsqrt_rn(s)) < theta);
        if (pass) act = ACT_FAR;
        else if (kind == CELL_OPEN) act = ACT_OPEN;
        else if (kind == CELL_OPEN_P2P) act = ACT_P2PN;
      }
      // every lane's next cell strictly increases, so a walk ends within
      // n_cells iterations whatever the cell records hold
      next = (act == ACT_OPEN) ? q + 1 : max(skp, q + 1);
    }
    if (act == ACT_FAR) {
      if (kMixed) {
        // bytes 104-127 are 8-byte aligned: three float2 loads
        const float2 f0 = *reinterpret_cast<const float2*>(&cp->f_g[0]);  // g0 g1
        const float2 f1 = *reinterpret_cast<const float2*>(&cp->f_g[2]);  // g2 m02
        const float2 f2 = *reinterpret_cast<const float2*>(&cp->f_m12);   // m12 m22
        float vx, vy, vz;
        expansion32(f0.x, f0.y, f1.x, __int_as_float(h.x), f1.y, f2.x, f2.y, (float)(rp.x - t0.y),
                    (float)(rp.y - t1.x), (float)(rp.z - t1.y), vx, vy, vz);
        ax += vx; ay += vy; az += vz;
      } else {
        d3 v = expansion64(cp->y, cp->m, mk3(rp.x - t0.y, rp.y - t1.x, rp.z - t1.y));
        ax += v.x; ay += v.y; az += v.z;
      }
    } else if (act == ACT_P2P1) {
      // skip rule of calculate_vs_shift (src/tangle.c:567-569)
      if (h.y != -1 && h.x != skip && h.y != skip)
        p2p_one<kMixed>(P, mk3(t0.y, t1.x, t1.y), mk3(cp->y[0], cp->y[1], cp->y[2]), rp, ax, ay, az);
    }
    const unsigned far_mask = __ballot_sync(FULL, act == ACT_FAR);
    const unsigned p1_mask = __ballot_sync(FULL, act == ACT_P2P1);
    const unsigned pn_mask = __ballot_sync(FULL, act == ACT_P2PN);
    if (lane == 0) {
      n_far += __popc(far_mask);
      n_p2p += __popc(p1_mask);
      ++n_iter;
    }
    if (pn_mask) {
      const int2 rg = T.cell_range[q];
      const int end = min(rg.x + rg.y, T.n_nodes);
      if (lane == 0) n_p2p += (unsigned long long)__popc(pn_mask) * rg.y;
      for (int i = max(rg.x, 0); i < end; ++i) {
        const int2 id = T.nodeids[i];
        if (act != ACT_P2PN) continue;
        if (id.y == -1 || id.x == skip || id.y == skip) continue;
        const double* nd = T.nodes64 + 6 * (size_t)i;
        p2p_one<kMixed>(P, mk3(nd[0], nd[1], nd[2]), mk3(nd[3], nd[4], nd[5]), rp, ax, ay, az);
      }
    }
  }
  return mk3(ax, ay, az);
}

// ----------------------------------------------------------------------
// Multi-image walk (tables of periodic shifts in {-1,0,1}^3, no mirrors).
//
// The reference walks the tree once per image point r - L s (27 walks for
// periodic-26), each with its own opening decisions, because the opening
// distance is |r - L s - com| after a single box wrap of the centre of mass
// (src/octree.c:286).  Per axis that distance is the minimum image for s = 0
// and either the same value or a larger one for s = +-1, so every image's
// walk visits a subset of the cells of the s = 0 walk.  One traversal per
// target therefore serves all images: each lane keeps, per tree level, the
// 27-bit mask of images that opened the parent, makes each image's decision
// exactly as the reference would (per-axis wrapped distances with its FP64
// operations), evaluates every image that accepts the cell or reaches a leaf
// from the same cell load, and descends while any image opens.
//
// combo c = 9 (sx+1) + 3 (sy+1) + (sz+1); c = 13 is the tangle itself.

constexpr int kCombos = 27;
constexpr int kPrimary = 13;
// up to this many open images besides the target's own are decided one by
// one; more take all 27 decisions at once (mac_exact)
constexpr int kFewImages = 4;
constexpr unsigned kAllImages = (1u << 27) - 1;
constexpr int kLevelSlots = 34;

// Parameters of the walk's shortcut decisions (every image from the
// target's own distance): on = no image shifts along a non-periodic axis
// (whose images may lie nearer than the target); hw[a] = the largest
// |c - r| along axis a at which every image's wrap still undoes its shift
// (half a box less a rounding allowance; DBL_MAX on axes without shifts).
struct ImageShortcut {
  double hw[3];
  double wr[3];     // the smallest |c - r| at which the target's own image surely wraps (DBL_MAX: no shifts)
  double half[3];   // L / 2 on periodic axes (the reference's wrap test), DBL_MAX otherwise
  int on;
};

// wrapped component u and its square for one image coordinate v
__device__ __forceinline__ double wrapped_sq(const OvParams& P, int a, double v, double c) {
  double cc = c;
  if (P.periodic[a]) {
    double d = __dsub_rn(c, v);
    if (d > P.L[a] * 0.5) cc = __dsub_rn(c, P.L[a]);
    else if (d < -P.L[a] * 0.5) cc = __dadd_rn(c, P.L[a]);
  }
  double u = __dsub_rn(v, cc);
  return __dmul_rn(u, u);
}

__device__ __forceinline__ float sel3f(int i, float a, float b, float c) {
  return i == 0 ? a : (i == 1 ? b : c);
}

// FP64 reference formula for one segment at one image point, and the FP64
// expansion at one image offset.  Inlined: out of line (__noinline__) the
// calls' register saves made the mixed walk 52.1 ms per launch at 1M points
// against 37.9 ms.
__device__ __forceinline__ d3 seg64_at(double f4pi, d3 r1, d3 r2, d3 t) {
  return seg_vel64_nr(f4pi, r1, r2, t);
}
__device__ __forceinline__ d3 expansion64_at(const Cell* cp, d3 R) { return expansion64(cp->y, cp->m, R); }

// One segment r1 -> r2 for every image in `mask`: FP64 with the reference's
// cut-offs and skip rule (the skip applies to the tangle itself only), or in
// the mixed form FP32 beyond the near radius.  Images are visited as nine
// (x, y) columns of three z shifts, the z loop unrolled.
// image coordinate r - L s along one axis, s = i - 1, with the reference's
// single rounding (shifted, src/tangle.c:51-53)
__device__ __forceinline__ double img_coord(double r, double L, int i) {
  return i == 1 ? r : (i == 0 ? __dsub_rn(r, -L) : __dsub_rn(r, L));
}

// The 27 opening decisions of a cell (wrapped squared distance of each
// image point to the centre of mass >= thr), exactly with the reference's
// FP64 operations: per axis and shift the wrapped square, summed x + y then
// + z as segment_len does (src/octree.c:284-296).  All 27 are independent.
__device__ __forceinline__ unsigned mac_exact(const OvParams& P, d3 r, double cx, double cy,
                                              double cz, double thr) {
  const double qx[3] = {wrapped_sq(P, 0, img_coord(r.x, P.L[0], 0), cx), wrapped_sq(P, 0, r.x, cx),
                        wrapped_sq(P, 0, img_coord(r.x, P.L[0], 2), cx)};
  const double qy[3] = {wrapped_sq(P, 1, img_coord(r.y, P.L[1], 0), cy), wrapped_sq(P, 1, r.y, cy),
                        wrapped_sq(P, 1, img_coord(r.y, P.L[1], 2), cy)};
  const double qz[3] = {wrapped_sq(P, 2, img_coord(r.z, P.L[2], 0), cz), wrapped_sq(P, 2, r.z, cz),
                        wrapped_sq(P, 2, img_coord(r.z, P.L[2], 2), cz)};
  unsigned pass = 0;
#pragma unroll
  for (int ix = 0; ix < 3; ++ix) {
#pragma unroll
    for (int iy = 0; iy < 3; ++iy) {
      const double qxy = __dadd_rn(qx[ix], qy[iy]);
#pragma unroll
      for (int iz = 0; iz < 3; ++iz)
        pass |= (__dadd_rn(qxy, qz[iz]) >= thr ? 1u : 0u) << (9 * ix + 3 * iy + iz);
    }
  }
  return pass;
}

// The images of a cell whose opening test the target's own image fails by
// the margin E, from two distances per axis (dx = cx - r.x and so on, not
// wrapped).  Along an axis where |d| <= hw every image's wrapped distance is
// |d|.  Where |d| >= wr the target's own image wraps, to |d| - L: the image
// shifted towards the cell has that distance too, and the one shifted away
// wraps back to |d|.  So the images fall into the products of "same" and
// "away" along the wrapped axes.  Each product's squared distance is formed
// here within the rounding that E covers (mac_margin: every component within
// e of its exact value), so it decides its images when it is E away from the
// threshold.  False when a product is not, or an axis lies between hw and wr:
// the caller then takes the images' decisions in full.
// (22.4k nodes, theta = 0.4: 248 of a group's 1478 visits took mac_exact for
// such cells.)
__device__ __forceinline__ bool wrapped_decisions(const OvParams& P, const ImageShortcut& S, d3 r, double cx,
                                                  double cy, double cz, double dx, double dy, double dz, double thr,
                                                  double E, unsigned& pass) {
  const double ax = fabs(dx), ay = fabs(dy), az = fabs(dz);
  const bool wx = ax > S.hw[0], wy = ay > S.hw[1], wz = az > S.hw[2];
  pass = 0;
  if (!(wx || wy || wz)) return true;   // every image as near as the target
  if ((wx && ax < S.wr[0]) || (wy && ay < S.wr[1]) || (wz && az < S.wr[2])) return false;
  // images shifted away along a wrapped axis: shift index 2 for d > 0
  const unsigned mx = wx ? (dx > 0 ? 0x1ffu << 18 : 0x1ffu) : 0u;
  const unsigned my = wy ? (dy > 0 ? 0x1c0e07u << 6 : 0x1c0e07u) : 0u;
  const unsigned mz = wz ? (dz > 0 ? 0x1249249u << 2 : 0x1249249u) : 0u;
  const double qx = wrapped_sq(P, 0, r.x, cx), qy = wrapped_sq(P, 1, r.y, cy), qz = wrapped_sq(P, 2, r.z, cz);
  const double hi = thr + E, lo = thr - E;
  bool clear = true;
#pragma unroll
  for (int b = 1; b < 8; ++b) {
    const unsigned set = ((b & 4) ? mx : ~mx) & ((b & 2) ? my : ~my) & ((b & 1) ? mz : ~mz);
    if (!(set & kAllImages) || ((b & 4) && !wx) || ((b & 2) && !wy) || ((b & 1) && !wz)) continue;
    const double q = ((b & 4) ? dx * dx : qx) + ((b & 2) ? dy * dy : qy) + ((b & 1) ? dz * dz : qz);
    if (q >= hi) pass |= set;
    else if (q >= lo) clear = false;
  }
  pass &= kAllImages;
  return clear;
}

template <bool kMixed>
__device__ __forceinline__ void p2p_images(const OvParams& P, unsigned mask, d3 r, d3 r1, d3 r2,
                                           int id, int fw, int skip, double near2, d3& nl, d3& im,
                                           unsigned& n_p2p) {
  if (fw == -1) return;
  if (id == skip || fw == skip) mask &= ~(1u << kPrimary);
  n_p2p += __popc(mask);
  const d3 ds = r2 - r1;
  const double ds2 = dot3(ds, ds);
  const double far2 = fmax(16.0 * ds2, near2);
  const float dsx = (float)ds.x, dsy = (float)ds.y, dsz = (float)ds.z;
  const float f4 = (float)P.f4pi;
  float fx = 0, fy = 0, fz = 0;
  // one image per iteration, rolled: a single copy of each formula
#pragma unroll 1
  while (mask) {
    const int c = __ffs(mask) - 1;
    mask &= mask - 1;
    const int ix = (c * 57) >> 9, rem = c - 9 * ix, iy = (rem * 11) >> 5, iz = rem - 3 * iy;
    const d3 t = mk3(img_coord(r.x, P.L[0], ix), img_coord(r.y, P.L[1], iy), img_coord(r.z, P.L[2], iz));
    if (kMixed) {
      const d3 R = r1 - t;
      const double R2 = dot3(R, R);
      float vx, vy, vz;
      if (R2 >= far2 && ds2 > 0 &&
          seg_vel32(f4, (float)R.x, (float)R.y, (float)R.z, dsx, dsy, dsz, vx, vy, vz)) {
        fx += vx; fy += vy; fz += vz;
        continue;
      }
      // the mixed form keeps one sum for the tangle and its images
      nl = nl + seg64_at(P.f4pi, r1, r2, t);
      continue;
    }
    // the reference's formula with refined reciprocals (its own operations
    // near the cut-offs), as the FP64 direct sum
    const d3 v = seg_vel64_nr(P.f4pi, r1, r2, t);
    if (c == kPrimary) nl = nl + v;
    else im = im + v;
  }
  if (kMixed) nl = nl + mk3(fx, fy, fz);
}

// Mixed form of one segment r1 -> r2 at every image in `mask` with many
// images: the images' offsets R = r1 - (r - L s) per axis and shift are
// formed in FP64 and rounded once, and two (x, y) image columns share each
// packed FP32 pair (columns 2g and 2g + 1, their three z images one after
// the other), as in cell_mixed.  Per image, with d = r2 - r1, a = |R|,
// b = |R + d|, u = 1/(ab), w = u / (1 + R.(R + d) u):
//   v = kappa/4pi (1/a + 1/b) w (R x d),   1 - cos = |R x d|^2 u w
// (the reference's segment formula, src/tangle.c:486-517, and its
// colinearity cut-off, zero inside it).  R x d, R.d and |R|^2 share their
// x and y parts along a column.  Images nearer than the far radius, or
// within 2.5e-3 of the cut-off, take the FP64 formula afterwards.  The skip
// rule (calculate_vs_shift, src/tangle.c:567-569) drops the tangle's own
// image for the target's own segments.
__device__ __forceinline__ void p2p_mixed_columns(const OvParams& P, unsigned mask, d3 r, d3 r1, d3 r2,
                                                  int id, int fw, int skip, double near2, d3& nl,
                                                  unsigned& n_p2p) {
  if (fw == -1) return;
  if (id == skip || fw == skip) mask &= ~(1u << kPrimary);
  n_p2p += __popc(mask);
  const d3 ds = r2 - r1;
  const double ds2 = dot3(ds, ds);
  const float far2 = (float)fmax(16.0 * ds2, near2);
  const float dx = (float)ds.x, dy = (float)ds.y, dz = (float)ds.z;
  const f2 Dx = f2_splat(dx), Dz = f2_splat(dz), nDy = f2_splat(-dy);
  const f2 D2 = f2_splat(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
  const f2 one = f2_splat(1.0f), two = f2_splat(2.0f);
  // FP32 copies of r1 - (r - L s) per axis and shift
  const float Fx[3] = {(float)__dsub_rn(r1.x, img_coord(r.x, P.L[0], 0)), (float)__dsub_rn(r1.x, r.x),
                       (float)__dsub_rn(r1.x, img_coord(r.x, P.L[0], 2))};
  const float Fy[3] = {(float)__dsub_rn(r1.y, img_coord(r.y, P.L[1], 0)), (float)__dsub_rn(r1.y, r.y),
                       (float)__dsub_rn(r1.y, img_coord(r.y, P.L[1], 2))};
  const float Fz[3] = {(float)__dsub_rn(r1.z, img_coord(r.z, P.L[2], 0)), (float)__dsub_rn(r1.z, r.z),
                       (float)__dsub_rn(r1.z, img_coord(r.z, P.L[2], 2))};
  f2 bx = f2_splat(0.f), by = bx, bz = bx;
  unsigned special = 0;   // images left to the FP64 formula
#pragma unroll
  for (int grp = 0; grp < 5; ++grp) {
    const int xa = 2 * grp, xb = grp < 4 ? xa + 1 : xa;
    const unsigned bits_a = (mask >> (3 * xa)) & 7u;
    const unsigned bits_b = grp < 4 ? (mask >> (3 * xb)) & 7u : 0u;
    if (!(bits_a | bits_b)) continue;
    const int ixa = (xa * 11) >> 5, iya = xa - 3 * ixa;
    const int ixb = (xb * 11) >> 5, iyb = xb - 3 * ixb;
    const f2 X = f2_pack(sel3f(ixa, Fx[0], Fx[1], Fx[2]), sel3f(ixb, Fx[0], Fx[1], Fx[2]));
    const f2 Y = f2_pack(sel3f(iya, Fy[0], Fy[1], Fy[2]), sel3f(iyb, Fy[0], Fy[1], Fy[2]));
    const f2 XY2 = f2_fma(X, X, Y * Y);
    const f2 XYd = f2_fma(X, Dx, Y * f2_splat(dy));
    const f2 Ydz = Y * Dz, mXdz = X * f2_splat(-dz);
    const f2 Cz = f2_fma(X, f2_splat(dy), Y * f2_splat(-dx));
    const f2 Cz2 = Cz * Cz;
#pragma unroll
    for (int iz = 0; iz < 3; ++iz) {
      const f2 Zs = f2_splat(Fz[iz]);
      const f2 R2 = f2_fma(Zs, Zs, XY2);
      const f2 Rd = f2_fma(Zs, Dz, XYd);
      const f2 Q2 = f2_fma(two, Rd, R2 + D2);
      const f2 ia = f2_rsqrt(R2), ib = f2_rsqrt(Q2);
      const f2 u = ia * ib;
      const f2 w = u * f2_rcp(f2_fma(R2 + Rd, u, one));
      const f2 s = (ia + ib) * w;
      const f2 Cx = f2_fma(Zs, nDy, Ydz);
      const f2 Cy = f2_fma(Zs, Dx, mXdz);
      const f2 tc = f2_fma(Cy, Cy, f2_fma(Cx, Cx, Cz2)) * (u * w);   // 1 - cos
      float tc0, tc1, r20, r21, s0, s1;
      f2_unpack(tc, tc0, tc1);
      f2_unpack(R2, r20, r21);
      f2_unpack(s, s0, s1);
      const bool in0 = (bits_a >> iz) & 1u, in1 = (bits_b >> iz) & 1u;
      const bool far0 = r20 >= far2, far1 = r21 >= far2;
      const bool ok0 = in0 && far0 && tc0 > kColHi, ok1 = in1 && far1 && tc1 > kColHi;
      // colinear (zero), masked-out and FP64 images add nothing here
      const f2 sk = f2_pack(ok0 ? s0 : 0.f, ok1 ? s1 : 0.f);
      bx = f2_fma(Cx, sk, bx);
      by = f2_fma(Cy, sk, by);
      bz = f2_fma(Cz, sk, bz);
      if (in0 && !ok0 && !(far0 && tc0 < kColLo)) special |= 1u << (3 * xa + iz);
      if (in1 && !ok1 && !(far1 && tc1 < kColLo)) special |= 1u << (3 * xb + iz);
    }
  }
  float lo, hi;
  const float f4 = (float)P.f4pi;
  f2_unpack(bx, lo, hi);
  const float fx = f4 * (lo + hi);
  f2_unpack(by, lo, hi);
  const float fy = f4 * (lo + hi);
  f2_unpack(bz, lo, hi);
  const float fz = f4 * (lo + hi);
  nl = nl + mk3(fx, fy, fz);
#pragma unroll 1
  while (special) {
    const int c = __ffs(special) - 1;
    special &= special - 1;
    const int ix = (c * 57) >> 9, rem = c - 9 * ix, iy = (rem * 11) >> 5, iz = rem - 3 * iy;
    nl = nl + seg64_at(P.f4pi, r1, r2,
                       mk3(img_coord(r.x, P.L[0], ix), img_coord(r.y, P.L[1], iy), img_coord(r.z, P.L[2], iz)));
  }
}

// images at which a segment is evaluated by columns rather than one by one
constexpr int kColumnImages = 8;

// images from which a product of shift sets takes the unrolled image loop
// (1M nodes mixed, ms per walk: 27.7 from 4, 6 or 8 images, 28.0 from 12,
// 28.5 from 18, 32.2 with only full masks; fewer images run only a few
// groups of the masked loop, the tangle's own image alone just one)
constexpr int kProductImages = 6;

// Whether an image mask is a product of per-axis shift sets (bit i of
// mx: shift i - 1 along x, and so on).  The masks of partly accepted cells
// mostly are: an opening test's images differ along the axes where the
// target's offset wraps.
__device__ __forceinline__ bool product_mask(unsigned m, unsigned& mx, unsigned& my, unsigned& mz) {
  const unsigned a = m & 511u, b = (m >> 9) & 511u, c = (m >> 18) & 511u, u = a | b | c;
  mx = (a ? 1u : 0u) | (b ? 2u : 0u) | (c ? 4u : 0u);
  my = (u & 7u ? 1u : 0u) | (u & 56u ? 2u : 0u) | (u & 448u ? 4u : 0u);
  mz = (u | (u >> 3) | (u >> 6)) & 7u;
  return __popc(m) == __popc(mx) * __popc(my) * __popc(mz);
}

// Mixed form of one accepted cell at every image in `pass` (a 27-bit mask
// of the combos 9 (sx+1) + 3 (sy+1) + (sz+1)): FP32 expansions from the FP32
// moments at R = r - L s - com formed in FP64 and rounded once, summed in
// factored form and added to nl; images within the near radius in FP64
// (expansion64_at, added to nl as they come).  m21 is the FP32 m21 moment
// (the cell header's first word), thr the cell's opening threshold, dc the
// opening test's FP64 difference com - r.
__device__ __forceinline__ void cell_mixed(const OvParams& P, const Cell* cp, float m21, double cx, double cy,
                                           double cz, double thr, d3 r, d3 dc, unsigned pass, double near2,
                                           d3& nl) {
  const float2 q0f = *reinterpret_cast<const float2*>(&cp->f_g[0]);
  const float2 q1f = *reinterpret_cast<const float2*>(&cp->f_g[2]);
  const float2 q2f = *reinterpret_cast<const float2*>(&cp->f_m12);
  const float g0 = q0f.x, g1 = q0f.y, g2 = q1f.x, m02 = q1f.y, m12 = q2f.x, m22 = q2f.y;
  float ax, ay, az;
  {
    // FP32 copies of the FP64-formed offsets r - L s - com per axis and shift
    float Fx[3] = {(float)__dsub_rn(img_coord(r.x, P.L[0], 0), cx),
                   -(float)dc.x,
                   (float)__dsub_rn(img_coord(r.x, P.L[0], 2), cx)};
    float Fy[3] = {(float)__dsub_rn(img_coord(r.y, P.L[1], 0), cy),
                   -(float)dc.y,
                   (float)__dsub_rn(img_coord(r.y, P.L[1], 2), cy)};
    float Fz[3] = {(float)__dsub_rn(img_coord(r.z, P.L[2], 0), cz),
                   -(float)dc.z,
                   (float)__dsub_rn(img_coord(r.z, P.L[2], 2), cz)};
    // an accepting image has |R|^2 >= its wrapped squared distance >=
    // thr, so a cell whose thr reaches the near radius needs no test
    const bool test_near = thr < near2;
    const float fnear2 = (float)near2;
    // two (x, y) columns per packed FP32 pair: columns 2g and 2g + 1
    // (the last group has column 8 only), their three z images
    // evaluated side by side (independent chains).  The 27 image
    // terms are summed in factored form: with i3 = |R|^-3 and
    // i5 = R_z |R|^-5 per image, the reference's
    // ((g + m R_z/|R|^2) x R + (m21, 0, 0)) i3 summed over the images
    // is g x P + m x Q + (m21 S, 0, 0), P = sum i3 R, Q = sum i5 R,
    // S = sum i3; since R_x and R_y are constant along a column,
    // P_x, P_y, Q_x, Q_y take each column's sums of i3 and i5 once.
    float Px, Py, Pz, Qx, Qy, Qz, Sv;
    // All 27 images accept (the usual case: the wrapped opening test
    // treats every image point like the target), or a product of per-axis
    // shift sets, and none but the tangle's own image is near: no per-image
    // masks or near-field tests.  A shift outside its set takes an offset of
    // 1e18, whose |R|^-3 underflows to an exact zero.  An image shifted
    // along an axis has |R|^2 >= that axis offset squared (FP32
    // rounding of sums of non-negative terms is monotonic), so when
    // every shifted offset reaches the near radius, only the tangle's own
    // image can take the FP64 path; its weight here is then zero.
    // (1M nodes: 922 visits of a group have a lane with all images, 246 one
    // with 14 to 26 of them.)
    bool all = pass == kAllImages, near0 = false;
    if (!all && __popc(pass) >= kProductImages) {
      unsigned mx, my, mz;
      all = product_mask(pass, mx, my, mz);
      if (all) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if (!((mx >> i) & 1u)) Fx[i] = 1e18f;
          if (!((my >> i) & 1u)) Fy[i] = 1e18f;
          if (!((mz >> i) & 1u)) Fz[i] = 1e18f;
        }
      }
    }
    if (all && test_near) {
      const float X = Fx[1], Y = Fy[1], Z = Fz[1];
      near0 = fmaf(Z, Z, fmaf(X, X, Y * Y)) < fnear2;
      all = Fx[0] * Fx[0] >= fnear2 && Fx[2] * Fx[2] >= fnear2 && Fy[0] * Fy[0] >= fnear2 &&
            Fy[2] * Fy[2] >= fnear2 && Fz[0] * Fz[0] >= fnear2 && Fz[2] * Fz[2] >= fnear2;
    }
    if (all) {
      // unrolled: the column offsets are chosen at compile time.  The sums
      // over a shift along z are kept per shift, so R_z multiplies each once
      // at the end, and column 8 goes by itself: its z shifts 0 and 1 as a
      // pair, shift 2 alone.
      f2 px = f2_splat(0.f), py = px, qx = px, qy = px, z3[3] = {px, px, px}, z5[3] = {px, px, px};
#pragma unroll
      for (int grp = 0; grp < 4; ++grp) {
        const int xa = 2 * grp, xb = xa + 1;
        const int ixa = (xa * 11) >> 5, iya = xa - 3 * ixa;
        const int ixb = (xb * 11) >> 5, iyb = xb - 3 * ixb;
        const f2 X = f2_pack(Fx[ixa], Fx[ixb]), Y = f2_pack(Fy[iya], Fy[iyb]);
        const f2 XY2 = f2_fma(X, X, Y * Y);
        f2 c3 = f2_splat(0.f), c5 = c3;
#pragma unroll
        for (int iz = 0; iz < 3; ++iz) {
          const f2 Zs = f2_splat(Fz[iz]);
          f2 inv = f2_rsqrt(f2_fma(Zs, Zs, XY2));
          if (grp == 2 && iz == 1) inv = inv * f2_pack(near0 ? 0.f : 1.f, 1.f);
          const f2 inv2 = inv * inv;
          const f2 i3 = inv2 * inv;
          const f2 t5 = i3 * inv2;
          c3 = iz ? c3 + i3 : i3;
          c5 = iz ? f2_fma(t5, Zs, c5) : t5 * Zs;
          z3[iz] = grp ? z3[iz] + i3 : i3;
          z5[iz] = grp ? z5[iz] + t5 : t5;
        }
        px = grp ? f2_fma(c3, X, px) : c3 * X;
        py = grp ? f2_fma(c3, Y, py) : c3 * Y;
        qx = grp ? f2_fma(c5, X, qx) : c5 * X;
        qy = grp ? f2_fma(c5, Y, qy) : c5 * Y;
      }
      const float X8 = Fx[2], Y8 = Fy[2], xy2 = fmaf(X8, X8, Y8 * Y8);
      const f2 Z01 = f2_pack(Fz[0], Fz[1]);
      const f2 inv = f2_rsqrt(f2_fma(Z01, Z01, f2_splat(xy2)));
      const f2 inv2 = inv * inv;
      const f2 i3 = inv2 * inv, t5 = i3 * inv2;
      const float inv_2 = rsqrt_approx(fmaf(Fz[2], Fz[2], xy2)), i3_2 = (inv_2 * inv_2) * inv_2;
      const float t5_2 = i3_2 * (inv_2 * inv_2);
      float i3_0, i3_1, t5_0, t5_1, lo, hi;
      f2_unpack(i3, i3_0, i3_1);
      f2_unpack(t5, t5_0, t5_1);
      const float c3 = (i3_0 + i3_1) + i3_2, c5 = fmaf(t5_2, Fz[2], fmaf(t5_1, Fz[1], t5_0 * Fz[0]));
      f2_unpack(px, lo, hi);
      Px = fmaf(c3, X8, lo + hi);
      f2_unpack(py, lo, hi);
      Py = fmaf(c3, Y8, lo + hi);
      f2_unpack(qx, lo, hi);
      Qx = fmaf(c5, X8, lo + hi);
      f2_unpack(qy, lo, hi);
      Qy = fmaf(c5, Y8, lo + hi);
      f2_unpack(z3[0], lo, hi);
      const float s0 = (lo + hi) + i3_0;
      f2_unpack(z3[1], lo, hi);
      const float s1 = (lo + hi) + i3_1;
      f2_unpack(z3[2], lo, hi);
      const float s2 = (lo + hi) + i3_2;
      Sv = (s0 + s1) + s2;
      Pz = fmaf(s2, Fz[2], fmaf(s1, Fz[1], s0 * Fz[0]));
      f2_unpack(z5[0], lo, hi);
      const float w0 = ((lo + hi) + t5_0) * Fz[0];
      f2_unpack(z5[1], lo, hi);
      const float w1 = ((lo + hi) + t5_1) * Fz[1];
      f2_unpack(z5[2], lo, hi);
      const float w2 = ((lo + hi) + t5_2) * Fz[2];
      Qz = fmaf(w2, Fz[2], fmaf(w1, Fz[1], w0 * Fz[0]));
      if (near0)
        nl = nl + expansion64_at(cp, mk3(__dsub_rn(r.x, cx), __dsub_rn(r.y, cy), __dsub_rn(r.z, cz)));
    } else {
    f2 px = f2_splat(0.f), py = px, pz = px, qx = px, qy = px, qz = px, sv = px;
#pragma unroll 1
    for (int grp = 0; grp < 5; ++grp) {
      const int xa = 2 * grp, xb = grp < 4 ? xa + 1 : xa;
      const unsigned bits_a = (pass >> (3 * xa)) & 7u;
      const unsigned bits_b = grp < 4 ? (pass >> (3 * xb)) & 7u : 0u;
      if (!(bits_a | bits_b)) continue;
      const int ixa = (xa * 11) >> 5, iya = xa - 3 * ixa;
      const int ixb = (xb * 11) >> 5, iyb = xb - 3 * ixb;
      const float Xa = sel3f(ixa, Fx[0], Fx[1], Fx[2]), Xb = sel3f(ixb, Fx[0], Fx[1], Fx[2]);
      const float Ya = sel3f(iya, Fy[0], Fy[1], Fy[2]), Yb = sel3f(iyb, Fy[0], Fy[1], Fy[2]);
      const f2 X = f2_pack(Xa, Xb), Y = f2_pack(Ya, Yb);
      const f2 XY2 = f2_fma(X, X, Y * Y);
      float xy2a, xy2b;
      f2_unpack(XY2, xy2a, xy2b);
      // no z image of a column is nearer than its (x, y) distance
      const bool near_a = test_near && xy2a < fnear2, near_b = test_near && xy2b < fnear2;
      f2 c3 = f2_splat(0.f), c5 = c3;
#pragma unroll
      for (int iz = 0; iz < 3; ++iz) {
        const float Z = Fz[iz];
        const f2 Zs = f2_splat(Z);
        const f2 R2 = f2_fma(Zs, Zs, XY2);
        float r2a, r2b;
        f2_unpack(R2, r2a, r2b);
        bool on_a = (bits_a >> iz) & 1u, on_b = (bits_b >> iz) & 1u;
        if ((on_a && near_a) || (on_b && near_b)) {
          // near field: FP64 expansion from the FP64 offsets
          if (on_a && near_a && r2a < fnear2) {
            nl = nl + expansion64_at(cp, mk3(__dsub_rn(img_coord(r.x, P.L[0], ixa), cx),
                                             __dsub_rn(img_coord(r.y, P.L[1], iya), cy),
                                             __dsub_rn(img_coord(r.z, P.L[2], iz), cz)));
            on_a = false;
          }
          if (on_b && near_b && r2b < fnear2) {
            nl = nl + expansion64_at(cp, mk3(__dsub_rn(img_coord(r.x, P.L[0], ixb), cx),
                                             __dsub_rn(img_coord(r.y, P.L[1], iyb), cy),
                                             __dsub_rn(img_coord(r.z, P.L[2], iz), cz)));
            on_b = false;
          }
        }
        // images not evaluated here contribute exact zeros
        const f2 inv = f2_pack(on_a ? rsqrt_approx(r2a) : 0.f, on_b ? rsqrt_approx(r2b) : 0.f);
        const f2 inv2 = inv * inv;
        const f2 i3 = inv2 * inv;
        const f2 i5 = (i3 * inv2) * Zs;
        c3 = c3 + i3;
        c5 = c5 + i5;
        pz = f2_fma(i3, Zs, pz);
        qz = f2_fma(i5, Zs, qz);
      }
      px = f2_fma(c3, X, px);
      py = f2_fma(c3, Y, py);
      qx = f2_fma(c5, X, qx);
      qy = f2_fma(c5, Y, qy);
      sv = sv + c3;
    }
    float a0, a1;
    f2_unpack(px, a0, a1);
    Px = a0 + a1;
    f2_unpack(py, a0, a1);
    Py = a0 + a1;
    f2_unpack(pz, a0, a1);
    Pz = a0 + a1;
    f2_unpack(qx, a0, a1);
    Qx = a0 + a1;
    f2_unpack(qy, a0, a1);
    Qy = a0 + a1;
    f2_unpack(qz, a0, a1);
    Qz = a0 + a1;
    f2_unpack(sv, a0, a1);
    Sv = a0 + a1;
    }
    // g x P + m x Q + (m21 S, 0, 0), m = (m02, m12, m22)
    ax = fmaf(g1, Pz, fmaf(-g2, Py, fmaf(m12, Qz, fmaf(-m22, Qy, m21 * Sv))));
    ay = fmaf(g2, Px, fmaf(-g0, Pz, fmaf(m22, Qx, -m02 * Qz)));
    az = fmaf(g0, Py, fmaf(-g1, Px, fmaf(m02, Qy, -m12 * Qx)));
  }
  // the mixed form keeps one sum for the tangle and its images
  nl = nl + mk3(ax, ay, az);
}

// FP64 form of one accepted cell at every image in `pass`: the reference's
// expansion (src/octree.c:303-328) at R = r - L s - com.  The tangle's own
// image goes into nl as one evaluation; the other images are summed in
// factored form into im, as in cell_mixed: with i3 = |R|^-3 and
// i5 = R_z |R|^-5 per image, the sum of ((g + m R_z/|R|^2) x R + (m21, 0, 0)) i3
// is g x P + m x Q + (m21 S, 0, 0), P = sum i3 R, Q = sum i5 R, S = sum i3.
// All images, or a product of shift sets: no branch per image, as in
// cell_mixed (a shift outside its set takes an offset of 1e150, whose |R|^-3
// underflows to an exact zero).
__device__ __forceinline__ void cell_fp64(const OvParams& P, const Cell* cp, double cx, double cy, double cz, d3 r,
                                          unsigned pass, d3& nl, d3& im) {
  const double g[3] = {cp->y[0], cp->y[1], cp->y[2]};
  const double mm[4] = {cp->m[0], cp->m[1], cp->m[2], cp->m[3]};
  if (pass & (1u << kPrimary))
    nl = nl + expansion64(g, mm, mk3(__dsub_rn(r.x, cx), __dsub_rn(r.y, cy), __dsub_rn(r.z, cz)));
  const unsigned rest = pass & ~(1u << kPrimary);
  if (!rest) return;
  double Rx[3] = {__dsub_rn(img_coord(r.x, P.L[0], 0), cx), __dsub_rn(r.x, cx),
                  __dsub_rn(img_coord(r.x, P.L[0], 2), cx)};
  double Ry[3] = {__dsub_rn(img_coord(r.y, P.L[1], 0), cy), __dsub_rn(r.y, cy),
                  __dsub_rn(img_coord(r.y, P.L[1], 2), cy)};
  double Rz[3] = {__dsub_rn(img_coord(r.z, P.L[2], 0), cz), __dsub_rn(r.z, cz),
                  __dsub_rn(img_coord(r.z, P.L[2], 2), cz)};
  double px = 0, py = 0, pz = 0, qx = 0, qy = 0, qz = 0, sv = 0;
  bool all = pass == kAllImages;
  if (!all && __popc(pass) >= kProductImages) {
    unsigned mx, my, mz;
    all = product_mask(pass, mx, my, mz);
    if (all) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (!((mx >> i) & 1u)) Rx[i] = 1e150;
        if (!((my >> i) & 1u)) Ry[i] = 1e150;
        if (!((mz >> i) & 1u)) Rz[i] = 1e150;
      }
    }
  }
  if (all) {
    // sums over a shift along z kept per shift, as in cell_mixed
    double z3[3] = {0, 0, 0}, z5[3] = {0, 0, 0};
#pragma unroll
    for (int xy = 0; xy < 9; ++xy) {
      const double X = Rx[xy / 3], Y = Ry[xy % 3];
      const double XY2 = fma(X, X, Y * Y);
      double c3 = 0, c5 = 0;
#pragma unroll
      for (int iz = 0; iz < 3; ++iz) {
        if (3 * xy + iz == kPrimary) continue;
        const double Z = Rz[iz];
        const double inv = rsqrt_nr(fma(Z, Z, XY2));
        const double inv2 = inv * inv;
        const double i3 = inv2 * inv;
        const double t5 = i3 * inv2;
        c3 = iz ? c3 + i3 : i3;
        c5 = iz ? fma(t5, Z, c5) : t5 * Z;
        z3[iz] = xy ? z3[iz] + i3 : i3;
        z5[iz] = xy ? z5[iz] + t5 : t5;
      }
      px = xy ? fma(c3, X, px) : c3 * X;
      py = xy ? fma(c3, Y, py) : c3 * Y;
      qx = xy ? fma(c5, X, qx) : c5 * X;
      qy = xy ? fma(c5, Y, qy) : c5 * Y;
    }
    sv = (z3[0] + z3[1]) + z3[2];
    pz = fma(z3[2], Rz[2], fma(z3[1], Rz[1], z3[0] * Rz[0]));
    qz = fma(z5[2] * Rz[2], Rz[2], fma(z5[1] * Rz[1], Rz[1], (z5[0] * Rz[0]) * Rz[0]));
  } else {
#pragma unroll 1
    for (int xy = 0; xy < 9; ++xy) {
      const unsigned bits = (rest >> (3 * xy)) & 7u;
      if (!bits) continue;
      const int ix = (xy * 11) >> 5, iy = xy - 3 * ix;
      const double X = ix == 0 ? Rx[0] : (ix == 1 ? Rx[1] : Rx[2]);
      const double Y = iy == 0 ? Ry[0] : (iy == 1 ? Ry[1] : Ry[2]);
      const double XY2 = fma(X, X, Y * Y);
      double c3 = 0, c5 = 0;
#pragma unroll
      for (int iz = 0; iz < 3; ++iz) {
        if (!((bits >> iz) & 1u)) continue;
        const double Z = Rz[iz];
        const double inv = rsqrt_nr(fma(Z, Z, XY2));
        const double inv2 = inv * inv;
        const double i3 = inv2 * inv;
        const double i5 = (i3 * inv2) * Z;
        c3 += i3;
        c5 += i5;
        pz = fma(i3, Z, pz);
        qz = fma(i5, Z, qz);
      }
      px = fma(c3, X, px);
      py = fma(c3, Y, py);
      qx = fma(c5, X, qx);
      qy = fma(c5, Y, qy);
      sv += c3;
    }
  }
  // g x P + m x Q + (m21 S, 0, 0), m = (m02, m12, m22)
  const double m21 = mm[0], m02 = mm[1], m12 = mm[2], m22 = mm[3];
  im = im + mk3(fma(g[1], pz, fma(-g[2], py, fma(m12, qz, fma(-m22, qy, m21 * sv)))),
                fma(g[2], px, fma(-g[0], pz, fma(m22, qx, -m02 * qz))),
                fma(g[0], py, fma(-g[1], px, fma(m02, qy, -m12 * qx))));
}

// resident warps per SM the register allocation must allow.  ms per launch for
// 12 / 16 / 20 / 24 warps: mixed 1M nodes 31.5 / 27.7 / 28.0 before the sums
// per z shift and the segments' queue (25.7 and 23.8 at 16 since); FP64 in one
// part per group 1M 46.2 / 41.6 / 38.8 / 42.0, 200k 8.4 / 7.6 / 7.6 / 8.0, in
// parts 60k 3.91 / 3.34 / 3.26.  20 warps spill some 90 bytes; the split form
// stays at 16, where a wave holds fewer parts.
// Blocks are one warp each: a block of four kept its place until its slowest
// warp ended (200k nodes FP64, two parts, a first walk: 16.9 ms against 15.9;
// 1M mixed 35.8 against 35.1).
constexpr int kWalkWarps = 16;
constexpr int kWalkWarpsFp64 = 20;

// A group's walk split over `parts` warps (a power of two), for launches with
// too few groups to fill the GPU.  Every part traverses the cells whose
// subtree holds more than `frontier` cells and takes their decisions; those
// cells' evaluations and the smaller subtrees below them are dealt to the
// parts by their place in the preorder, a stretch of 2^deal cells each in
// turn.  Cells near the targets, where most of the work lies, are close
// together in the preorder, so dealing them in turn spreads them.  A target's
// terms are thus dealt by the cells alone, whatever group it is in.  Part p
// of target i writes its sums to nl[p * n_t + i]; k_walk_reduce adds the
// parts in order, so the result depends on neither the grouping nor the
// scheduling.
struct WalkSplit {
  int parts;       // 1, 2, 4, ...
  int frontier;    // cells
  int deal;        // log2 of the stretch of cells dealt at a time
  const int* skip; // points: slot skipped per point (null: none); nodes: unused
  double* nl;      // partial sums, 3 doubles per part and target
  double* im;
};

__device__ __forceinline__ d3 shfl3(d3 v, int src) {
  return mk3(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
             __shfl_sync(0xffffffffu, v.z, src));
}

// Pairs of cell and target waiting to be evaluated 32 at a time, one by each
// lane of the warp, whichever lane's target they belong to.  A leaf is near 8
// to 10 of a group's 32 targets and an accepted cell is one for 20 to 24 of
// them, so evaluated at the visit they leave the other lanes idle.  A target's
// pairs are taken in preorder and added in that order by its own lane.  When a
// queue's are depends on the other targets of the group, so each queue's pairs
// have a sum of their own, to which nothing else is added, and a target's sums
// do not depend on its group.  A grain leaf's node range waits with the
// segments where cells wait.  Segments wait in both forms: 200k / 1M nodes mixed
// 5.04 -> 4.62 / 25.7 -> 23.8 ms, FP64 10.0 -> 8.3 / 51.2 -> 43.5.  Cells wait
// in the FP64 form, where their evaluation takes the FP64 pipe some 400
// operations: 8.3 -> 7.6 / 43.5 -> 38.8; in the mixed form the queue costs more
// than the idle lanes (23.8 -> 27.7).
struct WalkQueue {
  int cell[64];
  unsigned mask[64];   // lane of the target << 27 | image mask
};
struct WalkBatch {
  bool on;
  int cell, own;   // own: lane of the target
  unsigned mask;
};

// every lane with a mask adds the pair of cell q and its target; n < 32
__device__ __forceinline__ void queue_put(WalkQueue& Q, int& n, int q, unsigned mask, int lane) {
  const unsigned who = __ballot_sync(0xffffffffu, mask != 0);
  if (mask) {
    const int at = n + __popc(who & ((1u << lane) - 1u));
    Q.cell[at] = q;
    Q.mask[at] = mask | ((unsigned)lane << 27);
  }
  n += __popc(who);
  __syncwarp();
}

// the first 32 entries (or all n), one per lane; of[l]: which of them are
// of lane l's target, to be read after a __syncwarp()
__device__ __forceinline__ WalkBatch queue_take(WalkQueue& Q, int& n, unsigned* of, int lane) {
  const int cnt = min(n, 32);
  WalkBatch e;
  e.on = lane < cnt;
  e.cell = e.on ? Q.cell[lane] : 0;
  const unsigned m = e.on ? Q.mask[lane] : 0u;
  e.own = e.on ? (int)(m >> 27) : lane;
  e.mask = m & kAllImages;
  const unsigned same = __match_any_sync(0xffffffffu, e.on ? e.own : 32 + lane);
  of[lane] = 0;
  const bool more = lane + 32 < n;
  const int c1 = more ? Q.cell[lane + 32] : 0;
  const unsigned m1 = more ? Q.mask[lane + 32] : 0u;
  __syncwarp();
  if (e.on && lane == __ffs(same) - 1) of[e.own] = same;
  if (more) {
    Q.cell[lane] = c1;
    Q.mask[lane] = m1;
  }
  n -= cnt;
  return e;
}

// kRanges: the tree has grain leaves of several nodes.  The FP64 form has
// kernels of its own without them: with the loop over a node range they take
// 2% longer over trees that have none (200k nodes 7.93 ms, against 7.74).
template <bool kMixed, bool kSplit, bool kRanges>
__global__ void __launch_bounds__(32, kMixed || kSplit ? kWalkWarps : kWalkWarpsFp64)
    k_walk_multi(
    OvParams P, TreeView T, const int* __restrict__ order, const int2* __restrict__ status,
    const double* __restrict__ pos, int n_t, unsigned combos, ImageShortcut S, double near2,
    double* v_nl, double* v_img, unsigned long long* counters, const int* __restrict__ warp_perm,
    unsigned* __restrict__ warp_cost, WalkSplit W) {
  __shared__ unsigned sh_mask[kLevelSlots][32];
  __shared__ WalkQueue leaves;                    // segments and the targets they are near
  __shared__ WalkQueue cells;                     // accepted cells and their targets
  __shared__ unsigned sh_of[32];                  // entries of each lane's target
  __shared__ double sh_seg[kMixed ? 3 : 6][32];   // each lane's sums over segments
  constexpr bool kQueueCells = !kMixed, kQueueRanges = kQueueCells && kRanges;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x;
  const long long t_start = clock64();
  // the group of 32 consecutive targets this warp takes (and its part of a
  // split group): block b runs unit warp_perm[b] (the units by decreasing
  // time in the previous evaluation), or unit b
  const int unit = warp_perm ? warp_perm[blockIdx.x] : blockIdx.x;
  const int gw = kSplit ? unit / W.parts : unit;
  const int i = gw * 32 + lane;
  const int k = i < n_t ? (order ? order[i] : i) : -1;
  const bool live =
      k >= 0 && ((kSplit && !status) || (status[k].x != OV_PINNED && status[k].x != OV_EMPTY));
  // the slot whose own segments the tangle's sum leaves out
  const int skip = kSplit && !status ? (W.skip && live ? W.skip[k] : -1) : k;
  const int part = kSplit ? unit % W.parts : 0;
  int own_end = 0;   // end of the subtree this part walks
  const d3 r = live ? ld3(pos, k) : mk3(0, 0, 0);
  // the shortcuts' bound on rounding holds for targets within a quarter box
  // of the box (a node further out takes every decision in full)
  bool sane = S.on;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double v = a == 0 ? r.x : (a == 1 ? r.y : r.z);
    sane = sane && v >= P.lo[a] - 0.25 * P.L[a] && v <= P.hi[a] + 0.25 * P.L[a];
  }
  unsigned* lvl_mask = &sh_mask[0][lane];   // level l at lvl_mask[32 l]
  lvl_mask[0] = combos;
  d3 nl = mk3(0, 0, 0), im = mk3(0, 0, 0);
  unsigned n_p2p = 0, n_far = 0, n_iter = 0;
  int next = live ? 0 : T.n_cells;
  int n_leaves = 0, n_cells = 0;   // entries waiting
#pragma unroll
  for (int c = 0; c < (kMixed ? 3 : 6); ++c) sh_seg[c][lane] = 0;
  __syncwarp();
  for (;;) {
    const int q = (int)__reduce_min_sync(FULL, (unsigned)next);
    const bool done = q >= T.n_cells;
    if (kQueueCells && (n_cells >= 32 || (done && n_cells > 0))) {
      const WalkBatch e = queue_take(cells, n_cells, sh_of, lane);
      const d3 rt = shfl3(r, e.own);
      d3 v = mk3(0, 0, 0), w = v;
      if (e.on) {
        const Cell* cp = T.cells + e.cell;
        cell_fp64(P, cp, cp->x[0], cp->x[1], cp->x[2], rt, e.mask, v, w);
      }
      __syncwarp();
      for (unsigned of = sh_of[lane]; __any_sync(FULL, of != 0); of &= of - 1) {
        const int src = of ? __ffs(of) - 1 : lane;
        const d3 a = shfl3(v, src), b = shfl3(w, src);
        if (of) {
          nl = nl + a;
          im = im + b;
        }
      }
      continue;
    }
    if (n_leaves >= 32 || (done && n_leaves > 0)) {
      const WalkBatch e = queue_take(leaves, n_leaves, sh_of, lane);
      const d3 rt = shfl3(r, e.own);
      const int skip_t = __shfl_sync(FULL, skip, e.own);
      d3 v = mk3(0, 0, 0), w = v;
      if (e.on) {
        const Cell* cp = T.cells + e.cell;
        const int4 eh = *reinterpret_cast<const int4*>(cp);
        int2 id = make_int2(eh.x, eh.y);
        d3 r1 = mk3(cp->x[0], cp->x[1], cp->x[2]), r2 = mk3(cp->y[0], cp->y[1], cp->y[2]);
        int j = 0, end = 1;
        auto load = [&]() {
          const double* nd = T.nodes64 + 6 * (size_t)j;
          id = T.nodeids[j];
          r1 = mk3(nd[0], nd[1], nd[2]);
          r2 = mk3(nd[3], nd[4], nd[5]);
        };
        if (kQueueRanges && cell_kind(eh.w) != CELL_LEAF1) {
          const int2 rg = T.cell_range[e.cell];
          j = max(rg.x, 0);
          end = min(rg.x + rg.y, T.n_nodes);
          if (j < end) load();
        }
        while (j < end) {
          if (kMixed && __popc(e.mask) >= kColumnImages)
            p2p_mixed_columns(P, e.mask, rt, r1, r2, id.x, id.y, skip_t, near2, v, n_p2p);
          else
            p2p_images<kMixed>(P, e.mask, rt, r1, r2, id.x, id.y, skip_t, near2, v, w, n_p2p);
          if (!kQueueRanges || ++j >= end) break;
          load();
        }
      }
      __syncwarp();
      for (unsigned of = sh_of[lane]; __any_sync(FULL, of != 0); of &= of - 1) {
        const int src = of ? __ffs(of) - 1 : lane;
        const d3 a = shfl3(v, src);
        if (of) {
          sh_seg[0][lane] += a.x;
          sh_seg[1][lane] += a.y;
          sh_seg[2][lane] += a.z;
        }
        if constexpr (!kMixed) {
          const d3 b = shfl3(w, src);
          if (of) {
            sh_seg[3][lane] += b.x;
            sh_seg[4][lane] += b.y;
            sh_seg[5][lane] += b.z;
          }
        }
      }
      continue;
    }
    if (done) break;
    const Cell* cp = T.cells + q;
    if (lane == 0 && q + 1 < T.n_cells) prefetch_l1(cp + 1);
    const int4 h = *reinterpret_cast<const int4*>(cp);
    const double2 t0 = *reinterpret_cast<const double2*>(&cp->thr);
    const double2 t1 = *reinterpret_cast<const double2*>(&cp->x[1]);
    const int kind = cell_kind(h.w);
    if (lane == 1 && h.z < T.n_cells) prefetch_l1(T.cells + h.z);
    bool mine = true;   // whether this part evaluates the cell
    if (kSplit && q >= own_end) {
      mine = ((q >> W.deal) & (W.parts - 1)) == part;
      if (h.z - q <= W.frontier) {
        if (!mine) {   // a subtree of another part
          if (next == q) next = max(h.z, q + 1);
          continue;
        }
        own_end = h.z;
      }
    }
    unsigned p2p_mask = 0;    // images summing this cell's node range directly
    unsigned leaf_mask = 0;   // images summing this leaf's segment
    unsigned cell_mask = 0;   // images accepting this cell
    if (next == q) {
      const unsigned m = lvl_mask[32 * cell_ltop(h.w)];
      unsigned open = 0;
      if (kind == CELL_LEAF1) {
        leaf_mask = h.y == -1 ? 0u : m;
      } else if (kind == CELL_LEAFN) {
        p2p_mask = mine ? m : 0;
      } else {
        // opening test per image (octree_get_vs, src/octree.c:284-296)
        const double cx = t0.y, cy = t1.x, cz = t1.y;
        // Per axis, an image point's exact wrapped distance to the centre
        // of mass is at least the target's, and equal to it when the
        // target's unwrapped difference c - r is below half a box (the
        // image's single wrap then undoes its shift).  The cell's margin E
        // (mac_margin) bounds the FP64 rounding of every image's squared
        // distance, so when the target's q0 passes by E every image passes,
        // and when q0 fails by E the images' decisions follow from the
        // per-axis distances (wrapped_decisions).  Otherwise (and at the
        // root, whose centre of mass may lie outside the box) all decisions
        // are taken in full.
        unsigned pass;
        // The reference wraps an axis when c - r lies outside [-L/2, L/2];
        // where no axis wraps its squared distance is that of c - r itself
        // (fl(r - c) = -fl(c - r)), bit for bit.
        const double dx = __dsub_rn(cx, r.x), dy = __dsub_rn(cy, r.y), dz = __dsub_rn(cz, r.z);
        double q0;
        if (fabs(dx) <= S.half[0] && fabs(dy) <= S.half[1] && fabs(dz) <= S.half[2])
          q0 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        else
          q0 = __dadd_rn(__dadd_rn(wrapped_sq(P, 0, r.x, cx), wrapped_sq(P, 1, r.y, cy)), wrapped_sq(P, 2, r.z, cz));
        const double E = (double)__int_as_float(h.y);
        const bool shortcut = sane && q > 0;
        if (shortcut && q0 >= t0.x + E) {
          pass = m;
        } else if (shortcut && q0 < t0.x - E && wrapped_decisions(P, S, r, cx, cy, cz, dx, dy, dz, t0.x, E, pass)) {
          // decided from the per-axis distances
        } else {
          // q0 is the target's own decision in mac_exact's operations; the
          // other images still open here are few below the top levels, so
          // they are decided one by one unless there are many
          pass = q0 >= t0.x ? (1u << kPrimary) : 0u;
          unsigned rest = m & ~(1u << kPrimary);
          if (__popc(rest) > kFewImages) {
            pass |= mac_exact(P, r, cx, cy, cz, t0.x) & rest;
          } else {
            while (rest) {
              const int c = __ffs(rest) - 1;
              rest &= rest - 1;
              const int ix = (c * 57) >> 9, rem = c - 9 * ix, iy = (rem * 11) >> 5, iz = rem - 3 * iy;
              const double q = __dadd_rn(__dadd_rn(wrapped_sq(P, 0, img_coord(r.x, P.L[0], ix), cx),
                                                   wrapped_sq(P, 1, img_coord(r.y, P.L[1], iy), cy)),
                                         wrapped_sq(P, 2, img_coord(r.z, P.L[2], iz), cz));
              if (q >= t0.x) pass |= 1u << c;
            }
          }
        }
        pass &= m;
        const unsigned fail = m & ~pass;
        if (kind == CELL_OPEN) open = fail;
        else if (kind == CELL_OPEN_P2P) p2p_mask = mine ? fail : 0;
        if (pass && mine) {
          n_far += __popc(pass);
          // expansion at every accepting image: R = r - L s - com, unwrapped
          if (kQueueCells)
            cell_mask = pass;
          else
            cell_mixed(P, cp, __int_as_float(h.x), cx, cy, cz, t0.x, r, mk3(dx, dy, dz), pass, near2, nl);
        }
      }
      if (open) lvl_mask[32 * (cell_lbot(h.w) + 1)] = open;
      // each lane's next cell strictly increases: the loop ends within n_cells
      next = open ? q + 1 : max(h.z, q + 1);
    }
    ++n_iter;
    if (kind == CELL_LEAF1) {
      queue_put(leaves, n_leaves, q, leaf_mask, lane);
      continue;
    }
    if (kQueueCells) queue_put(cells, n_cells, q, cell_mask, lane);
    // direct sums over a node range (grain leaves)
    if (kQueueRanges) {
      if (kind == CELL_LEAFN || kind == CELL_OPEN_P2P) queue_put(leaves, n_leaves, q, p2p_mask, lane);
    } else if (kRanges && __ballot_sync(FULL, p2p_mask != 0)) {   // shared by the warp
      const int2 rg = T.cell_range[q];
      const int end = min(rg.x + rg.y, T.n_nodes);
      for (int j = max(rg.x, 0); j < end; ++j) {
        const int2 id = T.nodeids[j];
        if (!p2p_mask) continue;
        const double* nd = T.nodes64 + 6 * (size_t)j;
        if (kMixed && __popc(p2p_mask) >= kColumnImages)
          p2p_mixed_columns(P, p2p_mask, r, mk3(nd[0], nd[1], nd[2]), mk3(nd[3], nd[4], nd[5]), id.x, id.y,
                            skip, near2, nl, n_p2p);
        else
          p2p_images<kMixed>(P, p2p_mask, r, mk3(nd[0], nd[1], nd[2]), mk3(nd[3], nd[4], nd[5]), id.x,
                             id.y, skip, near2, nl, im, n_p2p);
      }
    }
  }
  nl = nl + mk3(sh_seg[0][lane], sh_seg[1][lane], sh_seg[2][lane]);
  if constexpr (!kMixed) im = im + mk3(sh_seg[3][lane], sh_seg[4][lane], sh_seg[5][lane]);
  if (kSplit) {
    if (i < n_t) {
      st3(W.nl + 3 * (size_t)part * n_t, i, nl);
      if (!kMixed) st3(W.im + 3 * (size_t)part * n_t, i, im);
    }
  } else if (live) {
    st3(v_nl, k, nl);
    st3(v_img, k, im);
  }
  // counters: per-warp sums
  unsigned long long a = n_p2p, b = n_far;
  for (int off = 16; off > 0; off >>= 1) {
    a += __shfl_xor_sync(FULL, a, off);
    b += __shfl_xor_sync(FULL, b, off);
  }
  if (lane == 0) {
    atomicAdd(&counters[0], a);
    atomicAdd(&counters[1], b);
    atomicAdd(&counters[2], (unsigned long long)n_iter);
    // this unit's time in SM cycles / 64, for the next evaluation's order
    if (warp_cost) warp_cost[unit] = (unsigned)min((clock64() - t_start) >> 6, 0xffffffffll);
  }
}

// the parts of a split walk added in order: target i's sums into slot
// order[i] (or i); im null: the mixed form, whose one sum is in nl
__global__ void k_walk_reduce(const int* __restrict__ order, const int2* __restrict__ status, int n_t, int parts,
                              const double* __restrict__ nl, const double* __restrict__ im, double* v_nl,
                              double* v_img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_t) return;
  const int k = order ? order[i] : i;
  if (k < 0 || (status && (status[k].x == OV_PINNED || status[k].x == OV_EMPTY))) return;
  d3 a = ld3(nl, i);
  for (int p = 1; p < parts; ++p) a = a + ld3(nl + 3 * (size_t)p * n_t, i);
  st3(v_nl, k, a);
  if (!v_img) return;
  d3 b = im ? ld3(im, i) : mk3(0, 0, 0);
  for (int p = 1; im && p < parts; ++p) b = b + ld3(im + 3 * (size_t)p * n_t, i);
  st3(v_img, k, b);
}

// All nodes: warp w handles sorted targets 32w .. 32w+31, every image.
// Targets in `order` (the tree's key order, so a warp's targets are close in
// space), or slot order when order is null.
template <bool kMixed>
__global__ void __launch_bounds__(128) k_walk_nodes(OvParams P, TreeView T, const int* __restrict__ order,
                                                    const int2* __restrict__ status,
                                                    const double* __restrict__ pos, int n_t,
                                                    double* v_nl, double* v_img,
                                                    unsigned long long* counters) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int i = gw * 32 + lane;
  if (gw * 32 >= n_t) return;   // whole warp out of range
  int k = i < n_t ? (order ? order[i] : i) : -1;
  bool live = k >= 0 && status[k].x != OV_PINNED && status[k].x != OV_EMPTY;
  d3 r = live ? ld3(pos, k) : mk3(0, 0, 0);
  unsigned long long n_p2p = 0, n_far = 0, n_iter = 0;
  d3 nl = warp_walk<kMixed>(P, T, r, live, k, true, P.theta, n_p2p, n_far, n_iter);
  d3 im = mk3(0, 0, 0);
  for (int j = 0; j < P.n_img; ++j) {
    d3 rp = live ? image_point(P, j, r) : r;
    d3 v = warp_walk<kMixed>(P, T, rp, live, -1, true, P.theta, n_p2p, n_far, n_iter);
    int face = P.img[j][3];
    if (face > -1) v = mirror_dir(v, face);
    im = im + v;
  }
  if (live) {
    st3(v_nl, k, nl);
    st3(v_img, k, im);
  }
  if (lane == 0) {
    atomicAdd(&counters[0], n_p2p);
    atomicAdd(&counters[1], n_far);
    atomicAdd(&counters[2], n_iter);
  }
}

// Arbitrary points (octree_get_vs at user points), optionally with images.
template <bool kMixed>
__global__ void __launch_bounds__(128) k_walk_points(OvParams P, TreeView T, const double* __restrict__ pts,
                                                     const int* __restrict__ skip, int npts,
                                                     int use_thr, double theta, double* out_nl,
                                                     double* out_img, unsigned long long* counters) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int i = gw * 32 + lane;
  if (gw * 32 >= npts) return;
  bool live = i < npts;
  d3 r = live ? ld3(pts, i) : mk3(0, 0, 0);
  int sk = (live && skip) ? skip[i] : -1;
  unsigned long long n_p2p = 0, n_far = 0, n_iter = 0;
  d3 v = warp_walk<kMixed>(P, T, r, live, sk, use_thr != 0, theta, n_p2p, n_far, n_iter);
  if (out_img) {
    d3 im = mk3(0, 0, 0);
    for (int j = 0; j < P.n_img; ++j) {
      d3 rp = live ? image_point(P, j, r) : r;
      d3 w = warp_walk<kMixed>(P, T, rp, live, -1, use_thr != 0, theta, n_p2p, n_far, n_iter);
      int face = P.img[j][3];
      if (face > -1) w = mirror_dir(w, face);
      im = im + w;
    }
    if (live) st3(out_img, i, im);
  }
  if (live) st3(out_nl, i, v);
  if (lane == 0) {
    atomicAdd(&counters[0], n_p2p);
    atomicAdd(&counters[1], n_far);
    atomicAdd(&counters[2], n_iter);
  }
}

TreeView view_of(OvTree* t) {
  TreeView v;
  v.cells = t->cells.as<Cell>();
  v.cell_lm = t->cell_lm.as<double>();
  v.cell_range = t->cell_range.as<int2>();
  v.nodes64 = t->nodes64.as<double>();
  v.nodeids = t->nodeids.as<int2>();
  v.n_cells = t->n_cells;
  v.n_nodes = t->n_nodes;
  return v;
}

}  // namespace

// Target list with the nin nodes inside the root box after the nd outside
// it, each of those alone in a warp (lane 0; -1 marks an empty lane).
constexpr int kMaxDropWarps = 1024;
static __global__ void k_drop_first(const int* __restrict__ perm, int nin, int nd, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int pad = 32 * nd;
  if (i >= pad + nin) return;
  out[i] = i < pad ? ((i & 31) == 0 ? perm[nin + (i >> 5)] : -1) : perm[i - pad];
}

// sort keys for the units' order: decreasing time first, to 8 significant
// bits (the time as an FP32 number, its sign and low 15 bits dropped), so two
// passes of the radix sort order them
constexpr int kCostBits = 16;
static __global__ void k_cost_keys(const unsigned* cost, int n, uint64_t* keys, int* vals) {
  follow_early();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = 0xffffu - ((unsigned)__float_as_int((float)cost[i]) >> 15);
  vals[i] = i;
}

// Hilbert keys of points in the box, kCurveBits per axis (J. Skilling,
// "Programming the Hilbert curve", AIP Conf. Proc. 707, 2004: the transform
// of the axes into the curve's transposed index).  Points outside the box,
// whose coordinates clamp, and NaN, which converts to 0, sort somewhere: the
// order only decides which targets share a warp.
constexpr int kCurveBits = 10;
static __global__ void k_curve_keys(OvParams P, const double* pts, int n, uint64_t* keys, int* vals) {
  follow_early();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned x[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double f = (pts[3 * (size_t)i + a] - P.lo[a]) / P.L[a] * (1 << kCurveBits);
    x[a] = (unsigned)fmin(fmax(f, 0.0), (double)((1 << kCurveBits) - 1));
  }
  for (unsigned q = 1u << (kCurveBits - 1); q > 1; q >>= 1) {
    const unsigned m = q - 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (x[a] & q) {
        x[0] ^= m;
      } else {
        const unsigned t = (x[0] ^ x[a]) & m;
        x[0] ^= t;
        x[a] ^= t;
      }
    }
  }
  x[1] ^= x[0];
  x[2] ^= x[1];
  unsigned t = 0;
  for (unsigned q = 1u << (kCurveBits - 1); q > 1; q >>= 1)
    if (x[2] & q) t ^= q - 1;
  unsigned key = 0;
#pragma unroll
  for (int b = kCurveBits - 1; b >= 0; --b)
#pragma unroll
    for (int a = 0; a < 3; ++a) key = (key << 1) | (((x[a] ^ t) >> b) & 1u);
  keys[i] = key;
  vals[i] = i;
}

constexpr int kMaxParts = 16;        // warps a group of nodes' walk is split over, at most
constexpr int kMaxPointParts = 32;   // and a group of points'

static bool read_counters(ov_state_impl* s, const unsigned long long* ctr) {
  unsigned long long c[3] = {0, 0, 0};
  OV_TRY_CUDA(cudaMemcpyAsync(c, ctr, sizeof(c), cudaMemcpyDeviceToHost, s->stream));
  OV_TRY_CUDA(cudaStreamSynchronize(s->stream));
  OvStatsAcc& st = ov_stats_tls();
  st.interactions = (double)c[0];
  st.cell_interactions = (double)c[1];
  st.warp_iterations = (double)c[2];
  return true;
}

// The image table as a set of periodic shifts in {-1,0,1}^3 (bit 9 (sx+1) +
// 3 (sy+1) + (sz+1), the tangle itself included); false for a table with
// mirrors or repeated shifts, which the multi-image walk does not take.
static bool image_combos(const OvParams& P, int n_img, unsigned& combos) {
  combos = 1u << kPrimary;
  for (int j = 0; j < n_img; ++j) {
    const int* im = P.img[j];
    if (im[3] != -1 || im[0] < -1 || im[0] > 1 || im[1] < -1 || im[1] > 1 || im[2] < -1 || im[2] > 1)
      return false;
    const unsigned bit = 1u << (9 * (im[0] + 1) + 3 * (im[1] + 1) + (im[2] + 1));
    if (combos & bit) return false;
    combos |= bit;
  }
  return true;
}

// shortcut parameters: see ImageShortcut and mac_margin (the rounding
// allowance 8 u B with B the bound on magnitudes of mac_margin)
static ImageShortcut image_shortcut(const OvParams& P, unsigned combos) {
  ImageShortcut sc;
  double B = 0;
  for (int a = 0; a < 3; ++a) B = std::max(B, std::fabs(P.lo[a]) + std::fabs(P.hi[a]));
  const double allowance = 8 * 0x1p-53 * 3.5 * B;
  sc.on = 1;
  for (int a = 0; a < 3; ++a) {
    bool shifted = false;
    for (int c = 0; c < kCombos; ++c) {
      const int sa = a == 0 ? c / 9 : (a == 1 ? (c / 3) % 3 : c % 3);
      if (((combos >> c) & 1u) && sa != 1) shifted = true;
    }
    if (shifted && !P.periodic[a]) sc.on = 0;
    sc.hw[a] = shifted ? 0.5 * P.L[a] - allowance : DBL_MAX;
    sc.wr[a] = shifted ? 0.5 * P.L[a] + allowance : DBL_MAX;
    sc.half[a] = P.periodic[a] ? P.L[a] * 0.5 : DBL_MAX;
  }
  return sc;
}

// warps of one wave of a walk kernel: resident blocks on every SM
template <class K>
static int walk_wave(K kernel) {
  int dev = 0, sms = 0, nb = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, 32, 0) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return std::max(1, sms * nb);
}

// The multi-image walk of n_t targets at pos: nodes (status given: slots of
// `order`) or points (status null: order sorts them, skip per point).
// n_rule: the targets the split rule counts (a rank's share of a sharded
// evaluation counts all of them, so every rank adds its sums in the order
// one GPU would).  v_img null: no image sums wanted.
static bool launch_multi(ov_state_impl* s, OvTree* t, const OvParams& P, const int* order, const int2* status,
                         const int* skip, const double* pos, int n_t, int n_rule, unsigned combos, double* v_nl,
                         double* v_img, unsigned long long* ctr, bool timed) {
  const bool mixed = P.precision == OV_PREC_MIXED;
  const ImageShortcut sc = image_shortcut(P, combos);
  const TreeView tv = view_of(t);
  static const int wave_mixed = walk_wave(k_walk_multi<true, true, true>);
  static const int wave_fp64 = walk_wave(k_walk_multi<false, true, true>);
  const int wave = mixed ? wave_mixed : wave_fp64;
  // Parts per group.  Nodes: enough that the units make two waves (of 2368
  // warps), so the last wave's slow units are short, but no more than 16, as
  // each part takes the decisions above the frontier again.  26 images, theta
  // = 0.4, ms per walk of a tangle stepped on: 8 / 16 / 32 parts at 3000 nodes
  // mixed 0.25 / 0.23 / 0.32, at 8000 0.37 / 0.34 / 0.65; targets of one, two
  // and four waves at 22.4k 0.96 / 0.85 / 1.52, at 100k 4.06 / 3.48 / 3.56.
  // Points are fewer and their groups wider: 5/6 of a wave, so that it is one
  // wave whatever power of two the parts come to, and up to 32 parts: queries
  // of 512 points over 20k nodes 0.74 ms, 16 parts 0.85; of 4096 over 50k 1.15
  // ms in 16 parts, 1.29 in 32.
  int parts = 1;
  const int groups = (n_t + 31) / 32;
  const long long groups_rule = (n_rule + 31) / 32;
  const long long units = status ? 2LL * wave : 5LL * wave / 6;
  while (parts < (status ? kMaxParts : kMaxPointParts) && groups_rule * parts < units) parts *= 2;
  // Frontier: a smaller one deals the work out more evenly, but its cells'
  // decisions are taken again in every part.  Nodes 1/32 of the cells, ms at
  // 1/8, 1/16, 1/32, 1/64, 1/128: mixed 8000 nodes 0.34 (1/32), 0.35, 0.40;
  // 22.4k 0.92, 0.76, 0.79, 0.85, 1.06; 60k 1.83, 1.88, 1.87, 2.09, 2.30; FP64
  // 22.4k 1.29, 1.20, 1.17, 1.24, 1.48.  Points 1/96 (512 over 20k nodes 0.77
  // at 1/64, 0.74, 0.75 at 1/128, 0.77 at 1/192).
  const int frontier = std::max(1, t->n_cells / (status ? 32 : 96));
  // Stretches of a quarter of the frontier.  Chosen when a walk evaluated its
  // leaves and cells at the visit (22.4k nodes FP64, 8 parts: 2.52 ms, against
  // 2.66 with a sixteenth).  With the queues a sixteenth is the faster one:
  // theta = 0.4, FP64 1.14 ms against 1.21 now and mixed 0.78 against 0.92 at
  // 22.4k nodes, 3.46 / 3.53 and 2.29 / 2.34 at 59k, 0.58 / 0.60 and 0.35 /
  // 0.34 at 7.9k.  It would change the order of the sums and is not taken here.
  int deal = 0;
  while ((8 << deal) <= frontier) ++deal;
  const bool split = parts > 1 || !status;
  const int warps = groups * parts;
  WalkSplit W{parts, frontier, deal, skip, nullptr, nullptr};
  if (split) {
    const size_t per = 3 * (size_t)n_t * parts;
    if (!s->walk_part.reserve(sizeof(double) * (mixed ? 1 : 2) * per)) return false;
    W.nl = s->walk_part.as<double>();
    W.im = mixed ? nullptr : W.nl + per;
  }
  // Longest first: the launch runs the warps' units (groups of 32 targets,
  // or their parts) in the order of their times in the previous walk of this
  // tree (the same regions of the key order, a few node moves apart), so the
  // slow ones do not start in the last wave.  The sums do not depend on the
  // order.  A launch within one wave starts every unit at once and needs no
  // order.  A rank's share of a sharded evaluation is the same key range at
  // every evaluation, so its units are ordered the same way.
  timed = timed && warps > wave;
  const int* wperm = timed && t->n_perm_warps == warps ? t->wvals.as<int>() : nullptr;
  unsigned* wcost = nullptr;
  if (timed) {
    if (!t->warp_cost.reserve(sizeof(unsigned) * (size_t)warps)) return false;
    wcost = t->warp_cost.as<unsigned>();
  }
  auto kernel = split ? (mixed         ? k_walk_multi<true, true, true>
                         : t->has_ranges ? k_walk_multi<false, true, true>
                                         : k_walk_multi<false, true, false>)
                      : (mixed         ? k_walk_multi<true, false, true>
                         : t->has_ranges ? k_walk_multi<false, false, true>
                                         : k_walk_multi<false, false, false>);
  kernel<<<warps, 32, 0, s->stream>>>(P, tv, order, status, pos, n_t, combos, sc, P.near2, v_nl, v_img, ctr, wperm,
                                      wcost, W);
  OV_LAUNCHED();
  OV_TRY_CUDA(cudaGetLastError());
  if (split) {
    k_walk_reduce<<<(n_t + 127) / 128, 128, 0, s->stream>>>(order, status, n_t, parts, W.nl, W.im, v_nl, v_img);
    OV_LAUNCHED();
    OV_TRY_CUDA(cudaGetLastError());
  }
  if (status) ov_mark(s, s->ev2);   // of an evaluation; a point query is none
  if (timed) {
    // the order for the next walk (after the timed kernel)
    const size_t nw = (size_t)warps;
    if (!t->wkeys.reserve(sizeof(uint64_t) * nw) || !t->wkeys2.reserve(sizeof(uint64_t) * nw) ||
        !t->wvals.reserve(sizeof(int) * nw) || !t->wvals2.reserve(sizeof(int) * nw))
      return false;
    OV_TRY_CUDA(ov_launch_early(k_cost_keys, dim3((warps + 255) / 256), 256, s->stream, wcost, warps,
                                t->wkeys.as<uint64_t>(), t->wvals.as<int>()));
    OV_LAUNCHED();
    if (!ov_radix_sort_u64(t->wkeys.as<uint64_t>(), t->wvals.as<int>(), t->wkeys2.as<uint64_t>(),
                           t->wvals2.as<int>(), warps, kCostBits, t->whist, t->wscan, s->stream))
      return false;
    t->n_perm_warps = warps;
  }
  return true;
}

bool ov_tree_walk_nodes(ov_state_impl* s, OvTree* t, const double* pos, bool own_tree,
                        double* v_nl, double* v_img, int k0, int k_count) {
  unsigned long long* ctr = s->evctr.as<unsigned long long>() + 3 * s->pending;
  OV_TRY_CUDA(cudaMemsetAsync(ctr, 0, 24, s->stream));
  // a tree built from these positions: its key order; otherwise slot order
  const int* order = own_tree ? t->perm.as<int>() : nullptr;
  int n_t = own_tree ? t->n_nodes : s->n;
  if (n_t == 0 || t->n_cells == 0) {
    ov_mark(s, s->ev1);
    ov_mark(s, s->ev2);
    OV_TRY_CUDA(cudaMemsetAsync(v_nl, 0, sizeof(double) * 3 * s->n, s->stream));
    OV_TRY_CUDA(cudaMemsetAsync(v_img, 0, sizeof(double) * 3 * s->n, s->stream));
    return true;
  }
  // one rank's share: a contiguous range of the key order (each target's
  // walk depends only on its own position, so the range changes no result)
  int key_lo = 0;   // key position of order[0]
  if (own_tree && k_count >= 0) {
    const int lo = std::min(std::max(k0, 0), n_t);
    key_lo = lo;
    n_t = std::min(k_count, n_t - lo);
    order += lo;
    if (n_t <= 0) {
      ov_mark(s, s->ev1);
      ov_mark(s, s->ev2);
      return true;
    }
  }
  // Nodes outside the root box take key digit 8 at level 1 and sort after
  // every other node, so they would share the last warps whatever their
  // positions.  A warp of targets scattered over the box's faces walks the
  // union of their trees, and as the last block it ran almost alone at the
  // end of the launch: 20 such nodes made a 1M-point walk 28% longer.  Each
  // gets a warp of its own at the front of the list instead (the other lanes
  // empty); the sums do not depend on the order.  In a rank's share of the
  // key order these nodes are the share's last ones.
  const int nd = own_tree ? std::max(0, std::min(n_t, key_lo + n_t - (t->n_nodes - t->n_drop_root))) : 0;
  if (nd > 0 && t->n_drop_root <= kMaxDropWarps) {
    const int nin = n_t - nd;
    const int m = 32 * nd + nin;
    if (!t->walk_order.reserve(sizeof(int) * (size_t)m)) return false;
    k_drop_first<<<(m + 255) / 256, 256, 0, s->stream>>>(order, nin, nd, t->walk_order.as<int>());
    OV_LAUNCHED();
    OV_TRY_CUDA(cudaGetLastError());
    order = t->walk_order.as<int>();
    n_t = m;
  }
  OvParams P = t->P;
  // image table and precision of this call; geometry of the tree's build
  P.n_img = s->P.n_img;
  for (int j = 0; j < P.n_img; ++j)
    for (int c = 0; c < 4; ++c) P.img[j][c] = s->P.img[j][c];
  P.precision = s->P.precision;
  const bool mixed = s->P.precision == OV_PREC_MIXED;
  unsigned combos = 0;
  if (image_combos(P, P.n_img, combos)) {
    ov_mark(s, s->ev1);
    P.near2 = s->P.near2;
    if (!launch_multi(s, t, P, order, s->status.as<int2>(), nullptr, pos, n_t, own_tree ? t->n_nodes : n_t, combos,
                      v_nl, v_img, ctr, own_tree))
      return false;
    return true;
  }
  const TreeView tv = view_of(t);
  ov_mark(s, s->ev1);
  const int warps = (n_t + 31) / 32;
  const int blocks = (warps * 32 + 127) / 128;
  if (mixed) {
    k_walk_nodes<true><<<blocks, 128, 0, s->stream>>>(P, tv, order, s->status.as<int2>(), pos, n_t,
                                                        v_nl, v_img, ctr);
    OV_LAUNCHED();
  } else {
    k_walk_nodes<false><<<blocks, 128, 0, s->stream>>>(P, tv, order, s->status.as<int2>(), pos, n_t,
                                                        v_nl, v_img, ctr);
    OV_LAUNCHED();
  }
  OV_TRY_CUDA(cudaGetLastError());
  ov_mark(s, s->ev2);
  return true;
}

bool ov_tree_walk_points(ov_state_impl* s, OvTree* t, int npts, const double* pts, const int* skip,
                         double theta, double* out_nl, double* out_img) {
  if (npts <= 0) return true;
  if (t->n_cells == 0) {
    OV_TRY_CUDA(cudaMemsetAsync(out_nl, 0, sizeof(double) * 3 * npts, s->stream));
    if (out_img) OV_TRY_CUDA(cudaMemsetAsync(out_img, 0, sizeof(double) * 3 * npts, s->stream));
    return true;
  }
  unsigned long long* ctr = s->evctr.as<unsigned long long>() + 3 * kEvalSlots;
  OV_TRY_CUDA(cudaMemsetAsync(ctr, 0, 24, s->stream));
  OvParams P = t->P;
  P.n_img = s->P.n_img;
  for (int j = 0; j < P.n_img; ++j)
    for (int c = 0; c < 4; ++c) P.img[j][c] = s->P.img[j][c];
  const int use_thr = theta == t->theta;
  unsigned combos = 0;
  // One traversal per point for all its images, the points in Hilbert order
  // of the box so a warp's 32 are close together: 4096 probes of a 50k-node
  // tangle with 26 images take 1.06 ms with the build, against 129 ms with one
  // walk per image and the points as given.  FP64 in the mixed form too (a
  // query's cost is its traversal).  A table with mirrors, or an opening angle
  // other than the tree's, takes the walk per image.
  if (use_thr && image_combos(P, out_img ? P.n_img : 0, combos)) {
    const int* order = nullptr;
    if (npts > 32) {
      const size_t np = (size_t)npts;
      if (!s->pkeys.reserve(sizeof(uint64_t) * 2 * np) || !s->pvals.reserve(sizeof(int) * 2 * np)) return false;
      uint64_t* keys = s->pkeys.as<uint64_t>();
      int* vals = s->pvals.as<int>();
      OV_TRY_CUDA(ov_launch_early(k_curve_keys, dim3((npts + 255) / 256), 256, s->stream, P, pts, npts, keys,
                                  vals));
      OV_LAUNCHED();
      if (!ov_radix_sort_u64(keys, vals, keys + np, vals + np, npts, 3 * kCurveBits, s->phist, s->pscan, s->stream))
        return false;
      order = vals;
    }
    P.precision = OV_PREC_FP64;
    if (!launch_multi(s, t, P, order, nullptr, skip, pts, npts, npts, combos, out_nl, out_img, ctr, false))
      return false;
    return read_counters(s, ctr);
  }
  const int warps = (npts + 31) / 32;
  const int blocks = (warps * 32 + 127) / 128;
  const TreeView tv = view_of(t);
  if (s->P.precision == OV_PREC_MIXED) {
    k_walk_points<true><<<blocks, 128, 0, s->stream>>>(P, tv, pts, skip, npts, use_thr, theta,
                                                        out_nl, out_img, ctr);
    OV_LAUNCHED();
  }
  else {
    k_walk_points<false><<<blocks, 128, 0, s->stream>>>(P, tv, pts, skip, npts, use_thr, theta,
                                                         out_nl, out_img, ctr);
    OV_LAUNCHED();
  }
  OV_TRY_CUDA(cudaGetLastError());
  return read_counters(s, ctr);
}

// ---------------------------------------------------------------- shards
namespace {

__global__ void k_shard_pack(const int* __restrict__ perm, int k0, int count,
                             const double* __restrict__ v_nl, const double* __restrict__ v_img,
                             double* xbuf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int k = perm[k0 + i];
  double* o = xbuf + 6 * ((size_t)k0 + i);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    o[c] = v_nl[3 * (size_t)k + c];
    o[3 + c] = v_img[3 * (size_t)k + c];
  }
}

__global__ void k_shard_unpack(const int* __restrict__ perm, int n, const double* __restrict__ xbuf,
                               double* v_nl, double* v_img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = perm[i];
  const double* x = xbuf + 6 * (size_t)i;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    v_nl[3 * (size_t)k + c] = x[c];
    v_img[3 * (size_t)k + c] = x[3 + c];
  }
}

// the exchange buffer holds 6 doubles per key position of the tree
bool shard_fits(ov_state_impl* s, size_t xcap) {
  if (6 * (size_t)s->tree.n_nodes <= xcap) return true;
  ov_set_error(OV_ERR_INVALID, "tree of %d nodes beyond the exchange buffer (%zu doubles): call "
               "ov_state_shard after the upload", s->tree.n_nodes, xcap);
  return false;
}

}  // namespace

bool ov_shard_pack(ov_state_impl* s, int k0, int count, double* xbuf, size_t xcap) {
  if (!shard_fits(s, xcap)) return false;
  const int n = s->tree.n_nodes;
  k0 = std::min(std::max(k0, 0), n);
  count = std::min(count, n - k0);
  if (count <= 0) return true;
  k_shard_pack<<<(count + 255) / 256, 256, 0, s->stream>>>(s->tree.perm.as<int>(), k0, count,
                                                           s->v_nl.as<double>(), s->v_img.as<double>(), xbuf);
  OV_LAUNCHED();
  OV_TRY_CUDA(cudaGetLastError());
  return true;
}

bool ov_shard_unpack(ov_state_impl* s, const double* xbuf, size_t xcap) {
  if (!shard_fits(s, xcap)) return false;
  const int n = s->tree.n_nodes;
  if (n <= 0) return true;
  k_shard_unpack<<<(n + 255) / 256, 256, 0, s->stream>>>(s->tree.perm.as<int>(), n, xbuf,
                                                         s->v_nl.as<double>(), s->v_img.as<double>());
  OV_LAUNCHED();
  OV_TRY_CUDA(cudaGetLastError());
  return true;
}
