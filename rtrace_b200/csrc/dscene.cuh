// Device-resident scene layout and the intersection routines of the render
// path.  Each primitive test restates one reference function in the same
// IEEE operation order; see the comments for the reference lines.
//
// Acceleration.  The reference tests objects in scene order
// (World::hit, src/ray.rs:699-711) and walks each mesh's k-d tree without
// t-interval pruning (src/mesh.rs:399-465).  The device reaches the same
// answers faster:
//   * Meshes: a BVH over the mesh's triangles proposes candidates; a
//     candidate counts only if the reference's traversal would have tested
//     it, i.e. if one of the k-d leaves holding it is visited by the
//     reference's rules (near child always, far child iff t_split >= 0,
//     one side for axis-parallel rays, then the leaf's slab test).  Among
//     equal-t candidates the one the reference's depth-first walk meets
//     first wins (the strict `t < closest` test keeps the first).  When
//     verification cannot settle a closest-hit query (more ties than the
//     buffer holds, or no minimal candidate is visited), the exact k-d walk
//     runs instead.
//   * Runs of consecutive spheres: a BVH over the run.  Spheres accept
//     `root <= closest`, so the sequential scan's result is the minimal
//     accepted t with ties resolved to the latest sphere; the group search
//     returns exactly that.
//   * Shadow rays only ask `world.hit(..).is_some()`; every per-object
//     test is monotone in t_max, so any accepting object suffices.
// Boxes are padded and pruning uses a relative margin, so a box never
// rejects a primitive the exact test would accept.  Mesh BVH boxes are
// tested in single precision with margins that keep this (RayF).
#pragma once

#include "dmath.cuh"

namespace rtb {

#ifndef RTB_INF
#define RTB_INF __longlong_as_double(0x7ff0000000000000LL)
#endif

enum { OBJ_SPHERE = 0, OBJ_PLANE = 1, OBJ_CUBE = 2, OBJ_MESH = 3, OBJ_SPHERE_GROUP = 4 };

// Device error flags (bitmask in DFrame::err)
enum { ERR_WATCHDOG = 1, ERR_EMPTY_RANGE = 2, ERR_STACK = 4, ERR_RANGE_OVERFLOW = 8, ERR_BARRIER = 32 };

// Pruning: a box is skipped only when its entry exceeds t * REL + ABS.
#define RTB_PRUNE_REL 1.000001
#define RTB_PRUNE_ABS 1e-9
#define RTB_STACK 64
#define RTB_TIES 8

struct DCube {
  double c[3], half[3];
  double w2l[12];  // rows 0..2 of the world-to-local matrix
  double l2w[12];  // rows 0..2 of the local-to-world matrix
  double ntr[9];   // inverse-transpose of w2l's rotation part
  double bound[4];  // a world sphere around it, of infinite radius where none is known
  int identity;
  int pad;
};

// BVH node: 7 double2 = lmin, lmax, rmin, rmax (12 doubles) + int4
// {lidx, lcnt, ridx, rcnt} (cnt > 0 leaf range, 0 internal node, < 0 empty).
// Triangle records: 5 double2 = v0, e1 = v1 - v0, e2 = v2 - v0,
// meta = int2{triangle index, degenerate}.
// k-d nodes: 4 double2 = (bmin.x, bmin.y) (bmin.z, bmax.x) (bmax.y, bmax.z)
// (split, int2 meta): internal {right child, axis}, leaf {first, -1-count}.
struct DMesh {
  double bmin[3], bmax[3];
  // triangle BVH nodes in double precision: set only for meshes prepared on
  // the device (null for host-prepared ones) and read by no walk; the
  // walks test fbvh
  const double2* bvh;
  const float4* fbvh;      // the BVH in single precision (FNode), which the walks test
  const double2* btris;    // triangle records in BVH leaf order
  const double2* brute;    // triangle records in original order
  const double4* normals;  // normalize(e1 x e2) per triangle
  const double2* nodes;    // reference k-d tree, preorder
  const int* leaf_tris;    // k-d leaf triangle lists, leaf order (KdNode::Leaf.triangles)
  const int2* leaf_path;   // per k-d node: {path bits (bit k: right at depth k), depth}
  const double2* cells;    // per k-d leaf: its cell lo < p <= hi (3 double2: lo.xyz, hi.xyz)
  const int* occ_off;      // per triangle: occurrences [occ_off[t], occ_off[t+1])
  const int2* occ;         // {k-d leaf node, position in the leaf}
  int n_nodes;
  int n_tris;
};

// A run of consecutive spheres [first_obj, first_obj + count) in the World.
struct DSphGroup {
  const float4* fbvh;  // BVH over the run in single precision (FNode); leaves index `order`
  const int* order;    // BVH position -> position in the run
  int first_sphere;    // index of the run's first sphere in DScene::sph
  int first_obj;       // World index of the run's first sphere
  int count;
  int pad;
};

struct DMat {
  double color[3];
  double ambient, diffuse, specular, shininess;
  double refl;
  int has_refl;
  int texture;
  double grid_color[3];  // the grid colour after its #RRGGBB round trip
  double half_width, cell_size;
  double cb_color[3];
  double cb_ambient, cb_diffuse, cb_specular, cb_shininess;
};

struct DLight {
  double pos[3];
  double color[3];
  double intensity;
  double diameter;
  int disk;
  int pad;
};

struct DScene {
  int n_obj;  // entries of `obj` (a sphere group is one entry)
  int n_lights;
  const int4* obj;     // {kind, index in its kind array, material, World index}
  const double* sph;   // 5 per sphere: cx cy cz r r*r
  const int* sph_mat;  // per sphere: material index
  const double* pln;   // 12 per plane: p, n, u axis, v axis
  const DCube* cub;
  const DMesh* mesh;
  const DSphGroup* grp;
  const DMat* mat;
  const DLight* lights;
  double amb_color[3];
  double amb_int;
  double fog_color[3];
  double fog_density, fog_start, fog_end;
  double bg[3];
  int has_fog;
  int shadow_per_hit;
  int has_bvh;  // some entry of `obj` is a mesh or a run of spheres
};

struct DCam {
  double origin[3], hor[3], ver[3], llc[3], vdir[3];
  double campos[3];
  double pitch, half_th, gcolor[3];
  int persp;
  int grid;
};

// Work counters (profiling renders only).
struct Work {
  unsigned long long nodes, tris, spheres, verify;
};

// Per-ray constants shared by all object tests.
struct RayC {
  V3 o, d;
  double dd;  // d.d (sphere `a`)
  V3 inv;     // 1/d per axis
  int par;    // bit a: |d[a]| < 1e-9 (k-d slabs treat the axis as parallel)
};
__device__ __forceinline__ RayC make_rayc(V3 o, V3 d) {
  RayC r;
  r.o = o;
  r.d = d;
  r.dd = dot(d, d);
  r.inv = mk(1.0 / d.x, 1.0 / d.y, 1.0 / d.z);
  r.par = (fabs(d.x) < 1e-9 ? 1 : 0) | (fabs(d.y) < 1e-9 ? 2 : 0) | (fabs(d.z) < 1e-9 ? 4 : 0);
  return r;
}

// Sphere::hit (src/ray.rs:89-120): returns the accepted root
__device__ __forceinline__ bool sphere_t(const double* s, const RayC& r, double tmin, double tmax, double* t) {
  V3 oc = r.o - mk(s[0], s[1], s[2]);
  double a = r.dd;
  double hb = dot(oc, r.d);
  double c = dot(oc, oc) - s[4];
  double disc = hb * hb - a * c;
  if (disc < 0.0) return false;
  double sq = sqrt(disc);
  double root = (-hb - sq) / a;
  if (root < tmin || tmax < root) {
    root = (-hb + sq) / a;
    if (root < tmin || tmax < root) return false;
  }
  *t = root;
  return true;
}

// Plane::hit (src/ray.rs:136-148)
__device__ __forceinline__ bool plane_t(const double* p, const RayC& r, double tmin, double tmax, double* t) {
  V3 n = mk(p[3], p[4], p[5]);
  double denom = dot(n, r.d);
  if (fabs(denom) < 1e-8) return false;
  double tt = dot(mk(p[0], p[1], p[2]) - r.o, n) / denom;
  if (tt < tmin || tt > tmax) return false;
  *t = tt;
  return true;
}

// Cube::hit (src/ray.rs:411-465).  axis receives the index whose slab set
// the entry (the local normal is -e_axis), or 3 when none did.
__device__ __forceinline__ bool cube_t(const DCube& C, const RayC& r, double tmin, double tmax, double* t,
                                       int* axis) {
  V3 lo = gemv34(C.w2l, r.o - ld3(C.c), 0.0);
  V3 ld = gemv34(C.w2l, r.d, 0.0);
  if (norm(ld) < 1e-8) return false;
  V3 dn = normalize(ld);
  double tl = tmin, th = tmax;
  int ax = 3;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    double inv = 1.0 / dn[a];
    double t0 = (-C.half[a] - lo[a]) * inv;
    double t1 = (C.half[a] - lo[a]) * inv;
    if (inv < 0.0) {
      double tmp = t0;
      t0 = t1;
      t1 = tmp;
    }
    if (t0 > tl) {
      tl = t0;
      ax = a;
    }
    if (t1 < th) th = t1;
    if (tl > th) return false;
  }
  double tt = tl > tmin ? tl : th;
  if (tt < tmin || tt > tmax) return false;
  *t = tt;
  *axis = ax;
  return true;
}

// MeshObject::intersect_bounds (src/ray.rs:586-610)
__device__ __forceinline__ bool mesh_bounds(const DMesh& M, const RayC& r, double tmin, double tmax) {
  double tl = tmin, th = tmax;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    double inv = r.inv[a];
    double t0 = (M.bmin[a] - r.o[a]) * inv;
    double t1 = (M.bmax[a] - r.o[a]) * inv;
    if (inv < 0.0) {
      double tmp = t0;
      t0 = t1;
      t1 = tmp;
    }
    tl = rmax(tl, t0);
    th = rmin(th, t1);
    if (tl > th) return false;
  }
  return true;
}

// MeshObject::intersect_triangle (src/ray.rs:527-583) up to the acceptance
// test; the normal is looked up afterwards for the winning triangle.  Most
// triangles a walk tests are missed: they are rejected on the undivided
// numerators x = u a, y = v a and w = t a, with margins (1e-300 and 1e-14 of
// |a|) beyond which the reference's rounded quotients f x, f y
// and f w, f = 1 / a, are certain to fail the same comparison.
// The others, NaN included, divide as the reference does.
__device__ __forceinline__ bool tri_t(const double2* E, const RayC& r, double tmin, double tmax, double* t) {
  double2 q0 = __ldg(E + 0), q1 = __ldg(E + 1), q2 = __ldg(E + 2), q3 = __ldg(E + 3), q4 = __ldg(E + 4);
  V3 v0 = mk(q0.x, q0.y, q1.x);
  V3 e1 = mk(q1.y, q2.x, q2.y);
  V3 e2 = mk(q3.x, q3.y, q4.x);
  V3 h = cross(r.d, e2);
  double a = dot(e1, h);
  if (a > -1e-8 && a < 1e-8) return false;
  V3 s = r.o - v0;
  const double x = dot(s, h);
  const bool neg = a < 0.0;
  const double top = fabs(a) * (1.0 + 1e-14);
  const double sx = neg ? -x : x;
  const double low = -1e-300 * top;
  if (sx < low || sx > top) return false;
  V3 q = cross(s, e1);
  const double y = dot(r.d, q);
  const double sy = neg ? -y : y;
  if (sy < low || sx + sy > top) return false;
  const double w = dot(e2, q);
  const double sw = neg ? -w : w;
  if ((sw < 0.0 && tmin >= 0.0) || (sw > top * tmax && tmax >= 0.0)) return false;
  double f = 1.0 / a;
  double u = f * x;
  if (!(u >= 0.0 && u <= 1.0)) return false;
  double v = f * y;
  if (v < 0.0 || u + v > 1.0) return false;
  double tt = f * w;
  if (tt > tmin && tt < tmax) {
    if (hi32(q4.y)) return false;  // ||e1 x e2|| < 1e-8
    *t = tt;
    return true;
  }
  return false;
}

// KdTree::ray_intersects_bounds (src/mesh.rs:218-255); *te = slab entry
__device__ __forceinline__ bool kd_slab(const double2* N, const RayC& r, double* te) {
  double2 n0 = __ldg(N + 0), n1 = __ldg(N + 1), n2 = __ldg(N + 2);
  double bmin[3] = {n0.x, n0.y, n1.x}, bmax[3] = {n1.y, n2.x, n2.y};
  double tl = -RTB_INF, th = RTB_INF;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    double o = r.o[a];
    if (r.par & (1 << a)) {
      if (o < bmin[a] || o > bmax[a]) return false;
    } else {
      double inv = r.inv[a];
      double t0 = (bmin[a] - o) * inv;
      double t1 = (bmax[a] - o) * inv;
      if (t0 > t1) {
        double tmp = t0;
        t0 = t1;
        t1 = tmp;
      }
      tl = rmax(tl, t0);
      th = rmin(th, t1);
      if (tl > th) return false;
    }
  }
  *te = tl;
  return th >= 0.0;
}

// `(split - origin) / dir >= 0.0` without the division (src/mesh.rs:441,
// :448).  Here |dir| >= 1e-9 and |dir| <= 1 (a unit direction), so a
// non-zero numerator gives a quotient of magnitude at least the smallest
// subnormal: the quotient is non-negative exactly when the numerator is
// zero or both signs agree (and neither operand is NaN).
__device__ __forceinline__ bool split_ahead(double split, double origin, double dir) {
  double diff = split - origin;
  return (diff == 0.0 && dir == dir) || (diff > 0.0 && dir > 0.0) || (diff < 0.0 && dir < 0.0);
}

// Whether the reference's traversal tests k-d leaf `leaf` for this ray
// (src/mesh.rs:399-465, leaf test :411); *key orders visited leaves in the
// reference's depth-first visiting order (bit 31-k: far child at depth k).
__device__ __forceinline__ bool kd_leaf_visited(const DMesh& M, const RayC& r, int leaf, unsigned* key) {
  int2 lp = __ldg(M.leaf_path + leaf);
  unsigned path = (unsigned)lp.x;
  int depth = lp.y;
  int node = 0;
  unsigned k_out = 0;
  for (int k = 0; k < depth; k++) {
    double2 n3 = __ldg(M.nodes + 4 * (size_t)node + 3);
    int right = lo32(n3.y), axis = hi32(n3.y);
    double split = n3.x;
    bool go_right = (path >> k) & 1u;
    double op = r.o[axis];
    bool left_side = op <= split;
    if (r.par & (1 << axis)) {
      if (go_right == left_side) return false;  // only the origin's side
    } else if (go_right == left_side) {         // far child: needs t_split >= 0
      if (!split_ahead(split, op, r.d[axis])) return false;
      k_out |= 1u << (31 - k);
    }
    node = go_right ? right : node + 1;
  }
  double te;
  if (!kd_slab(M.nodes + 4 * (size_t)node, r, &te)) return false;
  *key = k_out;
  return true;
}

// kd_leaf_visited's answer without its root-to-leaf walk, from the leaf's
// cell: per axis, lo = the largest split the path turns right at and hi =
// the smallest it turns left at (k_prep_cells).  The walk fails at a
// right turn at split s only when o <= s and split_ahead(s, o, d) fails,
// and that happens at some right turn of an axis exactly when
// !(o > lo || d > 0 || (o == lo && d == d)); at a left turn only when
// o > s and d is not negative, i.e. when !(o <= hi || d < 0).  On an axis
// the reference treats as parallel, the origin must be on the leaf's side
// of every split: lo < o <= hi.  Then the leaf's slab test.  A cell that
// could not be built (NaN split on the path, marked by a NaN lo) or a
// non-finite origin takes the walk.
__device__ __forceinline__ bool kd_leaf_visited_cell(const DMesh& M, const RayC& r, int leaf, Work* w) {
  const double2* C = M.cells + 3 * (size_t)leaf;
  const double2 c0 = __ldg(C), c1 = __ldg(C + 1), c2 = __ldg(C + 2);
  const double lo[3] = {c0.x, c0.y, c1.x}, hi[3] = {c1.y, c2.x, c2.y};
  if (w) w->verify += 4;
  const bool finite_o = fabs(r.o.x) < RTB_INF && fabs(r.o.y) < RTB_INF && fabs(r.o.z) < RTB_INF;
  if (lo[0] != lo[0] || !finite_o) {
    if (w) w->verify += (unsigned)__ldg(M.leaf_path + leaf).y;
    unsigned key;
    return kd_leaf_visited(M, r, leaf, &key);
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double o = r.o[a], d = r.d[a];
    if (r.par & (1 << a)) {
      if (!(o > lo[a] && o <= hi[a])) return false;
    } else {
      if (!(o > lo[a] || d > 0.0 || (o == lo[a] && d == d))) return false;
      if (!(o <= hi[a] || d < 0.0)) return false;
    }
  }
  if (w) w->verify += 3;
  double te;
  return kd_slab(M.nodes + 4 * (size_t)leaf, r, &te);
}

// Whether the reference tests triangle `tri` for this ray: whether it
// visits some k-d leaf holding it.
__device__ __forceinline__ bool tri_visited(const DMesh& M, const RayC& r, int tri, Work* w) {
  const int b = __ldg(M.occ_off + tri), e = __ldg(M.occ_off + tri + 1);
  for (int k = b; k < e; k++)
    if (kd_leaf_visited_cell(M, r, __ldg(M.occ + k).x, w)) return true;
  return false;
}

// The reference's first test of triangle `tri` for this ray: the smallest
// (leaf key, position) over the visited leaves holding it.
__device__ __forceinline__ bool tri_first_visit(const DMesh& M, const RayC& r, int tri, unsigned long long* order,
                                                Work* w) {
  int b = __ldg(M.occ_off + tri), e = __ldg(M.occ_off + tri + 1);
  bool any = false;
  unsigned long long best = ~0ULL;
  for (int k = b; k < e; k++) {
    int2 oc = __ldg(M.occ + k);
    // work unit: one 16-byte read (occurrence, each ancestor's split record,
    // and three for the leaf box)
    if (w) w->verify += 4 + (unsigned)__ldg(M.leaf_path + oc.x).y;
    unsigned key;
    if (kd_leaf_visited(M, r, oc.x, &key)) {
      unsigned long long o = ((unsigned long long)key << 32) | (unsigned)oc.y;
      if (o < best) best = o;
      any = true;
    }
  }
  *order = best;
  return any;
}

// The exact reference k-d walk (MeshObject::hit with KdTree::traverse,
// src/ray.rs:614-649, src/mesh.rs:399-465) with exact subtree culling by
// node bounds and closest-t pruning.  Returns the winning triangle index.
__device__ bool mesh_kd_walk(const DMesh& M, const RayC& r, double tmin, double& closest, int& best_tri, int* err,
                             Work* w) {
  if (M.n_nodes == 0) return false;
  bool found = false;
  int stack[RTB_STACK];
  int sp = 0;
  int node = 0;
  for (;;) {
    const double2* N = M.nodes + 4 * (size_t)node;
    double te;
    if (w) w->nodes++;
    bool visit = kd_slab(N, r, &te) && !(te > closest * RTB_PRUNE_REL + RTB_PRUNE_ABS);
    if (visit) {
      double2 n3 = __ldg(N + 3);
      int ma = lo32(n3.y), mb = hi32(n3.y);
      if (mb < 0) {
        int first = ma, cnt = -1 - mb;
        for (int k = 0; k < cnt; k++) {
          double t;
          int tri = __ldg(M.leaf_tris + first + k);
          const double2* E = M.brute + 5 * (size_t)tri;
          if (w) w->tris++;
          if (tri_t(E, r, tmin, closest, &t) && t < closest) {
            closest = t;
            best_tri = tri;
            found = true;
          }
        }
      } else {
        int axis = mb;
        double split = n3.x;
        double op = r.o[axis];
        int near_c = op <= split ? node + 1 : ma;
        int far_c = op <= split ? ma : node + 1;
        if (r.par & (1 << axis)) {
          node = near_c;
          continue;
        }
        if (split_ahead(split, op, r.d[axis])) {
          if (sp >= RTB_STACK) {
            atomicOr(err, ERR_STACK);
            return found;
          }
          stack[sp++] = far_c;
        }
        node = near_c;
        continue;
      }
    }
    if (sp == 0) break;
    node = stack[--sp];
  }
  return found;
}

// A BVH node in single precision: the double node's child boxes rounded
// outwards to floats, the same child references.  Layout: fbvh[0].x is
// the largest |coordinate| of any child box (the scale the slab constants
// below need; elements 1-3 unused); node k is fbvh[H + 4k .. H + 3 + 4k]
// (H = RTB_FBVH_HEAD) = {lmn.xyz, lmx.x},
// {lmx.yz, rmn.xy}, {rmn.z, rmx.xyz}, {lidx, lcnt, ridx, rcnt as int bits}.
struct FNode {
  float lmn[3], lmx[3], rmn[3], rmx[3];
  int lidx, lcnt, ridx, rcnt;
};
__device__ __forceinline__ FNode load_fnode(const float4* fbvh, int node) {
  // two 32-byte loads (nodes lie on 64 bytes): a warp's lanes read 32 different
  // nodes, and each load instruction costs the L1 a tag look-up per lane
  const float4* N = fbvh + RTB_FBVH_HEAD + 4 * (size_t)node;
  float4 a, b, c, d;
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(N));
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w), "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
      : "l"(N + 2));
  FNode n;
  n.lmn[0] = a.x; n.lmn[1] = a.y; n.lmn[2] = a.z;
  n.lmx[0] = a.w; n.lmx[1] = b.x; n.lmx[2] = b.y;
  n.rmn[0] = b.z; n.rmn[1] = b.w; n.rmn[2] = c.x;
  n.rmx[0] = c.y; n.rmx[1] = c.z; n.rmx[2] = c.w;
  n.lidx = __float_as_int(d.x);
  n.lcnt = __float_as_int(d.y);
  n.ridx = __float_as_int(d.z);
  n.rcnt = __float_as_int(d.w);
  return n;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float m;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

// A ray's single-precision slab constants.  Entry distances are taken from
// hi = o + delta rounded up, exit distances from lo = o - delta rounded
// down: the distances of the box grown by delta on every side.  A slab plane
// is one fused multiply-add, plane * inv + c with c = -hi inv or -lo inv
// rounded.  The direction rounded to float, its rounded reciprocal, c's
// rounding and the fused one's move a computed plane by at most 2^-24 *
// (3 |box coordinate - hi| + |hi|) <= 2.4e-7 * (|box coordinate| + |hi|), so
// delta = 3e-7 * (scale + max |o|) keeps every computed interval around the
// exact interval of the float box (which holds the double box): a box the
// exact ray meets is never rejected.  An axis with d = 0 takes a reciprocal
// of 1e37 / (scale + max |o| + 1): the products stay finite, an origin within
// the slab's delta gives planes beyond any distance on both sides, one
// outside gives an empty interval.  all: the constants cannot bound the
// rounding (NaN, an origin or scale beyond 1e30, a component of d nonzero
// but below 1e-30 or with a reciprocal above that limit), so every box is
// accepted.
struct RayF {
  float lo[3], hi[3], inv[3];  // lo, hi: the constants c of the exit and entry planes
  bool all;
};
__device__ __forceinline__ RayF make_rayf(V3 ro, V3 rd, float scale) {
  RayF f;
  bool bad = !(scale < 1e30f);
  double om = 0.0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double o = ro[a], d = rd[a];
    bad = bad || !(fabs(o) < 1e30) || d != d || (d != 0.0 && fabs(d) < 1e-30);
    om = fmax(om, fabs(o));
  }
  const double delta = 3e-7 * ((double)scale + om) + 1e-30;
  const float cap = 1e37f / (scale + (float)om + 1.f);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float i = rd[a] == 0.0 ? cap : __frcp_rn(__double2float_rn(rd[a]));
    bad = bad || !(fabsf(i) <= cap);
    f.inv[a] = i;
    f.lo[a] = -(__double2float_rd(ro[a] - delta) * i);
    f.hi[a] = -(__double2float_ru(ro[a] + delta) * i);
  }
  f.all = bad;
  return f;
}

// Ray/box entry for BVH culling (padded boxes; not a reference test), in
// single precision: never rejects a box that the exact ray meets within
// tmax (see RayF); tmax is the rounded-up pruning bound
// t * RTB_PRUNE_REL + RTB_PRUNE_ABS.
__device__ __forceinline__ bool box_hit_f(const float* mn, const float* mx, const RayF& f, float tmax, float* te) {
  float n[3], x[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float t0 = __fmaf_rn(mn[a], f.inv[a], f.hi[a]);
    const float t1 = __fmaf_rn(mx[a], f.inv[a], f.lo[a]);
    n[a] = fminf(t0, t1);
    x[a] = fmaxf(t0, t1);
  }
  const float tl = max3(n[0], n[1], n[2]), th = min3(x[0], x[1], x[2]);
  *te = tl;
  return f.all || (tl <= th && th >= 0.0f && !(tl > tmax));
}

// BVH walks by one thread each, over references to children (walk_ref).  A
// walk descends until it meets a leaf or runs out of nodes and only then
// tests the leaf, so that the lanes of a warp run the (double) leaf tests
// together rather than one lane's leaf at a time between the others'
// (single-precision) node steps.  (Warp packets, one shared walk for the 16
// rays of a light, cost 2.5 ms where this costs 1.4 on the rays the icosphere
// frame's cones leave: those cones are wide, and their rays meet different
// leaves.)

// The pruning bound t * RTB_PRUNE_REL + RTB_PRUNE_ABS, rounded up.
__device__ __forceinline__ float prune_bound(double t) {
  return __double2float_ru(t * RTB_PRUNE_REL + RTB_PRUNE_ABS);
}

// Closest-hit walk of a BVH by one thread, nearer children first.  test(j)
// tests the primitive at position j and returns the pruning distance after
// it; tmax is the distance before the walk.  The stack keeps each entry's
// box distance: what lies beyond a hit found since is not loaded.
template <class Test>
__device__ __forceinline__ void closest_bvh(const float4* fbvh, V3 o, V3 d, double tmax, Test test, int* err,
                                            Work* w) {
  const RayF f = make_rayf(o, d, __ldg(fbvh).x);
  float bound = prune_bound(tmax);
  int2 stack[RTB_STACK];
  int sp = 0, cur = 0;
  for (;;) {
    while (cur >= 0 && cur != RTB_WALK_DONE) {
      const FNode nd = load_fnode(fbvh, cur);
      if (w) w->nodes++;
      float tl, tr;
      const bool hl = box_hit_f(nd.lmn, nd.lmx, f, bound, &tl) && nd.lcnt >= 0;
      const bool hr = box_hit_f(nd.rmn, nd.rmx, f, bound, &tr) && nd.rcnt >= 0;
      const int l = walk_ref(nd.lidx, nd.lcnt), r = walk_ref(nd.ridx, nd.rcnt);
      if (hl && hr) {
        if (sp >= RTB_STACK) {
          atomicOr(err, ERR_STACK);
          return;
        }
        const bool swap = tr < tl;
        stack[sp++] = swap ? make_int2(l, __float_as_int(tl)) : make_int2(r, __float_as_int(tr));
        cur = swap ? r : l;
      } else if (hl || hr) {
        cur = hl ? l : r;
      } else {
        cur = RTB_WALK_DONE;
        while (sp && cur == RTB_WALK_DONE) {
          const int2 e = stack[--sp];
          if (f.all || !(__int_as_float(e.y) > bound)) cur = e.x;
        }
      }
    }
    if (cur == RTB_WALK_DONE) return;
    const int first = leaf_first(cur), cnt = leaf_count(cur);
    double t = 0.0;
    for (int j = first; j < first + cnt; j++) t = test(j);
    bound = prune_bound(t);
    cur = RTB_WALK_DONE;
    while (sp && cur == RTB_WALK_DONE) {
      const int2 e = stack[--sp];
      if (f.all || !(__int_as_float(e.y) > bound)) cur = e.x;
    }
  }
}

// Closest hit on a mesh (MeshObject::hit, src/ray.rs:614-675).  On entry
// `closest` is the World's closest-so-far; on a hit it becomes the hit's t
// and best_tri the winning triangle (original index).
__device__ bool mesh_closest(const DMesh& M, V3 o, V3 d, double tmin, double& closest, int& best_tri,
                             bool use_kd, int* err, Work* w) {
  const double cin = closest;
  double bt = closest;
  bool have = false;
  int ties[RTB_TIES];
  int nt = 0;
  bool overflow = false;
  RayC r;
  r.o = o;
  r.d = d;
  closest_bvh(
      M.fbvh, o, d, closest,
      [&](int j) {
        const double2* E = M.btris + 5 * (size_t)j;
        double t;
        if (w) w->tris++;
        if (tri_t(E, r, tmin, cin, &t)) {
          int tri = lo32(__ldg(E + 4).y);
          if (!have || t < bt) {
            bt = t;
            have = true;
            nt = 0;
            ties[nt++] = tri;
            overflow = false;
          } else if (t == bt) {
            if (nt < RTB_TIES) ties[nt++] = tri;
            else overflow = true;
          }
        }
        return bt;
      },
      err, w);
  // No triangle meets t in (tmin, closest): the reference finds none either.
  if (!have) return false;
  r = make_rayc(o, d);
  if (!mesh_bounds(M, r, tmin, cin)) return false;
  if (!use_kd) {
    // brute force tests in original order: lowest index among the minimal t
    int bi = ties[0];
    for (int k = 1; k < nt; k++) bi = min(bi, ties[k]);
    if (overflow) {
      for (int i = 0; i < M.n_tris; i++) {
        double t;
        if (tri_t(M.brute + 5 * (size_t)i, r, tmin, cin, &t) && t == bt) {
          bi = i;
          break;
        }
      }
    }
    closest = bt;
    best_tri = bi;
    return true;
  }
  if (nt == 1 && tri_visited(M, r, ties[0], w)) {
    closest = bt;
    best_tri = ties[0];
    return true;
  }
  if (!overflow) {
    unsigned long long bo = ~0ULL;
    int bi = -1;
    for (int k = 0; k < nt; k++) {
      unsigned long long o;
      if (tri_first_visit(M, r, ties[k], &o, w) && o < bo) {
        bo = o;
        bi = ties[k];
      }
    }
    if (bi >= 0) {
      closest = bt;
      best_tri = bi;
      return true;
    }
  }
  // The reference does not test the nearest triangle (or too many tie):
  // answer with the reference's own walk.
  return mesh_kd_walk(M, r, tmin, closest, best_tri, err, w);
}

// A run of spheres: minimal accepted root, ties to the latest sphere.  On
// entry `closest` is the World's closest-so-far (an inclusive bound, as
// Sphere::hit accepts root == t_max).
__device__ bool group_hit(const DScene& S, const DSphGroup& G, const RayC& r, double tmin, double& closest,
                          int& best, int* err, Work* w) {
  bool have = false;
  double bt = closest;
  int bi = -1;
  closest_bvh(
      G.fbvh, r.o, r.d, closest,
      [&](int j) {
        const int sidx = __ldg(G.order + j);  // position in the run
        double t;
        if (w) w->spheres++;
        if (sphere_t(S.sph + 5 * (size_t)(G.first_sphere + sidx), r, tmin, bt, &t)) {
          if (!have || t < bt || sidx > bi) {
            bt = t;
            bi = sidx;
            have = true;
          }
        }
        return bt;
      },
      err, w);
  if (!have) return false;
  closest = bt;
  best = bi;
  return true;
}

struct WHit {
  int obj;  // World index of the winner, -1 = miss
  int aux;  // mesh triangle / cube axis
  double t;
  int ent;  // entry of DScene::obj that produced the hit
};

// World::hit (src/ray.rs:699-711): scene order, closest narrowing
__device__ __forceinline__ WHit world_closest(const DScene& S, const RayC& r, double tmin, bool use_kd, int* err,
                                             Work* w) {
  double closest = RTB_INF;
  WHit h{-1, 0, 0.0, -1};
  for (int i = 0; i < S.n_obj; i++) {
    int4 ob = __ldg(S.obj + i);
    double t;
    switch (ob.x) {
      case OBJ_SPHERE:
        if (w) w->spheres++;
        if (sphere_t(S.sph + 5 * (size_t)ob.y, r, tmin, closest, &t)) {
          closest = t;
          h = WHit{ob.w, 0, t, i};
        }
        break;
      case OBJ_PLANE:
        if (plane_t(S.pln + 12 * (size_t)ob.y, r, tmin, closest, &t)) {
          closest = t;
          h = WHit{ob.w, 0, t, i};
        }
        break;
      case OBJ_CUBE: {
        int ax;
        if (cube_t(S.cub[ob.y], r, tmin, closest, &t, &ax)) {
          closest = t;
          h = WHit{ob.w, ax, t, i};
        }
        break;
      }
      case OBJ_MESH: {
        int tri = -1;
        if (mesh_closest(S.mesh[ob.y], r.o, r.d, tmin, closest, tri, use_kd, err, w)) h = WHit{ob.w, tri, closest, i};
        break;
      }
      default: {
        int k = -1;
        if (group_hit(S, S.grp[ob.y], r, tmin, closest, k, err, w)) h = WHit{ob.w + k, 0, closest, i};
        break;
      }
    }
  }
  return h;
}

// ---------------------------------------------------------------------------
// Light cones.  The shadow rays of one shading point towards one disk light
// share their origin o = p + 0.001 n and end on a disk of radius R that is
// perpendicular to the axis c at axis distance D from o (their directions are
// sp - p with sp on the disk, so the rays from o end D along the axis too):
// they fill a cone with tangent R / D.  shaft_collect finds the primitives
// that any ray of the cone can meet.  None: every ray is unblocked.  A
// sphere that every ray must enter: every ray is blocked.  A few: the rays
// test those and nothing else (ray_blocked_by), with the tests the World's
// own queries run, so each ray's answer is shadow_walk's.  The tests here only
// ever keep too much: margins are far above the rounding of the exact tests
// (1e-6 relative for boxes and spheres, 1e-9 for planes and triangle planes,
// whose exact tests are double arithmetic at 1e-16).
// ---------------------------------------------------------------------------
// Candidates kept per cone.  A cone that finds one more stops there, which
// saves its walk's rest, and its rays walk the BVH; one that finds fewer
// spares them the walk.  Frames in ms with 1 / 2 / 3 / 4 / 8 / 16 candidates:
// 1080p mesh 4.44 / 4.47 / 4.48 / 4.51 / 4.61 / 4.78, 1,000 spheres at 4 spp
// 19.8 / 17.7 / 17.1 / 17.1 / 17.3 / 17.7, learned 23.6 / 19.7 / 18.7 / 18.9 /
// 19.5 / 20.3, 4K terrain 12.1 / 12.0 / 11.9 / 12.1 / 12.2 / 12.6.
#define RTB_CAND 3
// Nodes of a BVH over n primitives that a cone visits at most; beyond them its
// rays walk.  Wide cones along a surface meet the boxes of what lies below it
// for thousands of nodes, one thread's chain of loads: 161x93 icosphere under a
// light of diameter 10, 8.2 ms without a limit, 0.79 with 64, 1.1 with 128 (16
// rays' walks each: 0.98).  Cones that settle their light need fewer: 1080p
// icosphere 4.69 without, 4.39 with 64, 4.48 with 128, 4.50 with 32; terrain of
// 2 M triangles, four times its levels of nodes: 12.7 without, 12.05 with 64,
// 12.4 with 128, but 18.0 with 32.
__device__ __forceinline__ int cone_nodes(int n) { return max(64, 4 * (32 - __clz(n / RTB_LEAF))); }
enum { CONE_BLOCKED = -2, CONE_MANY = -1 };  // shaft_collect's results below zero

struct Cone {
  V3 o, c;
  double D, R;    // axis length, disk radius
  float T;        // tangent of the half angle, rounded up
  float ca, sa;   // its cosine and sine (to 1e-6)
  float h[3];     // normal of a plane through o with the cone on its positive side
};
// False when the margins cannot cover the cone (a light within its own
// radius of the point, huge or non-finite coordinates): the rays are traced.
// n: the surface's unit normal at the point.  Most of what lies near a
// shading point is the surface itself, below the cone: h is n where the
// whole light is above the point's horizon, else n turned towards the axis
// until it is (zero, which cuts nothing off, when n points away from it).
// The leaf tests use it; on the boxes it cost more than the nodes it saved.
__device__ __forceinline__ bool make_cone(V3 o, V3 n, V3 c, double D, double R, Cone* k) {
  k->o = o;
  k->c = c;
  k->D = D;
  k->R = R;
  const float t = (float)R / (float)D;
  k->T = t * (1.0f + 2e-6f) + 1e-7f;
  k->ca = rsqrtf(1.0f + t * t);
  k->sa = t * k->ca;
  const float nc = (float)dot(n, c), low = k->sa + 1e-5f;
  const float px = (float)n.x - nc * (float)c.x, py = (float)n.y - nc * (float)c.y, pz = (float)n.z - nc * (float)c.z;
  const float p2 = px * px + py * py + pz * pz;
  // h = u n' + v c, n' the part of n across the axis
  float u = nc >= low ? 1.f : rsqrtf(p2) * sqrtf(fmaxf(0.f, 1.f - low * low)), v = nc >= low ? nc : low;
  if (!(p2 > 1e-6f) && nc < low) u = v = 0.f;
  k->h[0] = u * px + v * (float)c.x;
  k->h[1] = u * py + v * (float)c.y;
  k->h[2] = u * pz + v * (float)c.z;
  return D > 1e-6 && D < 1e18 && R > 1e-30 && k->T <= 1.0f && fabs(o.x) < 1e18 && fabs(o.y) < 1e18 &&
         fabs(o.z) < 1e18 && fabs(c.x) <= 2.0 && fabs(c.y) <= 2.0 && fabs(c.z) <= 2.0;
}

// The cone's single-precision slab constants for one BVH.  At axis distance
// a the cone's cross-section spans o + a [dl, du] on each axis (dl, du = c
// -+ T sqrt(1 - c^2), widened by 2e-6 against their own rounding); a box
// meets the cone only where o + a dl <= max and o + a du >= min hold on
// every axis, six half-lines of a.  Rounding: as in RayF, each is one fused
// multiply-add, and the origin is moved by delta against its comparison.
struct ConeF {
  float lo[3], hi[3], il[3], iu[3];  // lo, hi: -(o - delta) il and -(o + delta) iu
  float len;
  bool all;
};
__device__ __forceinline__ void cone_slopes(const Cone& k, ConeF* f) {
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float c = (float)k.c[a];
    const float e = k.T * sqrtf(fmaxf(0.f, 1.f - c * c) + 1e-6f) + 2e-6f;
    float dl = c - e, du = c + e;
    if (fabsf(dl) < 1e-7f) dl = -1e-7f;
    if (fabsf(du) < 1e-7f) du = 1e-7f;
    f->il[a] = 1.f / dl;
    f->iu[a] = 1.f / du;
  }
  f->len = __double2float_ru(k.D * (1.0 + 1e-6));
}
__device__ __forceinline__ void cone_origin(const Cone& k, float scale, ConeF* f) {
  const double om = fmax(fabs(k.o.x), fmax(fabs(k.o.y), fabs(k.o.z)));
  const double delta = 3e-7 * ((double)scale + om) + 1e-30;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    f->lo[a] = -(__double2float_rd(k.o[a] - delta) * f->il[a]);
    f->hi[a] = -(__double2float_ru(k.o[a] + delta) * f->iu[a]);
  }
  f->all = !(scale < 1e30f);
}
__device__ __forceinline__ bool cone_box(const ConeF& f, const float* mn, const float* mx) {
  float tl = 0.f, th = f.len;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float t = __fmaf_rn(mx[a], f.il[a], f.lo[a]);
    const float s = __fmaf_rn(mn[a], f.iu[a], f.hi[a]);
    if (f.il[a] > 0.f) th = fminf(th, t);
    else tl = fmaxf(tl, t);
    if (f.iu[a] > 0.f) tl = fmaxf(tl, s);
    else th = fminf(th, s);
  }
  return tl <= th || f.all;
}

// Whether the cone can meet the sphere; *blocks: every ray of the cone is
// accepted by Sphere::hit (the directions lie inside the sphere's own cone,
// or o inside the sphere; one root beyond 0.001 and the whole sphere nearer
// than the disk).  endless: the cone goes on beyond the disk.
__device__ __forceinline__ bool cone_sphere(const Cone& k, const double* s, bool* blocks, bool endless = false) {
  const V3 v = mk(s[0], s[1], s[2]) - k.o;
  const double r = fabs(s[3]);
  const double a = dot(v, k.c), vv = dot(v, v);
  const double end = endless ? fmax(k.D, sum_abs(v) + r) : k.D;  // beyond all of the sphere
  const double m = 1e-6 * (2.0 * end + r);
  *blocks = false;
  if (!(vv < 1e200)) return true;  // the exact test's discriminant may overflow
  if (a < -(r + m) || a > end + r + m) return false;
  // apex margin: the point itself may lie on the sphere
  const double ma = 1e-8 * (end + r + sum_abs(k.o)), out2 = (r + ma) * (r + ma);
  if (v.x * k.h[0] + v.y * k.h[1] + v.z * k.h[2] < -(r + ma) * (1.0 + 1e-5)) return false;
  const double p2 = fmax(vv - a * a, 0.0);
  // behind the apex, whose distance then is the cone's: a ca + p sa < 0
  if (vv > out2 && a < 0.0 && a * a * k.ca * k.ca > p2 * k.sa * k.sa * (1.0 + 1e-5)) return false;
  const double reach = k.T * a + (r + m) / k.ca;
  if (reach < 0.0 || p2 > reach * reach) return false;
  if (a + r < k.D * (1.0 - 1e-6) - m) {
    const double in = r - 0.001 - m, out = r + 0.001 + m;
    if (in > 0.0 && vv < in * in) {
      *blocks = true;
    } else if (vv > out * out && a > 0.0) {
      const double p = sqrt(p2);
      *blocks = p * k.ca + a * k.sa < r * (1.0 - 1e-6) - m && a * k.ca - p * k.sa > 0.0;
    }
  }
  return true;
}

// Whether the cone can cross the plane through q with normal n (any
// length; `size`: the magnitude of the terms its distances are sums of).
__device__ __forceinline__ bool cone_plane(const Cone& k, V3 q, V3 n, double size) {
  const double nc = dot(n, k.c);
  const double h0 = dot(n, k.o - q), h1 = h0 + k.D * nc;
  // the disk's points are within e = R |n x c| of its centre's distance
  const double nn = dot(n, n);
  const double e2 = k.R * k.R * (fmax(nn - nc * nc, 0.0) * (1.0 + 1e-5) + 1e-14 * nn);
  const double m = 1e-9 * size, end = fabs(h1) - m;
  return !(fabs(h0) > m && end > 0.0 && end * end > e2 && (h0 > 0.0) == (h1 > 0.0));
}

// Whether the cone can meet a triangle record: its plane, then its box.
__device__ __forceinline__ bool cone_tri(const Cone& k, const ConeF& f, const double2* E) {
  const double2 q0 = __ldg(E + 0), q1 = __ldg(E + 1), q2 = __ldg(E + 2), q3 = __ldg(E + 3), q4 = __ldg(E + 4);
  if (hi32(q4.y)) return false;  // ||e1 x e2|| < 1e-8: never accepted
  const V3 v0 = mk(q0.x, q0.y, q1.x), e1 = mk(q1.y, q2.x, q2.y), e2 = mk(q3.x, q3.y, q4.x);
  const double coords = sum_abs(k.o) + sum_abs(v0) + k.D;
  const V3 h = mk(k.h[0], k.h[1], k.h[2]);
  const double h0 = dot(h, v0 - k.o), top = h0 + fmax(0.0, fmax(dot(h, e1), dot(h, e2)));
  if (top < -1e-7 * coords) return false;
  const double size = sum_abs(e1) * sum_abs(e2) * coords;
  if (!cone_plane(k, v0, cross(e1, e2), size)) return false;
  const V3 v1 = v0 + e1, v2 = v0 + e2;
  float mn[3], mx[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    mn[a] = __double2float_rd(fmin(v0[a], fmin(v1[a], v2[a])));
    mx[a] = __double2float_ru(fmax(v0[a], fmax(v1[a], v2[a])));
  }
  return cone_box(f, mn, mx);
}

// The primitives the cone can meet, as {entry of DScene::obj, index}: index =
// the triangle's position in the BVH order, the sphere's position in its
// run, 0 otherwise.  Writes candidate j to out[j * stride]; returns their
// number, CONE_MANY when there are more than RTB_CAND, or CONE_BLOCKED.
// One thread per cone: neighbouring hits' cones take similar walks, and one
// walk answers for all of a light's rays.
__device__ __forceinline__ int shaft_collect(const DScene& S, const Cone& k, int2* out, int stride, int* err,
                                             Work* w) {
  int n = 0;
  ConeF f;
  cone_slopes(k, &f);
  for (int i = 0; i < S.n_obj; i++) {
    const int4 ob = __ldg(S.obj + i);
    if (ob.x == OBJ_SPHERE || ob.x == OBJ_PLANE || ob.x == OBJ_CUBE) {
      if (ob.x != OBJ_PLANE) {
        // a cube by the sphere around it; its own test measures t in its local
        // frame, so that a scaled cube may block from beyond the light
        const bool sphere = ob.x == OBJ_SPHERE;
        bool blocks;
        if (w && sphere) w->spheres++;
        if (!cone_sphere(k, sphere ? S.sph + 5 * (size_t)ob.y : S.cub[ob.y].bound, &blocks,
                         !sphere && !S.cub[ob.y].identity))
          continue;
        if (blocks && sphere) return CONE_BLOCKED;
      } else {
        const double* p = S.pln + 12 * (size_t)ob.y;
        const V3 q = mk(p[0], p[1], p[2]), pn = mk(p[3], p[4], p[5]);
        if (!cone_plane(k, q, pn, sum_abs(pn) * (sum_abs(k.o) + sum_abs(q) + k.D))) continue;
      }
      if (n == RTB_CAND) return CONE_MANY;
      out[n * stride] = make_int2(i, 0);
      n++;
      continue;
    }
    const bool mesh = ob.x == OBJ_MESH;
    const float4* fbvh = mesh ? S.mesh[ob.y].fbvh : S.grp[ob.y].fbvh;
    int left = cone_nodes(mesh ? S.mesh[ob.y].n_tris : S.grp[ob.y].count);
    cone_origin(k, __ldg(fbvh).x, &f);
    int stack[RTB_STACK];
    int sp = 0, cur = 0;
    while (cur != RTB_WALK_DONE) {
      while (cur >= 0 && cur != RTB_WALK_DONE) {
        if (left-- == 0) return CONE_MANY;
        const FNode nd = load_fnode(fbvh, cur);
        if (w) w->nodes++;
        const bool hl = nd.lcnt >= 0 && cone_box(f, nd.lmn, nd.lmx);
        const bool hr = nd.rcnt >= 0 && cone_box(f, nd.rmn, nd.rmx);
        const int l = walk_ref(nd.lidx, nd.lcnt), r = walk_ref(nd.ridx, nd.rcnt);
        if (hl && hr) {
          if (sp >= RTB_STACK) {
            atomicOr(err, ERR_STACK);
            return CONE_MANY;
          }
          stack[sp++] = r;
          cur = l;
        } else if (hl || hr) {
          cur = hl ? l : r;
        } else {
          cur = sp ? stack[--sp] : RTB_WALK_DONE;
        }
      }
      if (cur == RTB_WALK_DONE) break;
      const int first = leaf_first(cur), cnt = leaf_count(cur);
      for (int j = first; j < first + cnt; j++) {
        int at = j;
        if (mesh) {
          if (w) w->tris++;
          if (!cone_tri(k, f, S.mesh[ob.y].btris + 5 * (size_t)j)) continue;
        } else {
          if (w) w->spheres++;
          bool blocks;
          at = __ldg(S.grp[ob.y].order + j);
          if (!cone_sphere(k, S.sph + 5 * (size_t)(S.grp[ob.y].first_sphere + at), &blocks)) continue;
          if (blocks) return CONE_BLOCKED;
        }
        if (n == RTB_CAND) return CONE_MANY;
        out[n * stride] = make_int2(i, at);
        n++;
      }
      cur = sp ? stack[--sp] : RTB_WALK_DONE;
    }
  }
  return n;
}

// A triangle in BVH order that the shadow ray meets within (tmin, tmax), as
// World::hit over its mesh decides it: the triangle's test, the mesh's
// bounds and a k-d leaf the reference visits.
__device__ __forceinline__ bool shadow_tri(const DMesh& M, int j, V3 o, V3 d, double tmin, double tmax, bool use_kd,
                                           Work* w) {
  const double2* E = M.btris + 5 * (size_t)j;
  RayC r;
  r.o = o;
  r.d = d;
  double t;
  if (w) w->tris++;
  if (!tri_t(E, r, tmin, tmax, &t)) return false;
  r = make_rayc(o, d);
  return mesh_bounds(M, r, tmin, tmax) && (!use_kd || tri_visited(M, r, lo32(__ldg(E + 4).y), w));
}

// Any hit in a BVH, each lane walking for itself (see walk_ref), nearer
// children first.  test(j): whether the primitive at position j is hit.
template <class Test>
__device__ __forceinline__ bool shadow_bvh(const float4* fbvh, V3 o, V3 d, double tmax, Test test, int* err,
                                           Work* w) {
  const RayF f = make_rayf(o, d, __ldg(fbvh).x);
  const float bound = prune_bound(tmax);
  int stack[RTB_STACK];
  int sp = 0, cur = 0;
  for (;;) {
    while (cur >= 0 && cur != RTB_WALK_DONE) {
      const FNode nd = load_fnode(fbvh, cur);
      if (w) w->nodes++;
      float tl, tr;
      const bool hl = box_hit_f(nd.lmn, nd.lmx, f, bound, &tl) && nd.lcnt >= 0;
      const bool hr = box_hit_f(nd.rmn, nd.rmx, f, bound, &tr) && nd.rcnt >= 0;
      const int l = walk_ref(nd.lidx, nd.lcnt), r = walk_ref(nd.ridx, nd.rcnt);
      if (hl && hr) {
        if (sp >= RTB_STACK) {
          atomicOr(err, ERR_STACK);
          return false;
        }
        const bool swap = tr < tl;
        stack[sp++] = swap ? l : r;
        cur = swap ? r : l;
      } else if (hl || hr) {
        cur = hl ? l : r;
      } else {
        cur = sp ? stack[--sp] : RTB_WALK_DONE;
      }
    }
    if (cur == RTB_WALK_DONE) return false;
    const int first = leaf_first(cur), cnt = leaf_count(cur);
    for (int j = first; j < first + cnt; j++)
      if (test(j)) return true;
    cur = sp ? stack[--sp] : RTB_WALK_DONE;
  }
}
__device__ __forceinline__ bool shadow_mesh(const DMesh& M, V3 o, V3 d, double tmin, double tmax, bool use_kd, int* err,
                                            Work* w) {
  return shadow_bvh(M.fbvh, o, d, tmax, [&](int j) { return shadow_tri(M, j, o, d, tmin, tmax, use_kd, w); }, err, w);
}

// world.hit(ray, t_min, t_max).is_some(): any object, in any order.
__device__ __forceinline__ bool shadow_walk(const DScene& S, V3 o, V3 d, double tmin, double tmax, bool use_kd,
                                            int* err, Work* w) {
  RayC rs;
  rs.o = o;
  rs.d = d;
  rs.dd = dot(d, d);
  for (int i = 0; i < S.n_obj; i++) {
    const int4 ob = __ldg(S.obj + i);
    double t;
    bool hit = false;
    switch (ob.x) {
      case OBJ_SPHERE:
        if (w) w->spheres++;
        hit = sphere_t(S.sph + 5 * (size_t)ob.y, rs, tmin, tmax, &t);
        break;
      case OBJ_PLANE:
        hit = plane_t(S.pln + 12 * (size_t)ob.y, rs, tmin, tmax, &t);
        break;
      case OBJ_CUBE: {
        int ax;
        hit = cube_t(S.cub[ob.y], rs, tmin, tmax, &t, &ax);
        break;
      }
      case OBJ_MESH:
        hit = shadow_mesh(S.mesh[ob.y], o, d, tmin, tmax, use_kd, err, w);
        break;
      default: {
        const DSphGroup& G = S.grp[ob.y];
        hit = shadow_bvh(
            G.fbvh, o, d, tmax,
            [&](int j) {
              if (w) w->spheres++;
              return sphere_t(S.sph + 5 * (size_t)(G.first_sphere + __ldg(G.order + j)), rs, tmin, tmax, &t);
            },
            err, w);
        break;
      }
    }
    if (hit) return true;
  }
  return false;
}

// Whether a shadow ray is blocked by one candidate of shaft_collect: the
// object's own test, as shadow_walk runs it.
__device__ __forceinline__ bool ray_blocked_by(const DScene& S, int2 cand, V3 o, V3 d, double tmin, double tmax,
                                               bool use_kd, Work* w) {
  const int4 ob = __ldg(S.obj + cand.x);
  RayC r;
  r.o = o;
  r.d = d;
  double t;
  switch (ob.x) {
    case OBJ_SPHERE:
    case OBJ_SPHERE_GROUP: {
      const int si = ob.x == OBJ_SPHERE ? ob.y : S.grp[ob.y].first_sphere + cand.y;
      r.dd = dot(d, d);
      if (w) w->spheres++;
      return sphere_t(S.sph + 5 * (size_t)si, r, tmin, tmax, &t);
    }
    case OBJ_PLANE:
      return plane_t(S.pln + 12 * (size_t)ob.y, r, tmin, tmax, &t);
    case OBJ_CUBE: {
      int ax;
      return cube_t(S.cub[ob.y], r, tmin, tmax, &t, &ax);
    }
    default:
      return shadow_tri(S.mesh[ob.y], cand.y, o, d, tmin, tmax, use_kd, w);
  }
}

struct HitRec {
  V3 p, n;
  int mat;
  int has_uv;
  double u, v;
};

// HitRecord::new (src/ray.rs:39-64)
__device__ __forceinline__ V3 face_normal(V3 d, V3 outward) {
  bool front = dot(d, outward) < 0.0;
  return front ? normalize(outward) : normalize(-outward);
}

// Rebuilds the winning object's HitRecord from (entry, aux, t).
__device__ __forceinline__ HitRec finalize_hit(const DScene& S, const RayC& r, const WHit& w) {
  HitRec h;
  int4 ob = __ldg(S.obj + w.ent);
  h.mat = ob.z;
  h.has_uv = 0;
  h.u = h.v = 0.0;
  double t = w.t;
  switch (ob.x) {
    case OBJ_SPHERE:
    case OBJ_SPHERE_GROUP: {
      int si = ob.x == OBJ_SPHERE ? ob.y : S.grp[ob.y].first_sphere + (w.obj - ob.w);
      const double* s = S.sph + 5 * (size_t)si;
      if (ob.x == OBJ_SPHERE_GROUP) h.mat = S.sph_mat[si];
      V3 c = mk(s[0], s[1], s[2]);
      h.p = r.o + t * r.d;
      h.n = face_normal(r.d, (h.p - c) / s[3]);
      break;
    }
    case OBJ_PLANE: {
      const double* p = S.pln + 12 * (size_t)ob.y;
      V3 n = mk(p[3], p[4], p[5]);
      h.p = r.o + t * r.d;
      h.n = face_normal(r.d, n);
      V3 rel = h.p - mk(p[0], p[1], p[2]);
      h.has_uv = 1;
      h.u = dot(rel, mk(p[6], p[7], p[8]));
      h.v = dot(rel, mk(p[9], p[10], p[11]));
      break;
    }
    case OBJ_CUBE: {
      const DCube& C = S.cub[ob.y];
      V3 lo = gemv34(C.w2l, r.o - ld3(C.c), 0.0);
      V3 dn = normalize(gemv34(C.w2l, r.d, 0.0));
      V3 lhp = lo + t * dn;
      h.p = ld3(C.c) + gemv34(C.l2w, lhp, 1.0);
      V3 ln = mk(0.0, 0.0, 0.0);
      if (w.aux == 0) ln.x = -1.0;
      if (w.aux == 1) ln.y = -1.0;
      if (w.aux == 2) ln.z = -1.0;
      V3 wn = C.identity ? ln : gemv33(C.ntr, ln);
      h.n = face_normal(r.d, wn);
      break;
    }
    default: {
      const DMesh& M = S.mesh[ob.y];
      const double2* E = M.brute + 5 * (size_t)w.aux;
      double2 q0 = E[0], q1 = E[1], q2 = E[2], q3 = E[3], q4 = E[4];
      V3 v0 = mk(q0.x, q0.y, q1.x), e1 = mk(q1.y, q2.x, q2.y), e2 = mk(q3.x, q3.y, q4.x);
      V3 hh = cross(r.d, e2);
      double a = dot(e1, hh);
      double f = 1.0 / a;
      V3 s = r.o - v0;
      double u = f * dot(s, hh);
      V3 q = cross(s, e1);
      double v = f * dot(r.d, q);
      double4 nn = M.normals[w.aux];
      V3 n = mk(nn.x, nn.y, nn.z);
      if (a < 0.0) n = -n;
      h.p = r.o + t * r.d;
      h.n = face_normal(r.d, n);
      h.has_uv = 1;
      h.u = u;
      h.v = v;
      break;
    }
  }
  return h;
}

// Camera::get_grid_color (src/camera.rs:171-254)
__device__ __forceinline__ bool grid_color(const DCam& c, V3 o, V3 d, V3* out) {
  if (!c.grid) return false;
  double p = c.pitch, half = c.half_th;
#pragma unroll
  for (int plane = 0; plane < 3; plane++) {
    int ax = plane == 0 ? 2 : (plane == 1 ? 1 : 0);
    int a1 = plane == 2 ? 1 : 0;
    int a2 = plane == 0 ? 1 : 2;
    if (fabs(d[ax]) > 1e-10) {
      double t = -o[ax] / d[ax];
      if (t > 0.0) {
        V3 ip = o + t * d;
        double m1 = fabs(rfract(ip[a1] / p));
        double m2 = fabs(rfract(ip[a2] / p));
        double d1 = rmin(m1 * p, (1.0 - m1) * p);
        double d2 = rmin(m2 * p, (1.0 - m2) * p);
        if (d1 <= half || d2 <= half) {
          *out = ld3(c.gcolor);
          return true;
        }
      }
    }
  }
  return false;
}

}  // namespace rtb
