// unbounded.cuh -- the nearest-triangle search of SDFGPU_MODE_UNBOUNDED and SDFGPU_MODE_LEARNED:
// the kernel arguments, the warp's search of a brick of 32 nodes over the LBVH (FP32, every node's
// triangles within the band of its minimum) and its FP64 resolution in ascending triangle index
// (k_unbounded, distance.cu; k_unbounded_multi, search_multi.cu; the training grid, learned.cu).
//
// Every search returns, for each node, the FP64 minimum over all triangles of the point-triangle
// distance (tri_step64 without the vertex-skip rule), ties to the lowest triangle index -- the
// result of folding every triangle in index order (dfOnTriangularMesh.jl:101-177 with the true
// minimum).  The FP32 search only decides which triangles can hold that minimum: a subtree or a
// triangle is dropped only when its lower bound exceeds every node's bound plus the FP32 margin
// of the test (wide_bound).

#pragma once

#include "common.cuh"

namespace sdfgpu {
namespace {

constexpr double kBig = 1.0e10;  // abs(-1.0e10), the reference's initial running minimum

__device__ __forceinline__ float3 local32(const GridP& g, const d3& p) {
  return make_float3((float)(p.x - g.center[0]), (float)(p.y - g.center[1]), (float)(p.z - g.center[2]));
}

__device__ __forceinline__ void child_box(const BNode& nd, int side, float3& lo, float3& hi) {
  if (side == 0) {
    lo = make_float3(nd.a.x, nd.a.y, nd.a.z);
    hi = make_float3(nd.a.w, nd.b.x, nd.b.y);
  } else {
    lo = make_float3(nd.b.z, nd.b.w, nd.c.x);
    hi = make_float3(nd.c.y, nd.c.z, nd.c.w);
  }
}

constexpr int kUnbWarps = 8;     // warps per CTA of k_unbounded
constexpr int kUnbThreads = kUnbWarps * 32;
constexpr int kWarpStack = 64;   // per-warp stack of the FP64 re-search (shared memory)
constexpr int kKeep = 16;         // per-lane triangles kept for the FP64 resolution

struct UnbArgs {
  GridP g;
  const BNode* nodes;
  LeafTris ltri;        // leaf-ordered FP32 triangle records
  const TriRec64* rec;
  float pad;              // FP32 margin of the FP64 re-search's box tests
  float eD_abs, eD_rel;   // FP32 point-triangle distance error: eD_abs + eD_rel d
  float wpad_abs;         // FP32 margin of the brick search's tests: wpad_abs + kWidePadRel d
  int64_t max_visits;
  const float* radius;  // learned radius per brick, at its centre (nullable)
  double* dist;
  double* xp;
  int64_t* counters;
  int32_t b[3];         // brick of one warp: nodes along x, y, z (product 32)
  int64_t nb[3];        // bricks per axis
  int64_t nbricks;
  unsigned long long* next;  // brick queue: warps take the next brick with one atomic (zeroed per launch)
  const OBox* obb;           // oriented boxes of the LBVH children (obb[2 node + side])
  const int64_t* bricks = nullptr;               // nullable: search only these bricks ...
  const unsigned long long* bricks_n = nullptr;  // ... this many (read on the device)
  int64_t* redo = nullptr;                       // the radius-bounded search lists here the bricks ...
  unsigned long long* redo_n = nullptr;          // ... it did not certify (a counter zeroed per launch)
  int64_t redo_base = 0;                         // added to the listed brick index (a batch's item offset)
  const float4* lv32 = nullptr;                  // leaf-ordered FP32 vertices, three per triangle
  const float4* v32 = nullptr;                   // the same by triangle index; .w the global vertex id
  bool local = false;                            // the mesh lies near the coordinate origin (see unb_mesh)
  // the brick's lattice: node p (lane bits b = 0..4) lies at node 0 + the sum over set bits of lat[b]
  float lat[5][3] = {};
  float E = 0.f;                                 // the frame's scale
  int* spill = nullptr;                          // kWideSpill queue entries per resident warp of the launch
};

inline LeafTris leaf_tris(sdfgpu_ctx* ctx) { return {buf<float4>(ctx, "ltri"), ctx->mesh.nel}; }

// The mesh's arrays of a search beyond its positional fields.  lane_resolve compares plain FP64 distances
// only while the mesh lies within 64 of its own half-extents of the coordinate origin: far from it the
// reference's barycentric solve, which works on absolute coordinates, loses the digits it relies on.  And from
// 1e-15 on, below which the FP32 root in its tolerance can underflow.
inline void unb_mesh(sdfgpu_ctx* ctx, UnbArgs& A) {
  const MeshDev& M = ctx->mesh;
  double off = 0.0;
  for (int a = 0; a < 3; ++a) off = M.center[a] > off ? M.center[a] : (-M.center[a] > off ? -M.center[a] : off);
  A.lv32 = buf<float4>(ctx, "lv32");
  A.v32 = buf<float4>(ctx, "v32");
  A.local = off <= 64.0 * M.E && M.E >= 1e-15;
}

// Error model of the FP32 searches, u = 2^-24.  Coordinates in the mesh-local frame are within E, so
// each carries at most u E.  The point-triangle distance (view_d2 and its approximate square root) is
// within 4e-7 E + 1e-6 (d + e) of the exact one, e the triangle's longest edge (4e7 random, sliver and needle
// triangles: 1.9e-7 (E + d + e));
// kUnbDistRel (E + d) plus the share of the mesh's longest edge bounds it.
constexpr float kUnbDistRel = 1.5e-6f;
// A test of the brick search compares a lower bound LB of the true distance with the bound of the FP32
// distances that matter.  The box and plane evaluations, the FP32 rounding of the boxes' axes, the
// approximate reciprocal square root and the lattice sums stay below 2.5e-6 E + 1.5e-6 d, the triangle's
// plane and edge lines below 1e-6 E + 1e-6 (d + its edges); with the error of the distance itself,
// kWidePadRel (E + d) plus the share of the longest edge covers both.
constexpr float kWidePadRel = 4.0e-6f;
// What underflow takes from a squared distance of up to 16 terms, 16 * 2^-149, as a distance; it enters both.
constexpr float kUnbUnderflow = 2.0e-22f;
// FP32 margin of the box tests of the FP64 re-search, as a multiple of E (per-lane box distances).
constexpr float kUnbPadRel = 2.2e-5f;

// The arguments that follow from the error model, for a grid frame of scale E.
inline void unb_errors(const MeshDev& M, double E, UnbArgs& A) {
  A.E = (float)E;
  A.pad = kUnbPadRel * (float)E;
  // edges are at most 2 rho_max long
  A.eD_abs = kUnbDistRel * (float)E + 2.0e-6f * (float)M.rho_max + kUnbUnderflow;
  A.eD_rel = kUnbDistRel;
  A.wpad_abs = kWidePadRel * (float)E + 2.0e-6f * (float)M.rho_max + kUnbUnderflow;
}

// Squared lower bound on the distance from p to the child `side` of an LBVH node: the larger of its
// axis-aligned and its oriented box (leaves: the axis-aligned box only).
__device__ __forceinline__ float child_d2(const BNode& nd, const OBox& o, int side, float3 p, float3 lo, float3 hi) {
  const float d = box_d2(p, lo, hi);
  const int c = side ? nd.d.y : nd.d.x;
  if (c & kLeafBit) return d;
  return fmaxf(d, obox_d2(p, o));
}

// Instantiations of the grid searches (k_unbounded, distance.cu; k_unbounded_multi, search_multi.cu):
// kUnbPlain every brick unbounded; kUnbRadius each lane started from its learned radius;
// kUnbListed the plain search over listed bricks.
constexpr int kUnbPlain = 0, kUnbRadius = 1, kUnbListed = 2;
// Lane `lane`'s node (lx, ly, lz) in a warp brick of shape b, and the brick's central lane rep.
__device__ __forceinline__ void brick_lane(const int32_t b[3], int lane, int& lx, int& ly, int& lz, int& rep) {
  lx = lane % b[0];
  ly = (lane / b[0]) % b[1];
  lz = lane / (b[0] * b[1]);
  rep = b[0] / 2 + b[0] * (b[1] / 2 + b[1] * (b[2] / 2));
}

// The warp's next brick from the launch's queue (bricks differ widely in cost, so a static split
// leaves warps idle at the end); every lane gets the same index.
__device__ __forceinline__ int64_t next_brick(const UnbArgs& A, int lane) {
  unsigned long long b = 0ULL;
  if (lane == 0) b = atomicAdd(A.next, 1ULL);
  return (int64_t)__shfl_sync(0xffffffffu, b, 0);
}

// FP32 square root of a leaf's squared distance by the approximate instruction (sqrt.approx.f32:
// relative error at most 2^-23, part of the error model above), one MUFU operation instead of the
// correctly rounded sequence.
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The FP64 step out of line (inlining it would size the registers of the whole search for it).
__device__ __noinline__ void step64_call(const TriRec64* rec, int prim, const d3& p, double& m64, d3& proj) {
  tri_step64(rec[prim], p, m64, proj, false);
}

// Per-lane state of the FP32 search.  m bounds the lane's FP32 minimum point-triangle distance from
// above by at most a few roundings (a triangle's FP32 distance, or that of one of its vertices), and
// the triangles whose FP32 distance lies within band(m) = m + 2 err(m) hold the true (FP64) nearest:
// |FP32 - FP64| <= err for every distance, so the FP64 winner t* has D32(t*) <= d64(t*) + err <=
// m + 2 err.  Their indices are kept in shared memory (slot q of thread x at q * S + x, S the CTA's
// thread count: consecutive threads, consecutive banks); n counts them, and n > kKeep means that more
// were in the band than there are slots.  Some kept early may lie outside the final band, which costs
// an FP64 step and changes nothing.
struct LaneBest {
  float m;
  int n;
  int* t;  // shared: kept triangle ids
};

template <class P>
__device__ __forceinline__ float band_of(const P& A, float m) { return m + 2.f * (A.eD_abs + A.eD_rel * m); }
// What the brick search's tests compare lower bounds with: the band of m plus their margin.
template <class P>
__device__ __forceinline__ float wide_bound(const P& A, float m) {
  return fmaf(m, 1.f + 2.f * kUnbDistRel + kWidePadRel, 2.f * A.eD_abs + A.wpad_abs);
}

// Squared distance from p to the triangle of r in FP64 by the regions of its Voronoi diagram (Ericson,
// Real-Time Collision Detection, 5.1.5), from differences of coordinates, and the Feature that the
// reference step certainly takes its value from, or -1:
//   vertex: p's feet on its two edges lie beyond it by more than tol, and the triangle's height over the
//     third edge is above 1e-6 of the distance;
//   edge: the foot lies within the middle 0.998 of it, p's projection beyond its line by more than tol,
//     and the triangle's heights are above 1e-3 of the distance;
//   face: the barycentric coordinates are above 1e-4.
// Then the step's barycentric signs and edge parameters are far from their limits against FP64
// rounding, and every foot or vertex other than the feature's is farther by more than 1e-12 of the
// distance (for a convex set |p - x|^2 >= |p - q|^2 + |x - q|^2, q the closest point).
__device__ __noinline__ double near64(const TriRec64* __restrict__ rec, int t, const d3& p, double tol2, int& feat) {
  const TriRec64& r = rec[t];
  const d3 v0 = rec_v(r, 0), v1 = rec_v(r, 1), v2 = rec_v(r, 2);
  const double wx = p.x - v0.x, wy = p.y - v0.y, wz = p.z - v0.z;
  const double ax = v1.x - v0.x, ay = v1.y - v0.y, az = v1.z - v0.z;
  const double bx = v2.x - v0.x, by = v2.y - v0.y, bz = v2.z - v0.z;
  const double aa = ax * ax + ay * ay + az * az, ab = ax * bx + ay * by + az * bz, bb = bx * bx + by * by + bz * bz;
  const double d1 = ax * wx + ay * wy + az * wz, d2 = bx * wx + by * wy + bz * wz;
  // the same dot products at v1 (w - a) and at v2 (w - b)
  const double p3 = d1 - aa, p4 = d2 - ab, p5 = d1 - ab, p6 = d2 - bb;
  const double nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
  const double nn = nx * nx + ny * ny + nz * nz, cc = aa + bb - 2.0 * ab;
  feat = -1;
  // a foot (dot / edge length) beyond the limit by more than tol
  auto past = [&](double dot, double ee) { return dot < 0.0 && dot * dot > tol2 * ee; };
  if (d1 <= 0.0 && d2 <= 0.0) {
    const double uu = wx * wx + wy * wy + wz * wz;
    if (past(d1, aa) && past(d2, bb) && nn > 1e-12 * uu * cc) feat = F_VERT0;
    return uu;
  }
  if (p3 >= 0.0 && p4 <= p3) {
    const double ux = wx - ax, uy = wy - ay, uz = wz - az, uu = ux * ux + uy * uy + uz * uz;
    if (past(-p3, aa) && past(p4 - p3, cc) && nn > 1e-12 * uu * bb) feat = F_VERT1;
    return uu;
  }
  if (p6 >= 0.0 && p5 <= p6) {
    const double ux = wx - bx, uy = wy - by, uz = wz - bz, uu = ux * ux + uy * uy + uz * uz;
    if (past(-p6, bb) && past(p5 - p6, cc) && nn > 1e-12 * uu * aa) feat = F_VERT2;
    return uu;
  }
  // barycentric coordinates times nn, of v2, v1 and v0
  const double vc = d1 * p4 - p3 * d2, vb = p5 * d2 - d1 * p6, va = p3 * p6 - p5 * p4;
  double s, ee, ex, ey, ez, qx = wx, qy = wy, qz = wz, out;
  if (vc <= 0.0 && d1 >= 0.0 && p3 <= 0.0) {
    s = d1; ee = aa; ex = ax; ey = ay; ez = az; out = vc; feat = F_EDGE0;
  } else if (vb <= 0.0 && d2 >= 0.0 && p6 <= 0.0) {
    s = d2; ee = bb; ex = bx; ey = by; ez = bz; out = vb; feat = F_EDGE2;
  } else if (va <= 0.0 && p4 - p3 >= 0.0 && p5 - p6 >= 0.0) {
    s = p4 - p3; ee = cc; ex = bx - ax; ey = by - ay; ez = bz - az; out = va; feat = F_EDGE1;
    qx -= ax; qy -= ay; qz -= az;
  } else {
    const double h = wx * nx + wy * ny + wz * nz, lim = 1e-4 * nn;
    if (va > lim && vb > lim && vc > lim) feat = F_FACE;
    return h * h / nn;
  }
  const double f = s / ee;
  qx -= f * ex; qy -= f * ey; qz -= f * ez;
  const double uu = qx * qx + qy * qy + qz * qz;
  // out / (nn / edge length) is p's projection beyond the edge line; heights squared are nn / edge^2
  const double emax = fmax(aa, fmax(bb, cc));
  if (!(f > 1e-3 && f < 1.0 - 1e-3 && out < 0.0 && out * out > tol2 * nn * ee && nn > 1e-6 * uu * emax)) feat = -1;
  return uu;
}

constexpr int kFeatShift = 29;  // a pruned slot holds the triangle index and its feature (7: unknown) above it
constexpr int kTriMask = (1 << kFeatShift) - 1;

// Drops the kept triangles that cannot hold the FP64 minimum and returns how many are left (all of them
// where that cannot be told: a triangle unfit for FP32 decisions among them, or a mesh far from the
// coordinate origin).  The FP32 band holds a few triangles per node -- all around the nearest vertex or
// edge -- of which only those that share the nearest feature can win: a plain FP64 distance from the
// vertices (72 of the record's 352 bytes, a tenth of the reference step's work) is within 1e-11 E of the
// step's value on triangles fit for FP32 decisions, and the ones farther than the nearest by more than
// 1e-9 E go.  gid: the global id of the certain nearest vertex that all of them share, or -1.
template <int S>
__device__ __forceinline__ int lane_filter(const UnbArgs& A, const LaneBest& L, const d3& p, int& gid, bool keep_id) {
  const int n = min(L.n, kKeep);
  gid = -1;
  if (!A.local) return n;
  for (int q = 0; q < n; ++q)
    if (L.t[q * S] & kWeakTri) return n;
  const double tol = 1e-9 * (double)A.E, tol2 = tol * tol;
  double best = 1e300, lim = 1e300;
  int left = 0;
#pragma unroll 1
  for (int q = 0; q < n; ++q) {
    const int t = L.t[q * S];
    int feat;
    const double d2 = near64(A.rec, t, p, tol2, feat);
    if (d2 > lim) continue;
    const int g = feat >= F_VERT0 ? __float_as_int(A.v32[3 * (int64_t)t + (feat - F_VERT0)].w) : -1;
    if (d2 < best) {
      const double dl = 2.0 * tol * (double)sqrtf((float)d2) * (1.0 + 1e-6) + tol2;
      if (d2 + dl < best) left = 0;  // everything left so far is farther
      best = d2;
      lim = d2 + dl;
    }
    gid = left == 0 || g == gid ? g : -1;
    L.t[left++ * S] = keep_id ? t : (int)((unsigned)t | (unsigned)(feat < 0 ? 7 : feat) << kFeatShift);  // left <= q
  }
  if (left == 0) gid = -1;
  return keep_id ? left : left | (1 << 16);  // bit 16: the slots carry features
}
template <int S>
__device__ __noinline__ void lane_prune(const UnbArgs& A, LaneBest& L, const d3& p) {
  int gid;
  L.n = lane_filter<S>(A, L, p, gid, true);
}

// The fold of a lane's n slots in ascending triangle index (so exact ties keep the lowest index): the reference
// step, or where `known` the expression that it certainly takes its value from, unless the step's box test passes
// the triangle over, as it can a value that is a few roundings below the minimum so far (never at kBig).  Out of
// line with the steps inlined: in the search's own code the test cost 0.7 of 27.1 ms on 16.8M nodes (B200),
// wherever it stood; here nothing.
template <int S>
__device__ __noinline__ void resolve_many(const TriRec64* rec, const int* slots, int n, bool known, const d3& p,
                                          double& m64, d3& proj) {
  int last = -1;
#pragma unroll 1
  for (int it = 0; it < n; ++it) {
    unsigned best = 0xffffffffu;
    int tri = 0x7fffffff;
#pragma unroll 1
    for (int q = 0; q < n; ++q) {
      const unsigned s = (unsigned)slots[q * S];
      const int t = known ? (int)(s & kTriMask) : (int)(s & ~(unsigned)kWeakTri);
      if (t > last && t < tri) { tri = t; best = s; }
    }
    if (tri == 0x7fffffff) break;
    last = tri;
    const int feat = known ? (int)(best >> kFeatShift) : 7;
    if (feat == 7) {
      tri_step64(rec[tri], p, m64, proj, false);
    } else {
      double d;
      d3 x;
      feature64(rec[tri], p, feat, d, x);
      if (d < m64 && !(m64 < kBig && step_skips(rec[tri], p, m64))) {
        m64 = d;
        proj = x;
      }
    }
  }
}

// The FP64 minimum over the kept triangles.  Triangles left with the same certain nearest vertex all have its
// distance: the first stands for all.
template <int S>
__device__ __forceinline__ void lane_resolve(const UnbArgs& A, LaneBest& L, const d3& p, double& m64, d3& proj,
                                             uint32_t& fp64) {
  int gid;
  const int got = lane_filter<S>(A, L, p, gid, false);
  const bool known = (got >> 16) != 0;
  int n = got & 0xffff;
  if (gid >= 0) n = 1;
  fp64 += n;
  resolve_many<S>(A.rec, L.t, n, known, p, m64, proj);
}

// ---- the FP32 pass: one warp, one brick of 32 nodes -------------------------------------------------
//
// Three stages run on queues in shared memory, each with 32 full lanes where the work allows it:
//   open   up to kWideNodes LBVH nodes per step, two levels at once: each lane takes ONE grandchild and
//          tests it against ALL 32 nodes of the brick.  A convex set S at distance LB from the brick's
//          centre c, in unit direction u from its closest point to c, has dist(p, S) >= LB + u . (p - c)
//          for every p, so it matters only when LB <= max over the nodes of (ub(p) - u . (p - c)), ub(p)
//          the band of the lane's minimum plus the FP32 margin.  The nodes form a lattice, so the 32
//          values of u . (p - c) are sums of five per-bit terms.  The queue is first in, first out -- a
//          level is opened before the next one -- and the minimum of every node is first lowered to its
//          distance from a vertex of each opened subtree's middle triangle, so that the bounds are as
//          tight as the boxes of the level: no seed and no nearest-first order is needed.
//   leaves of subtrees of up to kWideLeafs triangles, 32 triangles at a time: a triangle lies on the
//          inner side of its three edge lines, so dist(p, T)^2 >= (plane distance)^2 + (largest distance
//          outside an edge line)^2, four lattice functions of p; the lane keeps a bit per node.
//   eval   of the triangles that are left, 32 at a time, a lane per triangle with its record in
//          registers: the distances of all triangles to one node, their minimum (REDUX) and the ones
//          within its band (a ballot) at a time, for the nodes that any of the 32 can matter to.
// The packet search before it (a lane per node, one child or one triangle per step) spent its time on
// broadcast loads: a 128-bit load costs four cycles of the load pipe even when every lane reads the same
// address.  Here the per-(child, node) work reads one word.
constexpr int kWideNodes = 8;     // LBVH nodes opened per step (four grandchildren each: one per lane)
constexpr int kWideQueue = 256;   // nodes waiting per warp in shared memory (a ring), 160 of them in use ...
constexpr int kWideSpill = 2048;  // ... and behind them in device memory (a ring per resident warp; the
                                  // nearest-vertex search has one of kKnnSpill)
constexpr int kKnnSpill = 512;
constexpr int kWideLeafs = 4;     // subtrees of up to this many triangles are queued whole
constexpr int kWideLeafQ = 32 * kWideLeafs + 32;  // a step adds at most 32 kWideLeafs to at most 31
static_assert(kWideLeafs < 8, "three bits of triangle counts");

struct __align__(16) WideShared {
  float ub[32];           // per node: bound on the FP32 distances that matter, -3e38 for unused lanes
  float4 node[32];        // the nodes relative to node 0
  float4 rep[3 * kWideNodes]; // sample vertices of a step relative to the centre, .w = -|x|^2 (1 + 1e-6)
  int queue[kWideQueue];
  int leaf[kWideLeafQ];
  int2 cand[64];          // triangles left to evaluate: (sorted leaf, bit per node)
  int prim[32];           // triangle indices of the 32 being evaluated
};

// Whether three leaf-ordered vertices are distinct (global ids in .w).
__device__ __forceinline__ bool differ3(const float4& a, const float4& b, const float4& c) {
  const int i = __float_as_int(a.w), j = __float_as_int(b.w), k = __float_as_int(c.w);
  return i != j && j != k && i != k;
}

// The linear function base + g . (p - p0) over the brick's lattice by the bits of the node index: lo
// (bits 0-1) + hi (bits 2-3) + top (bit 4).  The loops over bit 4 stay rolled: the kernel's code is
// bound by instruction fetch where all of it is laid out.
struct Lattice {
  float lo[4], hi[4], top;
};
template <class P>
__device__ __forceinline__ Lattice lattice_terms(const P& A, float3 g, float base) {
  float t[5];
#pragma unroll
  for (int b = 0; b < 5; ++b) t[b] = fmaf(g.x, A.lat[b][0], fmaf(g.y, A.lat[b][1], g.z * A.lat[b][2]));
  Lattice L;
  L.lo[0] = 0.f; L.lo[1] = t[0]; L.lo[2] = t[1]; L.lo[3] = t[0] + t[1];
  L.hi[0] = base; L.hi[1] = base + t[2]; L.hi[2] = base + t[3]; L.hi[3] = L.hi[1] + t[3];
  L.top = t[4];
  return L;
}
__device__ __forceinline__ void lattice_next(Lattice& f) {
#pragma unroll
  for (int k = 0; k < 4; ++k) f.hi[k] += f.top;
}

// Whether LB + u . (p - c) <= ub(p) for some node p (base = LB + u . (p0 - c)); NaN means yes.
template <class P>
__device__ __forceinline__ bool plane_wanted(const P& A, const WideShared& W, float3 u, float base) {
  Lattice f = lattice_terms(A, u, base);
  const float4* ub = reinterpret_cast<const float4*>(W.ub);
  bool far = true;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 b = ub[4 * h + k];
      const float m = fmaxf(fmaxf(b.x - f.lo[0], b.y - f.lo[1]), fmaxf(b.z - f.lo[2], b.w - f.lo[3]));
      far = far && f.hi[k] > m;
    }
    lattice_next(f);
  }
  return !far;
}

// Lower bound LB at c and direction u (at most unit length) of the child `side` of LBVH node nid: its
// axis-aligned or its oriented box (inner children), whichever is farther.  LB comes from the same
// components as u, so the plane bound above holds to the rounding of those components.  Squares
// beyond FP32 make LB NaN, which every test here reads as "open it".
template <class P>
__device__ __forceinline__ void child_plane(const P& A, int nid, int side, bool inner, float3 c, float& LB, float3& u) {
  const float4* n4 = reinterpret_cast<const float4*>(A.nodes + nid);
  const float4 b = n4[1], o = n4[side ? 2 : 0];
  const float3 lo = side ? make_float3(b.z, b.w, o.x) : make_float3(o.x, o.y, o.z);
  const float3 hi = side ? make_float3(o.y, o.z, o.w) : make_float3(o.w, b.x, b.y);
  // c minus its closest point of the axis-aligned box
  float3 v = make_float3(c.x - fminf(fmaxf(c.x, lo.x), hi.x), c.y - fminf(fmaxf(c.y, lo.y), hi.y),
                         c.z - fminf(fmaxf(c.z, lo.z), hi.z));
  float d2 = dot3f(v, v);
  if (inner) {
    const OBox q = A.obb[2 * (int64_t)nid + side];
    const float t0 = fmaf(c.x, q.a0.x, fmaf(c.y, q.a0.y, fmaf(c.z, q.a0.z, -q.a0.w)));
    const float t1 = fmaf(c.x, q.a1.x, fmaf(c.y, q.a1.y, fmaf(c.z, q.a1.z, -q.a1.w)));
    const float t2 = fmaf(c.x, q.a2.x, fmaf(c.y, q.a2.y, fmaf(c.z, q.a2.z, -q.a2.w)));
    const float s0 = copysignf(fmaxf(fabsf(t0) - q.e.x, 0.f), t0);
    const float s1 = copysignf(fmaxf(fabsf(t1) - q.e.y, 0.f), t1);
    const float s2 = copysignf(fmaxf(fabsf(t2) - q.e.z, 0.f), t2);
    const float o2 = fmaf(s0, s0, fmaf(s1, s1, s2 * s2));
    if (o2 > d2) {
      d2 = o2;
      v = make_float3(fmaf(s0, q.a0.x, fmaf(s1, q.a1.x, s2 * q.a2.x)), fmaf(s0, q.a0.y, fmaf(s1, q.a1.y, s2 * q.a2.y)),
                      fmaf(s0, q.a0.z, fmaf(s1, q.a1.z, s2 * q.a2.z)));
    }
  }
  const float r = rsqrtf(fmaxf(d2, 1.0e-30f));
  LB = d2 * r;
  u = v * r;
}

// The FP32 pass over the LBVH from L's initial minimum (INFINITY, or the learned radius).  On return L
// holds the FP32 minimum and the triangles of its band.  Returns false when the visit or queue bound is
// exceeded.
//
// Queue: a step opens the n <= kWideNodes oldest nodes of the shared ring and adds at most 4n, to the
// ring while at most kWideQueue - 96 wait there and nothing is spilled, else to the warp's ring in device
// memory, which refills the shared one when that is empty (a brick near a medial axis of the surface has
// hundreds of nodes of a level at its distance).  When the spilled nodes leave no room for a step, the
// newest node of the shared ring is opened alone instead and its children stay there: depth-first
// steps grow it by at most 3 per two levels of the tree (at most 62 levels: unique keys of 30 Morton bits
// and a 32-bit index), which the 96 reserved entries hold.
//
// kKnn: the search for each lane's three nearest vertices (k_knn_bricks, distance.cu).  m then bounds
// the distance of the third: a triangle's farthest vertex, where its vertices differ; the queued
// leaves go to the evaluation as they are, and a triangle is kept when its nearest vertex lies
// within band(m).  flush(): makes room in the slots (kKnn: called by all lanes, and empties them).
template <int S, bool kKnn, class P, class Flush>
__device__ __forceinline__ bool wide_search(const P& A, WideShared& W, int* spill, int lane, const d3& p,
                                            const float3& p32, bool active, LaneBest& L, uint32_t& visits_out,
                                            Flush flush) {
  constexpr unsigned kSpill = kKnn ? kKnnSpill : kWideSpill;
  const float3 p0 = make_float3(__shfl_sync(0xffffffffu, p32.x, 0), __shfl_sync(0xffffffffu, p32.y, 0),
                                __shfl_sync(0xffffffffu, p32.z, 0));
  // the brick's centre: half of every lattice step from node 0
  const float3 hc = make_float3(0.5f * (A.lat[0][0] + A.lat[1][0] + A.lat[2][0] + A.lat[3][0] + A.lat[4][0]),
                                0.5f * (A.lat[0][1] + A.lat[1][1] + A.lat[2][1] + A.lat[3][1] + A.lat[4][1]),
                                0.5f * (A.lat[0][2] + A.lat[1][2] + A.lat[2][2] + A.lat[3][2] + A.lat[4][2]));
  const float3 c = p0 + hc;
  if (lane == 0) W.queue[0] = 0;
  W.node[lane] = make_float4(p32.x - p0.x, p32.y - p0.y, p32.z - p0.z, 0.f);
  W.ub[lane] = active ? wide_bound(A, L.m) : -3.0e38f;
  unsigned head = 0, tail = 1;    // shared ring positions (mod kWideQueue)
  unsigned shead = 0, stail = 0;  // spilled ring positions (mod kWideSpill)
  int nl = 0, nc = 0;
  uint32_t visits = 0;  // at most max_visits = 2 nel + 64 < 2^30
  bool ok = true;
  const unsigned below = (1u << lane) - 1u;
  __syncwarp();
  while (true) {
    int waiting = (int)(tail - head);
    if (waiting == 0 && stail != shead) {  // refill the shared ring
      waiting = (int)min(stail - shead, (unsigned)(kWideQueue - 96));
      for (int i = lane; i < waiting; i += 32) W.queue[i] = spill[(shead + i) % kSpill];
      shead += waiting;
      head = 0;
      tail = waiting;
      __syncwarp();
    }
    if constexpr (kKnn) {
      if (nl >= 32 || (waiting == 0 && nl > 0)) {
        // ---- eval of three vertices: lane = triangle, one node at a time
        const int cnt = min(nl, 32);
        nl -= cnt;
        const int li = lane < cnt ? W.leaf[nl + lane] : 0;
        const float4 a4 = A.lv32[3 * (int64_t)li], b4 = A.lv32[3 * (int64_t)li + 1], c4 = A.lv32[3 * (int64_t)li + 2];
        const float3 a = f3(a4) - p0, b = f3(b4) - p0, e = f3(c4) - p0;
        const bool three = lane < cnt && differ3(a4, b4, c4);
        W.prim[lane] = __float_as_int(A.ltri.at(0, li).w) & ~kWeakTri;
        unsigned mine = 0u;
        float mnew = L.m;
        __syncwarp();
        for (unsigned todo = __ballot_sync(0xffffffffu, active); todo; todo &= todo - 1u) {
          const int q = __ffs(todo) - 1;
          const float3 P3 = f3(W.node[q]);
          const float3 da = P3 - a, db = P3 - b, dc = P3 - e;
          const float xa = dot3f(da, da), xb = dot3f(db, db), xc = dot3f(dc, dc);
          const unsigned key = three ? __float_as_uint(fmaxf(xa, fmaxf(xb, xc))) : 0x7f800000u;
          const float best = sqrt_approx(__uint_as_float(__reduce_min_sync(0xffffffffu, key)));
          const float m = fminf(__shfl_sync(0xffffffffu, L.m, q), best);
          const float bd = band_of(A, m);
          const unsigned in = __ballot_sync(0xffffffffu, lane < cnt && !(fminf(xa, fminf(xb, xc)) > bd * bd));
          if (lane == q) {
            mine = in;
            mnew = m;
          }
        }
        if (!active) mine = 0u;
        L.m = mnew;
        while (true) {
          for (; mine && L.n < kKeep; mine &= mine - 1u) L.t[L.n++ * S] = W.prim[__ffs(mine) - 1];
          if (!__any_sync(0xffffffffu, mine != 0u)) break;
          flush();  // all lanes together: one lane at a time took most of the kernel
        }
        if (active) W.ub[lane] = wide_bound(A, L.m);
        __syncwarp();
        continue;
      }
    }
    if (!kKnn && (nc >= 32 || (waiting == 0 && nl == 0 && nc > 0))) {
      // ---- eval: lane = triangle, one node at a time
      const int cnt = min(nc, 32);
      nc -= cnt;
      const int2 e = lane < cnt ? W.cand[nc + lane] : make_int2(0, 0);
      const LeafTri T = A.ltri.load(e.x);
      W.prim[lane] = __float_as_int(T.a.w);
      const LeafView V = leaf_view(T, p0);
      unsigned mine = 0u;  // this lane's node: the triangles within its band
      float mnew = L.m;
      __syncwarp();
      for (unsigned todo = __reduce_or_sync(0xffffffffu, (unsigned)e.y); todo; todo &= todo - 1u) {
        const int q = __ffs(todo) - 1;
        const float4 P4 = W.node[q];
        const float d2 = view_d2(V, make_float3(P4.x, P4.y, P4.z));
        // non-negative: bit order = value order (a lane without a triangle, or NaN, never wins)
        const unsigned key = lane < cnt ? __float_as_uint(d2) : 0x7fffffffu;
        const float best = sqrt_approx(__uint_as_float(__reduce_min_sync(0xffffffffu, key)));
        const float m = fminf(__shfl_sync(0xffffffffu, L.m, q), best);
        const float bd = band_of(A, m);
        const unsigned in = __ballot_sync(0xffffffffu, lane < cnt && !(d2 > bd * bd));
        if (lane == q) {
          mine = in;
          mnew = m;
        }
      }
      if (active) {
        if (L.m > band_of(A, mnew)) L.n = 0;  // everything kept so far is outside the new band
        L.m = mnew;
        if (L.n + __popc(mine) > kKeep && L.n <= kKeep) flush();  // make room
        for (; mine; mine &= mine - 1u) {
          if (L.n < kKeep) L.t[L.n * S] = W.prim[__ffs(mine) - 1];
          ++L.n;
        }
        W.ub[lane] = wide_bound(A, L.m);
      }
      __syncwarp();
      continue;
    }
    if (!kKnn && (nl >= 32 || (waiting == 0 && nl > 0))) {
      // ---- leaves: lane = triangle, its plane and edge lines against every node
      const int cnt = min(nl, 32);
      nl -= cnt;
      const int li = lane < cnt ? W.leaf[nl + lane] : 0;
      unsigned bits = 0u;
      {
        const LeafTri T = A.ltri.load(li);
        const float3 w = p0 - f3(T.a);
        Lattice fn = lattice_terms(A, f3(T.n), dot3f(w, f3(T.n)));
        Lattice f0 = lattice_terms(A, f3(T.m0), dot3f(w, f3(T.m0)));
        Lattice f1 = lattice_terms(A, f3(T.m1), dot3f(w, f3(T.m1)) - T.m1.w);
        Lattice f2 = lattice_terms(A, f3(T.m2), dot3f(w, f3(T.m2)));
        const bool flat = T.m2.w < 0.f;  // a triangle without area has no edge lines here: nothing is known
        const float4* ub = reinterpret_cast<const float4*>(W.ub);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          unsigned half = 0u;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 b = ub[4 * h + k];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float bj = j == 0 ? b.x : (j == 1 ? b.y : (j == 2 ? b.z : b.w));
              const float dn = fn.hi[k] + fn.lo[j];
              const float s = fminf(fminf(f0.hi[k] + f0.lo[j], f1.hi[k] + f1.lo[j]), fminf(f2.hi[k] + f2.lo[j], 0.f));
              // unused nodes carry a negative bound; NaN counts as near
              if (!(fmaf(dn, dn, s * s) > bj * fabsf(bj))) half |= 1u << (4 * k + j);
            }
          }
          bits |= half << (16 * h);
          lattice_next(fn);
          lattice_next(f0);
          lattice_next(f1);
          lattice_next(f2);
        }
        if (flat) bits = 0xffffffffu;
        if (lane >= cnt) bits = 0u;
      }
      const unsigned m = __ballot_sync(0xffffffffu, bits != 0u);
      if (bits) W.cand[nc + __popc(m & below)] = make_int2(li, (int)bits);
      nc += __popc(m);
      __syncwarp();
      continue;
    }
    if (waiting == 0) break;
    // ---- open
    int n = min(kWideNodes, waiting);
    const bool fifo = stail - shead + 4 * kWideNodes <= kSpill;
    if (!fifo) n = 1;
    visits += n;
    if (visits > A.max_visits || (!fifo && waiting + 3 > kWideQueue)) { ok = false; break; }
    const unsigned first = fifo ? head : tail - 1u;
    if (fifo) head += n;
    else tail -= 1u;
    // the lane's grandchild: child s1 of the node, then its child s2 -- or child s1 itself (one lane of
    // the pair) when that is a subtree of at most kWideLeafs triangles
    bool act = (lane >> 2) < n;
    int nid = act ? W.queue[(first + (lane >> 2)) % kWideQueue] : 0;
    int4 q = A.nodes[nid].d;
    if (kKnn ? (lane & 3) != 3 : (lane & 3) == 0) {  // the node's sample vertex (kKnn: all three of its triangle)
      const int64_t l = 3 * (int64_t)((q.z + q.w) >> 1);
      const float4 v = A.lv32[l + (kKnn ? lane & 3 : 0)];
      const bool use = act && (!kKnn || differ3(A.lv32[l], A.lv32[l + 1], A.lv32[l + 2]));
      const float3 r = make_float3(v.x - c.x, v.y - c.y, v.z - c.z);
      W.rep[kKnn ? 3 * (lane >> 2) + (lane & 3) : lane >> 2] =
          make_float4(r.x, r.y, r.z, use ? dot3f(r, r) * -(1.f + 1.0e-6f) : -3.0e38f);
    }
    int side = (lane >> 1) & 1;
    int gamma = q.x & 0x7fffffff;
    int lo = side ? gamma + 1 : q.z, num = side ? q.w - gamma : gamma - q.z + 1;
    if (num > kWideLeafs) {
      nid = side ? q.y : q.x;
      q = A.nodes[nid].d;
      side = lane & 1;
      gamma = q.x & 0x7fffffff;
      lo = side ? gamma + 1 : q.z;
      num = side ? q.w - gamma : gamma - q.z + 1;
    } else {
      act = act && (lane & 1) == 0 && num > 0;  // num 0: the right side of a one-triangle tree
    }
    const int child = side ? q.y : q.x;
    float LB;
    float3 u;
    child_plane(A, nid, side, num > 1, c, LB, u);
    __syncwarp();
    {
      // |p - v|^2 = |d|^2 + |r|^2 - 2 d . r with d = p - c, the squares raised by 1e-6 over the rounding
      const float3 d = p32 - c;
      float best = -3.0e38f;
#pragma unroll
      for (int k = 0; k < kWideNodes; ++k) {
        auto at = [&](int j) {
          const float4 r = W.rep[j];
          return fmaf(2.f * d.x, r.x, fmaf(2.f * d.y, r.y, fmaf(2.f * d.z, r.z, r.w)));
        };
        best = fmaxf(best, kKnn ? fminf(at(3 * k), fminf(at(3 * k + 1), at(3 * k + 2))) : at(k));
      }
      const float d2 = fmaf(dot3f(d, d), 1.f + 1.0e-6f, -best);
      L.m = fminf(L.m, sqrt_approx(fmaxf(d2, 0.f)) * (1.f + 2.0e-6f));
      if (active) W.ub[lane] = wide_bound(A, L.m);
    }
    __syncwarp();
    const bool want = act && plane_wanted(A, W, u, LB - dot3f(u, hc));
    const bool open = want && num > kWideLeafs;
    const unsigned mi = __ballot_sync(0xffffffffu, open);
    const unsigned more = __popc(mi);
    if (!fifo || (stail == shead && tail - head + more <= (unsigned)(kWideQueue - 96))) {
      if (open) W.queue[(tail + __popc(mi & below)) % kWideQueue] = child;
      tail += more;
    } else {
      if (open) spill[(stail + __popc(mi & below)) % kSpill] = child;
      stail += more;
    }
    const unsigned add = want && !open ? (unsigned)num : 0u;  // triangles to queue: 0..kWideLeafs
    int at = nl;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const unsigned mb = __ballot_sync(0xffffffffu, (add >> b) & 1u);
      at += __popc(mb & below) << b;
      nl += __popc(mb) << b;
    }
    for (unsigned k = 0; k < add; ++k) W.leaf[at + k] = lo + k;
    __syncwarp();
  }
  __syncwarp();
  visits_out += visits;
  return ok;
}

// The FP64 re-search of lanes whose band overflowed (rare): a packet traversal, one LBVH node per step with
// its two children tested per lane, where every leaf triangle within a lane's bound -- r0 = band of its FP32
// minimum, then its FP64 minimum -- runs the FP64 step at once.
//
// It finds the smallest value, its lowest triangle index, and the next larger value.  When that is farther off
// than roundings can matter, this is what the steps in ascending index come to.  Else (equally far triangles
// whose values differ by a few roundings, as two beside one edge: the steps' box test decides between them by
// their order) the steps of the triangles within tol of the smallest value are replayed in ascending index from
// the lane's share of the warp's spilled queue, which the FP32 pass has done with.  Where there are more of them
// than it holds (a node on the axis of a fan), the smallest value stays, which the box test could have kept from
// being reached by a few roundings.
constexpr int kTies = kWideSpill / 32;
template <class P>
__device__ __noinline__ bool exact_search(const P& A, int* stack, int* spill, int lane, int rep, const d3& p,
                                          const float3& p32, bool active, float r0, double& m64, d3& proj,
                                          uint32_t& fp64, uint32_t& visits_out) {
  int* ties = spill + lane;
  const double tol = 1e-9 * (double)A.E + 1e-14 * (fabs(p.x) + fabs(p.y) + fabs(p.z));
  double next = INFINITY;
  int at = -1, n = 0;  // the triangle of m64; triangles in `ties`
  int sp = 1;
  if (lane == 0) stack[0] = 0;
  __syncwarp();
  uint32_t visits = 0;  // at most max_visits = 2 nel + 64 < 2^30
  bool ok = true;
  while (sp > 0) {
    if (++visits > A.max_visits) { ok = false; break; }
    const int nid = stack[--sp];
    __syncwarp();
    // the node and both oriented boxes in one round of loads (leaf children carry kNoObb boxes)
    const BNode nd = A.nodes[nid];
    const OBox ob0 = A.obb[2 * nid], ob1 = A.obb[2 * nid + 1];
    float3 lo0, hi0, lo1, hi1;
    child_box(nd, 0, lo0, hi0);
    child_box(nd, 1, lo1, hi1);
    const bool e0 = lo0.x > hi0.x, e1 = lo1.x > hi1.x;  // empty child
    const float d0 = child_d2(nd, ob0, 0, p32, lo0, hi0), d1 = child_d2(nd, ob1, 1, p32, lo1, hi1);
    const float mf = (float)m64;
    const float b = fminf(r0, mf + A.eD_abs + A.eD_rel * mf) + A.pad;
    const float b2 = b * b;
    const bool w0 = active && !e0 && d0 <= b2, w1 = active && !e1 && d1 <= b2;
    const unsigned m0 = __ballot_sync(0xffffffffu, w0), m1 = __ballot_sync(0xffffffffu, w1);
    const float rd0 = __shfl_sync(0xffffffffu, e0 ? INFINITY : d0, rep);
    const float rd1 = __shfl_sync(0xffffffffu, e1 ? INFINITY : d1, rep);
    const bool swap = rd1 < rd0;
    const int cn = swap ? nd.d.y : nd.d.x, cf = swap ? nd.d.x : nd.d.y;
    const unsigned mn = swap ? m1 : m0, mfar = swap ? m0 : m1;
    const bool wn = swap ? w1 : w0, wf = swap ? w0 : w1;
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {  // leaves now, near one first
      const int ch = q == 0 ? cn : cf;
      const bool want = q == 0 ? wn : wf;
      if (!(ch & kLeafBit) || (q == 0 ? mn : mfar) == 0u) continue;
      const int64_t l = ch & 0x7fffffff;
      const float4* v = A.lv32 + 3 * l;
      const float D = sqrtf(pt_tri_d2(p32, f3(v[0]), f3(v[1]), f3(v[2])));
      const float mq = (float)m64;
      if (!want || D > fminf(r0, mq + A.eD_abs + A.eD_rel * mq) + A.pad) continue;
      const int prim = __float_as_int(A.ltri.at(0, (int)l).w) & ~kWeakTri;
      const double from = fmin(m64 + 2.0 * tol, kBig);
      double m = from;
      d3 x;
      step64_call(A.rec, prim, p, m, x);
      ++fp64;
      if (!(m < from)) continue;
      if (m < m64 - tol) n = 0;  // what was kept is farther
      if (n < kTies) ties[n * 32] = prim;
      ++n;
      if (m < m64 || (m == m64 && prim < at)) {
        if (m < m64) next = at < 0 ? INFINITY : m64;
        m64 = m;
        at = prim;
        proj = x;
      } else if (m > m64) {
        next = fmin(next, m);
      }
    }
    // inner children, the far one pushed first so the near one is popped next
    if (mfar != 0u && !(cf & kLeafBit)) {
      if (sp >= kWarpStack) { ok = false; break; }
      if (lane == 0) stack[sp] = cf;
      ++sp;
    }
    if (mn != 0u && !(cn & kLeafBit)) {
      if (sp >= kWarpStack) { ok = false; break; }
      if (lane == 0) stack[sp] = cn;
      ++sp;
    }
    __syncwarp();
  }
  __syncwarp();
  visits_out += visits;
  if (active && next <= m64 + tol && n <= kTies) {
    m64 = fmin(m64 + 2.0 * tol, kBig);
    int last = -1;
#pragma unroll 1
    for (int it = 0; it < n; ++it) {
      int t = 0x7fffffff;
      for (int q = 0; q < n; ++q)
        if (ties[q * 32] > last && ties[q * 32] < t) t = ties[q * 32];
      last = t;
      step64_call(A.rec, t, p, m64, proj);
    }
  }
  return ok;
}

}  // namespace
}  // namespace sdfgpu
