// geom32.cuh -- FP32 geometry for the bulk of the work: point-triangle distance and ray-box
// tests in mesh-local coordinates (vertices minus the mesh's bounding-box centre).  Every FP32
// result is used only as a filter with an explicit error margin; decisions that land inside the
// margin are re-made with the FP64 routines of exact64.cuh.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace sdfgpu {

__device__ __forceinline__ float3 f3(float4 a) { return make_float3(a.x, a.y, a.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot3f(float3 a, float3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ float3 cross3f(float3 a, float3 b) {
  return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// Squared distance from p to segment [a, a+e].
__device__ __forceinline__ float seg_d2(float3 p, float3 a, float3 e) {
  const float3 w = p - a;
  const float ee = dot3f(e, e);
  float t = ee > 0.f ? dot3f(w, e) / ee : 0.f;
  t = fminf(fmaxf(t, 0.f), 1.f);
  const float3 q = w - e * t;
  return dot3f(q, q);
}

// Squared distance from p to triangle (a, b, c): minimum of the three edge distances and, when
// p projects inside, the plane distance.  Degenerate triangles reduce to their edges.  The normal is formed
// from edges scaled to about 1: products of all the lengths would leave FP32 from some 1e6 on.
__device__ __forceinline__ float pt_tri_d2(float3 p, float3 a, float3 b, float3 c) {
  const float3 ab = b - a, bc = c - b, ca = a - c;
  float d2 = fminf(seg_d2(p, a, ab), fminf(seg_d2(p, b, bc), seg_d2(p, c, ca)));
  const float size = fmaxf(fmaxf(fmaxf(fabsf(ab.x), fabsf(ab.y)), fmaxf(fabsf(ab.z), fabsf(ca.x))),
                           fmaxf(fabsf(ca.y), fabsf(ca.z)));
  const float inv = 1.f / size;
  const float3 u = ab * inv, v = bc * inv, w = ca * inv, n = cross3f(w, u);
  const float nn = dot3f(n, n);
  if (nn > 0.f) {
    const float s1 = dot3f(cross3f(u, p - a), n);
    const float s2 = dot3f(cross3f(v, p - b), n);
    const float s3 = dot3f(cross3f(w, p - c), n);
    if (s1 >= 0.f && s2 >= 0.f && s3 >= 0.f) {
      const float pd = dot3f(p - a, n) / sqrtf(nn);
      d2 = fminf(d2, pd * pd);
    }
  }
  return d2;
}

// Oriented box of an LBVH child subtree (mesh-local FP32).  For every vertex x of the subtree's
// triangles, and so for every point of them, |x . a_k - c_k| <= e_k along the three stored axes
// a_k (the inequality holds in exact arithmetic on the stored FP32 values).  a0..a2 hold
// (a_k.x, a_k.y, a_k.z, c_k), e holds (e_0, e_1, e_2, 0).  A child without a fitted box carries
// extents kNoObb, for which the bound below is 0.
struct __align__(16) OBox {
  float4 a0, a1, a2, e;
};
constexpr float kNoObb = 3.0e38f;

// Squared lower bound on the distance from p to the points of an oriented box: the axes are
// orthonormal to FP32 rounding, so the sum over axes of (|p . a_k - c_k| - e_k)_+^2 is the squared
// distance to the box up to a relative 1e-6 (callers add an absolute margin for it and for the
// rounding of this evaluation).
__device__ __forceinline__ float obox_d2(float3 p, const OBox& o) {
  const float t0 = fabsf(fmaf(p.x, o.a0.x, fmaf(p.y, o.a0.y, fmaf(p.z, o.a0.z, -o.a0.w)))) - o.e.x;
  const float t1 = fabsf(fmaf(p.x, o.a1.x, fmaf(p.y, o.a1.y, fmaf(p.z, o.a1.z, -o.a1.w)))) - o.e.y;
  const float t2 = fabsf(fmaf(p.x, o.a2.x, fmaf(p.y, o.a2.y, fmaf(p.z, o.a2.z, -o.a2.w)))) - o.e.z;
  const float u0 = fmaxf(t0, 0.f), u1 = fmaxf(t1, 0.f), u2 = fmaxf(t2, 0.f);
  return fmaf(u0, u0, fmaf(u1, u1, u2 * u2));
}

// Leaf-ordered FP32 record of one triangle for the unbounded searches (mesh-local; every field rounded
// once from its FP64 value): vertex a, the unit normal n and, for the edges a -> b, b -> c and c -> a,
// the unit in-plane normals m_k pointing into the triangle and the lengths L_k.  With w = p - a the
// in-plane distances of p inside the edge lines are f0 = w.m0, f1 = w.m1 - o1, f2 = w.m2, and the edge
// directions are m_k x n.  A triangle without area is its longest edge: a, m0, n and L0 describe that
// edge's line (n and m0 any normals of it), and the other two edges lie kFlat away (L2 < 0 marks it).
constexpr float kFlat = 1.0e18f;
constexpr int kWeakTri = 1 << 30;  // above every triangle index (at most 2^29)
struct __align__(16) LeafTri {
  float4 a;   // a.xyz, triangle index | kWeakTri when it is not fit for FP32 decisions (int bits)
  float4 n;   // n.xyz, L0
  float4 m0;  // m0.xyz, L1
  float4 m1;  // m1.xyz, o1
  float4 m2;  // m2.xyz, L2
};

// The records of all sorted leaves as five planes of float4 (the fields of LeafTri in order, n per
// plane): the searches read runs of consecutive leaves, a lane per leaf.
struct LeafTris {
  const float4* p;
  int64_t n;
  __device__ __forceinline__ float4 at(int field, int leaf) const { return p[field * n + leaf]; }
  __device__ __forceinline__ LeafTri load(int leaf) const {
    return {at(0, leaf), at(1, leaf), at(2, leaf), at(3, leaf), at(4, leaf)};
  }
};

// The triangle of T as seen from points p0 + d: its plane distance, the distances inside its three edge
// lines and the coordinates along its edges as linear functions of d.
struct LeafView {
  float3 n, m0, m1, m2, u0, u1, u2;
  float bn, f0, f1, f2, g0, g1, g2;  // values at p0
  float L0, L1, L2;
};
__device__ __forceinline__ LeafView leaf_view(const LeafTri& T, float3 p0) {
  LeafView V;
  V.n = f3(T.n); V.m0 = f3(T.m0); V.m1 = f3(T.m1); V.m2 = f3(T.m2);
  V.L0 = T.n.w; V.L1 = T.m0.w; V.L2 = T.m2.w;
  V.u0 = cross3f(V.m0, V.n); V.u1 = cross3f(V.m1, V.n); V.u2 = cross3f(V.m2, V.n);
  const float3 w = p0 - f3(T.a);
  V.bn = dot3f(w, V.n);
  V.f0 = dot3f(w, V.m0); V.f1 = dot3f(w, V.m1) - T.m1.w; V.f2 = dot3f(w, V.m2);
  V.g0 = dot3f(w, V.u0); V.g1 = dot3f(w, V.u1) - V.L0 * dot3f(V.u0, V.u1); V.g2 = dot3f(w, V.u2) + V.L2;
  return V;
}
// Squared distance from p0 + d to the triangle, without division or branch: the plane distance and the
// in-plane one.  With e the squared in-plane distance to the nearest edge, the latter is e outside and
// e - s^2 = 0 inside, where s, the smallest distance inside an edge line, is that same distance.  (A
// point beyond a needle's tip that the rounding puts inside both lines has s far below its distance to
// the edges, so the difference stays its distance whatever the triangle's shape.)  Every rounding is
// relative to |p0 - a| + |d| + the edges.
__device__ __forceinline__ float view_d2(const LeafView& V, float3 d) {
  auto at = [&](float3 g, float c) { return fmaf(g.x, d.x, fmaf(g.y, d.y, fmaf(g.z, d.z, c))); };
  auto edge = [](float f, float g, float L) {
    const float t = fmaxf(fmaxf(-g, g - L), 0.f);
    return fmaf(t, t, __fmul_rn(f, f));
  };
  const float f0 = at(V.m0, V.f0), f1 = at(V.m1, V.f1), f2 = at(V.m2, V.f2), h = at(V.n, V.bn);
  const float e = fminf(fminf(edge(f0, at(V.u0, V.g0), V.L0), edge(f1, at(V.u1, V.g1), V.L1)),
                        edge(f2, at(V.u2, V.g2), V.L2));
  const float s = fmaxf(fminf(fminf(f0, f1), f2), 0.f);
  return fmaf(h, h, fmaxf(__fsub_rn(e, __fmul_rn(s, s)), 0.f));  // inside e is fl(s s): exactly 0
}

// Squared distance from p to the box [lo, hi].
__device__ __forceinline__ float box_d2(float3 p, float3 lo, float3 hi) {
  const float dx = fmaxf(fmaxf(lo.x - p.x, p.x - hi.x), 0.f);
  const float dy = fmaxf(fmaxf(lo.y - p.y, p.y - hi.y), 0.f);
  const float dz = fmaxf(fmaxf(lo.z - p.z, p.z - hi.z), 0.f);
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// Slab test of the half-line o + t d (t >= -tpad) against [lo - pad, hi + pad].  inv holds
// 1/d per axis (inf where d is 0; such axes test containment of o instead).
__device__ __forceinline__ bool ray_box(float3 o, float3 d, float3 inv, float3 lo, float3 hi, float pad,
                                        float tpad) {
  float t0 = -tpad, t1 = 3.0e38f;
  if (d.x != 0.f) {
    float a = (lo.x - pad - o.x) * inv.x, b = (hi.x + pad - o.x) * inv.x;
    t0 = fmaxf(t0, fminf(a, b)); t1 = fminf(t1, fmaxf(a, b));
  } else if (o.x < lo.x - pad || o.x > hi.x + pad) return false;
  if (d.y != 0.f) {
    float a = (lo.y - pad - o.y) * inv.y, b = (hi.y + pad - o.y) * inv.y;
    t0 = fmaxf(t0, fminf(a, b)); t1 = fminf(t1, fmaxf(a, b));
  } else if (o.y < lo.y - pad || o.y > hi.y + pad) return false;
  if (d.z != 0.f) {
    float a = (lo.z - pad - o.z) * inv.z, b = (hi.z + pad - o.z) * inv.z;
    t0 = fmaxf(t0, fminf(a, b)); t1 = fminf(t1, fmaxf(a, b));
  } else if (o.z < lo.z - pad || o.z > hi.z + pad) return false;
  return t0 <= t1 + tpad;
}

}  // namespace sdfgpu
