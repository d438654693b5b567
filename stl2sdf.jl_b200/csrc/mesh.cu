// mesh.cu -- TriangularMesh upload, per-triangle preparation and the LBVH build.
//
// Reference: TriangularMesh (src/MeshGrid/MeshInformations.jl:57-84), prepare_triangle_data
// (src/SignedDistances/dfOnTriangularMesh.jl:329-368) and the two acceleration structures the
// reference builds per call (KD-trees at dfOnTriangularMesh.jl:27,35; ImplicitBVH at
// RaycastingSignDetection.jl:35-56).  Here one LBVH over triangle boxes serves every query that
// is not grid-structured: arbitrary-direction rays, the 3-nearest-vertex fallback and the
// unbounded nearest-triangle search.
//
// LBVH (Karras 2012, "Maximizing parallelism in the construction of BVHs, octrees, and k-d
// trees"): 30-bit Morton codes of the triangle centroids with the triangle index in the low 32
// bits (unique 64-bit keys), a CUB radix sort, one thread per internal node to find its range
// and split, then a bottom-up refit with one atomic counter per internal node.
#include <cstddef>

#include <cub/cub.cuh>

#include "common.cuh"

namespace sdfgpu {

namespace {

// One set of atomics per block: with one per warp they took 35 of 44 us (0.7M vertices).
__global__ void __launch_bounds__(256) k_vertex_bbox(const double* __restrict__ X, int64_t nnp, unsigned long long* bb) {
  __shared__ double s_lo[8][3], s_hi[8][3];
  __shared__ int s_bad;
  if (threadIdx.x == 0) s_bad = 0;
  __syncthreads();
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  bool nonfinite = false;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nnp; v += (int64_t)gridDim.x * blockDim.x) {
    for (int a = 0; a < 3; ++a) {
      const double x = X[3 * v + a];
      if (!isfinite(x)) nonfinite = true;
      lo[a] = fmin(lo[a], x);
      hi[a] = fmax(hi[a], x);
    }
  }
  for (int a = 0; a < 3; ++a) {
    for (int off = 16; off > 0; off >>= 1) {
      lo[a] = fmin(lo[a], __shfl_down_sync(0xffffffffu, lo[a], off));
      hi[a] = fmax(hi[a], __shfl_down_sync(0xffffffffu, hi[a], off));
    }
    if ((threadIdx.x & 31) == 0) {
      s_lo[threadIdx.x >> 5][a] = lo[a];
      s_hi[threadIdx.x >> 5][a] = hi[a];
    }
  }
  if (nonfinite) s_bad = 1;
  __syncthreads();
  if (threadIdx.x < 3) {
    const int a = threadIdx.x;
    double l = s_lo[0][a], h = s_hi[0][a];
    for (int w = 1; w < 8; ++w) {
      l = fmin(l, s_lo[w][a]);
      h = fmax(h, s_hi[w][a]);
    }
    atomicMin(&bb[a], dbl_ord(l));
    atomicMax(&bb[3 + a], dbl_ord(h));
  }
  if (threadIdx.x == 3 && s_bad) atomicOr(&bb[6], 1ULL);
}

// The FP32 record of a triangle (LeafTri, geom32.cuh), computed in FP64 from its FP64 record, mesh-local,
// and rounded once; id: its index, with kWeakTri when it is not fit for FP32 decisions.
__device__ __forceinline__ LeafTri leaf_record(const TriRec64& r, int id, double cx, double cy, double cz) {
  const double* v = r.v;
  const double e0[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
  const double e1[3] = {v[6] - v[0], v[7] - v[1], v[8] - v[2]};
  const double e2[3] = {v[6] - v[3], v[7] - v[4], v[8] - v[5]};
  const double l0 = e0[0] * e0[0] + e0[1] * e0[1] + e0[2] * e0[2];
  const double l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
  const double l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
  const double nx = e0[1] * e1[2] - e0[2] * e1[1], ny = e0[2] * e1[0] - e0[0] * e1[2], nz = e0[0] * e1[1] - e0[1] * e1[0];
  const double nn = nx * nx + ny * ny + nz * nz;
  LeafTri T;
  T.a = make_float4((float)(v[0] - cx), (float)(v[1] - cy), (float)(v[2] - cz), __int_as_float(id));
  if (nn > 1e-20 * l0 * l1) {
    // inward in-plane edge normals: n x (unit edge), edges a->b, b->c, c->a; with the area above 1e-10 of the
    // edges' product, n is normal to the edges within 1e-5 and these are unit vectors within 1e-10
    double m[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double* u = r.u + 3 * k;
      m[k][0] = r.n[1] * u[2] - r.n[2] * u[1];
      m[k][1] = r.n[2] * u[0] - r.n[0] * u[2];
      m[k][2] = r.n[0] * u[1] - r.n[1] * u[0];
    }
    T.n = make_float4((float)r.n[0], (float)r.n[1], (float)r.n[2], (float)r.L[0]);
    T.m0 = make_float4((float)m[0][0], (float)m[0][1], (float)m[0][2], (float)r.L[1]);
    T.m1 = make_float4((float)m[1][0], (float)m[1][1], (float)m[1][2],
                       (float)(e0[0] * m[1][0] + e0[1] * m[1][1] + e0[2] * m[1][2]));
    T.m2 = make_float4((float)m[2][0], (float)m[2][1], (float)m[2][2], (float)r.L[2]);
  } else {  // no area: the longest edge (see LeafTri)
    const int k = l0 >= l1 && l0 >= l2 ? 0 : (l1 >= l2 ? 2 : 1);  // edge a->b, c->a or b->c
    const double len = sqrt(k == 0 ? l0 : (k == 1 ? l2 : l1));
    double u[3], o[3];  // the edge's direction, and its origin: b along b->c, else a
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double d = k == 0 ? e0[q] : (k == 1 ? e2[q] : e1[q]);
      u[q] = len > 0.0 ? d / len : (q == 0 ? 1.0 : 0.0);
      o[q] = k == 1 ? v[3 + q] : v[q];
    }
    // n: the coordinate axis least along u, made normal to it
    const int j = fabs(u[0]) <= fabs(u[1]) && fabs(u[0]) <= fabs(u[2]) ? 0 : (fabs(u[1]) <= fabs(u[2]) ? 1 : 2);
    const double uj = j == 0 ? u[0] : (j == 1 ? u[1] : u[2]);
    double un[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) un[q] = (q == j ? 1.0 : 0.0) - uj * u[q];
    const double rn = 1.0 / sqrt(un[0] * un[0] + un[1] * un[1] + un[2] * un[2]);
#pragma unroll
    for (int q = 0; q < 3; ++q) un[q] *= rn;
    T.a = make_float4((float)(o[0] - cx), (float)(o[1] - cy), (float)(o[2] - cz), __int_as_float(id));
    T.n = make_float4((float)un[0], (float)un[1], (float)un[2], (float)len);
    T.m0 = make_float4((float)(un[1] * u[2] - un[2] * u[1]), (float)(un[2] * u[0] - un[0] * u[2]),
                       (float)(un[0] * u[1] - un[1] * u[0]), k == 1 ? 1.f : 0.f);
    T.m1 = make_float4(0.f, 0.f, 0.f, kFlat);
    T.m2 = make_float4(0.f, 0.f, 0.f, -kFlat);
  }
  return T;
}

// The per-triangle data of a mesh, one thread per triangle: the FP64 record (dfOnTriangularMesh.jl:329-368)
// with the barycentric factorization, the centroid, and mesh-local FP32 copies: vertices, centroid,
// outward-rounded box and the FP32 record.
// v32[3*el+k].w carries the global (0-based) index of vertex k; c32[el].w is 1 when the triangle
// is well conditioned for FP32 decisions (no edge shorter than 1e-5 E, sine of the smallest
// angle above ~1e-3, distinct vertices) and 0 when every decision on it must be made in FP64; rho_ord
// receives rho = max vertex distance from the centroid (decides whether the centroid rule can miss a
// triangle within h), the same over such unfit triangles only, and their number.  tri32: the triangles'
// FP32 records (LeafTris by triangle index).  bb: k_vertex_bbox's result, from which every thread forms the
// centre and E as the host does.
//
// Bound: the 544 bytes a triangle it writes.  The records go through shared memory, a warp's at a time, so
// that each store instruction fills whole lines: written by their own threads, 16 bytes at a stride of 336, they
// and the pass that read them back for the FP32 copies took 0.51 ms on 1.43M triangles and 2.04 ms on 5.8M
// (B200), against 0.20 and 0.70 ms.  An odd stride in doubles keeps both sides free of bank conflicts.
constexpr int kPrepThreads = 128;
constexpr int kRecDoubles = sizeof(TriRec64) / 8, kRecStride = kRecDoubles + 1;
static_assert(sizeof(TriRec64) % 16 == 0 && kRecStride % 2 == 1, "records are copied 16 bytes at a time");
// A warp's stage: 32 records, or the FP32 copies as float4.
struct __align__(16) PrepStage {
  double d[32 * kRecStride];
};
static_assert(sizeof(PrepStage) % sizeof(float4) == 0 && alignof(PrepStage) >= alignof(float4) &&
                  sizeof(PrepStage) >= 5 * 32 * sizeof(float4),
              "the stage holds five float4 a triangle");
__global__ void __launch_bounds__(kPrepThreads) k_prep(const double* __restrict__ X, int64_t nnp,
                                                       const int64_t* __restrict__ IEN, int64_t nel,
                                                       const unsigned long long* __restrict__ bb,
                                                       TriRec64* __restrict__ rec, double4* __restrict__ cent,
                                                       float4* __restrict__ v32, float4* __restrict__ c32,
                                                       float4* __restrict__ box32, float4* __restrict__ tri32,
                                                       unsigned long long* bad, unsigned long long* rho_ord) {
  __shared__ PrepStage s_rec[kPrepThreads / 32];
  const int lane = threadIdx.x & 31;
  double* stage = s_rec[threadIdx.x >> 5].d;
  double ctr[3], E = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double lo = ord_dbl(bb[a]), hi = ord_dbl(bb[3 + a]);
    ctr[a] = dm(0.5, da(lo, hi));
    E = fmax(E, fmax(ds(hi, ctr[a]), ds(ctr[a], lo)));
  }
  double rho2 = 0.0, rho2_weak = 0.0;
  unsigned weak = 0u;
  for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; base < nel;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t el = base + lane;
    const int count = (int)min((int64_t)32, nel - base);
    TriRec64 r;
    if (lane < count) {
      d3 v[3];
      int32_t gid[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        int64_t vi = IEN[3 * el + k];
        if (vi < 1 || vi > nnp) {
          atomicOr(bad, 2ULL);
          vi = 1;
        }
        vi -= 1;
        gid[k] = (int32_t)vi;
        v[k] = {X[3 * vi], X[3 * vi + 1], X[3 * vi + 2]};
        r.v[3 * k] = v[k].x; r.v[3 * k + 1] = v[k].y; r.v[3 * k + 2] = v[k].z;
      }
      const d3 e[3] = {v_sub(v[1], v[0]), v_sub(v[2], v[1]), v_sub(v[0], v[2])};
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        r.L[j] = v_norm(e[j]);
        const d3 u = v_div(e[j], r.L[j]);
        r.u[3 * j] = u.x; r.u[3 * j + 1] = u.y; r.u[3 * j + 2] = u.z;
      }
      const d3 nn = v_cross(e[0], v_neg(e[2]));
      const double area2 = v_norm(nn);
      const d3 n = v_div(nn, area2);
      r.n[0] = n.x; r.n[1] = n.y; r.n[2] = n.z;
      const d3 c = v_div(v_add(v_add(v[0], v[1]), v[2]), 3.0);
      r.bmin[0] = fmin(v[0].x, fmin(v[1].x, v[2].x));
      r.bmin[1] = fmin(v[0].y, fmin(v[1].y, v[2].y));
      r.bmin[2] = fmin(v[0].z, fmin(v[1].z, v[2].z));
      r.bmax[0] = fmax(v[0].x, fmax(v[1].x, v[2].x));
      r.bmax[1] = fmax(v[0].y, fmax(v[1].y, v[2].y));
      r.bmax[2] = fmax(v[0].z, fmax(v[1].z, v[2].z));
      r.pad = 0;
      cent[el] = make_double4(c.x, c.y, c.z, 0.0);
      double rt2 = 0.0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double dx = v[k].x - c.x, dy = v[k].y - c.y, dz = v[k].z - c.z;
        rt2 = fmax(rt2, dx * dx + dy * dy + dz * dz);
      }
      rho2 = fmax(rho2, rt2);
      const double lmin = fmin(r.L[0], fmin(r.L[1], r.L[2])), lmax = fmax(r.L[0], fmax(r.L[1], r.L[2]));
      const bool ok = lmin > 1e-5 * E && area2 > 1e-3 * lmax * lmax && gid[0] != gid[1] && gid[1] != gid[2] &&
                      gid[0] != gid[2];
      if (!ok) {
        ++weak;
        rho2_weak = fmax(rho2_weak, rt2);
      }
      c32[el] = make_float4((float)(c.x - ctr[0]), (float)(c.y - ctr[1]), (float)(c.z - ctr[2]), ok ? 1.f : 0.f);
      const LeafTri T = leaf_record(r, ok ? (int)el : (int)el | kWeakTri, ctr[0], ctr[1], ctr[2]);
      const float4 f[5] = {T.a, T.n, T.m0, T.m1, T.m2};
#pragma unroll
      for (int k = 0; k < 5; ++k) tri32[(int64_t)k * nel + el] = f[k];
      // vertices and box, staged: 3 and 2 float4 a triangle
      float4* f4 = reinterpret_cast<float4*>(stage);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        f4[3 * lane + k] = make_float4((float)(v[k].x - ctr[0]), (float)(v[k].y - ctr[1]), (float)(v[k].z - ctr[2]),
                                       __int_as_float(gid[k]));
      f4[96 + 2 * lane] = make_float4(__double2float_rd(r.bmin[0] - ctr[0]), __double2float_rd(r.bmin[1] - ctr[1]),
                                      __double2float_rd(r.bmin[2] - ctr[2]), 0.f);
      f4[96 + 2 * lane + 1] = make_float4(__double2float_ru(r.bmax[0] - ctr[0]), __double2float_ru(r.bmax[1] - ctr[1]),
                                          __double2float_ru(r.bmax[2] - ctr[2]), 0.f);
      factor_bary(r);
    }
    __syncwarp();
    {
      const float4* f4 = reinterpret_cast<const float4*>(stage);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (32 * k + lane < 3 * count) v32[3 * base + 32 * k + lane] = f4[32 * k + lane];
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (32 * k + lane < 2 * count) box32[2 * base + 32 * k + lane] = f4[96 + 32 * k + lane];
    }
    __syncwarp();
    if (lane < count) {
      double* o = stage + kRecStride * lane;
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        o[q] = r.v[q];
        o[9 + q] = r.u[q];
        o[30 + q] = r.A[q];
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        o[18 + q] = r.L[q];
        o[21 + q] = r.n[q];
        o[24 + q] = r.bmin[q];
        o[27 + q] = r.bmax[q];
      }
      o[39] = __hiloint2double(r.imax, r.kind);
      o[40] = __hiloint2double(r.pad, r.piv);
      o[41] = 0.0;
    }
    __syncwarp();
    double2* out = reinterpret_cast<double2*>(rec + base);
    for (int q = lane; q < count * (kRecDoubles / 2); q += 32) {
      const int s = 2 * q + q / (kRecDoubles / 2);
      out[q] = make_double2(stage[s], stage[s + 1]);
    }
    __syncwarp();
  }
  double rho = sqrt(rho2), rho_weak = sqrt(rho2_weak);
  for (int off = 16; off > 0; off >>= 1) {
    rho = fmax(rho, __shfl_down_sync(0xffffffffu, rho, off));
    rho_weak = fmax(rho_weak, __shfl_down_sync(0xffffffffu, rho_weak, off));
    weak += __shfl_down_sync(0xffffffffu, weak, off);
  }
  if (lane == 0) {
    atomicMax(rho_ord, dbl_ord(rho * (1.0 + 1e-12)));
    if (weak) {
      atomicMax(rho_ord + 1, dbl_ord(rho_weak * (1.0 + 1e-12)));
      atomicAdd(rho_ord + 2, (unsigned long long)weak);
    }
  }
}
static_assert(offsetof(TriRec64, u) == 9 * 8 && offsetof(TriRec64, L) == 18 * 8 && offsetof(TriRec64, n) == 21 * 8 &&
                  offsetof(TriRec64, bmin) == 24 * 8 && offsetof(TriRec64, bmax) == 27 * 8 && offsetof(TriRec64, A) == 30 * 8 &&
                  offsetof(TriRec64, kind) == 39 * 8 && offsetof(TriRec64, imax) == 39 * 8 + 4 &&
                  offsetof(TriRec64, piv) == 40 * 8 && offsetof(TriRec64, pad) == 40 * 8 + 4 && kRecDoubles == 42,
              "k_prep stages the record by double");

__device__ __forceinline__ unsigned expand_bits10(unsigned v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

// 30-bit Morton code of each centroid and the triangle index; a stable sort of the codes (index as
// the value) orders the triangles exactly as the unique 64-bit keys (code << 32 | index) would, in
// half the radix passes.
__global__ void k_morton(const float4* __restrict__ c32, int64_t nel, float lox, float loy, float loz, float inv,
                         uint32_t* __restrict__ code, int32_t* __restrict__ idx) {
  for (int64_t el = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; el < nel; el += (int64_t)gridDim.x * blockDim.x) {
    const float4 c = c32[el];
    const float fx = fminf(fmaxf((c.x - lox) * inv, 0.f), 1023.f);
    const float fy = fminf(fmaxf((c.y - loy) * inv, 0.f), 1023.f);
    const float fz = fminf(fmaxf((c.z - loz) * inv, 0.f), 1023.f);
    code[el] = (expand_bits10((unsigned)fx) << 2) | (expand_bits10((unsigned)fy) << 1) | expand_bits10((unsigned)fz);
    idx[el] = (int32_t)el;
  }
}

// The sorted unique keys (code << 32 | index) the hierarchy build splits on.
__global__ void k_pack_keys(const uint32_t* __restrict__ code, const int32_t* __restrict__ idx, int n,
                            unsigned long long* __restrict__ keys) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    keys[i] = ((unsigned long long)code[i] << 32) | (unsigned long long)(uint32_t)idx[i];
}

__device__ __forceinline__ int kdelta(const unsigned long long* __restrict__ k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  return __clzll(k[i] ^ k[j]);
}

__global__ void k_karras(const unsigned long long* __restrict__ keys, int n, BNode* __restrict__ nodes,
                         int32_t* __restrict__ int_parent, int32_t* __restrict__ leaf_parent) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
    const int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = kdelta(keys, n, i, i - d);
    int lmax = 2;
    while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
      if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = kdelta(keys, n, i, j);
    int s = 0, t = l;
    while (true) {
      t = (t + 1) >> 1;
      if (kdelta(keys, n, i, i + (s + t) * d) > dnode) s += t;
      if (t <= 1) break;
    }
    const int gamma = i + s * d + (d < 0 ? -1 : 0);
    const int lo = min(i, j), hi = max(i, j);
    int left, right;
    if (lo == gamma) { left = kLeafBit | gamma; leaf_parent[gamma] = i; }
    else { left = gamma; int_parent[gamma] = i; }
    if (hi == gamma + 1) { right = kLeafBit | (gamma + 1); leaf_parent[gamma + 1] = i; }
    else { right = gamma + 1; int_parent[gamma + 1] = i; }
    // d.z, d.w: the node's range of sorted leaves [lo, hi]; its left child covers [lo, gamma] and its
    // right child [gamma + 1, hi], so a parent tells the size of both children's subtrees.
    nodes[i].d = make_int4(left, right, lo, hi);
  }
}

__global__ void k_refit(const unsigned long long* __restrict__ keys, const float4* __restrict__ box32, int n,
                        BNode* nodes, const int32_t* __restrict__ int_parent, const int32_t* __restrict__ leaf_parent,
                        int32_t* flags, int32_t* __restrict__ leaf_prim) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int prim = (int)(keys[i] & 0xffffffffULL);
    leaf_prim[i] = prim;
    float4 lo = box32[2 * prim], hi = box32[2 * prim + 1];
    int child = kLeafBit | i;
    int node = leaf_parent[i];
    int guard = 0;
    while (node >= 0 && ++guard <= 128) {  // LBVH depth <= 64 for unique 64-bit keys
      float* f = reinterpret_cast<float*>(&nodes[node]);
      const int left = __ldcg(reinterpret_cast<const int*>(&nodes[node].d.x));
      const int slot = (left == child) ? 0 : 6;
      __stcg(f + slot + 0, lo.x); __stcg(f + slot + 1, lo.y); __stcg(f + slot + 2, lo.z);
      __stcg(f + slot + 3, hi.x); __stcg(f + slot + 4, hi.y); __stcg(f + slot + 5, hi.z);
      __threadfence();
      if (atomicAdd(&flags[node], 1) == 0) break;
      __threadfence();
      float b[12];
      for (int q = 0; q < 12; ++q) b[q] = __ldcg(f + q);
      lo = make_float4(fminf(b[0], b[6]), fminf(b[1], b[7]), fminf(b[2], b[8]), 0.f);
      hi = make_float4(fmaxf(b[3], b[9]), fmaxf(b[4], b[10]), fmaxf(b[5], b[11]), 0.f);
      child = node;
      node = int_parent[node];
    }
  }
}

// A single-triangle mesh: root with the leaf on the left and an empty box on the right.
__global__ void k_single_root(const float4* __restrict__ box32, BNode* nodes, int32_t* leaf_prim) {
  const float4 lo = box32[0], hi = box32[1];
  BNode nd;
  nd.a = make_float4(lo.x, lo.y, lo.z, hi.x);
  nd.b = make_float4(hi.y, hi.z, 3.0e38f, 3.0e38f);
  nd.c = make_float4(3.0e38f, -3.0e38f, -3.0e38f, -3.0e38f);
  nd.d = make_int4(kLeafBit | 0, kLeafBit | 0, 0, 0);
  nodes[0] = nd;
  leaf_prim[0] = 0;
}

// Leaf-ordered copies for the unbounded searches and the oriented-box fit, which read the triangles of
// runs of consecutive leaves: the FP32 vertices (3 x float4, as v32) and the LeafTri record.
__global__ void k_leaf_order(const int32_t* __restrict__ leaf_prim, const float4* __restrict__ v32,
                             const float4* __restrict__ tri32, int n, float4* __restrict__ lv32,
                             float4* __restrict__ ltri) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int64_t prim = leaf_prim[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) lv32[3 * (int64_t)i + k] = v32[3 * prim + k];
#pragma unroll
    for (int k = 0; k < 5; ++k) ltri[(int64_t)k * n + i] = tri32[(int64_t)k * n + prim];
  }
}

// Eigenvectors of the symmetric 3x3 matrix A (cyclic Jacobi rotations in FP32, at most 8 sweeps):
// the columns of V, orthonormal to a few FP32 roundings.
__device__ void jacobi3f(float A[3][3], float V[3][3]) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) V[i][j] = i == j ? 1.f : 0.f;
#pragma unroll 1
  for (int sweep = 0; sweep < 8; ++sweep) {
    const float off = fabsf(A[0][1]) + fabsf(A[0][2]) + fabsf(A[1][2]);
    const float diag = fabsf(A[0][0]) + fabsf(A[1][1]) + fabsf(A[2][2]);
    if (!(off > 1e-7f * diag)) break;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int p = r == 2 ? 1 : 0, q = r == 0 ? 1 : 2;
      const float apq = A[p][q];
      if (apq == 0.f) continue;
      const float th = (A[q][q] - A[p][p]) / (2.f * apq);
      const float t = copysignf(1.f, th) / (fabsf(th) + sqrtf(fmaf(th, th, 1.f)));
      const float c = rsqrtf(fmaf(t, t, 1.f)), sn = t * c;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float akp = A[k][p], akq = A[k][q];
        A[k][p] = c * akp - sn * akq;
        A[k][q] = sn * akp + c * akq;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float apk = A[p][k], aqk = A[q][k];
        A[p][k] = c * apk - sn * aqk;
        A[q][k] = sn * apk + c * aqk;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float vkp = V[k][p], vkq = V[k][q];
        V[k][p] = c * vkp - sn * vkq;
        V[k][q] = sn * vkp + c * vkq;
      }
    }
  }
}

// The oriented box of the leaves [first, first + cnt) (see k_obb): kLanes neighbouring lanes share the
// loops over the vertices and all return the same box.
// kLanes above 32: a CTA of that many threads, through `red`.
template <int kLanes, class Op>
__device__ __forceinline__ double obb_reduce(double v, Op op, unsigned group, double* red) {
  for (int off = (kLanes < 32 ? kLanes : 32) / 2; off > 0; off >>= 1) v = op(v, __shfl_xor_sync(group, v, off));
  if (kLanes > 32) {
    __syncthreads();  // the last use of red is over
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
    for (int w = 1; w < kLanes / 32; ++w) v = op(v, red[w]);
  }
  return v;
}

template <int kLanes>
__device__ OBox fit_obox(const float4* __restrict__ lv32, int first, int cnt, double E, int lane, unsigned group,
                         double* red) {
  const int step = kLanes, start = first + lane, end = first + cnt;
  const float4 r4 = lv32[3 * first];
  const double rx = r4.x, ry = r4.y, rz = r4.z;
  double s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // sums of x, y, z, xx, xy, xz, yy, yz, zz about the first vertex
  for (int l = start; l < end; l += step)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 v = lv32[3 * l + k];
      const double x = v.x - rx, y = v.y - ry, z = v.z - rz;
      s[0] += x; s[1] += y; s[2] += z;
      s[3] = fma(x, x, s[3]); s[4] = fma(x, y, s[4]); s[5] = fma(x, z, s[5]);
      s[6] = fma(y, y, s[6]); s[7] = fma(y, z, s[7]); s[8] = fma(z, z, s[8]);
    }
#pragma unroll
  for (int k = 0; k < 9; ++k) s[k] = obb_reduce<kLanes>(s[k], [](double x, double y) { return x + y; }, group, red);
  const double nv = 3.0 * cnt, mx = s[0] / nv, my = s[1] / nv, mz = s[2] / nv;
  const double c00 = s[3] / nv - mx * mx, c01 = s[4] / nv - mx * my, c02 = s[5] / nv - mx * mz;
  const double c11 = s[6] / nv - my * my, c12 = s[7] / nv - my * mz, c22 = s[8] / nv - mz * mz;
  const double tr = c00 + c11 + c22;
  double ax[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  if (tr > 0.0) {  // principal axes of the trace-normalised covariance (FP32 is enough for a direction)
    const double inv = 1.0 / tr;
    float A[3][3] = {{(float)(c00 * inv), (float)(c01 * inv), (float)(c02 * inv)},
                     {(float)(c01 * inv), (float)(c11 * inv), (float)(c12 * inv)},
                     {(float)(c02 * inv), (float)(c12 * inv), (float)(c22 * inv)}};
    float V[3][3];
    jacobi3f(A, V);
    // Gram-Schmidt in FP64: the axes are orthonormal to FP64 rounding before they are stored in FP32
    double a[3] = {V[0][0], V[1][0], V[2][0]}, b[3] = {V[0][1], V[1][1], V[2][1]};
    const double na = 1.0 / sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    for (int k = 0; k < 3; ++k) a[k] *= na;
    const double ab = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
    for (int k = 0; k < 3; ++k) b[k] -= ab * a[k];
    const double bb = b[0] * b[0] + b[1] * b[1] + b[2] * b[2];
    if (bb > 1e-12) {
      const double nb = 1.0 / sqrt(bb);
      for (int k = 0; k < 3; ++k) {
        ax[0][k] = a[k];
        ax[1][k] = b[k] * nb;
      }
      ax[2][0] = ax[0][1] * ax[1][2] - ax[0][2] * ax[1][1];
      ax[2][1] = ax[0][2] * ax[1][0] - ax[0][0] * ax[1][2];
      ax[2][2] = ax[0][0] * ax[1][1] - ax[0][1] * ax[1][0];
    }
  }
  float af[3][3];
  for (int a = 0; a < 3; ++a)
    for (int k = 0; k < 3; ++k) af[a][k] = (float)ax[a][k];
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int l = start; l < end; l += step)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float4 v = lv32[3 * l + k];
#pragma unroll
      for (int a = 0; a < 3; ++a) {  // float x float products are exact in FP64
        const double t = (double)v.x * af[a][0] + (double)v.y * af[a][1] + (double)v.z * af[a][2];
        lo[a] = fmin(lo[a], t);
        hi[a] = fmax(hi[a], t);
      }
    }
  OBox o;
  float ce[3], ex[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = obb_reduce<kLanes>(lo[a], [](double x, double y) { return fmin(x, y); }, group, red);
    hi[a] = obb_reduce<kLanes>(hi[a], [](double x, double y) { return fmax(x, y); }, group, red);
    const double c = 0.5 * (lo[a] + hi[a]);
    ce[a] = (float)c;
    // the FP64 sums above round by at most ~1e-15 E; the margin 1e-9 E covers them
    ex[a] = __double2float_ru(0.5 * (hi[a] - lo[a]) + fabs(c - (double)ce[a]) + 1e-9 * E);
  }
  o.a0 = make_float4(af[0][0], af[0][1], af[0][2], ce[0]);
  o.a1 = make_float4(af[1][0], af[1][1], af[1][2], ce[1]);
  o.a2 = make_float4(af[2][0], af[2][1], af[2][2], ce[2]);
  o.e = make_float4(ex[0], ex[1], ex[2], 0.f);
  return o;
}

// The child `side` of inner node i covers the sorted leaves [first, first + cnt): the left child
// [d.z, gamma], the right [gamma + 1, d.w].
__device__ __forceinline__ void child_range(const BNode* nodes, int i, int side, int& first, int& cnt) {
  const int4 d = nodes[i].d;
  const int gamma = d.x & 0x7fffffff;
  first = side ? gamma + 1 : d.z;
  cnt = side ? d.w - gamma : gamma - d.z + 1;
}

// Oriented boxes of the LBVH's children (OBox, two per inner node: obb[2 i + side]).  For each child
// subtree of 2..kObbMaxLeaves leaves (a contiguous run of the Morton-sorted leaves) the principal
// axes of its vertices -- the FP64 covariance about the run's first vertex, diagonalised by Jacobi
// rotations -- and then the exact extents of its FP32 vertices along the axes as stored.  The axes
// only decide how tight the box is; the extents make it a bound for whatever axes come out.  On a
// smooth surface the smallest axis is the patch normal and the box is a thin slab around the patch,
// so a point at distance D from the surface has a lower bound close to D for every patch away from
// its nearest point (an axis-aligned box of a tilted patch is as thick as the patch is wide).
// Leaves and larger subtrees get kNoObb.  One thread fits a child of up to kObbThread leaves, kObbLanes
// lanes one of up to kObbGroup, a CTA of kObbCta threads a larger one, from lists that k_obb_small writes:
// the diagonalisation is redundant work of all threads of a child, and the loops over the vertices are the
// serial chain.  Measured on 131k and 1.43M triangles (B200): 114 and 929 us together, against 226 and 1320
// with a thread for up to 32 leaves and a warp for the rest, which the largest children bound.
constexpr int kObbThread = 12, kObbLanes = 8, kObbGroup = 128, kObbCta = 128;

__global__ void k_obb_small(const BNode* __restrict__ nodes, const float4* __restrict__ lv32, int n_inner, double E,
                            OBox* __restrict__ obb, int32_t* __restrict__ list, int32_t* __restrict__ list_n) {
  const int lane = threadIdx.x & 31;
  for (int base = blockIdx.x * blockDim.x; base < 2 * n_inner; base += gridDim.x * blockDim.x) {
    const int ci = base + threadIdx.x;
    int first = 0, cnt = 0;
    if (ci < 2 * n_inner) child_range(nodes, ci >> 1, ci & 1, first, cnt);
    // lists: children for a group from the front, for a CTA from the back
    const bool fit = cnt >= 2 && cnt <= kObbMaxLeaves, wide = fit && cnt > kObbThread, big = wide && cnt > kObbGroup;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bool mine = wide && big == (k == 1);
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      if (!m) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(list_n + k, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
      if (mine) list[k == 0 ? at : 2 * n_inner - 1 - at] = ci;
    }
    if (ci >= 2 * n_inner || wide) continue;
    OBox o;
    if (fit) {
      o = fit_obox<1>(lv32, first, cnt, E, 0, 0u, nullptr);
    } else {
      o.a0 = make_float4(1.f, 0.f, 0.f, 0.f);
      o.a1 = make_float4(0.f, 1.f, 0.f, 0.f);
      o.a2 = make_float4(0.f, 0.f, 1.f, 0.f);
      o.e = make_float4(kNoObb, kNoObb, kNoObb, 0.f);
    }
    obb[ci] = o;
  }
}

// The listed children: blocks below `split` of the grid take the group list, the others the CTA list.
__global__ void __launch_bounds__(kObbCta) k_obb_large(const BNode* __restrict__ nodes, const float4* __restrict__ lv32,
                                                       int n_inner, double E, OBox* __restrict__ obb,
                                                       const int32_t* __restrict__ list,
                                                       const int32_t* __restrict__ list_n, int split) {
  __shared__ double red[kObbCta / 32];
  int first, cnt;
  if ((int)blockIdx.x >= split) {
    for (int q = blockIdx.x - split; q < list_n[1]; q += gridDim.x - split) {
      const int ci = list[2 * n_inner - 1 - q];
      child_range(nodes, ci >> 1, ci & 1, first, cnt);
      const OBox o = fit_obox<kObbCta>(lv32, first, cnt, E, threadIdx.x, 0xffffffffu, red);
      if (threadIdx.x == 0) obb[ci] = o;
    }
    return;
  }
  const int lane = threadIdx.x & (kObbLanes - 1);
  const unsigned group = ((1u << kObbLanes) - 1u) << ((threadIdx.x & 31) - lane);
  for (int q = (blockIdx.x * kObbCta + threadIdx.x) / kObbLanes; q < list_n[0]; q += split * kObbCta / kObbLanes) {
    const int ci = list[q];
    child_range(nodes, ci >> 1, ci & 1, first, cnt);
    const OBox o = fit_obox<kObbLanes>(lv32, first, cnt, E, lane, group, nullptr);
    if (lane == 0) obb[ci] = o;
  }
}

__global__ void k_ine_count(const int64_t* __restrict__ IEN, int64_t nel, int32_t* __restrict__ cnt) {
  for (int64_t el = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; el < nel; el += (int64_t)gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) atomicAdd(&cnt[IEN[3 * el + k] - 1], 1);
}

__global__ void k_ine_fill(const int64_t* __restrict__ IEN, int64_t nel, const int32_t* __restrict__ off,
                           int32_t* __restrict__ cur, int32_t* __restrict__ ine) {
  for (int64_t el = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; el < nel; el += (int64_t)gridDim.x * blockDim.x)
    for (int k = 0; k < 3; ++k) {
      const int64_t v = IEN[3 * el + k] - 1;
      ine[off[v] + atomicAdd(&cur[v], 1)] = (int32_t)el;
    }
}

}  // namespace

// The LBVH of the resident mesh and, with `boxes`, its oriented child boxes, built on first use on a stream
// of their own: only the unbounded searches, the 3-nearest-vertex fallback (both with the boxes) and the
// adaptive rays of many nodes read them, and wait for ev_obb or ev_bvh; the clamped distances and the
// axis rays do not.  (Building them for every mesh took a third of a reference-rule call on 1.4M
// triangles.)  set_mesh enqueues at once what the last mesh's calls used (ctx->tree_used), so that a
// program of unbounded calls overlaps the build as before.
static int build_tree(sdfgpu_ctx* ctx, bool boxes) {
  MeshDev& M = ctx->mesh;
  ctx->tree_used = std::max(ctx->tree_used, boxes ? 2 : 1);
  const int64_t nel = M.nel;
  const int n = (int)nel;
  cudaStream_t sb = ctx->bvh_stream;
  BNode* nodes = buf<BNode>(ctx, "nodes");
  float4* lv32 = buf<float4>(ctx, "lv32");
  if (M.tree < 1) {
    float4 *v32 = buf<float4>(ctx, "v32"), *c32 = buf<float4>(ctx, "c32"), *box32 = buf<float4>(ctx, "box32"),
           *tri32 = buf<float4>(ctx, "tri32");
    SDF_CUDA(ctx, cudaStreamWaitEvent(sb, ctx->ev_mesh, 0));
    unsigned long long* keys2;
    int32_t *int_parent, *leaf_parent, *flags, *leaf_prim;
    SDF_TRY(scratch_t(ctx, "keys2", (size_t)n, &keys2));
    SDF_TRY(scratch_t(ctx, "nodes", (size_t)std::max(1, n - 1), &nodes));
    SDF_TRY(scratch_t(ctx, "int_parent", (size_t)n, &int_parent));
    SDF_TRY(scratch_t(ctx, "leaf_parent", (size_t)n, &leaf_parent));
    SDF_TRY(scratch_t(ctx, "flags", (size_t)n, &flags));
    SDF_TRY(scratch_t(ctx, "leaf_prim", (size_t)n, &leaf_prim));
    if (n == 1) {
      k_single_root<<<1, 1, 0, sb>>>(box32, nodes, leaf_prim);
      SDF_KERNEL(ctx);
    } else {
      const float lox = (float)(M.bmin[0] - M.center[0]), loy = (float)(M.bmin[1] - M.center[1]),
                  loz = (float)(M.bmin[2] - M.center[2]);
      const double ext = std::max(M.bmax[0] - M.bmin[0], std::max(M.bmax[1] - M.bmin[1], M.bmax[2] - M.bmin[2]));
      const float inv = ext > 0 ? (float)(1024.0 / ext) : 1.0f;
      uint32_t *code, *code2;
      int32_t *idx, *idx2;
      SDF_TRY(scratch_t(ctx, "mcode", (size_t)n, &code));
      SDF_TRY(scratch_t(ctx, "mcode2", (size_t)n, &code2));
      SDF_TRY(scratch_t(ctx, "midx", (size_t)n, &idx));
      SDF_TRY(scratch_t(ctx, "midx2", (size_t)n, &idx2));
      k_morton<<<grid_for(nel, 256), 256, 0, sb>>>(c32, nel, lox, loy, loz, inv, code, idx);
      SDF_KERNEL(ctx);
      size_t tmp_bytes = 0;
      SDF_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, code, code2, idx, idx2, n, 0, 30, sb));
      void* tmp;
      SDF_TRY(scratch(ctx, "cub_tmp_bvh", tmp_bytes, &tmp));
      SDF_CUDA(ctx, cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, code, code2, idx, idx2, n, 0, 30, sb));
      k_pack_keys<<<grid_for(n, 256), 256, 0, sb>>>(code2, idx2, n, keys2);
      SDF_KERNEL(ctx);
      SDF_CUDA(ctx, cudaMemsetAsync(int_parent, 0xff, sizeof(int32_t) * n, sb));
      SDF_CUDA(ctx, cudaMemsetAsync(flags, 0, sizeof(int32_t) * n, sb));
      k_karras<<<grid_for(n - 1, 256), 256, 0, sb>>>(keys2, n, nodes, int_parent, leaf_parent);
      SDF_KERNEL(ctx);
      k_refit<<<grid_for(n, 256), 256, 0, sb>>>(keys2, box32, n, nodes, int_parent, leaf_parent, flags, leaf_prim);
      SDF_KERNEL(ctx);
    }
    float4* ltri;  // LeafTris: five planes
    SDF_TRY(scratch_t(ctx, "lv32", (size_t)n * 3, &lv32));
    SDF_TRY(scratch_t(ctx, "ltri", (size_t)n * 5, &ltri));
    k_leaf_order<<<grid_for(n, 256), 256, 0, sb>>>(leaf_prim, v32, tri32, n, lv32, ltri);
    SDF_KERNEL(ctx);
    SDF_CUDA(ctx, cudaEventRecord(ctx->ev_bvh, sb));
    M.tree = 1;
  }
  if (boxes && M.tree < 2) {
    OBox* obb;
    const int n_inner = std::max(1, n - 1);
    SDF_TRY(scratch_t(ctx, "obb", (size_t)2 * n_inner, &obb));
    int32_t* list;  // the children that more than one thread fits, and the lists' lengths
    SDF_TRY(scratch_t(ctx, "obb_list", (size_t)2 * n_inner + 2, &list));
    int32_t* list_n = list + 2 * (int64_t)n_inner;
    SDF_CUDA(ctx, cudaMemsetAsync(list_n, 0, 2 * sizeof(int32_t), sb));
    k_obb_small<<<grid_for(2 * n_inner, 256), 256, 0, sb>>>(nodes, lv32, n_inner, M.E, obb, list, list_n);
    SDF_KERNEL(ctx);
    // half the blocks for each list
    const unsigned blocks = 2 * grid_for(2 * n_inner, kObbCta, 148 * 8);
    k_obb_large<<<blocks, kObbCta, 0, sb>>>(nodes, lv32, n_inner, M.E, obb, list, list_n, (int)blocks / 2);
    SDF_KERNEL(ctx);
    SDF_CUDA(ctx, cudaEventRecord(ctx->ev_obb, sb));
    M.tree = 2;
  }
  return 0;
}

int ensure_tree(sdfgpu_ctx* ctx, bool boxes) {
  const int rc = build_tree(ctx, boxes);
  // no event covers what a failed build has enqueued: wait, so that nothing rewrites its inputs under it
  if (rc != 0) cudaStreamSynchronize(ctx->bvh_stream);
  return rc;
}

int mesh_upload_and_build(sdfgpu_ctx* ctx, const double* X, int64_t nnp, const int64_t* IEN, int64_t nel,
                          bool device_ptrs) {
  cudaStream_t st = ctx->stream;
  if (nel < 1 || nnp < 3) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "mesh needs at least 1 triangle and 3 vertices");
  if (nel > (int64_t)0x7fffffff / 4) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "too many triangles (limit 536870911)");
  if (!X || !IEN) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "X and IEN must not be NULL");
  ctx->has_mesh = false;
  ctx->mesh.ine_ready = false;
  ctx->launches = 0;
  const int eager = ctx->tree_used;  // what the last mesh's calls needed, before set_mesh's own host wait
  ctx->tree_used = 0;
  ctx->mesh.tree = 0;
  // the previous mesh's LBVH build reads the buffers rewritten below
  SDF_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_bvh, 0));
  SDF_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_obb, 0));
  SDF_CUDA(ctx, cudaEventRecord(ctx->ev[4], st));

  double* dX;
  int64_t* dIEN;
  SDF_TRY(scratch_t(ctx, "X64", (size_t)nnp * 3, &dX));
  SDF_TRY(scratch_t(ctx, "IEN64", (size_t)nel * 3, &dIEN));
  const cudaMemcpyKind kind = device_ptrs ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  SDF_CUDA(ctx, cudaMemcpyAsync(dX, X, sizeof(double) * 3 * nnp, kind, st));
  SDF_CUDA(ctx, cudaMemcpyAsync(dIEN, IEN, sizeof(int64_t) * 3 * nel, kind, st));

  TriRec64* rec;
  double4* cent;
  float4 *v32, *c32, *box32;
  unsigned long long* bb;
  SDF_TRY(scratch_t(ctx, "rec", (size_t)nel, &rec));
  SDF_TRY(scratch_t(ctx, "cent64", (size_t)nel, &cent));
  SDF_TRY(scratch_t(ctx, "v32", (size_t)nel * 3, &v32));
  SDF_TRY(scratch_t(ctx, "c32", (size_t)nel, &c32));
  SDF_TRY(scratch_t(ctx, "box32", (size_t)nel * 2, &box32));
  SDF_TRY(scratch_t(ctx, "bbox", 10, &bb));

  float4* tri32;
  SDF_TRY(scratch_t(ctx, "tri32", (size_t)nel * 5, &tri32));

  // box; flags: 1 a vertex not finite, 2 an index out of range; rho, rho of the unfit triangles, their
  // number (0 is below the encoding of every non-negative double)
  unsigned long long init[10] = {~0ULL, ~0ULL, ~0ULL};
  SDF_CUDA(ctx, cudaMemcpyAsync(bb, init, sizeof(init), cudaMemcpyHostToDevice, st));
  k_vertex_bbox<<<grid_for(nnp, 256, 148 * 4), 256, 0, st>>>(dX, nnp, bb);
  SDF_KERNEL(ctx);
  k_prep<<<grid_for(nel, kPrepThreads), kPrepThreads, 0, st>>>(dX, nnp, dIEN, nel, bb, rec, cent, v32, c32, box32, tri32,
                                                              bb + 6, bb + 7);
  SDF_KERNEL(ctx);
  SDF_CUDA(ctx, cudaEventRecord(ctx->ev_mesh, st));
  static_assert(S_COUNTERS - S_MESH >= sizeof(init) / sizeof(init[0]), "the mesh's scalars have page-locked slots");
  SDF_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + S_MESH, bb, sizeof(init), cudaMemcpyDeviceToHost, st));
  SDF_CUDA(ctx, cudaEventRecord(ctx->ev[5], st));
  SDF_CUDA(ctx, cudaStreamSynchronize(st));
  unsigned long long hbb[10];
  std::memcpy(hbb, ctx->h_scalars + S_MESH, sizeof(hbb));
  if (hbb[6] & 1) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "mesh vertices must be finite");
  if (hbb[6] & 2) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "IEN holds an index outside 1..nnp");

  MeshDev& M = ctx->mesh;
  M.nnp = nnp;
  M.nel = nel;
  double E = 0.0;
  for (int a = 0; a < 3; ++a) {
    M.bmin[a] = ord_dbl(hbb[a]);
    M.bmax[a] = ord_dbl(hbb[3 + a]);
    M.center[a] = 0.5 * (M.bmin[a] + M.bmax[a]);
    E = std::max(E, std::max(M.bmax[a] - M.center[a], M.center[a] - M.bmin[a]));
  }
  M.E = E;
  M.rho_max = ord_dbl(hbb[7]);
  M.n_weak = (int64_t)hbb[9];
  M.rho_weak = M.n_weak ? ord_dbl(hbb[8]) : 0.0;
  if (eager) {
    const int rc = ensure_tree(ctx, eager > 1);
    if (rc == SDFGPU_ERR_OUT_OF_MEMORY) ctx->err.clear();  // this mesh's calls may not need it; those that do report it
    else SDF_TRY(rc);
  }
  ctx->tree_used = 0;
  float ms = 0.f;
  SDF_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev[4], ctx->ev[5]));
  ctx->stats.ms_mesh = ms;
  ctx->stats.mesh_launches = ctx->launches;
  ctx->stats.nel = nel;
  ctx->stats.rho_max = M.rho_max;
  ctx->has_mesh = true;
  return 0;
}

int ensure_ine(sdfgpu_ctx* ctx) {
  MeshDev& M = ctx->mesh;
  if (M.ine_ready) return 0;
  cudaStream_t st = ctx->stream;
  int32_t *cnt, *off, *cur, *ine;
  SDF_TRY(scratch_t(ctx, "ine_cnt", (size_t)M.nnp + 1, &cnt));
  SDF_TRY(scratch_t(ctx, "ine_off", (size_t)M.nnp + 1, &off));
  SDF_TRY(scratch_t(ctx, "ine_cur", (size_t)M.nnp + 1, &cur));
  SDF_TRY(scratch_t(ctx, "ine", (size_t)M.nel * 3, &ine));
  const int64_t* dIEN = buf<int64_t>(ctx, "IEN64");
  SDF_CUDA(ctx, cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (M.nnp + 1), st));
  SDF_CUDA(ctx, cudaMemsetAsync(cur, 0, sizeof(int32_t) * (M.nnp + 1), st));
  k_ine_count<<<grid_for(M.nel, 256), 256, 0, st>>>(dIEN, M.nel, cnt);
  SDF_KERNEL(ctx);
  SDF_TRY(cub_scan_i32(ctx, cnt, off, M.nnp + 1));
  k_ine_fill<<<grid_for(M.nel, 256), 256, 0, st>>>(dIEN, M.nel, off, cur, ine);
  SDF_KERNEL(ctx);
  M.ine_ready = true;
  return 0;
}

int cub_scan_i32(sdfgpu_ctx* ctx, const int32_t* in, int32_t* out, int64_t n, cudaStream_t st, const char* tmp_name) {
  if (!st) st = ctx->stream;
  size_t bytes = 0;
  SDF_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int)n, st));
  void* tmp;
  SDF_TRY(scratch(ctx, tmp_name, bytes, &tmp));
  SDF_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, bytes, in, out, (int)n, st));
  return 0;
}

int cub_scan_i64(sdfgpu_ctx* ctx, const int64_t* in, int64_t* out, int64_t n) {
  size_t bytes = 0;
  SDF_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int)n, ctx->stream));
  void* tmp;
  SDF_TRY(scratch(ctx, "cub_tmp_scan", bytes, &tmp));
  SDF_CUDA(ctx, cub::DeviceScan::ExclusiveSum(tmp, bytes, in, out, (int)n, ctx->stream));
  return 0;
}

}  // namespace sdfgpu
