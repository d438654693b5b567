// near.cu -- the truncated distances (evalDistancesOnTriMesh, src/SignedDistances/dfOnTriangularMesh.jl:19-209)
// of meshes whose triangles are small against the cell, without closest points: a scatter from the
// triangles to the nodes within one cell of them instead of candidate lists.
//
// Every result is clamped to h (:202-206), and every value the fold can assign for a triangle is at
// least its true distance, so a node farther than h from all triangles gets h (or kBig, the fold's initial
// minimum, where the cells are larger than that).  For the others let D be
// the smallest true distance.  A candidate's step (:101-176) assigns, given the running minimum m,
//   its plane distance when p projects inside;
//   otherwise F, the smallest distance to a foot on its edges, when F < m;
//   otherwise V, the smallest distance to its vertices, when V < m.
// Unless V < F < m can happen, the value does not depend on m: it is face, F or V.  So with the
// triangles whose distance can equal D (the "ties") the fold's result is the smallest of their values
// whenever no value depends on m, or those that do cannot go below the others -- or when they share
// one V and, in index order, some F is not below the F before it: after the earlier one m is at most its
// F, so the later one's feet do not improve it and V is taken.  (The ties are taken in index order with the box
// test of the step, which decides between values a few roundings apart.)  Nodes for which none of this holds, and
// nodes next to a triangle unfit for FP32 decisions, replay the whole fold (k_hard_*); when their candidates do
// not fit the lists (hundreds of coincident triangles, a fan of a thousand in a large mesh), the tile fold takes
// the call, whose work is bounded by the candidates' number.
// SDFGPU_MODE_EXACT takes the true minimum, so its ties' smallest value is the result.
//
// A triangle within h of a node has its centroid within h + rho of it (rho the mesh's largest
// vertex-to-centroid distance), so for rho < 1.5 h all ties are candidates of the reference rule.
//
// Work: the (triangle, node) pairs of the triangles' boxes grown by h -- about 27 a triangle where
// triangles are small against h -- against the 64 nodes of every tile each triangle's 2.5 h ball reaches.
// Whole field calls on a B200, tile fold -> scatter with the other stages alike (all nodes of the boxes in both
// scatters; the kernels' comments have what the masks gave): 16.8M nodes, 1.4M triangles, reference rule 7.25 ->
// 3.61 ms; 33M nodes, 5.8M triangles, true minimum 25.6 -> 16.3 ms; 590k nodes, 131k triangles 1.33 ->
// 0.77 ms; level at 149k nodes and 5k triangles (0.52 ms, launches).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "unbounded.cuh"

namespace sdfgpu {
namespace {

constexpr int kSlots = 16;        // triangles kept per near node
constexpr int kHardCap = 1024;    // candidates listed per hard node (more: the mesh is scanned)
constexpr int64_t kHardPool = 16 << 20;  // candidates listed in all (likewise)
// A scan is a warp's walk of the mesh, 20 ns a triangle by its latency, for as many nodes as there are resident
// warps; the tile fold with its lists takes 0.3 ms and 4.5 ns a triangle for the whole call (2.1M triangles of
// which 2000 meet in one point, B200: 43.7 ms with scans, 10.2 ms handed over).  They meet at about 19k triangles.
constexpr int64_t kScanTriangles = 16384;
constexpr int kScanNodes = 4096;
constexpr int kTileShift = 2;     // flags of 4 x 4 x 4 node tiles with hard nodes

struct NearArgs {
  GridP g;
  LeafTris tri;         // FP32 records by triangle index
  const TriRec64* rec;
  const double4* cent;
  const float4* box32;  // mesh-local outward-rounded boxes
  const float4* c32;    // and centroids
  int64_t nel;
  bool ref;             // the reference rule, else the true minimum
  double reach;         // box growth: h plus the margin
  double ih;            // 1 / h
  // the grid in FP32: node = ihf * (mesh-local coordinate) + bo, within rm cells; mesh-local node
  // coordinates o32 + hf * node; the near nodes' distance, with the FP32 error of a box and a node in it
  float ihf, hf, bo[3], rm, o32[3], limb;
  float mk;             // see k_near_scatter
  uint64_t* mask;       // per triangle: the nodes of its box that its second scatter looks at
  float lim2, eD;       // squared FP32 distance of a near node; error of the FP32 distances
  float E;
  double rho;           // the mesh's largest vertex-to-centroid distance (edges are at most 2 rho)
  double r2, rball;     // the reference's squared candidate radius; a radius that surely contains its ball
  uint32_t* m2;         // per node: smallest squared FP32 distance (float bits)
  int32_t* map;         // per near node: its slot index
  int32_t* near_n;      // number of near nodes
  int32_t* node;        // near nodes
  int32_t* cnt;         // triangles in the band of each
  int32_t* slot;        // kSlots each
  int32_t* hidx;        // per near node: its hard index, or -1
  int32_t* hard_n;
  int32_t* hard;        // near indices of hard nodes
  int32_t* unbounded_n; // hard nodes whose hbound is not known from their slots
  int32_t* scan_n;      // hard nodes without a list
  int32_t scan_max;     // how many of them are scanned for; with more the tile fold takes the call
  uint8_t* tflag;       // tiles with hard nodes
  uint8_t* tcand;       // tiles in which a candidate of a hard node can have its centroid
  int64_t tn[3];
  float* hbound;        // per hard node: bound on the distances that matter to its fold
  int32_t* hcnt;        // its candidates within it (listed if they fit)
  int64_t* hoff;        // their place in the pool, -1: none
  int32_t* pool;
  unsigned long long* pool_n;
  double* dist;
  int64_t* counters;
};

// Nodes of axis a with coordinate in [x0, x1] (grown by the grid's pad), as in the tile lists.
__device__ __forceinline__ bool near_range(const NearArgs& A, int a, double x0, double x1, int& lo, int& hi) {
  const GridP& g = A.g;
  const double shift = (double)gidx(g, a, 0);
  const double f0 = fmax((x0 - g.o[a]) * A.ih - shift - g.pad, -1.0);
  const double f1 = fmin((x1 - g.o[a]) * A.ih - shift + g.pad, (double)g.N[a] + 1.0);
  if (!(f0 <= f1)) return false;
  lo = max((int)ceil(f0), 0);
  hi = (int)min((int64_t)floor(f1), g.N[a]);
  return lo <= hi;
}

// Node of axis a at a mesh-local coordinate, in FP32 (within A.rm), moved by `off`, clamped to one node beyond
// the grid.
__device__ __forceinline__ float node32(const NearArgs& A, int a, float x, float off) {
  return fminf(fmaxf(fmaf(x, A.ihf, A.bo[a]) + off, -1.f), (float)A.g.N[a] + 1.f);
}

// kFill false: every node's smallest squared distance, over the nodes near each triangle.  kFill true:
// each near node's triangles within the band of its minimum.  A thread per triangle: the boxes of one
// mesh differ little in size, and the triangle's frame stays in registers.  The nodes within h of the
// triangle's box (a chord per grid row) are the bits of a 64-bit mask, so a warp takes as many steps as its
// largest count, about half of the box's nodes.  The first scatter keeps the bits of the pairs that were
// within the band of the node's minimum at that time; it only falls, so the second needs no others: about
// two pairs a triangle instead of thirty.  Triangles of more than 64 nodes go through 64 at a time, both
// times.  Bound: instruction issue, about 70 a pair, and the latency of the triangles' reads, for which the
// registers are limited to 64 (8 blocks an SM).  Both scatters of 1.4M and of 5.8M triangles (B200): 0.43 and
// 1.9 ms when each took all nodes of the boxes, 0.30 and 1.22 ms with the masks, 0.27 and 1.11 ms at 64 registers
// instead of the compiler's 80.
template <bool kFill>
__global__ void __launch_bounds__(128, 8) k_near_scatter(const __grid_constant__ NearArgs A) {
  const GridP& g = A.g;
  for (int64_t el = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; el < A.nel; el += (int64_t)gridDim.x * blockDim.x) {
    uint64_t kept = 0;
    if (kFill) {
      kept = A.mask[el];
      if (!kept) continue;
    }
    const float4 b0 = A.box32[2 * el], b1 = A.box32[2 * el + 1];
    const float blo[3] = {b0.x, b0.y, b0.z}, bhi[3] = {b1.x, b1.y, b1.z};
    const float grow = fmaf(A.limb, A.ihf, A.rm);
    int lo[3], n[3];
    bool any = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = max((int)ceilf(node32(A, a, blo[a], -grow)), 0);
      n[a] = min((int)floorf(node32(A, a, bhi[a], grow)), (int)g.N[a]) - lo[a] + 1;
      any = any && n[a] > 0;
    }
    uint64_t next = 0;
    if (any) {
      const LeafTri T = A.tri.load((int)el);
      // the record's vertex a: v1, or the end of the longest edge of a triangle without area
      const double* va = A.rec[el].v + (T.m2.w < 0.f && T.m0.w != 0.f ? 3 : 0);
      const LeafView V = leaf_view(T, f3(T.a));  // from points a + d
      // nodes relative to a: an FP64 difference rounded once, then FP32 steps
      const float x0 = (float)(g.o[0] + g.h * (double)lo[0] - va[0]), y0 = (float)(g.o[1] + g.h * (double)lo[1] - va[1]),
                  z0 = (float)(g.o[2] + g.h * (double)gidx(g, 2, lo[2]) - va[2]);
      const int rows = n[1] * n[2], per = max(64 / n[0], 1);  // near_applies keeps n[0] below 16
      const float inx = 1.f / (float)n[0], iny = 1.f / (float)n[1];
      const float limb2 = A.limb * A.limb;
#pragma unroll 1
      for (int row0 = 0; row0 < rows; row0 += per) {
        uint64_t bits = kept;
        if (!kFill || rows > per) {
          bits = 0;
          int at = 0;
          const int row1 = min(rows, row0 + per);
          int k = (int)(((float)row0 + 0.5f) * iny), j = row0 - k * n[1];
#pragma unroll 1
          for (int r = row0; r < row1; ++r, at += n[0]) {
            const float y = fmaf(A.hf, (float)(lo[1] + j), A.o32[1]), z = fmaf(A.hf, (float)(lo[2] + k), A.o32[2]);
            const float dy = fmaxf(fmaxf(blo[1] - y, y - bhi[1]), 0.f), dz = fmaxf(fmaxf(blo[2] - z, z - bhi[2]), 0.f);
            const float rem = limb2 - dy * dy - dz * dz;
            if (rem >= 0.f) {
              const float half = fmaf(sqrt_approx(rem) * (1.f + 1e-5f), A.ihf, A.rm);
              const int i0 = max((int)ceilf(node32(A, 0, blo[0], -half)), lo[0]) - lo[0];
              const int i1 = min((int)floorf(node32(A, 0, bhi[0], half)) - lo[0], n[0] - 1);
              if (i1 >= i0) bits |= ((2ull << (i1 - i0)) - 1ull) << (at + i0);
            }
            if (++j == n[1]) { j = 0; ++k; }
          }
        }
        while (bits) {
          const int b = __ffsll((long long)bits) - 1;
          bits &= bits - 1ull;
          const int br = (int)(((float)b + 0.5f) * inx), i = b - br * n[0], r = row0 + br;
          const int k = (int)(((float)r + 0.5f) * iny), j = r - k * n[1];
          const float d2 = view_d2(V, make_float3(fmaf(A.hf, (float)i, x0), fmaf(A.hf, (float)j, y0), fmaf(A.hf, (float)k, z0)));
          if (!(d2 <= A.lim2)) continue;
          const int64_t lin = lo[0] + i + g.n[0] * (lo[1] + j + g.n[1] * (int64_t)(lo[2] + k));
          const uint32_t m = __ldcg(A.m2 + lin);
          if (!kFill) {
            // (sqrt(m) + 2 eD)^2 with sqrt(m) at most the near nodes' distance
            if (d2 <= fmaf(__uint_as_float(m), 1.f + 4e-6f, A.mk)) next |= 1ull << b;
            if (__float_as_uint(d2) < m) atomicMin(A.m2 + lin, __float_as_uint(d2));
          } else {
            const float w = sqrt_approx(__uint_as_float(m)) * (1.f + 1e-6f) + 2.f * A.eD;
            if (d2 > w * w) continue;
            const int32_t q = A.map[lin];
            const int c = atomicAdd(A.cnt + q, 1);
            if (c < kSlots) A.slot[(int64_t)q * kSlots + c] = __float_as_int(T.a.w);
          }
        }
      }
    }
    if (!kFill) A.mask[el] = next;  // of several masks: whether any has a bit
  }
}

// Lists the near nodes; all others get h.  A block takes kNodes nodes a thread and one place in the list for
// them: an atomic per warp on the list's length took 0.31 ms for 33M nodes, this 0.11 (B200).  Bound: 12
// bytes a node.
constexpr int kNodes = 8, kNodesThreads = 256;
__global__ void __launch_bounds__(kNodesThreads) k_near_nodes(const __grid_constant__ NearArgs A) {
  __shared__ int s_n[kNodesThreads / 32], s_first;
  const GridP& g = A.g;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t base = blockIdx.x * (int64_t)(kNodes * kNodesThreads); base < g.ngp;
       base += (int64_t)gridDim.x * (kNodes * kNodesThreads)) {
    unsigned near = 0u;
    int before[kNodes], total = 0;  // near nodes of this warp before mine
#pragma unroll
    for (int q = 0; q < kNodes; ++q) {
      const int64_t lin = base + q * kNodesThreads + threadIdx.x;
      const bool in = lin < g.ngp, is = in && A.m2[lin] != 0x7f7f7f7fu;
      if (in && !is) A.dist[lin] = fmin(g.h, kBig);
      const unsigned mask = __ballot_sync(0xffffffffu, is);
      before[q] = total + __popc(mask & ((1u << lane) - 1u));
      total += __popc(mask);
      near |= (unsigned)is << q;
    }
    if (lane == 0) s_n[w] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
      int sum = 0;
#pragma unroll
      for (int v = 0; v < kNodesThreads / 32; ++v) {
        const int c = s_n[v];
        s_n[v] = sum;
        sum += c;
      }
      s_first = sum ? atomicAdd(A.near_n, sum) : 0;
    }
    __syncthreads();
    const int first = s_first + s_n[w];
#pragma unroll
    for (int q = 0; q < kNodes; ++q)
      if ((near >> q) & 1u) {
        const int64_t lin = base + q * kNodesThreads + threadIdx.x;
        A.map[lin] = first + before[q];
        A.node[first + before[q]] = (int32_t)lin;
      }
    __syncthreads();
  }
}

__device__ __forceinline__ d3 near_point(const GridP& g, int64_t lin) {
  const int64_t i = lin % g.n[0], j = (lin / g.n[0]) % g.n[1], k = lin / (g.n[0] * g.n[1]);
  return gnode(g, i, j, k);
}

// What the reference's step can assign for a triangle: `face` its plane distance when p projects inside
// (else NaN), F the smallest distance to a valid foot (INFINITY: none) and V to a vertex -- the
// expressions of tri_step64 (dfOnTriangularMesh.jl:104-176).
__device__ __noinline__ void step_values(const TriRec64* __restrict__ rec, int t, const d3& p, double& face, double& F,
                                         double& V) {
  const TriRec64& r = rec[t];
  double lam[3];
  bary_solve(r, p, lam);
  const d3 v0 = rec_v(r, 0), v1 = rec_v(r, 1), v2 = rec_v(r, 2);
  face = nan("");
  F = V = INFINITY;
  if (lam[0] >= 0.0 && lam[1] >= 0.0 && lam[2] >= 0.0) {
    const d3 xp = v_add(v_add(v_scale(v0, lam[0]), v_scale(v1, lam[1])), v_scale(v2, lam[2]));
    face = v_norm(v_sub(p, xp));
    return;
  }
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const d3 vj = rec_v(r, j);
    const d3 u = {r.u[3 * j], r.u[3 * j + 1], r.u[3 * j + 2]};
    const double P = v_dot(v_sub(p, vj), u);
    if (P >= 0.0 && P <= r.L[j]) F = fmin(F, v_norm(v_sub(p, v_add(vj, v_scale(u, P)))));
    V = fmin(V, v_norm(v_sub(p, vj)));
  }
}

// One thread per near node: the result from its ties, or a place in the hard list.
__global__ void __launch_bounds__(128, 6) k_near_resolve(const __grid_constant__ NearArgs A) {
  const GridP& g = A.g;
  const int n_near = *A.near_n;
  const double tol = 1e-9 * (double)A.E, tol2 = tol * tol;
  uint32_t fp64 = 0;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n_near; q += gridDim.x * blockDim.x) {
    const int64_t lin = A.node[q];
    const d3 p = near_point(g, lin);
    int32_t* slot = A.slot + (int64_t)q * kSlots;
    const int n = A.cnt[q];
    bool hard = n < 1 || n > kSlots;
    for (int s = 0; s < n && !hard; ++s) hard = (slot[s] & kWeakTri) != 0;
    double m = kBig, nearest = INFINITY;  // nearest: a squared distance of a triangle fit for FP32 decisions
    if (hard) {
      for (int s = 0; s < min(n, kSlots); ++s) {
        int feat;
        if ((slot[s] & kWeakTri) == 0) nearest = fmin(nearest, near64(A.rec, slot[s], p, tol2, feat));
      }
    } else {
      // the ties, as in lane_filter (unbounded.cuh)
      double best = 1e300, lim = 1e300;
      int left = 0;
#pragma unroll 1
      for (int s = 0; s < n; ++s) {
        const int t = slot[s];
        int feat;
        const double d2 = near64(A.rec, t, p, tol2, feat);
        if (d2 > lim) continue;
        if (d2 < best) {
          const double dl = 2.0 * tol * (double)sqrtf((float)d2) * (1.0 + 1e-6) + tol2;
          if (d2 + dl < best) left = 0;
          best = d2;
          lim = d2 + dl;
        }
        slot[left++] = (int)((unsigned)t | (unsigned)(feat < 0 ? 7 : feat) << kFeatShift);
      }
      nearest = best;
      // in ascending triangle index
      double Vc = INFINITY, Fprev = INFINITY, Fmin = INFINITY;
      int dependent = 0, last = -1;
      bool sure = false, one_v = true;
#pragma unroll 1
      for (int it = 0; it < left; ++it) {
        unsigned pick = 0u;
        int tri = 0x7fffffff;
        for (int s = 0; s < left; ++s) {
          const unsigned u = (unsigned)slot[s];
          const int t = (int)(u & kTriMask);
          if (t > last && t < tri) { tri = t; pick = u; }
        }
        last = tri;
        const int feat = (int)(pick >> kFeatShift);
        ++fp64;
        // a value that the triangle's step takes unless its box test passes it over at m (never at kBig)
        auto take = [&](double v) {
          if (v < m && !(m < kBig && step_skips(A.rec[tri], p, m))) m = v;
        };
        if (feat <= F_EDGE2 || (feat != 7 && !A.ref)) {  // face or edge: whatever m
          double d;
          d3 x;
          feature64(A.rec[tri], p, feat, d, x);
          take(d);
          continue;
        }
        double face, F, V;
        step_values(A.rec, tri, p, face, F, V);
        if (face == face) take(face);
        else if (!A.ref || !(V < F) || isinf(F)) take(fmin(F, V));
        else {  // V < F: depends on m
          if (dependent++ == 0) Vc = V;
          else {
            one_v = one_v && V == Vc;
            sure = sure || F >= Fprev;
          }
          if (V < Vc) Vc = V;
          Fmin = fmin(Fmin, F);
          Fprev = F;
        }
      }
      if (dependent) {
        // the values that depend on m can go below the others; and where values lie closer together than the
        // box test resolves, which of them are taken depends on the order (tol is far above that).  Below Vc
        // it does not when the test passes over none of the ties at Vc: then all of them are taken as here.
        const bool apart = Fmin - Vc > tol;
        if (m == Vc) {
          hard = !apart;
        } else if (m < Vc) {
          if (Vc - m <= tol)
            for (int s = 0; s < left && !hard; ++s) hard = step_skips(A.rec[(unsigned)slot[s] & kTriMask], p, Vc);
        } else {
          hard = !(one_v && sure && apart && m - Vc > tol);
          m = Vc;
        }
      }
    }
    A.hidx[q] = -1;
    if (hard) {
      const int hq = atomicAdd(A.hard_n, 1);
      A.hard[hq] = q;
      A.hidx[q] = hq;
      A.hcnt[hq] = 0;
      A.hbound[hq] = __double2float_ru(sqrt(nearest) + 4.0 * A.rho + 4.0 * tol);
      if (isinf(nearest)) atomicAdd(A.unbounded_n, 1);
      const int64_t at[3] = {lin % g.n[0], (lin / g.n[0]) % g.n[1], lin / (g.n[0] * g.n[1])};
      A.tflag[((at[2] >> kTileShift) * A.tn[1] + (at[1] >> kTileShift)) * A.tn[0] + (at[0] >> kTileShift)] = 1;
      const double rc = (A.ref ? A.rball : A.reach + A.rho) * A.ih + (double)A.rm + 1.0;
      int t0[3], t1[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        t0[a] = max((int)((double)at[a] - rc), 0) >> kTileShift;
        t1[a] = (int)fmin((double)at[a] + rc, (double)g.N[a]) >> kTileShift;
      }
      for (int z = t0[2]; z <= t1[2]; ++z)
        for (int y = t0[1]; y <= t1[1]; ++y)
          for (int x = t0[0]; x <= t1[0]; ++x) A.tcand[((int64_t)z * A.tn[1] + y) * A.tn[0] + x] = 1;
      continue;
    }
    A.dist[lin] = m > g.h ? g.h : m;  // clamp (dfOnTriangularMesh.jl:202-206)
  }
  for (int off = 16; off > 0; off >>= 1) fp64 += __shfl_down_sync(0xffffffffu, fp64, off);
  if ((threadIdx.x & 31) == 0 && fp64) count_add(A.counters, C_FP64, fp64);
}

// Whether triangle t is a candidate of node p: its centroid in the reference's ball, or for the true
// minimum its box within reach.
__device__ __forceinline__ bool hard_candidate(const NearArgs& A, int64_t t, const d3& p) {
  if (A.ref) {
    const double4 c = A.cent[t];
    const double ex = ds(c.x, p.x), ey = ds(c.y, p.y), ez = ds(c.z, p.z);
    double s = dm(ex, ex);
    s = da(s, dm(ey, ey));
    s = da(s, dm(ez, ez));
    return s <= A.r2;
  }
  const TriRec64& r = A.rec[t];
  return p.x >= r.bmin[0] - A.reach && p.x <= r.bmax[0] + A.reach && p.y >= r.bmin[1] - A.reach &&
         p.y <= r.bmax[1] + A.reach && p.z >= r.bmin[2] - A.reach && p.z <= r.bmax[2] + A.reach;
}

// The hard nodes' candidates that matter: the triangles with their centroid in a tile where a hard node can
// have candidates visit the tiles with hard nodes that their candidate region reaches.  A step assigns at
// most the distance to the farthest point of its triangle, so the fold ends at or below U = min over the
// triangles fit for FP32 decisions of (their distance + 2 rho); a value that can be the result comes from
// a triangle within U, and whether its feet improve the minimum depends on values up to U + 2 rho.
// k_near_resolve has that bound from a node's slots, unless all of them are unfit.  kPhase 0: it is found
// for those nodes (else returns at once); 1: the candidates within it counted (returns at once when every
// node can have kHardCap places); 2: listed.  Bound: 16 bytes and one flag a triangle; three passes that each
// formed the triangles' regions in FP64 took 0.81 ms on 5.8M triangles, this 0.09 (B200).
__device__ __forceinline__ bool hard_uniform(int n_hard) { return (int64_t)n_hard * kHardCap <= kHardPool; }

template <int kPhase>
__global__ void __launch_bounds__(128) k_hard_collect(const __grid_constant__ NearArgs A) {
  if (*A.hard_n == 0) return;
  if (kPhase == 0 && *A.unbounded_n == 0) return;
  if (kPhase == 1 && hard_uniform(*A.hard_n)) return;
  if (kPhase == 2 && *A.scan_n > A.scan_max) return;
  const GridP& g = A.g;
  const double tol = 1e-9 * (double)A.E;
  for (int64_t el = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; el < A.nel; el += (int64_t)gridDim.x * blockDim.x) {
    {
      const float4 c = A.c32[el];
      const float f[3] = {node32(A, 0, c.x, 0.f), node32(A, 1, c.y, 0.f), node32(A, 2, c.z, 0.f)};
      int t[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) t[a] = min(max((int)f[a], 0), (int)g.N[a]) >> kTileShift;
      if (!A.tcand[((int64_t)t[2] * A.tn[1] + t[1]) * A.tn[0] + t[0]]) continue;
    }
    int lo[3], hi[3];
    bool any = true;
    if (A.ref) {
      const double4 c4 = A.cent[el];
      const double c[3] = {c4.x, c4.y, c4.z};
#pragma unroll
      for (int a = 0; a < 3; ++a) any = any && near_range(A, a, c[a] - A.rball, c[a] + A.rball, lo[a], hi[a]);
    } else {
#pragma unroll
      for (int a = 0; a < 3; ++a)
        any = any && near_range(A, a, A.rec[el].bmin[a] - A.reach, A.rec[el].bmax[a] + A.reach, lo[a], hi[a]);
    }
    if (!any) continue;
    for (int tz = lo[2] >> kTileShift; tz <= hi[2] >> kTileShift; ++tz)
      for (int ty = lo[1] >> kTileShift; ty <= hi[1] >> kTileShift; ++ty)
        for (int tx = lo[0] >> kTileShift; tx <= hi[0] >> kTileShift; ++tx) {
          if (!A.tflag[((int64_t)tz * A.tn[1] + ty) * A.tn[0] + tx]) continue;
          constexpr int kT = 1 << kTileShift;
          for (int k = max(lo[2], tz * kT); k <= min(hi[2], tz * kT + kT - 1); ++k)
            for (int j = max(lo[1], ty * kT); j <= min(hi[1], ty * kT + kT - 1); ++j)
              for (int i = max(lo[0], tx * kT); i <= min(hi[0], tx * kT + kT - 1); ++i) {
                const int64_t lin = i + g.n[0] * (j + g.n[1] * (int64_t)k);
                if (A.m2[lin] == 0x7f7f7f7fu) continue;
                const int hq = A.hidx[A.map[lin]];
                if (hq < 0) continue;
                const d3 p = gnode(g, i, j, k);
                if (!hard_candidate(A, el, p)) continue;
                const bool weak = (__float_as_int(A.tri.at(0, (int)el).w) & kWeakTri) != 0;
                int feat;
                const double d = weak ? 0.0 : sqrt(near64(A.rec, (int)el, p, tol * tol, feat));
                if (kPhase == 0) {
                  const float b = __double2float_ru(d + 4.0 * A.rho + 4.0 * tol);
                  if (!weak) atomicMin(reinterpret_cast<int*>(A.hbound + hq), __float_as_int(b));  // non-negative
                  continue;
                }
                if (d - tol > (double)A.hbound[hq]) continue;
                if (kPhase == 1) {
                  atomicAdd(A.hcnt + hq, 1);
                } else if (A.hoff[hq] >= 0) {
                  const int c = atomicAdd(A.hcnt + hq, 1);
                  if (c == kHardCap) atomicAdd(A.scan_n, 1);
                  if (c < kHardCap) A.pool[A.hoff[hq] + c] = (int32_t)el;
                }
              }
        }
  }
}

// Places for the lists (between counting and listing); the counts start again at 0.
__global__ void k_hard_place(const __grid_constant__ NearArgs A) {
  const int n_hard = *A.hard_n;
  for (int hq = blockIdx.x * blockDim.x + threadIdx.x; hq < n_hard; hq += gridDim.x * blockDim.x) {
    const int c = A.hcnt[hq];
    int64_t off = -1;
    if (hard_uniform(n_hard)) {
      off = (int64_t)hq * kHardCap;
    } else if (c <= kHardCap) {
      off = (int64_t)atomicAdd(A.pool_n, (unsigned long long)c);
      if (off + c > kHardPool) off = -1;
    }
    if (off < 0) atomicAdd(A.scan_n, 1);
    A.hoff[hq] = off;
    A.hcnt[hq] = 0;
  }
}

// Replays the fold of a hard node, one warp each: the candidates in ascending index 32 at a time, a lane
// per candidate bounding its distance from below (near64; 0 where that is not certain), and the
// reference step on those that the running minimum does not exclude (every value a step can assign is at
// least the true distance).  Nodes without a list scan the mesh instead, where that is the cheaper way.
__global__ void __launch_bounds__(128) k_hard_replay(const __grid_constant__ NearArgs A) {
  __shared__ int s_list[4][kHardCap];
  const GridP& g = A.g;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (*A.scan_n > A.scan_max) {
    if (blockIdx.x == 0 && threadIdx.x == 0) count_add(A.counters, C_HARD_LEFT, *A.scan_n);
    return;
  }
  const int n_hard = *A.hard_n;
  const double tol = 1e-9 * (double)A.E;
  uint32_t fp64 = 0;
  for (int hq = blockIdx.x * 4 + w; hq < n_hard; hq += gridDim.x * 4) {
    const int64_t lin = A.node[A.hard[hq]];
    const d3 p = near_point(g, lin);
    double m = kBig;
    d3 proj = {0.0, 0.0, 0.0};
    auto batch = [&](int t) {  // this lane's candidate, or -1; ascending over the lanes
      double lb = INFINITY;
      if (t >= 0) {
        int feat;
        lb = (__float_as_int(A.tri.at(0, t).w) & kWeakTri) ? 0.0
                                                           : sqrt(near64(A.rec, t, p, tol * tol, feat)) - tol;
      }
      for (unsigned todo = __ballot_sync(0xffffffffu, lb <= m); todo; todo &= todo - 1u) {
        const int src = __ffs(todo) - 1;
        if (!(__shfl_sync(0xffffffffu, lb, src) <= m)) continue;
        tri_step64(A.rec[__shfl_sync(0xffffffffu, t, src)], p, m, proj, A.ref);
        ++fp64;
      }
    };
    const int n = A.hcnt[hq];
    if (A.hoff[hq] >= 0 && n <= kHardCap) {
      int *list = s_list[w], *sorted = A.pool + A.hoff[hq];
      for (int s = lane; s < n; s += 32) list[s] = sorted[s];
      __syncwarp();
      for (int s = lane; s < n; s += 32) {  // rank sort (the indices are distinct)
        const int t = list[s];
        int rank = 0;
        for (int o = 0; o < n; ++o) rank += list[o] < t;
        sorted[rank] = t;
      }
      __syncwarp();
      for (int base = 0; base < n; base += 32) batch(base + lane < n ? sorted[base + lane] : -1);
    } else {
      for (int64_t base = 0; base < A.nel; base += 32) {
        const int64_t t = base + lane;
        const bool in = t < A.nel && hard_candidate(A, t, p);
        if (__any_sync(0xffffffffu, in)) batch(in ? (int)t : -1);
      }
    }
    if (lane == 0) A.dist[lin] = m > g.h ? g.h : m;
    __syncwarp();
  }
  if (lane == 0 && fp64) count_add(A.counters, C_FP64, fp64);
}

}  // namespace

// Whether near_prepare and near_run take this call: triangles of at most 1.5 (reference rule) or 4 cells from their
// centroid, the mesh near the coordinate origin (see unb_mesh), mesh and grid within 1e5 cells of the mesh's
// centre (FP32 node indices within half a cell, and a box's rows within a mask), and few and small triangles
// unfit for FP32 decisions, each of which sends the nodes nearest to it to the replay.  And cells whose squares
// FP32 holds with all their digits: from 1e-15 the error of a square of a few cells by underflow, at most
// sqrt(16 * 2^-149) = 1.5e-22 of distance, is below a tenth of eD, and up to 1e15 nothing overflows.
bool near_applies(const sdfgpu_ctx* ctx, const GridP& g, int mode) {
  const MeshDev& M = ctx->mesh;
  double off = 0.0;
  for (int a = 0; a < 3; ++a) off = std::max(off, std::fabs(M.center[a]));
  const double rho = M.rho_max * (1.0 + 1e-9) + 1e-6 * g.E;
  return off <= 64.0 * M.E && g.h >= 1e-15 && g.h <= 1e15 && g.E <= 1e5 * g.h && rho < (mode == SDFGPU_MODE_REF_RULE ? 1.5 : 4.0) * g.h && M.rho_weak <= 1.5 * g.h &&
         M.n_weak <= M.nel / 64;
}

// The two parts of the stage: near_prepare finds every node's nearest distance in FP32 and the near nodes
// (whose number the host waits for, to size their slots); near_run the results.
static_assert(sizeof(NearArgs) <= sizeof(DistPlan::fold), "DistPlan::fold holds a NearArgs");

int near_prepare(sdfgpu_ctx* ctx, const GridP& g, int mode, double* d_dist, DistPlan& Pl) {
  cudaStream_t st = ctx->stream;
  const MeshDev& M = ctx->mesh;
  NearArgs A{};
  A.g = g;
  A.tri = LeafTris{buf<float4>(ctx, "tri32"), M.nel};
  A.rec = buf<TriRec64>(ctx, "rec");
  A.cent = buf<double4>(ctx, "cent64");
  A.box32 = buf<float4>(ctx, "box32");
  A.c32 = buf<float4>(ctx, "c32");
  A.nel = M.nel;
  A.ref = mode == SDFGPU_MODE_REF_RULE;
  // FP32 distances in the triangle's own frame: every rounding is relative to |p - a| + the edges, at most
  // d + 4 rho + 2 rho; below 1e-6 of that in all (see view_d2)
  A.eD = (float)(1.5e-6 * (g.h + 6.0 * M.rho_max));
  const double lim = (g.h + 4.0 * (double)A.eD) * (1.0 + 1e-6);
  A.lim2 = (float)(lim * lim);
  A.reach = lim * (1.0 + 1e-9) + 1e-9 * g.E;
  A.ih = 1.0 / g.h;
  A.E = (float)g.E;
  A.ihf = (float)A.ih;
  A.hf = (float)g.h;
  for (int a = 0; a < 3; ++a) {
    const double o = g.o[a] + g.h * (double)gidx(g, a, 0) - M.center[a];  // mesh-local
    A.o32[a] = (float)o;
    A.bo[a] = (float)(-o * A.ih);
  }
  // FP32 coordinates of boxes and nodes are within 3 roundings of E each
  A.limb = (float)(lim * (1.0 + 1e-6) + 1e-6 * g.E);
  A.rm = (float)(2e-6 * g.E * A.ih + 1e-4);
  A.mk = (float)(4.1 * A.eD * lim + 4.1 * A.eD * A.eD);
  A.rho = M.rho_max;
  const double sr = 2.5 * g.h;
  A.r2 = sr * sr;
  A.rball = sr * (1.0 + 1e-9) + 1e-6 * g.E;
  A.dist = d_dist;
  A.counters = ctx->d_counters;
  int64_t tiles = 1;
  for (int a = 0; a < 3; ++a) {
    A.tn[a] = (g.n[a] >> kTileShift) + 1;
    tiles *= A.tn[a];
  }
  int32_t* counts;  // near nodes, hard nodes, hard nodes without a bound, without a list; the pool's length
  SDF_TRY(scratch_t(ctx, "near_m2", (size_t)g.ngp, &A.m2));
  SDF_TRY(scratch_t(ctx, "near_map", (size_t)g.ngp, &A.map));
  SDF_TRY(scratch_t(ctx, "near_node", (size_t)g.ngp, &A.node));
  SDF_TRY(scratch_t(ctx, "near_counts", 6, &counts));
  SDF_TRY(scratch_t(ctx, "near_tflag", (size_t)tiles * 2, &A.tflag));
  SDF_TRY(scratch_t(ctx, "near_mask", (size_t)M.nel, &A.mask));
  A.tcand = A.tflag + tiles;
  A.near_n = counts;
  A.hard_n = counts + 1;
  A.unbounded_n = counts + 2;
  A.scan_n = counts + 3;
  A.scan_max = M.nel <= kScanTriangles ? kScanNodes : 0;
  A.pool_n = reinterpret_cast<unsigned long long*>(counts + 4);
  SDF_CUDA(ctx, cudaMemsetAsync(A.m2, 0x7f, sizeof(uint32_t) * g.ngp, st));  // 3.39e38
  SDF_CUDA(ctx, cudaMemsetAsync(counts, 0, 6 * sizeof(int32_t), st));
  SDF_CUDA(ctx, cudaMemsetAsync(A.tflag, 0, (size_t)tiles * 2, st));
  const unsigned gt = grid_for(M.nel, 128, 148 * 64);
  k_near_scatter<false><<<gt, 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  k_near_nodes<<<grid_for(cdiv(g.ngp, kNodes), kNodesThreads, 148 * 16), kNodesThreads, 0, st>>>(A);
  SDF_KERNEL(ctx);
  SDF_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + S_NEAR, A.near_n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  SDF_CUDA(ctx, cudaStreamSynchronize(st));
  int32_t n_near;
  std::memcpy(&n_near, ctx->h_scalars + S_NEAR, sizeof(n_near));
  SDF_TRY(scratch_t(ctx, "near_cnt", (size_t)n_near, &A.cnt));
  SDF_TRY(scratch_t(ctx, "near_slot", (size_t)n_near * kSlots, &A.slot));
  SDF_TRY(scratch_t(ctx, "near_hidx", (size_t)n_near, &A.hidx));
  SDF_TRY(scratch_t(ctx, "near_hard", (size_t)n_near, &A.hard));
  SDF_TRY(scratch_t(ctx, "near_hbound", (size_t)n_near, &A.hbound));
  SDF_TRY(scratch_t(ctx, "near_hcnt", (size_t)n_near, &A.hcnt));
  SDF_TRY(scratch_t(ctx, "near_hoff", (size_t)n_near, &A.hoff));
  SDF_TRY(scratch_t(ctx, "near_pool", (size_t)kHardPool, &A.pool));
  std::memcpy(Pl.fold, &A, sizeof(A));
  Pl.g = g;
  Pl.nonempty = n_near;
  return 0;
}

int near_run(sdfgpu_ctx* ctx, const DistPlan& Pl) {
  cudaStream_t st = ctx->stream;
  NearArgs A;
  std::memcpy(&A, Pl.fold, sizeof(A));
  const int64_t n = Pl.nonempty;
  ctx->h_counters[C_BAND] = n;
  if (n == 0) return 0;
  SDF_CUDA(ctx, cudaMemsetAsync(A.cnt, 0, sizeof(int32_t) * n, st));
  const unsigned gt = grid_for(A.nel, 128, 148 * 64);
  k_near_scatter<true><<<gt, 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  k_near_resolve<<<grid_for(n, 128, 148 * 32), 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  // these return at once when no node is hard
  k_hard_collect<0><<<gt, 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  k_hard_collect<1><<<gt, 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  k_hard_place<<<grid_for(n, 256, 148), 256, 0, st>>>(A);
  SDF_KERNEL(ctx);
  k_hard_collect<2><<<gt, 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  k_hard_replay<<<grid_for(n, 4, 148 * 8), 128, 0, st>>>(A);
  SDF_KERNEL(ctx);
  return 0;
}

}  // namespace sdfgpu
