// sign.cu -- raycast_sign_detection (src/SignedDistances/RaycastingSignDetection.jl:337-404).
//
// Per node the reference casts the prioritized directions (:162-227) and votes by the parity of
// the distinct Möller–Trumbore hits (:114-154): 6 axis rays, then batches of 4 until the vote
// is confident (:234-288), then the generalized winding number when confidence < 0.6 (:376-380).
//
// B200 layout of the work:
//   * The 6 axis rays are the only rays every node casts, and they are grid-structured.  For a
//     ray along +x from node (i, j, k) every Möller–Trumbore decision except t > eps depends only
//     on the row (j, k): h = cross(e_x, e2) has an exactly zero x component, so u and v never see
//     the node's x.  And the -x ray of the same node sees a = -a, f = -f, the same u and v, and
//     t = -t exactly.  So one list of (row, triangle) hits per axis serves both directions of
//     every node of the row.  The lists are built by a triangle scatter over the rows its
//     projected box covers (FP64 decisions, exactly the reference's).  t is linear in the node's
//     coordinate with slope -1, so a hit's coordinate and a bound of the rounding of t split the row's
//     nodes into those certainly below the hit, those certainly above it, and a node or none within the
//     bound; and the gaps between the row's hits say which of them merge within eps.  So a row's parities
//     are bit masks over its nodes, made of one prefix per distinct hit.  Where a node lies within the
//     bound of a hit, or a gap is near eps, the node evaluates t for all hits of the row with the
//     reference's formula, sorts, de-duplicates within eps and takes parities.
//   * Nodes whose 6 votes disagree continue with the reference's batches on the LBVH: FP32 slab
//     tests with an explicit margin prune, FP64 Möller–Trumbore decides.
//   * Nodes left with confidence < threshold sum the winding number over all triangles, one CTA
//     per node with a fixed-order block reduction.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "common.cuh"

namespace sdfgpu {

__constant__ double c_dirs[36 * 3];
__constant__ float c_dirs32[36 * 3];  // the same, rounded

namespace {

constexpr double kEps = 1e-8;  // check_ray_inside_bvh default (:118), passed to MT (:132)
constexpr int kRowCap = 64;    // hits per row a node sorts in registers/local memory
constexpr int kRayCap = 256;   // hits per generic ray
constexpr int kAllPairsNodes = 24;  // undecided nodes whose rays test every triangle
constexpr int kStack = 64;

// A row hit: the Möller–Trumbore constants of one triangle for one grid row, from which each node
// of the row gets t with the reference's operation order (see the per-axis formulas below).
struct RowHit {
  double v1a;  // v1 coordinate along the row axis
  double K1, K2, P;
  double ea, eb, fa, fb;
  double f;
};

template <int AX>
__device__ __forceinline__ double row_t(const RowHit& r, double xa) {
  const double s = ds(xa, r.v1a);
  if (AX == 0) {
    const double qy = ds(r.K1, dm(s, r.ea));
    const double qz = ds(dm(s, r.eb), r.K2);
    return dm(r.f, da(da(r.P, dm(r.fa, qy)), dm(r.fb, qz)));
  } else if (AX == 1) {
    const double qx = ds(dm(s, r.ea), r.K1);
    const double qz = ds(r.K2, dm(s, r.eb));
    return dm(r.f, da(da(dm(r.fa, qx), r.P), dm(r.fb, qz)));
  } else {
    const double qx = ds(r.K1, dm(s, r.ea));
    const double qy = ds(dm(s, r.eb), r.K2);
    return dm(r.f, da(da(dm(r.fa, qx), dm(r.fb, qy)), r.P));
  }
}

// Möller–Trumbore decisions of the +AX ray through (ob, oc) against the triangle; on a pass fills
// the row-hit constants.  The along-axis origin is v1's own coordinate (any value gives the same
// decisions, see the file comment).
template <int AX>
__device__ __forceinline__ bool row_test(const TriRec64& r, double ob, double oc, RowHit* out) {
  const d3 v1 = rec_v(r, 0), v2 = rec_v(r, 1), v3 = rec_v(r, 2);
  d3 o, d;
  if (AX == 0) { o = {v1.x, ob, oc}; d = {1.0, 0.0, 0.0}; }
  else if (AX == 1) { o = {ob, v1.y, oc}; d = {0.0, 1.0, 0.0}; }
  else { o = {ob, oc, v1.z}; d = {0.0, 0.0, 1.0}; }
  const d3 e1 = v_sub(v2, v1), e2 = v_sub(v3, v1);
  const d3 h = v_cross(d, e2);
  const double a = v_dot(e1, h);
  if (fabs(a) < kEps) return false;
  const double f = dd(1.0, a);
  const d3 s = v_sub(o, v1);
  const double u = dm(f, v_dot(s, h));
  if (u < 0.0 || u > 1.0) return false;
  const d3 q = v_cross(s, e1);
  const double v = dm(f, v_dot(d, q));
  if (v < 0.0 || da(u, v) > 1.0) return false;
  if (out) {
    RowHit R;
    R.f = f;
    if (AX == 0) {
      R.v1a = v1.x; R.K1 = dm(s.z, e1.x); R.K2 = dm(s.y, e1.x); R.P = dm(e2.x, q.x);
      R.ea = e1.z; R.eb = e1.y; R.fa = e2.y; R.fb = e2.z;
    } else if (AX == 1) {
      R.v1a = v1.y; R.K1 = dm(s.z, e1.y); R.K2 = dm(s.x, e1.y); R.P = dm(e2.y, q.y);
      R.ea = e1.z; R.eb = e1.x; R.fa = e2.x; R.fb = e2.z;
    } else {
      R.v1a = v1.z; R.K1 = dm(s.y, e1.z); R.K2 = dm(s.x, e1.z); R.P = dm(e2.z, q.z);
      R.ea = e1.y; R.eb = e1.x; R.fa = e2.x; R.fb = e2.y;
    }
    *out = R;
  }
  return true;
}

// The decisions of row_test in FP32 with explicit error bands (the bulk of the sign stage's
// arithmetic).  Returns 0 when the FP64 test certainly misses, 1 when it certainly hits, 2 when a
// decision lies inside its band (the caller replays row_test in FP64).
//
// With (P, Q) the transverse axes in cyclic order after AX, the +AX ray gives h = d x e2 with
// h_P = -e2_Q, h_Q = e2_P, h_AX = 0, so a = e1_Q e2_P - e1_P e2_Q, s.h = s_Q e2_P - s_P e2_Q and
// d.q = s_P e1_Q - s_Q e1_P (s_AX = 0).  The six inputs are the FP64 differences the reference
// forms, rounded once to FP32 (relative error u = 2^-24 each).  A difference of two products of
// rounded inputs is then within 4u (|p1| + |p2|) of the FP64 value (whose own error, ~2^-51 of the
// same sum, is far below); 6u is used.  With err_a, err_p those bounds, |A| >= 3 err_a (else the
// test is undecided) and den = |A| - err_a, the quotient U = fl(P_u / A) satisfies
//   |u - U| <= E_u = (1.5 err_p + 2 (|U| + 1) err_a) / den + 2u (|U| + 1)
// (|u| <= 2 (|U| + 1) follows from err_a <= den / 2), the same for v, and
// |(u + v) - fl(U + V)| <= E_u + E_v + 2u |U + V|.
constexpr float kU32 = 5.9604645e-8f;  // 2^-24

template <int AX>
__device__ __forceinline__ int row_test32(const TriRec64& r, double ob, double oc) {
  constexpr int P = AX == 0 ? 1 : (AX == 1 ? 2 : 0), Q = AX == 0 ? 2 : (AX == 1 ? 0 : 1);
  // row origin along P and Q (row_test's o: AX = 0 -> (y, z) = (ob, oc); AX = 1 -> (z, x) = (oc, ob);
  // AX = 2 -> (x, y) = (ob, oc))
  const double oP = AX == 1 ? oc : ob, oQ = AX == 1 ? ob : oc;
  const float e1P = (float)ds(r.v[3 + P], r.v[P]), e1Q = (float)ds(r.v[3 + Q], r.v[Q]);
  const float e2P = (float)ds(r.v[6 + P], r.v[P]), e2Q = (float)ds(r.v[6 + Q], r.v[Q]);
  const float sP = (float)ds(oP, r.v[P]), sQ = (float)ds(oQ, r.v[Q]);
  const float a1 = __fmul_rn(e1Q, e2P), a2 = __fmul_rn(e1P, e2Q);
  const float A = __fsub_rn(a1, a2);
  const float ea = 6.f * kU32 * (fabsf(a1) + fabsf(a2));
  const float aA = fabsf(A);
  if (aA + ea < (float)kEps) return 0;                          // |a| < eps certainly
  if (!(aA - ea >= (float)kEps) || !(aA >= 3.f * ea)) return 2;  // |a| near eps, or a ill-conditioned
  const float den = aA - ea;
  const float u1 = __fmul_rn(sQ, e2P), u2 = __fmul_rn(sP, e2Q);
  const float U = __fdiv_rn(__fsub_rn(u1, u2), A);
  const float Eu = (1.5f * 6.f * kU32 * (fabsf(u1) + fabsf(u2)) + 2.f * (fabsf(U) + 1.f) * ea) / den +
                   2.f * kU32 * (fabsf(U) + 1.f);
  if (U < -Eu || U > 1.f + Eu) return 0;
  const float v1 = __fmul_rn(sP, e1Q), v2 = __fmul_rn(sQ, e1P);
  const float V = __fdiv_rn(__fsub_rn(v1, v2), A);
  const float Ev = (1.5f * 6.f * kU32 * (fabsf(v1) + fabsf(v2)) + 2.f * (fabsf(V) + 1.f) * ea) / den +
                   2.f * kU32 * (fabsf(V) + 1.f);
  if (V < -Ev) return 0;
  const float UV = __fadd_rn(U, V);
  const float Euv = Eu + Ev + 2.f * kU32 * fabsf(UV);
  if (UV > 1.f + Euv) return 0;
  if (U >= Eu && U <= 1.f - Eu && V >= Ev && UV <= 1.f - Euv) return 1;
  return 2;
}

__device__ __forceinline__ bool axis_range2(const GridP& g, int a, double x0, double x1, int64_t& lo, int64_t& hi) {
  const double shift = (double)gidx(g, a, 0);
  double f0 = (x0 - g.o[a]) / g.h - shift - g.pad, f1 = (x1 - g.o[a]) / g.h - shift + g.pad;
  f0 = fmax(f0, -1.0);
  f1 = fmin(f1, (double)g.N[a] + 1.0);
  if (!(f0 <= f1)) return false;
  lo = (int64_t)ceil(f0);
  hi = (int64_t)floor(f1);
  if (lo < 0) lo = 0;
  if (hi > g.N[a]) hi = g.N[a];
  return lo <= hi;
}

struct RowArgs {
  GridP g;
  const TriRec64* rec;
  const float4* box32;
  int64_t nel;
  int chunk;            // triangles per block, a multiple of 32
  int lanes;            // threads per triangle and axis, a power of two; times gridDim.z blocks
  float ihf, bo[3], rm;  // node = ihf * (mesh-local FP32 coordinate) + bo, within rm cells
  int64_t base_y, base_z;
  int32_t* row_cnt;
  const int32_t* row_off;
  int32_t* row_cur;
  RowHit* hits;
  double2* where;
  int32_t* hrow;
  uint32_t* flags[3];   // per axis a bit per triangle: whether it has hits
  int64_t* counters;
};

template <int AX, bool kFill>
__device__ __forceinline__ bool tri_rows(const RowArgs& A, const TriRec64& r, uint32_t sub, uint32_t stride, int64_t& nhit,
                                         int64_t& nband) {
  const GridP& g = A.g;
  const int b = AX == 0 ? 1 : 0, c = AX == 2 ? 1 : 2;
  const int64_t row_base = AX == 0 ? 0 : (AX == 1 ? A.base_y : A.base_z);
  int64_t b0, b1, c0, c1;
  if (!axis_range2(g, b, fmin(r.v[b], fmin(r.v[3 + b], r.v[6 + b])), fmax(r.v[b], fmax(r.v[3 + b], r.v[6 + b])), b0, b1))
    return false;
  if (!axis_range2(g, c, fmin(r.v[c], fmin(r.v[3 + c], r.v[6 + c])), fmax(r.v[c], fmax(r.v[3 + c], r.v[6 + c])), c0, c1))
    return false;
  bool hit = false;
  const uint32_t nb = (uint32_t)(b1 - b0 + 1), rows = nb * (uint32_t)(c1 - c0 + 1);
  for (uint32_t q = sub; q < rows; q += stride) {
    const uint32_t qc = q / nb;
    const int64_t jc = c0 + qc, jb = b0 + (q - qc * nb);
    const double oc = da(g.o[c], dm(g.h, (double)gidx(g, c, jc))), ob = da(g.o[b], dm(g.h, (double)gidx(g, b, jb)));
    const int64_t row = row_base + jc * g.n[b] + jb;
    const int dec = row_test32<AX>(r, ob, oc);
    if (dec == 0) continue;
    if (!kFill) {
      if (dec == 2) ++nband;  // inside the FP32 band: the FP64 test decides
      if (dec == 1 || row_test<AX>(r, ob, oc, nullptr)) {
        atomicAdd(&A.row_cnt[row], 1);
        ++nhit;
        hit = true;
      }
    } else {
      RowHit R;
      if (row_test<AX>(r, ob, oc, &R)) {  // the hit's FP64 constants (and the band's decision)
        const int32_t pos = A.row_off[row] + atomicAdd(&A.row_cur[row], 1);
        A.hits[pos] = R;
        // the hit's coordinate, and a bound on |t - (coordinate - xa)| over the row's nodes: t is formed
        // from terms of these absolute sums by at most a dozen roundings, f's own error among them
        const double x0 = g.o[AX] + g.h * (double)gidx(g, AX, 0), x1 = g.o[AX] + g.h * (double)gidx(g, AX, g.N[AX]);
        const double S = fmax(fabs(x0 - R.v1a), fabs(x1 - R.v1a));
        const double sum = fabs(R.P) + fabs(R.fa) * (fabs(R.K1) + S * fabs(R.ea)) +
                           fabs(R.fb) * (fabs(R.K2) + S * fabs(R.eb));
        const double x = R.v1a + row_t<AX>(R, R.v1a), e = 7.2e-15 * (fabs(R.f) * sum + S + fabs(R.v1a));
        A.where[pos] = make_double2(x, e);
        A.hrow[pos] = (int32_t)row;
      }
    }
  }
  return hit;
}

// The row hits: counted per row, then (kFill) written to their places.  A block lists its triangles per
// axis -- those with a row of the grid across their box (FP32, with a margin), in the second pass those
// that had hits -- and works the lists off, so that the warps of the FP64 part are full whatever share of
// the triangles reaches a row.  Measured for both passes on 1.4M and 5.8M triangles (B200): 106 and 428 us,
// against 209 and 800 with a thread per triangle for all axes.  Bound: the latency of the records' reads.
// Meshes too small to fill the GPU that way get a block per axis (gridDim.y) and several threads and blocks
// (gridDim.z) for the rows of one triangle: 5k triangles on 149k nodes 54 -> 14 us.
constexpr int kRowThreads = 128, kRowChunk = 8 * kRowThreads;

template <bool kFill>
__global__ void __launch_bounds__(kRowThreads) k_rows(const __grid_constant__ RowArgs A) {
  __shared__ uint16_t s_list[3][kRowChunk];
  __shared__ uint32_t s_flag[3][kRowChunk / 32];
  __shared__ int s_n[3];
  const int lane = threadIdx.x & 31;
  const int64_t first = (int64_t)blockIdx.x * A.chunk;
  const int m = (int)min((int64_t)A.chunk, A.nel - first);
  const unsigned axes = gridDim.y == 1 ? 7u : 1u << blockIdx.y;
  if (threadIdx.x < 3) s_n[threadIdx.x] = 0;
  for (int t = threadIdx.x; t < 3 * (kRowChunk / 32); t += kRowThreads) s_flag[0][t] = 0u;
  __syncthreads();
  for (int t0 = 0; t0 < m; t0 += kRowThreads) {
    const int t = t0 + threadIdx.x;
    unsigned want = 0u;  // axes whose rows may meet the triangle
    if (t < m) {
      if (kFill) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if ((axes >> a) & 1u) want |= ((A.flags[a][(first + t) >> 5] >> (t & 31)) & 1u) << a;
      } else {
        const float4 b0 = A.box32[2 * (first + t)], b1 = A.box32[2 * (first + t) + 1];
        const float lo[3] = {b0.x, b0.y, b0.z}, hi[3] = {b1.x, b1.y, b1.z};
        bool some[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float f0 = fmaf(lo[a], A.ihf, A.bo[a]) - A.rm, f1 = fmaf(hi[a], A.ihf, A.bo[a]) + A.rm;
          some[a] = !(floorf(f1) < ceilf(f0) || f1 < 0.f || f0 > (float)A.g.N[a]);
        }
        want = axes & ((unsigned)(some[1] && some[2]) | (unsigned)(some[0] && some[2]) << 1 | (unsigned)(some[0] && some[1]) << 2);
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned in = __ballot_sync(0xffffffffu, (want >> a) & 1u);
      if (!in) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(&s_n[a], __popc(in));
      at = __shfl_sync(0xffffffffu, at, 0);
      if ((want >> a) & 1u) s_list[a][at + __popc(in & ((1u << lane) - 1u))] = (uint16_t)t;
    }
  }
  __syncthreads();
  int64_t nhit = 0, nband = 0;
  auto axis = [&](auto ax) {
    constexpr int AX = decltype(ax)::value;
    const uint32_t L = (uint32_t)A.lanes, sub = threadIdx.x & (L - 1u);
    for (int q = threadIdx.x / L; q < s_n[AX]; q += kRowThreads / L) {
      const int t = s_list[AX][q];
      if (tri_rows<AX, kFill>(A, A.rec[first + t], sub + L * blockIdx.z, L * gridDim.z, nhit, nband))
        atomicOr(&s_flag[AX][t >> 5], 1u << (t & 31));
    }
  };
  axis(std::integral_constant<int, 0>());
  axis(std::integral_constant<int, 1>());
  axis(std::integral_constant<int, 2>());
  if (!kFill) {
    __syncthreads();
    for (int t = threadIdx.x; t < 3 * (kRowChunk / 32); t += kRowThreads)
      if (s_flag[0][t]) atomicOr(A.flags[t / (kRowChunk / 32)] + (first >> 5) + t % (kRowChunk / 32), s_flag[0][t]);
    for (int off = 16; off > 0; off >>= 1) {
      nhit += __shfl_down_sync(0xffffffffu, nhit, off);
      nband += __shfl_down_sync(0xffffffffu, nband, off);
    }
    if (lane == 0 && nhit) count_add(A.counters, C_ROW_HITS, nhit);
    if (lane == 0 && nband) count_add(A.counters, C_SIGN_BAND, nband);
  }
}

// Per row two flags, from its hits, a thread per hit against those before it.  Hits certainly within eps / 4
// of one another are one hit to every node outside their bounds: all but the first get a negative bound (its
// magnitude stays), and kRowOdd says whether their number is odd.  kRowClose: two hits of the row are neither
// that close nor certainly more than eps apart, or there are too many of them to compare (then over[0] counts
// the row too).  A thread per row took 61 us where rows have up to a few dozen hits (131k triangles, 24k rows),
// this 6 us (B200).
constexpr unsigned kRowClose = 1u, kRowOdd = 2u;
__global__ void k_hit_info(int64_t total, const int32_t* __restrict__ hrow, const int32_t* __restrict__ row_off,
                           const int32_t* __restrict__ row_cnt, double2* __restrict__ where, uint32_t* __restrict__ flag,
                           int32_t* __restrict__ over) {
  for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < total; h += (int64_t)gridDim.x * blockDim.x) {
    const int row = hrow[h], off = row_off[row], n = row_cnt[row], a = (int)(h - off);
    if (n > kRowCap) {
      if (a == 0) {
        atomicAdd(over, 1);
        atomicOr(flag + row, kRowClose);
      }
      continue;
    }
    const double px = where[h].x, py = fabs(where[h].y);
    bool same = false, close = false;
    for (int b = 0; b < a; ++b) {
      const double gap = fabs(px - where[off + b].x), e = 2.0 * (py + fabs(where[off + b].y));
      const bool near = gap + e < 0.25 * kEps;
      same = same || near;
      close = close || (!near && !(gap > kEps + e));
    }
    if (close) atomicOr(flag + row, kRowClose);
    if (same) {
      where[h].y = -py;
      atomicXor(flag + row, kRowOdd);
    }
  }
}

// Number of distinct hits (gaps > eps) among sorted t values passing the direction's t > eps.
__device__ __forceinline__ int clusters_pos(const double* ts, int n) {
  int c = 0;
  double prev = 0.0;
  for (int a = 0; a < n; ++a) {
    if (!(ts[a] > kEps)) continue;
    if (c == 0 || fabs(ds(ts[a], prev)) > kEps) ++c;
    prev = ts[a];
  }
  return c;
}
__device__ __forceinline__ int clusters_neg(const double* ts, int n) {
  // the -axis ray sees t' = -t; ascending t' is descending t
  int c = 0;
  double prev = 0.0;
  for (int a = n - 1; a >= 0; --a) {
    const double tn = -ts[a];
    if (!(tn > kEps)) continue;
    if (c == 0 || fabs(ds(tn, prev)) > kEps) ++c;
    prev = tn;
  }
  return c;
}

// Parities of the +AX / -AX rays at coordinate xa of a row, from t of all its hits (bit 0: +AX, bit 1: -AX).
template <int AX>
__device__ __noinline__ uint8_t row_parity(const RowHit* __restrict__ hits, int n, double xa) {
  double ts[kRowCap];
  for (int q = 0; q < n; ++q) {
    const double tv = row_t<AX>(hits[q], xa);
    int p = q - 1;
    while (p >= 0 && ts[p] > tv) { ts[p + 1] = ts[p]; --p; }
    ts[p + 1] = tv;
  }
  return (uint8_t)((clusters_pos(ts, n) & 1) | ((clusters_neg(ts, n) & 1) << 1));
}

struct MaskArgs {
  GridP g;
  int64_t nrows[3], base[3];  // rows along x, y, z, and the first of each among all rows
  int64_t mbase[4];           // first mask word of each axis, and their number
  const int32_t *off, *cnt;   // per row: its first hit, their number
  const uint32_t* flag;       // and flags (k_hit_info)
  const RowHit* hits;
  const double2* where;
  uint2* mask;  // per axis [word of 32 nodes][row]: bits of the +AX and of the -AX ray
};

// One thread per row and 32 of its nodes.  Bound: the reads of the rows' hits, which the words of a row
// share in L2.
template <int AX>
__device__ __forceinline__ void row_mask(const MaskArgs& A, int64_t q) {
  const GridP& g = A.g;
  const int64_t word = q / A.nrows[AX], row = q - word * A.nrows[AX];
  const int64_t r0 = A.base[AX] + row;
  const int n = A.cnt[r0];
  uint2 m = make_uint2(0u, 0u);
  if (n > 0 && n <= kRowCap) {
    const int first = (int)(word * 32), last = (int)min((int64_t)31, g.n[AX] - 1 - first);  // this word's nodes
    const int off = A.off[r0];
    const unsigned flag = A.flag[r0];
    unsigned exact = (flag & kRowClose) ? 0xffffffffu : 0u;
    if (!exact) {
      const double o = g.o[AX] + g.h * (double)gidx(g, AX, 0), inv = 1.0 / g.h;
      const double slack = fabs(g.o[AX]) * inv + (double)g.n[AX] + 1.0;
      for (int a = 0; a < n; ++a) {
        const double2 c = A.where[off + a];
        // the hit in nodes from the row's first, and the half width of the window around it in which t's
        // sign against eps is open (eps, t's bound, and the roundings of this line and of the nodes)
        const double r = (c.x - o) * inv;
        const double w = 1.01 * (kEps + fabs(c.y)) * inv + 1e-13 * (fabs(r) + fabs(c.x) * inv + slack);
        if (!(fabs(r) + w < 1e9)) { exact = 0xffffffffu; break; }
        const int lo = max(0, min(32, (int)ceil(r - w) - first)), hi = max(-1, min(31, (int)floor(r + w) - first));
        const unsigned below = lo == 32 ? 0xffffffffu : (1u << lo) - 1u;  // nodes below the hit
        if (!signbit(c.y)) m.x ^= below;
        if (hi >= lo) exact |= (0xffffffffu >> (31 - hi)) & ~below;
      }
      m.y = (((unsigned)n & 1u) ^ ((flag & kRowOdd) ? 1u : 0u)) ? ~m.x : m.x;
    }
    exact &= 0xffffffffu >> (31 - last);
    while (exact) {
      const int b = __ffs(exact) - 1;
      exact &= exact - 1u;
      const unsigned par = row_parity<AX>(A.hits + off, n, da(g.o[AX], dm(g.h, (double)gidx(g, AX, first + b))));
      m.x = (m.x & ~(1u << b)) | ((par & 1u) << b);
      m.y = (m.y & ~(1u << b)) | ((par >> 1) << b);
    }
  }
  A.mask[A.mbase[AX] + q] = m;
}

__global__ void __launch_bounds__(128) k_row_masks(const __grid_constant__ MaskArgs A) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= A.mbase[3]) return;
  if (q < A.mbase[1]) row_mask<0>(A, q);
  else if (q < A.mbase[2]) row_mask<1>(A, q - A.mbase[1]);
  else row_mask<2>(A, q - A.mbase[2]);
}

// adaptive_point_in_mesh_raycast (:234-288).  cast(i) returns the parity of ray i (1-based) or
// -1 when that ray is not available to the caller.
template <class Cast>
__device__ __forceinline__ int vote_logic(int min_rays, int max_rays, Cast cast, double& sign, double& conf,
                                          int& total_out) {
  int inside = 0, total = 0;
  for (int i = 1; i <= min_rays; ++i) {
    const int r = cast(i);
    if (r < 0) return 1;
    inside += r;
    ++total;
  }
  double ratio = dd((double)inside, (double)total);
  double cf = fmax(ratio, ds(1.0, ratio));
  int used = min_rays;
  while (cf < 0.85 && used < max_rays) {
    const int batch = min(4, max_rays - used);
    for (int i = used + 1; i <= used + batch; ++i) {
      if (i <= 36) {
        const int r = cast(i);
        if (r < 0) return 1;
        inside += r;
        ++total;
      }
    }
    used += batch;
    ratio = dd((double)inside, (double)total);
    cf = fmax(ratio, ds(1.0, ratio));
    if (cf > 0.95) break;
  }
  sign = ratio > 0.5 ? 1.0 : -1.0;
  conf = cf;
  total_out = total;
  return 0;
}

__device__ __forceinline__ int axis_bit(unsigned px, unsigned py, unsigned pz, int i) {
  // rays 1..6: +X +Y +Z -X -Y -Z
  switch (i) {
    case 1: return px & 1;
    case 2: return py & 1;
    case 3: return pz & 1;
    case 4: return (px >> 1) & 1;
    case 5: return (py >> 1) & 1;
    default: return (pz >> 1) & 1;
  }
}

struct VoteArgs {
  GridP g;
  const uint2* mask[3];     // the axes' masks, [word][row]
  const int32_t* row_cnt;   // rows along x, then y, then z
  const int32_t* over;      // rows with more than kRowCap hits
  uint32_t tiles[3];
  int min_rays, max_rays;
  double conf_thresh;
  int use_winding;
  double* sign;
  double* conf;
  int32_t* und_list;
  uint64_t* und_have;
  uint64_t* und_par;
  int32_t* wind_list;
  int64_t* counters;
};

// The vote of a node whose six rays differ (or that cannot be decided here): the result, or its place in
// the lists of the nodes that go on.
__device__ __noinline__ void vote_node(const VoteArgs& A, int64_t lin, unsigned px, unsigned py, unsigned pz, bool ovf) {
  double s, cf;
  int total;
  if (vote_logic(A.min_rays, A.max_rays, [&](int r) { return (r <= 6 && !ovf) ? axis_bit(px, py, pz, r) : -1; }, s, cf,
                 total)) {
    const int64_t slot = atomicAdd((unsigned long long*)&A.counters[C_LIST_UNDECIDED], 1ULL);
    A.und_list[slot] = (int32_t)lin;
    uint64_t have = 0, par = 0;
    if (!ovf) {
      have = 0x3FULL;
      for (int r = 1; r <= 6; ++r) par |= (uint64_t)axis_bit(px, py, pz, r) << (r - 1);
    }
    A.und_have[slot] = have;
    A.und_par[slot] = par;
    return;
  }
  if (A.use_winding && cf < A.conf_thresh) {
    const int64_t slot = atomicAdd((unsigned long long*)&A.counters[C_LIST_WINDING], 1ULL);
    A.wind_list[slot] = (int32_t)lin;
    cf = 0.8;
  }
  A.sign[lin] = s;
  if (A.conf) A.conf[lin] = cf;
}

// The vote of every node from the rows' masks: one warp per 32 x kVoteJ x kVoteK nodes, a lane per column, so
// that a mask word is read once for kVoteJ or kVoteK nodes of a lane.  Measured on 16.8M nodes and 321k hits
// (B200): 52 us, and 23 us for the masks and the rows' flags, against 0.78 ms for a pass per axis in row order (which evaluated every
// t, and wrote its parities a sector per byte along y and z) and the vote, 0.10 ms for the radix sort of
// the hits that it needed, and 0.22 ms for comparing each node with its rows' hits.  Bound: the 8 or 16 bytes
// a node it writes.
constexpr int kVoteJ = 4, kVoteK = 4;
static_assert(32 % kVoteJ == 0 && 32 % kVoteK == 0 && kVoteJ * kVoteK <= 32, "a tile's rows lie in one word");
__global__ void __launch_bounds__(256) k_vote(const __grid_constant__ VoteArgs A) {
  const GridP& g = A.g;
  const int lane = threadIdx.x & 31;
  const int nx = (int)g.n[0], ny = (int)g.n[1], nz = (int)g.n[2];
  const bool over = *A.over != 0;
  const uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t tj = w / A.tiles[0], ti = w - tj * A.tiles[0], tk = tj / A.tiles[1];
  if (tk >= A.tiles[2]) return;
  const int i = (int)ti * 32 + lane, j0 = (int)(tj - tk * A.tiles[1]) * kVoteJ, k0 = (int)tk * kVoteK;
  const bool in = i < nx;
  uint2 mx = make_uint2(0u, 0u), my[kVoteK], mz[kVoteJ];
  {
    const int j = j0 + lane % kVoteJ, k = k0 + lane / kVoteJ;
    if (lane < kVoteJ * kVoteK && j < ny && k < nz) mx = A.mask[0][(int64_t)ti * ((int64_t)ny * nz) + (int64_t)k * ny + j];
  }
#pragma unroll
  for (int k = 0; k < kVoteK; ++k) {
    my[k] = make_uint2(0u, 0u);
    if (in && k0 + k < nz) my[k] = A.mask[1][(int64_t)(j0 >> 5) * ((int64_t)nx * nz) + (int64_t)(k0 + k) * nx + i];
    my[k].x >>= j0 & 31;
    my[k].y >>= j0 & 31;
  }
#pragma unroll
  for (int j = 0; j < kVoteJ; ++j) {
    mz[j] = make_uint2(0u, 0u);
    if (in && j0 + j < ny) mz[j] = A.mask[2][(int64_t)(k0 >> 5) * ((int64_t)nx * ny) + (int64_t)(j0 + j) * nx + i];
    mz[j].x >>= k0 & 31;
    mz[j].y >>= k0 & 31;
  }
#pragma unroll
  for (int k = 0; k < kVoteK; ++k) {
#pragma unroll
    for (int j = 0; j < kVoteJ; ++j) {
      const unsigned xp = __shfl_sync(0xffffffffu, mx.x, k * kVoteJ + j), xn = __shfl_sync(0xffffffffu, mx.y, k * kVoteJ + j);
      if (!in || j0 + j >= ny || k0 + k >= nz) continue;
      const int64_t lin = ((int64_t)(k0 + k) * ny + (j0 + j)) * nx + i;
      const unsigned px = ((xp >> lane) & 1u) | (((xn >> lane) & 1u) << 1);
      const unsigned py = ((my[k].x >> j) & 1u) | (((my[k].y >> j) & 1u) << 1);
      const unsigned pz = ((mz[j].x >> k) & 1u) | (((mz[j].y >> k) & 1u) << 1);
      bool ovf = false;
      if (over) {
        const int64_t Rx = (int64_t)ny * nz, Ry = (int64_t)nx * nz;
        ovf = A.row_cnt[(int64_t)(k0 + k) * ny + (j0 + j)] > kRowCap || A.row_cnt[Rx + (int64_t)(k0 + k) * nx + i] > kRowCap ||
              A.row_cnt[Rx + Ry + (int64_t)(j0 + j) * nx + i] > kRowCap;
      }
      const unsigned all = px & py & pz, any = px | py | pz;
      if (A.min_rays == 6 && !ovf && (all == 3u || any == 0u) && !(A.use_winding && 1.0 < A.conf_thresh)) {
        A.sign[lin] = any ? 1.0 : -1.0;  // six equal rays: ratio 1 or 0, confidence 1
        if (A.conf) A.conf[lin] = 1.0;
      } else {
        vote_node(A, lin, px, py, pz, ovf);
      }
    }
  }
}

struct RayArgs {
  GridP g;
  const BNode* nodes;
  const int32_t* leaf_prim;
  const TriRec64* rec;
  float pad;
  int64_t max_visits;
  const int32_t* list;
  int min_rays, max_rays;
  double conf_thresh;
  int use_winding;
  double* sign;
  double* conf;
  int32_t* wind_list;
  int64_t* counters;
  uint64_t* have;     // per undecided node: rays whose parity is known
  uint64_t* parbits;  // per undecided node: their parities
  uint8_t* done;
  int32_t* req_node;  // requests of the current round
  int8_t* req_ray;
  int64_t* rq_cnt;    // requests per round
  int speculative;    // request all remaining rays at once (latency-bound when few nodes remain)
  int last_ray;       // last ray index the vote can cast: min(36, max(min_rays, max_rays))
};

__device__ __forceinline__ void child_box2(const BNode& nd, int side, float3& lo, float3& hi) {
  if (side == 0) {
    lo = make_float3(nd.a.x, nd.a.y, nd.a.z);
    hi = make_float3(nd.a.w, nd.b.x, nd.b.y);
  } else {
    lo = make_float3(nd.b.z, nd.b.w, nd.c.x);
    hi = make_float3(nd.c.y, nd.c.z, nd.c.w);
  }
}

// ray_triangle_intersection (:64-106) for a ray of any direction decided in FP32 with explicit
// error bands: 0 = the FP64 test certainly misses, 1 = it certainly hits, 2 = a decision lies in
// its band.  Inputs are the FP64 differences the reference forms (e1, e2, s = o - v1) and the
// direction, each rounded once to FP32.  Each component of h = d x e2 and q = s x e1 is within
// 4u of its FP64 value times its absolute-value sum (u = 2^-24), and each three-term dot product
// over them within 12u times the dot product of the absolute-value sums; the quotients u, v, t
// then carry the bound of row_test32's comment.  The caller replays mt64 for every hit, certain or
// not: the hit's t in FP64 is what the reference sorts and de-duplicates within eps.
__device__ __forceinline__ int mt32(const d3& o, const d3& d, const d3& v1, const d3& v2, const d3& v3) {
  const float3 e1 = make_float3((float)ds(v2.x, v1.x), (float)ds(v2.y, v1.y), (float)ds(v2.z, v1.z));
  const float3 e2 = make_float3((float)ds(v3.x, v1.x), (float)ds(v3.y, v1.y), (float)ds(v3.z, v1.z));
  const float3 sv = make_float3((float)ds(o.x, v1.x), (float)ds(o.y, v1.y), (float)ds(o.z, v1.z));
  const float3 dv = make_float3((float)d.x, (float)d.y, (float)d.z);
  // h = d x e2 and the absolute-value sums of its terms
  const float3 h = make_float3(__fsub_rn(__fmul_rn(dv.y, e2.z), __fmul_rn(dv.z, e2.y)),
                               __fsub_rn(__fmul_rn(dv.z, e2.x), __fmul_rn(dv.x, e2.z)),
                               __fsub_rn(__fmul_rn(dv.x, e2.y), __fmul_rn(dv.y, e2.x)));
  const float3 th = make_float3(fabsf(dv.y * e2.z) + fabsf(dv.z * e2.y), fabsf(dv.z * e2.x) + fabsf(dv.x * e2.z),
                                fabsf(dv.x * e2.y) + fabsf(dv.y * e2.x));
  auto dot = [](float3 a, float3 b) { return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z)); };
  auto adot = [](float3 a, float3 t) { return fabsf(a.x) * t.x + fabsf(a.y) * t.y + fabsf(a.z) * t.z; };
  const float A = dot(e1, h);
  const float ea = 12.f * kU32 * adot(e1, th);
  const float aA = fabsf(A);
  if (aA + ea < (float)kEps) return 0;
  if (!(aA - ea >= (float)kEps) || !(aA >= 3.f * ea)) return 2;
  const float den = aA - ea;
  auto band = [&](float X, float e) { return (1.5f * e + 2.f * (fabsf(X) + 1.f) * ea) / den + 2.f * kU32 * (fabsf(X) + 1.f); };
  const float U = __fdiv_rn(dot(sv, h), A);
  const float Eu = band(U, 12.f * kU32 * adot(sv, th));
  if (U < -Eu || U > 1.f + Eu) return 0;
  const float3 q = make_float3(__fsub_rn(__fmul_rn(sv.y, e1.z), __fmul_rn(sv.z, e1.y)),
                               __fsub_rn(__fmul_rn(sv.z, e1.x), __fmul_rn(sv.x, e1.z)),
                               __fsub_rn(__fmul_rn(sv.x, e1.y), __fmul_rn(sv.y, e1.x)));
  const float3 tq = make_float3(fabsf(sv.y * e1.z) + fabsf(sv.z * e1.y), fabsf(sv.z * e1.x) + fabsf(sv.x * e1.z),
                                fabsf(sv.x * e1.y) + fabsf(sv.y * e1.x));
  const float V = __fdiv_rn(dot(dv, q), A);
  const float Ev = band(V, 12.f * kU32 * adot(dv, tq));
  if (V < -Ev) return 0;
  const float UV = __fadd_rn(U, V);
  const float Euv = Eu + Ev + 2.f * kU32 * fabsf(UV);
  if (UV > 1.f + Euv) return 0;
  const float T = __fdiv_rn(dot(e2, q), A);
  const float Et = band(T, 12.f * kU32 * adot(e2, tq));
  if (T + Et <= (float)kEps) return 0;
  if (U >= Eu && U <= 1.f - Eu && V >= Ev && UV <= 1.f - Euv && T - Et > (float)kEps) return 1;
  return 2;
}

// check_ray_inside_bvh (:114-154) on the LBVH.  Returns parity, or -1 on buffer/stack overflow.
// *band counts the ray-triangle tests whose FP32 decision fell in its band.
__device__ int ray_parity(const RayArgs& A, const d3& p, const float3& p32, int dir, int64_t* band) {
  const d3 d = {c_dirs[3 * dir], c_dirs[3 * dir + 1], c_dirs[3 * dir + 2]};
  const float3 d32 = make_float3((float)d.x, (float)d.y, (float)d.z);
  const float3 inv = make_float3(1.0f / d32.x, 1.0f / d32.y, 1.0f / d32.z);
  double ts[kRayCap];
  int n = 0;
  int stack[kStack];
  int sp = 0;
  stack[sp++] = 0;
  int64_t visits = 0;
  while (sp > 0) {
    if (++visits > A.max_visits) return -1;
    const BNode nd = A.nodes[stack[--sp]];
    const int ch[2] = {nd.d.x, nd.d.y};
    for (int side = 0; side < 2; ++side) {
      float3 lo, hi;
      child_box2(nd, side, lo, hi);
      if (lo.x > hi.x) continue;
      if (!ray_box(p32, d32, inv, lo, hi, A.pad, A.pad)) continue;
      if (ch[side] & kLeafBit) {
        const TriRec64& r = A.rec[A.leaf_prim[ch[side] & 0x7fffffff]];
        const int dec = mt32(p, d, rec_v(r, 0), rec_v(r, 1), rec_v(r, 2));
        if (dec == 0) continue;
        if (dec == 2) ++*band;
        double t;
        if (mt64(p, d, rec_v(r, 0), rec_v(r, 1), rec_v(r, 2), kEps, t)) {
          if (n >= kRayCap) return -1;
          int q = n - 1;
          while (q >= 0 && ts[q] > t) { ts[q + 1] = ts[q]; --q; }
          ts[q + 1] = t;
          ++n;
        }
      } else {
        if (sp >= kStack) return -1;
        stack[sp++] = ch[side];
      }
    }
  }
  if (n == 0) return 0;
  int unique = 1;
  for (int a = 1; a < n; ++a)
    if (fabs(ds(ts[a], ts[a - 1])) > kEps) ++unique;
  return unique & 1;
}

// The reference's vote (:234-288) replayed over the rays whose parity is already known (bit i-1
// of `have` / `par` for ray i).  Returns 0 with sign/conf when the vote is decided; otherwise 1
// with [need_lo, need_hi] = the rays of the first incomplete step (the initial min_rays, or the
// current batch of 4), which the caller requests all at once.
__device__ __forceinline__ int vote_known(uint64_t have, uint64_t par, int min_rays, int max_rays, double& sign,
                                          double& conf, int& need_lo, int& need_hi) {
  int inside = 0, total = 0;
  for (int i = 1; i <= min_rays; ++i) {
    if (!((have >> (i - 1)) & 1)) { need_lo = i; need_hi = min_rays; return 1; }
    inside += (int)((par >> (i - 1)) & 1);
    ++total;
  }
  double ratio = dd((double)inside, (double)total);
  double cf = fmax(ratio, ds(1.0, ratio));
  int used = min_rays;
  while (cf < 0.85 && used < max_rays) {
    const int batch = min(4, max_rays - used);
    for (int i = used + 1; i <= used + batch; ++i) {
      if (i <= 36) {
        if (!((have >> (i - 1)) & 1)) { need_lo = i; need_hi = min(used + batch, 36); return 1; }
        inside += (int)((par >> (i - 1)) & 1);
        ++total;
      }
    }
    used += batch;
    ratio = dd((double)inside, (double)total);
    cf = fmax(ratio, ds(1.0, ratio));
    if (cf > 0.95) break;
  }
  sign = ratio > 0.5 ? 1.0 : -1.0;
  conf = cf;
  return 0;
}

// One round of the adaptive vote over the undecided nodes: decide, or request the next rays.
__global__ void k_round(RayArgs A, int64_t nund, int round, int last) {
  const GridP& g = A.g;
  int64_t* rq_cnt = A.rq_cnt + round;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nund; q += (int64_t)gridDim.x * blockDim.x) {
    if (A.done[q]) continue;
    double s, cf;
    int lo, hi;
    const uint64_t have = A.have[q], par = A.parbits[q];
    if (vote_known(have, par, A.min_rays, A.max_rays, s, cf, lo, hi)) {
      if (last) {  // unreachable: the rounds cover every batch up to the 36th direction
        count_add(A.counters, C_ERR_CAPACITY, 1);
        continue;
      }
      if (A.speculative) hi = A.last_ray;  // few nodes: cast every ray the vote could still need
      for (int i = lo; i <= hi; ++i) {
        if ((have >> (i - 1)) & 1) continue;
        const int64_t slot = atomicAdd((unsigned long long*)rq_cnt, 1ULL);
        A.req_node[slot] = (int32_t)q;
        A.req_ray[slot] = (int8_t)i;
      }
      continue;
    }
    const int64_t lin = A.list[q];
    if (A.use_winding && cf < A.conf_thresh) {
      const int64_t slot = atomicAdd((unsigned long long*)&A.counters[C_LIST_WINDING], 1ULL);
      A.wind_list[slot] = (int32_t)lin;
      cf = 0.8;
    }
    A.sign[lin] = s;
    if (A.conf) A.conf[lin] = cf;
    A.done[q] = 1;
    (void)g;
  }
}

// Casts the requested rays of a round, one thread per (node, ray).
__global__ void __launch_bounds__(128) k_rays(RayArgs A, int round) {
  const GridP& g = A.g;
  const int64_t count = A.rq_cnt[round];
  int64_t rays = 0, band = 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = A.req_node[t];
    const int r = A.req_ray[t];
    const int64_t lin = A.list[q];
    const int64_t i = lin % g.n[0], j = (lin / g.n[0]) % g.n[1], k = lin / (g.n[0] * g.n[1]);
    const d3 p = gnode(g, i, j, k);
    const float3 p32 = make_float3((float)(p.x - g.center[0]), (float)(p.y - g.center[1]), (float)(p.z - g.center[2]));
    int v = ray_parity(A, p, p32, r - 1, &band);
    if (v < 0) { count_add(A.counters, C_ERR_CAPACITY, 1); v = 0; }
    const uint64_t bit = 1ULL << (r - 1);
    if (v) atomicOr((unsigned long long*)&A.parbits[q], (unsigned long long)bit);
    atomicOr((unsigned long long*)&A.have[q], (unsigned long long)bit);
    ++rays;
  }
  for (int off = 16; off > 0; off >>= 1) {
    rays += __shfl_down_sync(0xffffffffu, rays, off);
    band += __shfl_down_sync(0xffffffffu, band, off);
  }
  if ((threadIdx.x & 31) == 0 && rays) count_add(A.counters, C_EXTRA_RAYS, rays);
  if ((threadIdx.x & 31) == 0 && band) count_add(A.counters, C_SIGN_BAND, band);
}

// The rays of a few undecided nodes against every triangle, without the LBVH (which then need not be
// built): one thread per triangle, all requested rays.  Most pairs end at a distance test of the
// triangle's centroid from the ray's line; the rest take the tests of ray_parity, so the hits are the same.
// The node's terms are formed once for its rays, whose directions are constant operands.  Bound: the test's
// 7 instructions a pair; 24 rays of one node against 1.4M and 5.8M triangles 45 and 112 us (B200),
// against 61 and 240 with origins and directions read from shared memory a pair.
constexpr int kRayGroup = 6;
__global__ void __launch_bounds__(128) k_rays_all(const __grid_constant__ RayArgs A, int nund, const float4* __restrict__ c32,
                                                  int64_t nel, float reach, float lim2, int32_t* __restrict__ hit_n,
                                                  double* __restrict__ hit_t) {
  __shared__ float4 s_o[kAllPairsNodes];  // origin (mesh-local), .w: node index
  __shared__ unsigned long long s_want[kAllPairsNodes];
  const GridP& g = A.g;
  int64_t band = 0;
  for (int q = threadIdx.x; q < nund; q += blockDim.x) {
    const int64_t lin = A.list[q];
    const int64_t i = lin % g.n[0], j = (lin / g.n[0]) % g.n[1], k = lin / (g.n[0] * g.n[1]);
    const d3 p = gnode(g, i, j, k);
    s_o[q] = make_float4((float)(p.x - g.center[0]), (float)(p.y - g.center[1]), (float)(p.z - g.center[2]),
                         __int_as_float((int)lin));
    s_want[q] = 0ULL;
  }
  __syncthreads();
  const int count = (int)A.rq_cnt[0];
  for (int t = threadIdx.x; t < count; t += blockDim.x)
    atomicOr(&s_want[A.req_node[t]], 1ULL << (A.req_ray[t] - 1));
  __syncthreads();
  for (int64_t el = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; el < nel; el += (int64_t)gridDim.x * blockDim.x) {
    const float4 c = c32[el];
    for (int q = 0; q < nund; ++q) {
      const unsigned long long want = s_want[q];
      if (!want) continue;
      const float4 o = s_o[q];
      // squared distance of the centroid from the line: |w|^2 - (w . d)^2, d a unit vector
      const float wx = c.x - o.x, wy = c.y - o.y, wz = c.z - o.z, ww = fmaf(wx, wx, fmaf(wy, wy, fmaf(wz, wz, -lim2)));
      unsigned long long pass = 0ULL;
#pragma unroll
      for (int r0 = 0; r0 < 36; r0 += kRayGroup) {
        constexpr unsigned kGroup = (1u << kRayGroup) - 1u;
        if (!((unsigned)(want >> r0) & kGroup)) continue;
        unsigned in = 0u;
#pragma unroll
        for (int r = 0; r < kRayGroup; ++r) {
          const float s = fmaf(wx, c_dirs32[3 * (r0 + r)], fmaf(wy, c_dirs32[3 * (r0 + r) + 1], wz * c_dirs32[3 * (r0 + r) + 2]));
          in |= (unsigned)(!(fmaf(-s, s, ww) > 0.f) && !(s < -reach)) << r;
        }
        pass |= (unsigned long long)in << r0;
      }
      for (pass &= want; pass; pass &= pass - 1ULL) {
        const int ray = __ffsll((long long)pass) - 1;
        const int64_t lin = __float_as_int(o.w);
        const int64_t i = lin % g.n[0], j = (lin / g.n[0]) % g.n[1], k = lin / (g.n[0] * g.n[1]);
        const d3 p = gnode(g, i, j, k);
        const d3 dir = {c_dirs[3 * ray], c_dirs[3 * ray + 1], c_dirs[3 * ray + 2]};
        const TriRec64& r = A.rec[el];
        const int dec = mt32(p, dir, rec_v(r, 0), rec_v(r, 1), rec_v(r, 2));
        if (dec == 0) continue;
        if (dec == 2) ++band;
        double tt;
        if (mt64(p, dir, rec_v(r, 0), rec_v(r, 1), rec_v(r, 2), kEps, tt)) {
          const int h = atomicAdd(hit_n + q * 36 + ray, 1);
          if (h < kRayCap) hit_t[(int64_t)(q * 36 + ray) * kRayCap + h] = tt;
        }
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) band += __shfl_down_sync(0xffffffffu, band, off);
  if ((threadIdx.x & 31) == 0 && band) count_add(A.counters, C_SIGN_BAND, band);
}

// Parities of those rays from their hits: sorted, distinct within eps (:114-154).
__global__ void k_rays_parity(RayArgs A, const int32_t* __restrict__ hit_n, double* __restrict__ hit_t) {
  const int count = (int)A.rq_cnt[0];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
    const int at = A.req_node[t] * 36 + A.req_ray[t] - 1, n = hit_n[at];
    int parity = 0;
    if (n > kRayCap) {
      count_add(A.counters, C_ERR_CAPACITY, 1);
    } else if (n > 0) {
      double* ts = hit_t + (int64_t)at * kRayCap;
      for (int a = 1; a < n; ++a) {
        const double v = ts[a];
        int b = a;
        while (b > 0 && ts[b - 1] > v) { ts[b] = ts[b - 1]; --b; }
        ts[b] = v;
      }
      int unique = 1;
      for (int a = 1; a < n; ++a)
        if (fabs(ds(ts[a], ts[a - 1])) > kEps) ++unique;
      parity = unique & 1;
    }
    const int64_t q = A.req_node[t];
    const uint64_t bit = 1ULL << (A.req_ray[t] - 1);
    if (parity) atomicOr((unsigned long long*)&A.parbits[q], (unsigned long long)bit);
    atomicOr((unsigned long long*)&A.have[q], (unsigned long long)bit);
    count_add(A.counters, C_EXTRA_RAYS, 1);
  }
}

// generalized_winding_number (:295-328).  The triangles are cut into fixed chunks; one CTA sums
// one chunk for one node (fixed-order block reduction) and k_winding_final adds the chunk sums
// in chunk order, so the result does not depend on scheduling and one node still fills the GPU.
constexpr int kWindChunk = 8192;

__global__ void __launch_bounds__(256) k_winding(GridP g, const TriRec64* __restrict__ rec, int64_t nel,
                                                 const int32_t* __restrict__ list, int64_t count, int nchunks,
                                                 double* __restrict__ partial) {
  __shared__ double red[256];
  const int chunk = blockIdx.x;
  for (int64_t q = blockIdx.y; q < count; q += gridDim.y) {
    const int64_t lin = list[q];
    const int64_t i = lin % g.n[0], j = (lin / g.n[0]) % g.n[1], k = lin / (g.n[0] * g.n[1]);
    const d3 p = gnode(g, i, j, k);
    double w = 0.0;
    const int64_t e1 = min((int64_t)(chunk + 1) * kWindChunk, nel);
    for (int64_t el = (int64_t)chunk * kWindChunk + threadIdx.x; el < e1; el += blockDim.x) {
      const TriRec64& r = rec[el];
      const d3 a = v_normalize(v_sub(rec_v(r, 0), p));
      const d3 b = v_normalize(v_sub(rec_v(r, 1), p));
      const d3 c = v_normalize(v_sub(rec_v(r, 2), p));
      const double num = v_dot(a, v_cross(b, c));
      const double den = da(da(da(1.0, v_dot(a, b)), v_dot(b, c)), v_dot(c, a));
      if (fabs(den) > 1e-10) {
        double sa = dm(2.0, atan2(fabs(num), den));
        if (num < 0) sa = -sa;
        w = da(w, sa);
      }
    }
    red[threadIdx.x] = w;
    __syncthreads();
    for (int s2 = blockDim.x / 2; s2 > 0; s2 >>= 1) {
      if ((int)threadIdx.x < s2) red[threadIdx.x] = da(red[threadIdx.x], red[threadIdx.x + s2]);
      __syncthreads();
    }
    if (threadIdx.x == 0) partial[q * nchunks + chunk] = red[0];
    __syncthreads();
  }
}

__global__ void k_winding_final(const int32_t* __restrict__ list, int64_t count, int nchunks,
                                const double* __restrict__ partial, double* sign, int64_t* counters) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x) {
    double w = 0.0;
    for (int c = 0; c < nchunks; ++c) w = da(w, partial[q * nchunks + c]);
    const double wn = dd(w, 12.566370614359172);  // 4π
    sign[list[q]] = fabs(wn) > 0.5 ? 1.0 : -1.0;
    count_add(counters, C_WINDING, 1);
    if (fabs(fabs(wn) - 0.5) < 1e-9) count_add(counters, C_WIND_AMBIG, 1);
  }
}

__global__ void k_combine(int64_t n, const double* __restrict__ dist, const double* __restrict__ sign,
                          double* __restrict__ sdf) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    sdf[q] = dm(dist[q], sign[q]);
}

}  // namespace

int upload_directions(sdfgpu_ctx* ctx, const double* dirs) {
  SDF_CUDA(ctx, cudaMemcpyToSymbolAsync(c_dirs, dirs, sizeof(double) * 108, 0, cudaMemcpyHostToDevice, ctx->stream));
  float d32[108];
  for (int q = 0; q < 108; ++q) d32[q] = (float)dirs[q];
  SDF_CUDA(ctx, cudaMemcpyToSymbolAsync(c_dirs32, d32, sizeof(d32), 0, cudaMemcpyHostToDevice, ctx->stream));
  return 0;
}

static RowArgs row_args(sdfgpu_ctx* ctx, const GridP& g, const SignPlan& P) {
  const MeshDev& M = ctx->mesh;
  RowArgs A{};
  A.g = g;
  A.rec = buf<TriRec64>(ctx, "rec");
  A.box32 = buf<float4>(ctx, "box32");
  A.nel = M.nel;
  const double ih = 1.0 / g.h;
  A.ihf = (float)ih;
  for (int a = 0; a < 3; ++a) A.bo[a] = (float)((M.center[a] - (g.o[a] + g.h * (double)gidx(g, a, 0))) * ih);
  A.rm = (float)(2e-6 * g.E * ih + 1e-4);
  A.base_y = P.Rx;
  A.base_z = P.Rx + P.Ry;
  A.row_cnt = P.row_cnt;
  A.row_off = P.row_off;
  A.row_cur = P.row_cur;
  for (int a = 0; a < 3; ++a) A.flags[a] = P.row_flags + a * cdiv(M.nel, 32);
  A.counters = ctx->d_counters;
  return A;
}

// The launch shape: as many threads per triangle and axis as fill the GPU, up to half the rows that the
// mesh's largest triangle can meet; one block for all axes where the triangles alone fill it.
static dim3 row_grid(const sdfgpu_ctx* ctx, RowArgs& A) {
  const MeshDev& M = ctx->mesh;
  const double side = std::min(2.0 * M.rho_max / A.g.h + 1.0, 64.0);
  const int64_t threads = 148 * 2048;
  int64_t per = 1;
  while (2 * per <= 0.5 * side * side && M.nel * 3 * 2 * per <= threads) per *= 2;
  A.lanes = (int)std::min<int64_t>(per, kRowThreads);
  const int64_t z = per / A.lanes, y = M.nel * 3 <= threads ? 3 : 1;
  A.chunk = 32 * (int)std::min<int64_t>(kRowChunk / 32, 1 + M.nel * y * z / (32 * 148 * 8));
  return dim3((unsigned)cdiv(M.nel, A.chunk), (unsigned)y, (unsigned)z);
}

int sign_begin(sdfgpu_ctx* ctx, const GridP& g, SignPlan& P) {
  cudaStream_t st = ctx->sign_stream;
  const int64_t nel = ctx->mesh.nel;
  P.Rx = g.n[1] * g.n[2];
  P.Ry = g.n[0] * g.n[2];
  P.Rz = g.n[0] * g.n[1];
  P.nrows = P.Rx + P.Ry + P.Rz;
  if (P.nrows >= 0x7fffffffLL) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "grid has too many rows");
  SDF_TRY(scratch_t(ctx, "row_cnt", (size_t)P.nrows + 1, &P.row_cnt));
  SDF_TRY(scratch_t(ctx, "row_off", (size_t)P.nrows + 1, &P.row_off));
  SDF_TRY(scratch_t(ctx, "row_cur", (size_t)P.nrows + 1, &P.row_cur));
  SDF_CUDA(ctx, cudaMemsetAsync(P.row_cnt, 0, sizeof(int32_t) * (P.nrows + 1), st));
  SDF_CUDA(ctx, cudaMemsetAsync(P.row_cur, 0, sizeof(int32_t) * (P.nrows + 1), st));
  SDF_TRY(scratch_t(ctx, "row_flags", (size_t)cdiv(nel, 32) * 3, &P.row_flags));
  SDF_CUDA(ctx, cudaMemsetAsync(P.row_flags, 0, sizeof(uint32_t) * cdiv(nel, 32) * 3, st));
  RowArgs A = row_args(ctx, g, P);
  const dim3 grid = row_grid(ctx, A);
  k_rows<false><<<grid, kRowThreads, 0, st>>>(A);
  SDF_KERNEL(ctx);
  SDF_TRY(cub_scan_i32(ctx, P.row_cnt, P.row_off, P.nrows + 1, st, "cub_tmp_scan_sign"));
  ctx->h_scalars[S_ROW_TOTAL] = -1;
  SDF_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + S_ROW_TOTAL, P.row_off + P.nrows, sizeof(int32_t),
                                cudaMemcpyDeviceToHost, st));
  SDF_CUDA(ctx, cudaEventRecord(ctx->ev_rows, st));
  return 0;
}

int sign_vote(sdfgpu_ctx* ctx, const GridP& g, SignPlan& P, int min_rays, int max_rays, double conf_thresh,
              int use_winding, double* d_sign, double* d_conf) {
  cudaStream_t st = ctx->sign_stream;
  const int64_t Rx = P.Rx, Ry = P.Ry, nrows = P.nrows;
  int32_t *row_cnt = P.row_cnt, *row_off = P.row_off;
  SDF_CUDA(ctx, cudaEventSynchronize(ctx->ev_rows));
  int32_t total;
  std::memcpy(&total, ctx->h_scalars + S_ROW_TOTAL, sizeof(int32_t));  // the low 4 bytes hold the int32
  if (total < 0) return fail(ctx, SDFGPU_ERR_CAPACITY, "more than 2^31 row hits");
  RowHit* hits;
  double2* where;
  int32_t *hrow, *over;
  uint32_t* row_flag;
  MaskArgs K;
  const size_t H = (size_t)std::max(total, 1);
  SDF_TRY(scratch_t(ctx, "row_hits", H, &hits));
  SDF_TRY(scratch_t(ctx, "row_where", H, &where));
  SDF_TRY(scratch_t(ctx, "row_hrow", H, &hrow));
  SDF_TRY(scratch_t(ctx, "row_flag", (size_t)nrows + 1, &row_flag));  // and the number of overfull rows
  over = reinterpret_cast<int32_t*>(row_flag + nrows);
  SDF_CUDA(ctx, cudaMemsetAsync(row_flag, 0, sizeof(uint32_t) * (nrows + 1), st));
  K.nrows[0] = Rx;
  K.nrows[1] = Ry;
  K.nrows[2] = P.Rz;
  K.base[0] = 0;
  K.base[1] = Rx;
  K.base[2] = Rx + Ry;
  K.mbase[0] = 0;
  for (int a = 0; a < 3; ++a) K.mbase[a + 1] = K.mbase[a] + cdiv(g.n[a], 32) * K.nrows[a];
  SDF_TRY(scratch_t(ctx, "row_mask", (size_t)K.mbase[3], &K.mask));
  if (total > 0) {
    RowArgs A = row_args(ctx, g, P);
    A.hits = hits;
    A.where = where;
    A.hrow = hrow;
    const dim3 grid = row_grid(ctx, A);
    k_rows<true><<<grid, kRowThreads, 0, st>>>(A);
    SDF_KERNEL(ctx);
    k_hit_info<<<grid_for(total, 128), 128, 0, st>>>(total, hrow, row_off, row_cnt, where, row_flag, over);
    SDF_KERNEL(ctx);
  }
  SDF_MARK_ON(ctx, T_ROWS, st);
  K.g = g;
  K.off = row_off;
  K.cnt = row_cnt;
  K.flag = row_flag;
  K.hits = hits;
  K.where = where;
  k_row_masks<<<(unsigned)cdiv(K.mbase[3], 128), 128, 0, st>>>(K);
  SDF_KERNEL(ctx);

  SDF_TRY(scratch_t(ctx, "und_list", (size_t)g.ngp, &P.und));
  SDF_TRY(scratch_t(ctx, "und_have", (size_t)g.ngp, &P.und_have));
  SDF_TRY(scratch_t(ctx, "und_par", (size_t)g.ngp, &P.und_par));
  SDF_TRY(scratch_t(ctx, "wind_list", (size_t)g.ngp, &P.wind));
  VoteArgs V;
  V.g = g;
  for (int a = 0; a < 3; ++a) V.mask[a] = K.mask + K.mbase[a];
  V.row_cnt = row_cnt;
  V.over = over;
  V.tiles[0] = (uint32_t)cdiv(g.n[0], 32);
  V.tiles[1] = (uint32_t)cdiv(g.n[1], kVoteJ);
  V.tiles[2] = (uint32_t)cdiv(g.n[2], kVoteK);
  V.min_rays = min_rays;
  V.max_rays = max_rays;
  V.conf_thresh = conf_thresh;
  V.use_winding = use_winding;
  V.sign = d_sign;
  V.conf = d_conf;
  V.und_list = P.und;
  V.und_have = P.und_have;
  V.und_par = P.und_par;
  V.wind_list = P.wind;
  V.counters = ctx->d_counters;
  const int64_t vote_warps = (int64_t)V.tiles[0] * V.tiles[1] * V.tiles[2];
  k_vote<<<(unsigned)cdiv(vote_warps, 8), 256, 0, st>>>(V);
  SDF_KERNEL(ctx);
  SDF_MARK_ON(ctx, T_PARITY, st);
  SDF_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + S_UNDECIDED, ctx->d_counters + C_LIST_UNDECIDED, 2 * sizeof(int64_t),
                                cudaMemcpyDeviceToHost, st));
  return 0;
}

int sign_finish(sdfgpu_ctx* ctx, const GridP& g, SignPlan& P, int min_rays, int max_rays, double conf_thresh,
                int use_winding, double* d_sign, double* d_conf) {
  cudaStream_t st = ctx->sign_stream;
  const MeshDev& M = ctx->mesh;
  const int64_t nel = M.nel;
  const TriRec64* rec = buf<TriRec64>(ctx, "rec");
  int32_t *und = P.und, *wind = P.wind;
  uint64_t *und_have = P.und_have, *und_par = P.und_par;
  SDF_CUDA(ctx, cudaStreamSynchronize(st));
  const int64_t nund = ctx->h_scalars[S_UNDECIDED];
  if (nund > 0) {
    // Rounds of the adaptive vote: decide what is decidable, cast the next requested rays.
    constexpr int kRounds = 12;  // initial rays + at most 8 batches reach the 36 directions
    uint8_t* done;
    int32_t* req_node;
    int8_t* req_ray;
    int64_t* rq_cnt;
    SDF_TRY(scratch_t(ctx, "und_done", (size_t)nund, &done));
    SDF_TRY(scratch_t(ctx, "req_node", (size_t)nund * 36, &req_node));
    SDF_TRY(scratch_t(ctx, "req_ray", (size_t)nund * 36, &req_ray));
    SDF_TRY(scratch_t(ctx, "rq_cnt", (size_t)kRounds + 1, &rq_cnt));
    SDF_CUDA(ctx, cudaMemsetAsync(done, 0, (size_t)nund, st));
    SDF_CUDA(ctx, cudaMemsetAsync(rq_cnt, 0, sizeof(int64_t) * (kRounds + 1), st));
    // Few nodes: their rays against all triangles, about 19 ps a node and triangle (0.11 ms for one node and
    // 5.8M triangles), instead of walks of the LBVH, which take 0.28 ms by their latency and the build that
    // nothing else in such a call needs (0.47 ms for 1.4M triangles, 0.33 ns a triangle): the sides meet at
    // about 20 nodes for many triangles, and at more for few.
    const bool all_pairs = nund <= kAllPairsNodes;
    if (!all_pairs) {
      SDF_TRY(ensure_tree(ctx, false));
      SDF_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_bvh, 0));  // the adaptive rays walk the LBVH
    }
    RayArgs R;
    R.g = g;
    R.nodes = buf<BNode>(ctx, "nodes");
    R.leaf_prim = buf<int32_t>(ctx, "leaf_prim");
    R.rec = rec;
    R.pad = (float)(2e-6 * g.E);
    R.max_visits = 2 * nel + 64;
    R.list = und;
    R.min_rays = min_rays;
    R.max_rays = max_rays;
    R.conf_thresh = conf_thresh;
    R.use_winding = use_winding;
    R.sign = d_sign;
    R.conf = d_conf;
    R.wind_list = wind;
    R.counters = ctx->d_counters;
    R.have = und_have;
    R.parbits = und_par;
    R.done = done;
    R.req_node = req_node;
    R.req_ray = req_ray;
    R.rq_cnt = rq_cnt;
    R.speculative = nund <= 8192;
    R.last_ray = std::min(36, std::max(min_rays, max_rays));
    const int rounds = R.speculative ? 1 : kRounds;
    for (int r = 0; r < rounds; ++r) {
      k_round<<<grid_for(nund, 128), 128, 0, st>>>(R, nund, r, 0);
      SDF_KERNEL(ctx);
      if (all_pairs) {
        int32_t* hit_n;
        double* hit_t;
        SDF_TRY(scratch_t(ctx, "ray_hit_n", (size_t)nund * 36, &hit_n));
        SDF_TRY(scratch_t(ctx, "ray_hit_t", (size_t)nund * 36 * kRayCap, &hit_t));
        SDF_CUDA(ctx, cudaMemsetAsync(hit_n, 0, sizeof(int32_t) * nund * 36, st));
        // a hit triangle's centroid is within rho of the line: with the errors of the FP32 coordinates in
        // it (4e-6 E), and of |w|^2 - (w . d)^2 (|w| at most 3.5 E: below 1e-5 E^2)
        const double rho = M.rho_max * (1.0 + 1e-5) + 4e-6 * g.E, lim2 = rho * rho + 1.5e-5 * g.E * g.E;
        k_rays_all<<<grid_for(nel, 128, 148 * 16), 128, 0, st>>>(R, (int)nund, buf<float4>(ctx, "c32"), nel,
                                                                 (float)std::sqrt(lim2), (float)lim2, hit_n, hit_t);
        SDF_KERNEL(ctx);
        k_rays_parity<<<grid_for(nund * 36, 64), 64, 0, st>>>(R, hit_n, hit_t);
      } else {
        k_rays<<<grid_for(nund * 8, 128, 148 * 32), 128, 0, st>>>(R, r);
      }
      SDF_KERNEL(ctx);
    }
    k_round<<<grid_for(nund, 128), 128, 0, st>>>(R, nund, kRounds, 1);
    SDF_KERNEL(ctx);
  }
  if (use_winding) {
    if (nund > 0) {  // their votes may have added to the list
      SDF_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + S_WINDING, ctx->d_counters + C_LIST_WINDING, sizeof(int64_t),
                                    cudaMemcpyDeviceToHost, st));
      SDF_CUDA(ctx, cudaStreamSynchronize(st));
    }
    const int64_t nw = ctx->h_scalars[S_WINDING];
    if (nw > 0) {
      const int nchunks = (int)cdiv(nel, kWindChunk);
      double* partial;
      SDF_TRY(scratch_t(ctx, "wind_partial", (size_t)nw * nchunks, &partial));
      dim3 grid((unsigned)nchunks, (unsigned)std::min<int64_t>(nw, 65535));
      k_winding<<<grid, 256, 0, st>>>(g, rec, nel, wind, nw, nchunks, partial);
      SDF_KERNEL(ctx);
      k_winding_final<<<grid_for(nw, 128), 128, 0, st>>>(wind, nw, nchunks, partial, d_sign, ctx->d_counters);
      SDF_KERNEL(ctx);
    }
  }
  return 0;
}

// sdf = dist .* sign (stl_to_sdf.jl:119) on the context stream.
int run_combine(sdfgpu_ctx* ctx, const GridP& g, const double* d_dist, const double* d_sign, double* d_sdf) {
  return launch_combine(ctx, g.ngp, d_dist, d_sign, d_sdf, ctx->stream);
}

int launch_combine(sdfgpu_ctx* ctx, int64_t ngp, const double* d_dist, const double* d_sign, double* d_sdf,
                   cudaStream_t st) {
  k_combine<<<grid_for(ngp, 256, 148 * 16), 256, 0, st>>>(ngp, d_dist, d_sign, d_sdf);
  SDF_KERNEL(ctx);
  return 0;
}

}  // namespace sdfgpu
