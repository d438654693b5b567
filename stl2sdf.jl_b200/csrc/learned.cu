// learned.cu -- the exact unbounded distances the learned radius trains on (SDFGPU_MODE_LEARNED):
// the true minimum point-triangle distance (dfOnTriangularMesh.jl:101-177 without the clamp at
// :202-206) at the nodes of a sparse coarse grid, one warp per node.  The learned-radius search over
// the full grid is the brick search of SDFGPU_MODE_UNBOUNDED (k_unbounded, distance.cu) with every
// lane's minimum started at its radius r(p).
#include "common.cuh"
#include "unbounded.cuh"

namespace sdfgpu {

namespace {

// Exact unbounded distances of a sparse node set (the coarse grid the radius network trains on): one
// warp per node, through the brick search (wide_search) with one lane's node in use.  On a coarse grid
// neighbouring nodes are far apart, so a brick of them would take the union of very different regions;
// the warp-wide steps (32 children or 32 triangles at a time) serve a single node as well.
// Results are those of the other unbounded searches (FP64 resolution of the FP32 band in ascending
// triangle index; FP64 re-search of a node whose band overflowed).
__global__ void __launch_bounds__(kUnbThreads, 4) k_nearest_points(const __grid_constant__ UnbArgs A) {
  __shared__ WideShared s_wide[kUnbWarps];
  __shared__ int s_keep[kKeep * kUnbThreads];
  const GridP& g = A.g;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* spill = A.spill + (int64_t)(blockIdx.x * kUnbWarps + w) * kWideSpill;
  uint32_t fp64 = 0, errs = 0, visits = 0;  // per-thread statistics (far below 2^32)
  for (int64_t lin = blockIdx.x * (int64_t)kUnbWarps + w; lin < g.ngp; lin += (int64_t)gridDim.x * kUnbWarps) {
    const int64_t i = lin % g.n[0], j = (lin / g.n[0]) % g.n[1], k = lin / (g.n[0] * g.n[1]);
    const d3 p = gnode(g, i, j, k);
    const float3 p32 = local32(g, p);
    const bool mine = lane == 0;
    LaneBest L;
    L.m = INFINITY;
    L.n = 0;
    L.t = s_keep + threadIdx.x;
    double m64 = kBig;
    d3 proj = {0.0, 0.0, 0.0};
    bool ok = wide_search<kUnbThreads, false>(A, s_wide[w], spill, lane, p, p32, mine, L, visits,
                                                [&] { lane_prune<kUnbThreads>(A, L, p); });
    const bool over = mine && L.n > kKeep;
    if (ok && __any_sync(0xffffffffu, over))
      ok = exact_search(A, s_wide[w].queue, spill, lane, 0, p, p32, over, band_of(A, L.m), m64, proj, fp64, visits);
    if (mine) {
      if (!over) lane_resolve<kUnbThreads>(A, L, p, m64, proj, fp64);
      if (!ok) ++errs;
      A.dist[lin] = m64;
    }
    __syncwarp();
  }
  if (lane == 0) {
    if (fp64) count_add(A.counters, C_FP64, fp64);
    if (errs) count_add(A.counters, C_ERR_STACK, errs);
    if (visits) count_add(A.counters, C_VISITS, visits);
  }
}

}  // namespace

namespace {

// The search's arguments for the nodes of g, one at a time: the lattice steps stay zero.
UnbArgs point_args(sdfgpu_ctx* ctx, const GridP& g, double* d_dist) {
  UnbArgs A{};
  A.g = g;
  A.nodes = buf<BNode>(ctx, "nodes");
  A.obb = buf<OBox>(ctx, "obb");
  A.rec = buf<TriRec64>(ctx, "rec");
  unb_errors(ctx->mesh, g.E, A);
  A.max_visits = 2 * ctx->mesh.nel + 64;
  A.dist = d_dist;
  A.counters = ctx->d_counters;
  A.ltri = leaf_tris(ctx);
  unb_mesh(ctx, A);
  return A;
}

}  // namespace

// Exact unbounded distances of the nodes of a sparse grid, one warp per node (no closest points).
int run_nearest_points(sdfgpu_ctx* ctx, const GridP& g, double* d_dist) {
  UnbArgs A = point_args(ctx, g, d_dist);
  const unsigned grid = grid_for(g.ngp, kUnbWarps, 148 * 4);
  SDF_TRY(scratch_ctx(ctx, "unb_spill", (size_t)grid * kUnbWarps * kWideSpill, &A.spill));
  k_nearest_points<<<grid, kUnbThreads, 0, ctx->stream>>>(A);
  SDF_KERNEL(ctx);
  return 0;
}

}  // namespace sdfgpu
