// artifacts.cu -- remove_sdf_artifacts! / analyze_sdf_components
// (src/SignedDistances/SdfArtifactRemoval.jl:134-318) on the GPU.
//
// Interior nodes are sdf >= threshold (a NaN is exterior).  Their 6-connected components are found
// in two levels.  A CTA labels a tile of 32 x 8 x 8 nodes in shared memory: a row's runs of interior
// nodes are its starting sets, joined once per overlapping pair of runs with the row below and behind.
// Then the tiles' faces are joined by a lock-free union-find over the grid (the hooking and
// pointer-jumping scheme of ECL-CC, Jaiganesh and Burtscher 2018): parent[i] <= i always holds, a
// union links the larger of the two roots under the smaller one with one compare-and-swap, and a find
// shortens the path it walks.
// So when every union has completed, the root of a component is its smallest linear node index,
// whatever order the unions ran in -- the labelling is deterministic, while the reference's
// union-by-rank inside @threads (:164-182) is racy.  Components smaller than
// max(1, round(ratio * largest)) that are not the largest one are flipped to -|sdf| (:201-230).
// Ties for the largest component are broken towards the smallest root; they change a result only
// when ratio > 1, where the reference's choice depends on its Dict's iteration order.
//
// Measured on 14.2M nodes with 0.1% of stray signs (B200): 295 us (tiles 108, faces 112, flip 62, the
// roots 12) against 3.9 ms for one union-find over all nodes with a size count per node, most of whose
// atomics went to the one large component.  The tiles' pass moves 12 bytes a node and is bound by the
// latency of its shared-memory unions, the faces' by that of the chains it follows.
//
// Every loop walks strictly decreasing indices, so it ends within ngp steps; the loops still carry
// that bound and report SDFGPU_ERR_CAPACITY instead of spinning.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace sdfgpu {
namespace {

__device__ __forceinline__ int32_t ld_parent(const int32_t* p, int64_t i) { return __ldcg(p + i); }

// Root of x, halving the path on the way (every store writes an ancestor, so parent[i] <= i and the
// ancestor relation survive concurrent unions).
__device__ __forceinline__ int32_t find_root(int32_t* p, int32_t x, int64_t cap, bool& bad) {
  int32_t cur = ld_parent(p, x);
  if (cur == x) return x;
  int32_t prev = x;
  int64_t steps = 0;
  int32_t nxt;
  while (cur > (nxt = ld_parent(p, cur))) {
    if (++steps > cap) { bad = true; break; }
    __stcg(p + prev, nxt);
    prev = cur;
    cur = nxt;
  }
  return cur;
}

__device__ __forceinline__ void unite(int32_t* p, int32_t a, int32_t b, int64_t cap, bool& bad) {
  int32_t ra = find_root(p, a, cap, bad), rb = find_root(p, b, cap, bad);
  int64_t steps = 0;
  while (ra != rb && !bad) {
    if (++steps > cap) { bad = true; break; }
    if (ra < rb) {  // hook rb under ra
      const int32_t old = atomicCAS(p + rb, rb, ra);
      if (old == rb) break;
      rb = old;
    } else {
      const int32_t old = atomicCAS(p + ra, ra, rb);
      if (old == ra) break;
      ra = old;
    }
  }
}

constexpr int kTX = 32, kTY = 8, kTZ = 8;  // nodes of a tile: a warp per row of 32
constexpr int kTile = kTX * kTY * kTZ;

// Device counters of a call.
enum CCCounter : int { CC_LIST = 0, CC_BAD, CC_ROOTS, CC_FLIPPED, CC_NUM };

__device__ __forceinline__ int tile_find(const volatile int* l, int x) {
  while (l[x] != x) x = l[x];  // l[x] <= x: strictly decreasing
  return x;
}
__device__ __forceinline__ void tile_unite(int* l, int a, int b) {
  while (true) {
    a = tile_find(l, a);
    b = tile_find(l, b);
    if (a == b) return;
    if (a < b) { const int t = a; a = b; b = t; }
    const int old = atomicMin(&l[a], b);
    if (old == a) return;
    a = old;  // a was linked meanwhile: join what it was linked under
  }
}

// Components within each tile: parent[i] = the smallest linear index of i's component in its tile (the
// order of the tile's own indices is that of the linear ones), -1 outside; that root's size; the list of
// roots.  One read of sdf and one write of parent: bound by HBM (12 bytes a node).
__global__ void __launch_bounds__(256) k_cc_tiles(const double* __restrict__ sdf, int64_t nx, int64_t ny, int64_t nz,
                                                  double thr, int32_t* __restrict__ parent,
                                                  int32_t* __restrict__ size, int32_t* __restrict__ list,
                                                  int64_t* counters) {
  __shared__ int lab[kTile], cnt[kTile];
  __shared__ unsigned mask[kTY * kTZ];
  __shared__ int n_roots;
  __shared__ long long base;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t tnx = (nx + kTX - 1) / kTX, tny = (ny + kTY - 1) / kTY;
  const int64_t x0 = blockIdx.x % tnx * kTX, y0 = blockIdx.x / tnx % tny * kTY, z0 = blockIdx.x / (tnx * tny) * kTZ;
  if (threadIdx.x == 0) n_roots = 0;
  auto linear = [&](int t) { return x0 + (t & 31) + nx * (y0 + ((t >> 5) & (kTY - 1)) + ny * (z0 + (t >> 8))); };
#pragma unroll
  for (int q = 0; q < kTZ; ++q) {  // row w of layer q
    const int t = (q * kTY + w) * 32 + lane;
    bool in = x0 + lane < nx && y0 + w < ny && z0 + q < nz;
    in = in && sdf[linear(t)] >= thr;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    const unsigned gap = ~m & ((1u << lane) - 1u);
    lab[t] = t - lane + (gap ? 32 - __clz(gap) : 0);  // the run's first node
    cnt[t] = 0;
    if (lane == 0) mask[q * kTY + w] = m;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kTZ; ++q) {
    const int r = q * kTY + w, t = r * 32 + lane;
    const unsigned m = mask[r];
    if (w > 0) {
      const unsigned both = m & mask[r - 1];
      if (both & ~(both << 1) & (1u << lane)) tile_unite(lab, t, t - 32);  // once per overlap of two runs
    }
    if (q > 0) {
      const unsigned both = m & mask[r - kTY];
      if (both & ~(both << 1) & (1u << lane)) tile_unite(lab, t, t - 32 * kTY);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kTZ; ++q) {
    const int r = q * kTY + w, t = r * 32 + lane;
    const unsigned m = mask[r];
    const bool in = (m >> lane) & 1u;
    int root = t;
    if (in) {
      root = tile_find(lab, t);
      if (lane == 0 || !((m >> (lane - 1)) & 1u)) {  // the run's first node adds its length
        const unsigned rest = ~(m >> lane);
        atomicAdd(&cnt[root], rest ? __ffs(rest) - 1 : 32 - lane);
      }
    }
    if (x0 + lane < nx && y0 + w < ny && z0 + q < nz) parent[linear(t)] = in ? (int32_t)linear(root) : -1;
  }
  __syncthreads();
  int pos[kTZ];
#pragma unroll
  for (int q = 0; q < kTZ; ++q) {
    const int t = (q * kTY + w) * 32 + lane;
    pos[q] = cnt[t] > 0 ? atomicAdd(&n_roots, 1) : -1;
  }
  __syncthreads();
  if (threadIdx.x == 0 && n_roots > 0)
    base = (long long)atomicAdd((unsigned long long*)&counters[CC_LIST], (unsigned long long)n_roots);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kTZ; ++q)
    if (pos[q] >= 0) {
      const int t = (q * kTY + w) * 32 + lane;
      const int64_t i = linear(t);
      list[base + pos[q]] = (int32_t)i;
      size[i] = cnt[t];
    }
}

// Unions across the tiles' faces: each interior node on a tile's low face with its interior neighbour in
// the tile before.  A pair whose neighbour pair (one node back along the face, in the same two tiles) is
// interior too is already joined through it.
// All indices fit 32 bits (a grid has fewer than 2^31 nodes), and 32-bit divisions matter here.
__global__ void k_cc_faces(int32_t* parent, uint32_t nx, uint32_t ny, uint32_t nz, int64_t* counters) {
  const uint32_t nxy = nx * ny;
  const uint32_t fx = (nx - 1) / kTX, fy = (ny - 1) / kTY, fz = (nz - 1) / kTZ;  // faces per axis
  const uint32_t cx = fx * ny * nz, cy = fy * nx * nz, all = cx + cy + fz * nxy;
  bool bad = false;
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < all; t += gridDim.x * blockDim.x) {
    uint32_t i, step, back;  // the node, its neighbour i - step, and the face step back (0: none)
    if (t < cx) {
      const uint32_t v = t / ny, y = t - v * ny, f = v / nz, z = v - f * nz;
      i = (f + 1) * kTX + nx * (y + ny * z);
      step = 1;
      back = y % kTY ? nx : 0;
    } else {
      const bool isy = t < cx + cy;
      const uint32_t u = isy ? t - cx : t - cx - cy, v = u / nx, x = u - v * nx;
      const uint32_t d = isy ? fy : ny, hi = v / d, lo = v - hi * d;  // (z, face) or (face, y)
      i = isy ? x + nx * ((lo + 1) * kTY + ny * hi) : x + nx * (lo + ny * ((hi + 1) * kTZ));
      step = isy ? nx : nxy;
      back = x % kTX ? 1 : 0;
    }
    const bool in = ld_parent(parent, i) >= 0, in2 = ld_parent(parent, i - step) >= 0;
    if (!in || !in2) continue;
    if (back) {
      const bool b1 = ld_parent(parent, i - back) >= 0, b2 = ld_parent(parent, i - back - step) >= 0;
      if (b1 && b2) continue;
    }
    unite(parent, (int32_t)i, (int32_t)(i - step), (int64_t)nxy * nz, bad);
  }
  if (bad) count_add(counters, CC_BAD, 1);
}

// The tiles' roots point at their component's root and add their sizes to it.  The unions have all
// completed, so an entry only changes here to another ancestor of itself.
__global__ void k_cc_roots(int32_t* parent, int64_t ngp, int32_t* __restrict__ size, const int32_t* __restrict__ list,
                           int64_t* counters) {
  bool bad = false;
  int64_t roots = 0;
  const int64_t n = counters[CC_LIST];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = list[q];
    int32_t r = i, up;
    int64_t steps = 0;
    while ((up = ld_parent(parent, r)) != r) {
      if (++steps > ngp) { bad = true; break; }
      r = up;
    }
    if (r != i) {
      __stcg(parent + i, r);
      atomicAdd(size + r, size[i]);
    }
    roots += r == i;
  }
  for (int off = 16; off > 0; off >>= 1) roots += __shfl_down_sync(0xffffffffu, roots, off);
  if ((threadIdx.x & 31) == 0 && roots) count_add(counters, CC_ROOTS, roots);
  if (bad) count_add(counters, CC_BAD, 1);
}

// Largest component: max of (size << 32 | 0x7fffffff - root), i.e. ties to the smallest root.
__global__ void k_cc_largest(const int32_t* __restrict__ parent, const int32_t* __restrict__ size,
                             const int32_t* __restrict__ list, const int64_t* __restrict__ counters,
                             unsigned long long* best) {
  unsigned long long b = 0;
  const int64_t n = counters[CC_LIST];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = list[q];
    if (parent[i] != i) continue;
    const unsigned long long key = ((unsigned long long)(uint32_t)size[i] << 32) | (uint32_t)(0x7fffffff - i);
    b = key > b ? key : b;
  }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_down_sync(0xffffffffu, b, off);
    b = o > b ? o : b;
  }
  if ((threadIdx.x & 31) == 0 && b) atomicMax(best, b);
}

// A node's component root: its entry is a tile root, whose entry is the root (k_cc_roots).
__device__ __forceinline__ int32_t node_root(const int32_t* __restrict__ parent, int64_t i) {
  const int32_t v = parent[i];
  return v < 0 ? v : parent[v];
}

__global__ void k_cc_label(const int32_t* __restrict__ parent, int64_t ngp, int32_t* __restrict__ root) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ngp; i += (int64_t)gridDim.x * blockDim.x)
    root[i] = node_root(parent, i);
}

// Flips the components smaller than max(1, round(Int, ratio * largest)) (round to nearest, ties to
// even) other than the largest; the threshold is formed here, so the host need not wait for it.
__global__ void k_cc_flip(double* __restrict__ sdf, const int32_t* __restrict__ parent, const int32_t* __restrict__ size,
                          int64_t ngp, double ratio, const unsigned long long* __restrict__ best, int64_t* counters) {
  const unsigned long long b = *best;
  if (!b || counters[CC_BAD]) return;
  const int32_t keep_root = 0x7fffffff - (int32_t)(b & 0xffffffffULL);
  const double ms = rint(__dmul_rn(ratio, (double)(int64_t)(b >> 32)));
  const int64_t min_size = max((int64_t)1, ms > 9.0e18 ? (int64_t)9e18 : (int64_t)ms);
  int64_t flipped = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ngp; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t r = node_root(parent, i);
    if (r < 0 || r == keep_root || (int64_t)size[r] >= min_size) continue;
    sdf[i] = -fabs(sdf[i]);
    ++flipped;
  }
  for (int off = 16; off > 0; off >>= 1) flipped += __shfl_down_sync(0xffffffffu, flipped, off);
  if ((threadIdx.x & 31) == 0 && flipped) count_add(counters, CC_FLIPPED, flipped);
}

struct CCResult {
  int64_t components = 0, largest = 0, flipped = 0;
};

// Labels the interior components of d_sdf (grid N); when ratio >= 0 also flips the small ones.
int run_components(sdfgpu_ctx* ctx, const int64_t N[3], double* d_sdf, double thr, double ratio, CCResult& R,
                   int32_t** d_root_out) {
  if (!N) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "N must not be NULL");
  double cells = 1.0;
  for (int a = 0; a < 3; ++a) {
    if (N[a] < 0) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "N must be >= 0");
    cells *= (double)(N[a] + 1);
  }
  if (cells > 2147483647.0) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "grid has more than 2^31-1 nodes");
  const int64_t nx = N[0] + 1, ny = N[1] + 1, nz = N[2] + 1, ngp = nx * ny * nz;
  cudaStream_t st = ctx->stream;
  int32_t *parent, *size, *list;
  int64_t* cnt;  // the counters, then the largest component's key
  const int64_t tiles = cdiv(nx, kTX) * cdiv(ny, kTY) * cdiv(nz, kTZ);
  if (tiles > 0x7fffffffLL) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "grid has too many tiles");
  SDF_TRY(scratch_t(ctx, "cc_parent", (size_t)ngp, &parent));
  SDF_TRY(scratch_t(ctx, "cc_size", (size_t)ngp, &size));
  SDF_TRY(scratch_t(ctx, "cc_list", (size_t)ngp, &list));
  SDF_TRY(scratch_t(ctx, "cc_counters", CC_NUM + 1, &cnt));
  unsigned long long* best = reinterpret_cast<unsigned long long*>(cnt + CC_NUM);
  SDF_CUDA(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (CC_NUM + 1), st));
  k_cc_tiles<<<(unsigned)tiles, 256, 0, st>>>(d_sdf, nx, ny, nz, thr, parent, size, list, cnt);
  SDF_KERNEL(ctx);
  k_cc_faces<<<grid_for(cdiv(ngp, 3), 256, 148 * 8), 256, 0, st>>>(parent, (uint32_t)nx, (uint32_t)ny, (uint32_t)nz,
                                                                   cnt);
  SDF_KERNEL(ctx);
  k_cc_roots<<<grid_for(cdiv(ngp, 64), 256, 148 * 8), 256, 0, st>>>(parent, ngp, size, list, cnt);
  SDF_KERNEL(ctx);
  k_cc_largest<<<grid_for(cdiv(ngp, 64), 256, 148 * 8), 256, 0, st>>>(parent, size, list, cnt, best);
  SDF_KERNEL(ctx);
  const unsigned grid = grid_for(ngp, 256, 148 * 8);
  if (ratio >= 0.0) {
    k_cc_flip<<<grid, 256, 0, st>>>(d_sdf, parent, size, ngp, ratio, best, cnt);
    SDF_KERNEL(ctx);
  }
  if (d_root_out) {
    SDF_TRY(scratch_t(ctx, "cc_root", (size_t)ngp, d_root_out));
    k_cc_label<<<grid, 256, 0, st>>>(parent, ngp, *d_root_out);
    SDF_KERNEL(ctx);
  }
  int64_t h_cnt[CC_NUM + 1];
  SDF_CUDA(ctx, cudaMemcpyAsync(h_cnt, cnt, sizeof(h_cnt), cudaMemcpyDeviceToHost, st));
  SDF_CUDA(ctx, cudaStreamSynchronize(st));
  if (h_cnt[CC_BAD]) return fail(ctx, SDFGPU_ERR_CAPACITY, "component labelling exceeded its step bound");
  R.components = h_cnt[CC_ROOTS];
  R.largest = (int64_t)((unsigned long long)h_cnt[CC_NUM] >> 32);
  R.flipped = h_cnt[CC_FLIPPED];
  return 0;
}

void write_out(const CCResult& R, int64_t* flipped, int64_t* components, int64_t* largest) {
  if (flipped) *flipped = R.flipped;
  if (components) *components = R.components;
  if (largest) *largest = R.largest;
}

}  // namespace
}  // namespace sdfgpu

using namespace sdfgpu;

extern "C" {

int sdfgpu_remove_artifacts_device(sdfgpu_ctx* ctx, const int64_t N[3], double* d_sdf, double threshold,
                                   double min_component_ratio, int64_t* flipped, int64_t* components,
                                   int64_t* largest) {
  SDF_TRY(begin_call(ctx));
  if (!d_sdf) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "sdf must not be NULL");
  if (!(min_component_ratio >= 0.0) || !std::isfinite(min_component_ratio))
    return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "min_component_ratio must be finite and >= 0");
  CCResult R;
  SDF_TRY(run_components(ctx, N, d_sdf, threshold, min_component_ratio, R, nullptr));
  write_out(R, flipped, components, largest);
  return SDFGPU_OK;
}

int sdfgpu_remove_artifacts(sdfgpu_ctx* ctx, const int64_t N[3], double* sdf, double threshold,
                            double min_component_ratio, int64_t* flipped, int64_t* components, int64_t* largest) {
  SDF_TRY(begin_call(ctx));
  if (!sdf || !N) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "sdf and N must not be NULL");
  if (!(min_component_ratio >= 0.0) || !std::isfinite(min_component_ratio))
    return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "min_component_ratio must be finite and >= 0");
  double cells = 1.0;
  for (int a = 0; a < 3; ++a) cells *= (double)(std::max<int64_t>(N[a], -1) + 1);
  if (cells > 2147483647.0 || cells < 0.0) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "bad grid size");
  const size_t ngp = (size_t)cells;
  double* d;
  SDF_TRY(scratch_t(ctx, "cc_sdf", ngp, &d));
  SDF_CUDA(ctx, cudaMemcpyAsync(d, sdf, sizeof(double) * ngp, cudaMemcpyHostToDevice, ctx->stream));
  CCResult R;
  SDF_TRY(run_components(ctx, N, d, threshold, min_component_ratio, R, nullptr));
  if (R.flipped) {
    SDF_CUDA(ctx, cudaMemcpyAsync(sdf, d, sizeof(double) * ngp, cudaMemcpyDeviceToHost, ctx->stream));
    SDF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  write_out(R, flipped, components, largest);
  return SDFGPU_OK;
}

int sdfgpu_sdf_components(sdfgpu_ctx* ctx, const int64_t N[3], const double* sdf, double threshold, int32_t* root_out,
                          int64_t* components, int64_t* largest) {
  SDF_TRY(begin_call(ctx));
  if (!sdf || !N) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "sdf and N must not be NULL");
  double cells = 1.0;
  for (int a = 0; a < 3; ++a) cells *= (double)(std::max<int64_t>(N[a], -1) + 1);
  if (cells > 2147483647.0 || cells < 0.0) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "bad grid size");
  const size_t ngp = (size_t)cells;
  double* d;
  SDF_TRY(scratch_t(ctx, "cc_sdf", ngp, &d));
  SDF_CUDA(ctx, cudaMemcpyAsync(d, sdf, sizeof(double) * ngp, cudaMemcpyHostToDevice, ctx->stream));
  CCResult R;
  int32_t* root = nullptr;
  SDF_TRY(run_components(ctx, N, d, threshold, -1.0, R, root_out ? &root : nullptr));
  if (root_out) {
    SDF_CUDA(ctx, cudaMemcpyAsync(root_out, root, sizeof(int32_t) * ngp, cudaMemcpyDeviceToHost, ctx->stream));
    SDF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  write_out(R, nullptr, components, largest);
  return SDFGPU_OK;
}

}  // extern "C"
