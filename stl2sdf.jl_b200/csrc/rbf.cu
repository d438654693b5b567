// rbf.cu -- RBFs_smoothing (src/SdfSmoothing/RBFs4Smoothing.jl:275-320) on the GPU.
//
// The reference interpolates the SDF of the coarse grid with Gaussian RBFs of width sigma = cell
// size cut off below `threshold` (exp(-(r/sigma)^2) > threshold, i.e. r < sigma sqrt(-ln thr)),
// solving K w = sdf with conjugate gradients (interpolation) or taking w = sdf (approximation),
// and evaluates sum_j w_j exp(-(|p - c_j| / sigma)^2) on a grid refined `smooth` times.
//
// On a regular grid K is a fixed 3-D stencil, so nothing is assembled: the matrix-vector product
// reads the neighbourhood of each node (the cut-off keeps the 81 nodes with |offset|^2 <= 6 cells^2
// at the default threshold) with per-axis Gaussian factors taken from the nodes' actual Float32
// coordinates, K = Kx Ky Kz (FP64 product, rounded to FP32 as the reference stores K).  CG follows
// IterativeSolvers.cg: x0 = 0, u = r + (|r|^2/|r_prev|^2) u, c = K u, alpha = |r|^2 / (u . c), stop
// when |r| <= sqrt(eps(Float32)) |b| or after n iterations; FP32 vectors, dot products accumulated in
// FP64 in a fixed order (deterministic).  The new search direction is formed on the fly inside the
// product (double-buffered) and the scalars by the last block of each pass, so one CG iteration is two
// launches.  The last block raises a device flag when the stopping rule holds and every kernel after it
// returns at once, so the result is that of stopping exactly there, and the host reads the flag once per
// kBatchIters iterations.  The fine evaluation sums, per fine point, every coarse node within the
// cut-off distance (the reference's 124-nearest query always contains them all): which ones is decided
// by the FP32 distances the reference's KD-tree computes, and the terms are FP64 products of per-axis
// factors of the FP32 coordinate differences.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace sdfgpu {
namespace {

constexpr int kRbfMaxR = 4;      // stencil radius in cells (threshold >= exp(-16) ~ 1.1e-7)
constexpr int kRbfBlocks = 592;  // fixed grid of the update's reduction (4 per SM): fixed sum order
constexpr int kRbfThreads = 256;
constexpr int kBatchIters = 16;  // CG iterations enqueued per read of the stop flag (even: the u buffers swap back)
constexpr int kMX = 32, kMY = 8, kMZ = 4;  // nodes of a product's tile: one thread per (x, y), kMZ along z
constexpr int kTaps = 2 * kRbfMaxR + 4;    // coarse nodes considered along one axis, at most (from floor - R - 1 to floor + R + 2)

// Scalars of the CG loop (device): rr = |r|^2, beta, alpha, rr_prev, the stop flag (0/1), the
// iteration count and the stopping bound on rr.
enum CgScalar : int { CG_RR = 0, CG_BETA, CG_ALPHA, CG_RR_PREV, CG_DONE, CG_ITERS, CG_TOL2, CG_MAXIT, CG_NUM };

struct Axis3 {
  const float* x[3];
  int64_t n[3];
};

// process_vector (RBFs4Smoothing.jl:15-22), pass 1: max |v| over |v| < 1e9 (as ordered bits).
__global__ void k_rbf_absmax(const double* __restrict__ d, int64_t n, unsigned* out) {
  float m = 0.f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = fabsf((float)d[i]);
    if (v < 1.0e9f) m = fmaxf(m, v);
  }
  for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));  // m >= 0: bit order = value order
}

// pass 2: Float32 values, |v| ~ 1e10 (isapprox, rtol sqrt(eps(Float32))) -> sign(v) max.
__global__ void k_rbf_process(const double* __restrict__ d, int64_t n, const unsigned* mx, float* __restrict__ b) {
  const float big = 1.0e10f, rtol = 3.4526698e-4f, m = __uint_as_float(*mx);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = (float)d[i];
    const float a = fabsf(v);
    const bool near = fabsf(a - big) <= rtol * fmaxf(a, big);
    b[i] = near ? copysignf(m, v) : v;
  }
}

// The scalars of a CG step from the sum over all blocks' partials.  which = 0: alpha = rr / (u . c);
// which = 1: new rr, the next beta = rr_new / rr_old, one more iteration counted and the stop flag raised
// when rr <= tol^2 or the iteration cap is reached; which = 2: the initial rr = |b|^2 (no iteration,
// stop when b = 0).
__device__ __forceinline__ void cg_scalar(double sum, double* sc, int which) {
  if (which == 0) {
    sc[CG_ALPHA] = sc[CG_RR] / sum;
  } else if (which == 1) {
    sc[CG_RR_PREV] = sc[CG_RR];
    sc[CG_RR] = sum;
    sc[CG_BETA] = sum / sc[CG_RR_PREV];
    sc[CG_ITERS] += 1.0;
    if (!(sum > sc[CG_TOL2]) || sc[CG_ITERS] >= sc[CG_MAXIT]) sc[CG_DONE] = 1.0;
  } else {
    // IterativeSolvers: prev_residual = 1 at the start, so the first beta is |b|^2 (u is 0)
    sc[CG_RR] = sum;
    sc[CG_RR_PREV] = 1.0;
    sc[CG_BETA] = sum;
    sc[CG_TOL2] = (double)FLT_EPSILON * sum;  // (sqrt(eps(Float32)) |b|)^2
    if (!(sum > sc[CG_TOL2])) sc[CG_DONE] = 1.0;
  }
}

// Sum of acc over the block, then -- in the last block to arrive -- over all blocks' partials in a fixed
// order, and the step's scalars.  Every block has read the scalars before the last one changes them.
__device__ __forceinline__ void cg_reduce(double acc, double* partial, unsigned* arrived, double* sc, int which) {
  __shared__ double red[kRbfThreads];
  __shared__ bool last;
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kRbfThreads / 32; ++w) t += red[w];
    __stcg(partial + blockIdx.x, t);
    __threadfence();
    last = atomicAdd(arrived, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += kRbfThreads) t += __ldcg(partial + i);
  red[threadIdx.x] = t;
  __syncthreads();
  for (int s = kRbfThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *arrived = 0u;
    cg_scalar(red[0], sc, which);
  }
}

// c = K u_new with u_new = r + beta u_old; writes u_new and, through the partial sums of u_new . c,
// alpha.  A CTA forms u_new once for its tile and the halo of RE nodes in shared memory (RE: the
// farthest offset along an axis with a factor above the cut-off), and a thread walks kMZ nodes along
// z with its x and y factors in registers; products below the cut-off, and all outside the grid (factor
// 0), add nothing.  Same terms and order per node as the form that read 2 x 81 values from memory and
// formed u_new for each: 130 -> 32 us on 590k nodes.  Bound: instruction issue (60% of the slots) and the
// conversions of the FP64 products (48% of their pipe); FP64 29%, shared memory 22%.
template <int RE>
__global__ void __launch_bounds__(kRbfThreads) k_rbf_matvec(Axis3 ax, const double* __restrict__ kt, int R,
                                                            double thr, const float* __restrict__ r,
                                                            const float* __restrict__ u_old, float* __restrict__ u_new,
                                                            float* __restrict__ c, double* __restrict__ sc,
                                                            double* __restrict__ partial, unsigned* arrived) {
  if (sc[CG_DONE] != 0.0) return;  // converged in an earlier iteration
  constexpr int SX = kMX + 2 * RE, SY = kMY + 2 * RE, SZ = kMZ + 2 * RE;
  __shared__ float s_u[SZ * SY * SX];
  const int nx = (int)ax.n[0], ny = (int)ax.n[1], nz = (int)ax.n[2];
  const int bx = (nx + kMX - 1) / kMX, by = (ny + kMY - 1) / kMY;
  const int x0 = blockIdx.x % bx * kMX, y0 = blockIdx.x / bx % by * kMY, z0 = blockIdx.x / (bx * by) * kMZ;
  const float beta = (float)sc[CG_BETA];
  for (int q = threadIdx.x; q < SZ * SY * SX; q += kRbfThreads) {
    const int x = x0 - RE + q % SX, y = y0 - RE + q / SX % SY, z = z0 - RE + q / (SX * SY);
    float v = 0.f;
    if (x >= 0 && x < nx && y >= 0 && y < ny && z >= 0 && z < nz) {
      const int64_t i = ((int64_t)z * ny + y) * nx + x;
      v = fmaf(beta, u_old[i], r[i]);
    }
    s_u[q] = v;
  }
  __syncthreads();
  const int tx = threadIdx.x & (kMX - 1), ty = threadIdx.x / kMX, x = x0 + tx, y = y0 + ty;
  double acc = 0.0;
  if (x < nx && y < ny) {
    const int W = 2 * R + 1;
    double fx[2 * RE + 1], fy[2 * RE + 1];
#pragma unroll
    for (int o = 0; o < 2 * RE + 1; ++o) {
      fx[o] = kt[(int64_t)x * W + R - RE + o];
      fy[o] = kt[(int64_t)(nx + y) * W + R - RE + o];
    }
#pragma unroll 1
    for (int q = 0; q < kMZ && z0 + q < nz; ++q) {
      const double* tz = kt + (int64_t)(nx + ny + z0 + q) * W + R - RE;
      float s = 0.f;
#pragma unroll 1
      for (int oz = 0; oz < 2 * RE + 1; ++oz) {
        const double fz = tz[oz];
        const float* row = s_u + (q + oz) * SY * SX + ty * SX + tx;
#pragma unroll
        for (int oy = 0; oy < 2 * RE + 1; ++oy) {
          const double fzy = fz * fy[oy];
          if (!(fzy > thr)) continue;
#pragma unroll
          for (int ox = 0; ox < 2 * RE + 1; ++ox) {
            const double k = fzy * fx[ox];
            if (k > thr) s = fmaf((float)k, row[oy * SX + ox], s);
          }
        }
      }
      const float ui = s_u[(q + RE) * SY * SX + (ty + RE) * SX + tx + RE];
      const int64_t i = ((int64_t)(z0 + q) * ny + y) * nx + x;
      u_new[i] = ui;
      c[i] = s;
      acc += (double)ui * (double)s;
    }
  }
  cg_reduce(acc, partial, arrived, sc, 0);
}

// x += alpha u, r -= alpha c, and |r|^2 with the step's scalars (which = 1, or 2 at the start).
__global__ void __launch_bounds__(kRbfThreads) k_rbf_update(int64_t n, double* __restrict__ sc,
                                                            const float* __restrict__ u, const float* __restrict__ c,
                                                            float* __restrict__ x, float* __restrict__ r,
                                                            double* __restrict__ partial, unsigned* arrived, int which) {
  if (which != 2 && sc[CG_DONE] != 0.0) return;
  const float alpha = (float)sc[CG_ALPHA];
  double acc = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] = fmaf(alpha, u[i], x[i]);
    const float ri = fmaf(-alpha, c[i], r[i]);
    r[i] = ri;
    acc += (double)ri * (double)ri;
  }
  cg_reduce(acc, partial, arrived, sc, which);
}

// The coarse nodes within the cut-off of every fine index along each axis: the first one, the squared
// FP32 differences the distance is formed from (beyond the last: NaN; a square that overflows is an ordinary
// tap that no distance bound admits) and the factors exp(-(dx / sigma)^2).
struct EvalAxis {
  int32_t first[3];  // offset of the axis in the arrays below
  const int32_t* start;
  const float* d2;   // kTaps per fine index
  const double* g;
};
__global__ void k_rbf_taps(Axis3 fine, Axis3 coarse, double h, double sigma, float maxd, int R, EvalAxis E,
                           int32_t* __restrict__ start, float* __restrict__ d2, double* __restrict__ g) {
  const int a = blockIdx.y;
  const double inv_s2 = 1.0 / (sigma * sigma);
  const double reach = (double)maxd * (double)maxd * 1.0001;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < fine.n[a]; i += (int64_t)gridDim.x * blockDim.x) {
    const float p = fine.x[a][i];
    const int64_t m = (int64_t)floor(((double)p - (double)coarse.x[a][0]) / h);
    const int64_t lo = m - R - 1 > 0 ? m - R - 1 : 0, hi = m + R + 2 < coarse.n[a] - 1 ? m + R + 2 : coarse.n[a] - 1;
    const int64_t at = E.first[a] + i;
    int n = 0;
    int64_t first = 0;
    for (int64_t c = lo; c <= hi && n < kTaps; ++c) {
      const float d = __fsub_rn(p, coarse.x[a][c]);
      if ((double)d * (double)d > reach) {
        if (n > 0) break;  // past the cut-off
        continue;
      }
      if (n == 0) first = c;
      d2[at * kTaps + n] = __fmul_rn(d, d);
      g[at * kTaps + n] = exp(-((double)d * (double)d) * inv_s2);
      ++n;
    }
    start[at] = (int32_t)first;
    for (; n < kTaps; ++n) {
      d2[at * kTaps + n] = NAN;
      g[at * kTaps + n] = 0.0;
    }
  }
}

__global__ void k_rbf_double(const float* __restrict__ w, int64_t n, double* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)w[i];
}

// Fine grid: every coarse node with FP32 squared distance up to smax (the largest whose square root is
// within the cut-off), FP64 terms.  A thread takes one (x, y) and kEZ points along z, so that its x
// and y taps are read once (T >= the taps of any x).  An exp per term, and index arithmetic over all
// nodes of the bounding cube, took 2.4 ms on 4.6M points of 590k nodes; with the factors per axis
// 310 us.  Bound: the FP64 multiply-adds and the loads of the weights from L1.
constexpr int kEZ = 8;
template <int T>
__global__ void __launch_bounds__(kRbfThreads) k_rbf_eval(Axis3 fine, Axis3 coarse, EvalAxis E, float smax,
                                                          const double* __restrict__ w, float* __restrict__ out) {
  const int nx = (int)fine.n[0], ny = (int)fine.n[1], nz = (int)fine.n[2];
  const int bx = (nx + 31) / 32, by = (ny + 7) / 8;
  const int x = (int)(blockIdx.x % bx) * 32 + (threadIdx.x & 31);
  const int y = (int)(blockIdx.x / bx % by) * 8 + (threadIdx.x >> 5);
  const int z0 = (int)(blockIdx.x / (bx * by)) * kEZ;
  if (x >= nx || y >= ny) return;
  const int64_t ix = E.first[0] + x, iy = E.first[1] + y, cnx = coarse.n[0], cny = coarse.n[1];
  float dx2[T];
  double gx[T];
#pragma unroll
  for (int k = 0; k < T; ++k) {
    dx2[k] = E.d2[ix * kTaps + k];
    gx[k] = E.g[ix * kTaps + k];
  }
  const double* wxy = w + E.start[ix] + E.start[iy] * cnx;
#pragma unroll 1
  for (int z = z0; z < z0 + kEZ && z < nz; ++z) {
    const int64_t iz = E.first[2] + z, cz = E.start[iz];
    double acc = 0.0;
#pragma unroll 1
    for (int kz = 0; kz < kTaps; ++kz) {
      const float dz2 = E.d2[iz * kTaps + kz];
      if (isnan(dz2)) break;  // past the axis' taps
      if (!(dz2 <= smax)) continue;
      const double gz = E.g[iz * kTaps + kz];
#pragma unroll 1
      for (int ky = 0; ky < kTaps; ++ky) {
        const float dy2 = E.d2[iy * kTaps + ky];
        if (isnan(dy2)) break;
        if (!(__fadd_rn(dy2, dz2) <= smax)) continue;  // rounding is monotone: no x can pass
        const double* row = wxy + ((cz + kz) * cny + ky) * cnx;
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < T; ++k)
          if (__fadd_rn(__fadd_rn(dx2[k], dy2), dz2) <= smax) sum = fma(row[k], gx[k], sum);
        acc = fma(gz * E.g[iy * kTaps + ky], sum, acc);
      }
    }
    out[((int64_t)z * ny + y) * nx + x] = (float)acc;
  }
}

}  // namespace
}  // namespace sdfgpu

using namespace sdfgpu;

extern "C" int sdfgpu_rbf_smoothing(sdfgpu_ctx* ctx, const double aabb_min[3], const double aabb_max[3],
                                    const int64_t N[3], double cell_size, const double* dist, int32_t interpolation,
                                    int32_t smooth, double threshold, float* fine_out, float* weights_out,
                                    int32_t* cg_iterations, double* cg_residual) {
  SDF_TRY(begin_call(ctx));
  if (!aabb_min || !aabb_max || !N || !dist || !fine_out)
    return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "rbf_smoothing: NULL argument");
  if (!(cell_size > 0.0) || !std::isfinite(cell_size) || smooth < 1 || smooth > 16 || !(threshold > 1.2e-7) ||
      !(threshold < 1.0))
    return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT,
                "rbf_smoothing: need cell_size > 0, 1 <= smooth <= 16 and exp(-16) < threshold < 1");
  double cells = 1.0, fcells = 1.0;
  int64_t nc[3], nf[3];
  for (int a = 0; a < 3; ++a) {
    if (N[a] < 1) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "rbf_smoothing: every N must be >= 1");
    nc[a] = N[a] + 1;
    nf[a] = N[a] * smooth + 1;
    cells *= (double)nc[a];
    fcells *= (double)nf[a];
  }
  if (fcells > 2147483647.0) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "rbf_smoothing: fine grid too large");
  const int64_t n = (int64_t)cells, m = (int64_t)fcells;
  const double sigma = cell_size;
  const double rcut = std::sqrt(-std::log(threshold));  // cut-off radius in units of sigma
  const int R = std::min(kRbfMaxR, (int)std::ceil(rcut));
  const float maxd = (float)std::sqrt(-std::log(threshold) * sigma * sigma);
  // Coordinates (Float32) on the host: coarse = range(min, max, length = N+1); fine = min + i dx
  // with dx = (xmax - xmin) / (nx - 1) from the x axis, in Float32 arithmetic.
  std::vector<float> hc, hf;
  for (int a = 0; a < 3; ++a) {
    const double lo = (double)(float)aabb_min[a], hi = (double)(float)aabb_max[a];  // Float32 end points
    for (int64_t i = 0; i < nc[a]; ++i) hc.push_back((float)(lo + (hi - lo) * (double)i / (double)N[a]));
  }
  volatile float fx0 = (float)aabb_min[0], fx1 = (float)aabb_max[0];
  volatile float span = fx1 - fx0;
  volatile float dxf = span / (float)(nf[0] - 1);
  for (int a = 0; a < 3; ++a) {
    const float f0 = (float)aabb_min[a];
    for (int64_t i = 0; i < nf[a]; ++i) {
      volatile float step = (float)i * dxf;
      hf.push_back(f0 + step);
    }
  }
  // Per-axis Gaussian factors exp(-(dx/sigma)^2) of the coarse stencil (0 outside the grid).
  const int W = 2 * R + 1;
  std::vector<double> hk((size_t)(nc[0] + nc[1] + nc[2]) * W, 0.0);
  {
    size_t base = 0, off = 0;
    for (int a = 0; a < 3; ++a) {
      for (int64_t i = 0; i < nc[a]; ++i)
        for (int o = -R; o <= R; ++o) {
          const int64_t j = i + o;
          if (j < 0 || j >= nc[a]) continue;
          volatile float d = hc[off + j] - hc[off + i];
          const double t = (double)d / sigma;
          hk[base + (size_t)i * W + (o + R)] = std::exp(-t * t);
        }
      base += (size_t)nc[a] * W;
      off += (size_t)nc[a];
    }
  }
  // the farthest offset along an axis whose factor is above the cut-off (the product reads no farther)
  int reach = 1;
  for (size_t q = 0; q < hk.size(); ++q)
    if (hk[q] > threshold) reach = std::max(reach, std::abs((int)(q % W) - R));
  cudaStream_t st = ctx->stream;
  float *dc, *df, *b, *x, *r, *u0, *u1, *c, *out;
  double *kt, *dd, *part, *sc;
  unsigned* mx;
  SDF_TRY(scratch_t(ctx, "rbf_cx", hc.size(), &dc));
  SDF_TRY(scratch_t(ctx, "rbf_fx", hf.size(), &df));
  SDF_TRY(scratch_t(ctx, "rbf_kt", hk.size(), &kt));
  SDF_TRY(scratch_t(ctx, "rbf_dist", (size_t)n, &dd));
  SDF_TRY(scratch_t(ctx, "rbf_b", (size_t)n, &b));
  SDF_TRY(scratch_t(ctx, "rbf_x", (size_t)n, &x));
  SDF_TRY(scratch_t(ctx, "rbf_r", (size_t)n, &r));
  SDF_TRY(scratch_t(ctx, "rbf_u0", (size_t)n, &u0));
  SDF_TRY(scratch_t(ctx, "rbf_u1", (size_t)n, &u1));
  SDF_TRY(scratch_t(ctx, "rbf_c", (size_t)n, &c));
  SDF_TRY(scratch_t(ctx, "rbf_out", (size_t)m, &out));
  const int64_t mtiles = cdiv(nc[0], kMX) * cdiv(nc[1], kMY) * cdiv(nc[2], kMZ);
  if (mtiles > 0x7fffffffLL) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "rbf_smoothing: coarse grid too large");
  const unsigned mblocks = (unsigned)mtiles;
  unsigned* arrived;
  SDF_TRY(scratch_t(ctx, "rbf_part", (size_t)std::max<int64_t>(mtiles, kRbfBlocks), &part));
  SDF_TRY(scratch_t(ctx, "rbf_arrived", 1, &arrived));
  SDF_CUDA(ctx, cudaMemsetAsync(arrived, 0, sizeof(unsigned), st));
  SDF_TRY(scratch_t(ctx, "rbf_sc", CG_NUM, &sc));
  SDF_TRY(scratch_t(ctx, "rbf_mx", 1, &mx));
  SDF_CUDA(ctx, cudaMemcpyAsync(dc, hc.data(), sizeof(float) * hc.size(), cudaMemcpyHostToDevice, st));
  SDF_CUDA(ctx, cudaMemcpyAsync(df, hf.data(), sizeof(float) * hf.size(), cudaMemcpyHostToDevice, st));
  SDF_CUDA(ctx, cudaMemcpyAsync(kt, hk.data(), sizeof(double) * hk.size(), cudaMemcpyHostToDevice, st));
  SDF_CUDA(ctx, cudaMemcpyAsync(dd, dist, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  SDF_CUDA(ctx, cudaMemsetAsync(mx, 0, sizeof(unsigned), st));
  const unsigned g = grid_for(n, kRbfThreads, 148 * 8);
  k_rbf_absmax<<<g, kRbfThreads, 0, st>>>(dd, n, mx);
  SDF_KERNEL(ctx);
  k_rbf_process<<<g, kRbfThreads, 0, st>>>(dd, n, mx, b);
  SDF_KERNEL(ctx);
  Axis3 ac{{dc, dc + nc[0], dc + nc[0] + nc[1]}, {nc[0], nc[1], nc[2]}};
  Axis3 af{{df, df + nf[0], df + nf[0] + nf[1]}, {nf[0], nf[1], nf[2]}};
  const float* weights = b;
  int iters = 0;
  double res = 0.0;
  if (interpolation) {
    // x = 0, r = b, u = 0; |b|^2 through the update's reduction with alpha = 0 (x and r unchanged)
    SDF_CUDA(ctx, cudaMemsetAsync(x, 0, sizeof(float) * n, st));
    SDF_CUDA(ctx, cudaMemsetAsync(u0, 0, sizeof(float) * n, st));
    SDF_CUDA(ctx, cudaMemcpyAsync(r, b, sizeof(float) * n, cudaMemcpyDeviceToDevice, st));
    double h_sc[CG_NUM] = {0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, (double)n};
    SDF_CUDA(ctx, cudaMemcpyAsync(sc, h_sc, sizeof(h_sc), cudaMemcpyHostToDevice, st));
    k_rbf_update<<<kRbfBlocks, kRbfThreads, 0, st>>>(n, sc, u0, u0, x, r, part, arrived, 2);
    SDF_KERNEL(ctx);
    static_assert((int)CG_NUM <= (int)S_NUM, "the CG scalars are read back through the context's page-locked slots");
    double* h_out = reinterpret_cast<double*>(ctx->h_scalars);  // page-locked: read back per batch
    const int64_t max_batches = n / kBatchIters + 2;
    for (int64_t l = 0;; ++l) {
      for (int k = 0; k < kBatchIters; ++k) {
        float* ua = (k & 1) ? u1 : u0;
        float* ub = (k & 1) ? u0 : u1;
        auto product = [&](auto re) {
          k_rbf_matvec<decltype(re)::value><<<mblocks, kRbfThreads, 0, st>>>(ac, kt, R, threshold, r, ua, ub, c, sc,
                                                                            part, arrived);
        };
        if (reach <= 1) product(std::integral_constant<int, 1>());
        else if (reach == 2) product(std::integral_constant<int, 2>());
        else if (reach == 3) product(std::integral_constant<int, 3>());
        else product(std::integral_constant<int, 4>());
        SDF_KERNEL(ctx);
        k_rbf_update<<<kRbfBlocks, kRbfThreads, 0, st>>>(n, sc, ub, c, x, r, part, arrived, 1);
        SDF_KERNEL(ctx);
      }
      SDF_CUDA(ctx, cudaMemcpyAsync(h_out, sc, sizeof(double) * CG_NUM, cudaMemcpyDeviceToHost, st));
      SDF_CUDA(ctx, cudaStreamSynchronize(st));
      if (!std::isfinite(h_out[CG_RR]))
        return fail(ctx, SDFGPU_ERR_CUDA, "rbf_smoothing: CG diverged (non-finite residual)");
      if (h_out[CG_DONE] != 0.0 || l >= max_batches) break;
    }
    iters = (int)h_out[CG_ITERS];
    const double rr = h_out[CG_RR];
    res = std::sqrt(rr);
    weights = x;
  }
  // per-axis taps of the fine points; smax: the largest finite float whose correctly rounded square root is
  // within maxd (the root is monotone), so the terms are those of "sqrt(s) <= maxd" (a sum s that overflows
  // is an infinite distance, whose term is 0 where maxd is infinite too)
  EvalAxis E;
  E.first[0] = 0;
  E.first[1] = (int32_t)nf[0];
  E.first[2] = (int32_t)(nf[0] + nf[1]);
  const size_t nfa = (size_t)(nf[0] + nf[1] + nf[2]);
  int32_t* tstart;
  float* td2;
  double *tg, *wd;
  SDF_TRY(scratch_t(ctx, "rbf_tap_start", nfa, &tstart));
  SDF_TRY(scratch_t(ctx, "rbf_tap_d2", nfa * kTaps, &td2));
  SDF_TRY(scratch_t(ctx, "rbf_tap_g", nfa * kTaps, &tg));
  SDF_TRY(scratch_t(ctx, "rbf_w64", (size_t)n + kTaps, &wd));  // a row's unused taps may be read past the last node
  E.start = tstart;
  E.d2 = td2;
  E.g = tg;
  float smax = std::min(maxd * maxd, FLT_MAX);
  while (smax < FLT_MAX && std::sqrt(std::nextafter(smax, INFINITY)) <= maxd) smax = std::nextafter(smax, INFINITY);
  while (smax > 0.f && std::sqrt(smax) > maxd) smax = std::nextafter(smax, 0.f);
  k_rbf_taps<<<dim3(grid_for(std::max(nf[0], std::max(nf[1], nf[2])), 128), 3), 128, 0, st>>>(
      af, ac, cell_size, sigma, maxd, R, E, tstart, td2, tg);
  SDF_KERNEL(ctx);
  k_rbf_double<<<g, kRbfThreads, 0, st>>>(weights, n, wd);
  SDF_KERNEL(ctx);
  // taps along x: those within reach of a point at the smallest spacing of the coarse coordinates
  double gap = INFINITY;
  for (int64_t i = 0; i + 1 < nc[0]; ++i) gap = std::min(gap, (double)hc[i + 1] - (double)hc[i]);
  const double taps = gap > 0.0 ? 2.0 * (double)maxd * 1.0001 / gap + 1.0 : kTaps;
  const int64_t ecta = cdiv(nf[0], 32) * cdiv(nf[1], 8) * cdiv(nf[2], kEZ);
  if (ecta > 0x7fffffffLL) return fail(ctx, SDFGPU_ERR_INVALID_ARGUMENT, "rbf_smoothing: fine grid too large");
  if (taps < 7.0) k_rbf_eval<6><<<(unsigned)ecta, kRbfThreads, 0, st>>>(af, ac, E, smax, wd, out);
  else k_rbf_eval<kTaps><<<(unsigned)ecta, kRbfThreads, 0, st>>>(af, ac, E, smax, wd, out);
  SDF_KERNEL(ctx);
  SDF_CUDA(ctx, cudaMemcpyAsync(fine_out, out, sizeof(float) * m, cudaMemcpyDeviceToHost, st));
  if (weights_out) SDF_CUDA(ctx, cudaMemcpyAsync(weights_out, weights, sizeof(float) * n, cudaMemcpyDeviceToHost, st));
  SDF_CUDA(ctx, cudaStreamSynchronize(st));
  if (cg_iterations) *cg_iterations = iters;
  if (cg_residual) *cg_residual = res;
  return SDFGPU_OK;
}
