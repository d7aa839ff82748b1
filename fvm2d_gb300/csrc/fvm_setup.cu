// fvm_setup.cu -- FP64 set-up kernels, run once per mesh.  Compiled with
// --fmad=false so the results equal the serial FP64 arithmetic.
#include <climits>
#include <cstddef>

#include <cuda_runtime.h>

#include "fvm_launch.h"

namespace fvm {

// (ct, st, length) of every edge face from ds, as roe_flux.f:18-20 /
// kfvs_flux.f:16-18 / hllc_flux.f:18-20 compute them on every call.
__global__ void k_edge_csl(const double2 *__restrict__ ds, D4 *__restrict__ csl, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 d = ds[i];
  const double length = sqrt(d.x * d.x + d.y * d.y);
  D4 o;
  o.x = d.x / length;
  o.y = d.y / length;
  o.z = length;
  o.w = 0.0;
  csl[i] = o;
}

// dtlength.f:21-44: per triangle altitudes, min-scattered to its vertices.
// drmin holds positive doubles, whose bit patterns order like integers.
__global__ void k_dtlength(int nt, const double2 *__restrict__ coord, const int *__restrict__ elem,
                           const double *__restrict__ elarea, unsigned long long *drmin) {
  const int it = blockIdx.x * blockDim.x + threadIdx.x;
  if (it >= nt) return;
  const int n1 = elem[3 * it] - 1, n2 = elem[3 * it + 1] - 1, n3 = elem[3 * it + 2] - 1;
  const double2 c1 = coord[n1], c2 = coord[n2], c3 = coord[n3];
  const double ea = elarea[it];
  const double dx1 = c2.x - c3.x, dy1 = c2.y - c3.y;
  const double h1 = 2.0 * ea / sqrt(dx1 * dx1 + dy1 * dy1);
  const double dx2 = c3.x - c1.x, dy2 = c3.y - c1.y;
  const double h2 = 2.0 * ea / sqrt(dx2 * dx2 + dy2 * dy2);
  const double dx3 = c1.x - c2.x, dy3 = c1.y - c2.y;
  const double h3 = 2.0 * ea / sqrt(dx3 * dx3 + dy3 * dy3);
  atomicMin(drmin + n1, (unsigned long long)__double_as_longlong(h1));
  atomicMin(drmin + n2, (unsigned long long)__double_as_longlong(h2));
  atomicMin(drmin + n3, (unsigned long long)__double_as_longlong(h3));
}

__global__ void k_fill(double *a, double v, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

// wall_dist.f:28-61 and 87-92: each thread one point, the solid edges staged
// through shared memory in tiles.  The result is a minimum, so it depends
// neither on the order of the candidates nor on whether it is taken over the
// distances or over their squares (IEEE square roots are monotonic): one root
// per point remains.  FP64 runs at a 64th of the FP32 rate here, and nearly
// every edge is far from the nearest: a first FP32 sweep bounds the distance
// from above (`near`), a second drops every edge that lies farther, and the
// few left are done in FP64, eight at a time per thread so that the threads of
// a warp do theirs together.
//
// Why dropping is safe: an edge's candidates are its ends a, b and a point of
// the segment from a along the vector line 46 uses ((dx3, dx3) with
// bugcompat), so none is nearer than that segment or b.  The FP32 distances to
// those, relative to a common origin, are off by less than 2e-6 of the
// coordinates involved (rounding of a, p and the vector, and of the foot's
// place along it); `off` and `e1.z` hold 3e-6 of the point's and the edge's.
// `near` takes the distances of true candidates only (with bugcompat: the
// first ends).  Infinite or NaN distances compare as "not farther".  Where
// FP32 ends nothing is dropped: an edge or a point farther than kWallFar from
// the origin (squares overflow) gets an infinite margin, and `near` is never
// below kWallNear (squares underflow).  Far from zero the FP64 foot itself is
// rounded (an ulp of the edge's coordinates): `e1.z` holds that too.
// With every pair in FP64 (three roots and a quotient each) the pass took
// 15.8 ms for 196,608 points and 768 edges; now 0.82 ms
// (FP64 to FP32 conversions are as slow: with the edges' FP32 data formed by
// every CTA instead of once, 1.77 ms).
constexpr int kWallThreads = 128, kWallTile = 256, kWallList = 8;
constexpr float kWallFar = 1e15f, kWallNear = 1e-12f;

// squared distances to the candidates of one edge, folded into w
__device__ __forceinline__ void wall_edge(double2 ci, double2 a, double2 b, int bugcompat,
                                          double &w) {
  const double dx1 = a.x - ci.x, dy1 = a.y - ci.y;
  const double s1 = dx1 * dx1 + dy1 * dy1;
  w = (s1 < w) ? s1 : w;
  const double dx2 = b.x - ci.x, dy2 = b.y - ci.y;
  const double s2 = dx2 * dx2 + dy2 * dy2;
  w = (s2 < w) ? s2 : w;
  const double dx3 = b.x - a.x;
  const double dy3 = bugcompat ? (b.x - a.x) : (b.y - a.y);
  const double dl2 = dx3 * dx3 + dy3 * dy3;
  const double xi = -(dx1 * dx3 + dy1 * dy3) / dl2;
  if (xi >= 0.0 && xi <= 1.0) {
    const double xp = a.x + xi * dx3;
    const double yp = a.y + xi * dy3;
    const double ex = ci.x - xp, ey = ci.y - yp;
    const double s3 = ex * ex + ey * ey;
    w = (s3 < w) ? s3 : w;
  }
}

// The FP32 data of every edge: {a, vector}, {1/length^2, b.x, margin, b.y}.
__global__ void k_wall_edges(int nsedge, const double2 *__restrict__ coord,
                             const int2 *__restrict__ sedge, int bugcompat,
                             float4 *__restrict__ edge32) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nsedge) return;
  const double2 org = coord[sedge[0].x];
  const int2 e = sedge[k];
  const double2 a = coord[e.x], b = coord[e.y];
  const float ax = (float)(a.x - org.x), ay = (float)(a.y - org.y);
  const float bx = (float)(b.x - org.x), by = (float)(b.y - org.y);
  const float dx = (float)(b.x - a.x), dy = bugcompat ? dx : (float)(b.y - a.y);
  const float size = fabsf(ax) + fabsf(ay) + fabsf(bx) + fabsf(by) + fabsf(dx) + fabsf(dy);
  float margin = 3e-6f * size + (float)(1e-15 * (fabs(a.x) + fabs(a.y) + fabs(b.x) + fabs(b.y)));
  if (!(size <= kWallFar)) margin = __int_as_float(0x7f800000);
  edge32[2 * k] = make_float4(ax, ay, dx, dy);
  edge32[2 * k + 1] = make_float4(1.0f / (dx * dx + dy * dy), bx, margin, by);
}

__global__ void __launch_bounds__(kWallThreads) k_wall_dist(int np, int nsedge,
                                                            const double2 *__restrict__ coord,
                                                            const int2 *__restrict__ sedge,
                                                            const float4 *__restrict__ edge32,
                                                            const int *__restrict__ ptype,
                                                            int bugcompat,
                                                            double *__restrict__ wd) {
  __shared__ float4 s_e0[kWallTile], s_e1[kWallTile];   // k_wall_edges
  __shared__ int s_list[kWallList][kWallThreads];    // edges left to FP64
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool solid = i >= np || ptype[i] == 3;       // wd = 1 (or no point): nothing to find
  const double2 ci = (i < np) ? coord[i] : make_double2(0.0, 0.0);
  const double2 org = nsedge > 0 ? coord[sedge[0].x] : make_double2(0.0, 0.0);
  const float px = (float)(ci.x - org.x), py = (float)(ci.y - org.y);
  const float size = fabsf(px) + fabsf(py);
  const float off = size <= kWallFar ? 3e-6f * size : __int_as_float(0x7f800000);
  auto stage = [&](int t0) {
    __syncthreads();
    for (int k = threadIdx.x; k < kWallTile && t0 + k < nsedge; k += kWallThreads) {
      s_e0[k] = edge32[2 * (t0 + k)];
      s_e1[k] = edge32[2 * (t0 + k) + 1];
    }
    __syncthreads();
    return min(kWallTile, nsedge - t0);
  };
  auto end2 = [&](float x, float y) { return (px - x) * (px - x) + (py - y) * (py - y); };
  // squared distance to the segment (a degenerate one: to a)
  auto segment2 = [&](const float4 &e0, const float4 &e1) {
    const float rx = px - e0.x, ry = py - e0.y;
    const float t = fminf(fmaxf((rx * e0.z + ry * e0.w) * e1.x, 0.f), 1.f);
    const float ex = rx - t * e0.z, ey = ry - t * e0.w;
    return ex * ex + ey * ey;
  };
  float near = __int_as_float(0x7f800000);
  for (int t0 = 0; t0 < nsedge; t0 += kWallTile) {
    const int nk = stage(t0);
#pragma unroll 4
    for (int k = 0; k < nk; k++) {
      const float4 e0 = s_e0[k], e1 = s_e1[k];
      const float d2 = bugcompat ? end2(e0.x, e0.y) : segment2(e0, e1);
      near = fminf(near, sqrtf(d2) * 1.000001f + e1.z);
    }
  }
  near = fmaxf(near + 2.f * off, kWallNear);
  double w = 1.0e20;   // (1e10)^2
  int n = 0;
  auto flush = [&]() {
    for (int j = 0; __any_sync(0xffffffffu, j < n); j++)
      if (j < n) {
        const int2 e = sedge[s_list[j][threadIdx.x]];
        wall_edge(ci, coord[e.x], coord[e.y], bugcompat, w);
      }
    n = 0;
  };
  for (int t0 = 0; t0 < nsedge; t0 += kWallTile) {
    // (a single tile is still staged from the first sweep)
    const int nk = nsedge > kWallTile ? stage(t0) : nsedge;
    for (int k = 0; k < nk; k++) {
      const float4 e0 = s_e0[k], e1 = s_e1[k];
      float d2 = segment2(e0, e1);
      if (bugcompat) d2 = fminf(d2, end2(e1.y, e1.w));
      const float t = near + e1.z;
      if (!solid && !(d2 > t * t * 1.00001f)) s_list[n++][threadIdx.x] = t0 + k;
      if (__any_sync(0xffffffffu, n == kWallList)) flush();
    }
  }
  flush();
  if (i < np) wd[i] = solid ? 1.0 : sqrt(w);
}

cudaError_t launch_edge_csl(const double2 *ds, D4 *csl, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_edge_csl<<<(n + 255) / 256, 256, 0, s>>>(ds, csl, n);
  return cudaGetLastError();
}

cudaError_t launch_dtlength(int np, int nt, const double2 *coord, const int *elem,
                            const double *elarea, double *drmin, cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  k_fill<<<(np + 255) / 256, 256, 0, s>>>(drmin, 1.0e15, np);
  if (nt > 0)
    k_dtlength<<<(nt + 255) / 256, 256, 0, s>>>(nt, coord, elem, elarea,
                                               reinterpret_cast<unsigned long long *>(drmin));
  return cudaGetLastError();
}

size_t wall_scratch(int nsedge) { return 2 * sizeof(float4) * (size_t)nsedge; }

cudaError_t launch_wall_dist(int np, int nsedge, const double2 *coord, const int2 *sedge,
                             const int *ptype, int bugcompat, double *wd, void *scratch,
                             cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  float4 *edge32 = static_cast<float4 *>(scratch);
  if (nsedge > 0)
    k_wall_edges<<<(nsedge + 255) / 256, 256, 0, s>>>(nsedge, coord, sedge, bugcompat, edge32);
  k_wall_dist<<<(np + kWallThreads - 1) / kWallThreads, kWallThreads, 0, s>>>(
      np, nsedge, coord, sedge, edge32, ptype, bugcompat, wd);
  return cudaGetLastError();
}

// Driver-order FP64 arrays (k values per vertex) to and from a mesh's
// per-vertex arrays in arena order (rows of `stride` bytes, values of type R
// from column c0): orig holds each arena vertex's driver index (1-based).
// Conversions round to nearest, as the host's would (this unit does not
// flush subnormals).
template <typename R>
__global__ void k_get_vertex(double *dst, const unsigned char *src, size_t stride,
                             const int *__restrict__ orig, int np, int k, int c0) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < np; v += gridDim.x * blockDim.x) {
    const R *q = reinterpret_cast<const R *>(src + (size_t)v * stride) + c0;
    double *d = dst + (size_t)(orig[v] - 1) * k;
    for (int c = 0; c < k; c++) d[c] = (double)q[c];
  }
}

// The same transfers into / out of one of three buffers chosen on the
// device by *sel (a mesh's state phase or nu~ phase in its control block),
// so the host need not read the control block first.  off: the mesh's
// first row, in bytes.
template <typename R>
__global__ void k_put_vertex_sel(unsigned char *b0, unsigned char *b1, unsigned char *b2,
                                 const int *sel, size_t off, size_t stride,
                                 const double *__restrict__ src, const int *__restrict__ orig,
                                 int np, int k) {
  const int i = *sel;
  unsigned char *dst = (i == 0 ? b0 : i == 1 ? b1 : b2) + off;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < np; v += gridDim.x * blockDim.x) {
    const double *q = src + (size_t)(orig[v] - 1) * k;
    R *d = reinterpret_cast<R *>(dst + (size_t)v * stride);
    for (int c = 0; c < k; c++) d[c] = (R)q[c];
  }
}

template <typename R>
__global__ void k_get_vertex_sel(double *dst, const unsigned char *b0, const unsigned char *b1,
                                 const unsigned char *b2, const int *sel, size_t off,
                                 size_t stride, const int *__restrict__ orig, int np, int k,
                                 int c0) {
  const int i = *sel;
  const unsigned char *src = (i == 0 ? b0 : i == 1 ? b1 : b2) + off;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < np; v += gridDim.x * blockDim.x) {
    const R *q = reinterpret_cast<const R *>(src + (size_t)v * stride) + c0;
    double *d = dst + (size_t)(orig[v] - 1) * k;
    for (int c = 0; c < k; c++) d[c] = (double)q[c];
  }
}

// A mesh's control block set for a new state (what 0: iteration and
// iterlast = n, residual normaliser cleared, inactive) or for a start
// (what 1: up to n iterations stopping at fres <= minres), on the device.
__global__ void k_ctl_update(MeshCtl *c, int what, int n, double minres) {
  if (what == 0) {
    c->iter = n;
    c->iterlast = n;
    c->fres1 = 0.0;
    c->active = 0;
  } else {
    c->active = n > 0 ? 1 : 0;
    c->n_done = 0;
    c->n_max = n;
    c->minres = minres;
  }
  c->err = 0;
  c->err_point = INT_MAX;
}

cudaError_t launch_put_vertex_sel(int rsz, unsigned char *const b[3], const int *sel, size_t off,
                                  size_t stride, const double *src, const int *orig, int np,
                                  int k, cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  const int g = (np + 255) / 256;
  if (rsz == 8)
    k_put_vertex_sel<double><<<g, 256, 0, s>>>(b[0], b[1], b[2], sel, off, stride, src, orig, np, k);
  else
    k_put_vertex_sel<float><<<g, 256, 0, s>>>(b[0], b[1], b[2], sel, off, stride, src, orig, np, k);
  return cudaGetLastError();
}

cudaError_t launch_get_vertex_sel(int rsz, double *dst, unsigned char *const b[3], const int *sel,
                                  size_t off, size_t stride, const int *orig, int np, int k,
                                  int c0, cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  const int g = (np + 255) / 256;
  if (rsz == 8)
    k_get_vertex_sel<double><<<g, 256, 0, s>>>(dst, b[0], b[1], b[2], sel, off, stride, orig, np, k, c0);
  else
    k_get_vertex_sel<float><<<g, 256, 0, s>>>(dst, b[0], b[1], b[2], sel, off, stride, orig, np, k, c0);
  return cudaGetLastError();
}

cudaError_t launch_ctl_update(MeshCtl *c, int what, int n, double minres, cudaStream_t s) {
  k_ctl_update<<<1, 1, 0, s>>>(c, what, n, minres);
  return cudaGetLastError();
}

// every row of a mesh's per-vertex array set to the same k values
template <typename R>
__global__ void k_fill_vertex(unsigned char *dst, size_t stride, int np, int k, double a0,
                              double a1, double a2, double a3) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < np; v += gridDim.x * blockDim.x) {
    R *d = reinterpret_cast<R *>(dst + (size_t)v * stride);
    const double a[4] = {a0, a1, a2, a3};
    for (int c = 0; c < k; c++) d[c] = (R)a[c];
  }
}

cudaError_t launch_fill_vertex(int rsz, unsigned char *dst, size_t stride, int np, int k,
                               const double *values, cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  if (k < 1 || k > 4) return cudaErrorInvalidValue;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < k; c++) a[c] = values[c];
  const int g = (np + 255) / 256;
  if (rsz == 8) k_fill_vertex<double><<<g, 256, 0, s>>>(dst, stride, np, k, a[0], a[1], a[2], a[3]);
  else k_fill_vertex<float><<<g, 256, 0, s>>>(dst, stride, np, k, a[0], a[1], a[2], a[3]);
  return cudaGetLastError();
}

cudaError_t launch_get_vertex(int rsz, double *dst, const unsigned char *src, size_t stride,
                              const int *orig, int np, int k, int c0, cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  const int g = (np + 255) / 256;
  if (rsz == 8) k_get_vertex<double><<<g, 256, 0, s>>>(dst, src, stride, orig, np, k, c0);
  else k_get_vertex<float><<<g, 256, 0, s>>>(dst, src, stride, orig, np, k, c0);
  return cudaGetLastError();
}

// The work list's blocks copied in work-list order (the per-block kernels
// then read a block with one load instead of an index load and the block's).
__global__ void k_gather_blocks(const int *__restrict__ work, const BlockInfo *__restrict__ blocks,
                                BlockInfo *__restrict__ out, int n) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < n) out[w] = blocks[work[w]];
}

cudaError_t launch_gather_blocks(const int *work, const BlockInfo *blocks, BlockInfo *out, int n,
                                 cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_gather_blocks<<<(n + 255) / 256, 256, 0, s>>>(work, blocks, out, n);
  return cudaGetLastError();
}

}  // namespace fvm
