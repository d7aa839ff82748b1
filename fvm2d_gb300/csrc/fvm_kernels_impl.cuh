// fvm_kernels_impl.cuh -- launcher definitions for one state precision R.
// Included once per precision translation unit.
#pragma once

#include <cstring>

#include "fvm_kernels.cuh"
#include "fvm_launch.h"

namespace fvm {

// The arithmetic type of the kernels: F64 for FP64 states (products, quotients
// and roots on the integer pipes, the same bits), float for FP32.  The fused
// pass (off by default) keeps the hardware operations: it compiles for double.
template <typename R>
struct KernelType {
  using T = R;
};
template <>
struct KernelType<double> {
  using T = F64;
};
template <typename R>
using KT = typename KernelType<R>::T;
template <typename R>
inline ArenaPtrs<KT<R>> kptrs(const ArenaPtrs<R> &A) {
  static_assert(sizeof(ArenaPtrs<KT<R>>) == sizeof(ArenaPtrs<R>) && sizeof(KT<R>) == sizeof(R),
                "same arrays");
  ArenaPtrs<KT<R>> o;
  std::memcpy(&o, &A, sizeof(o));
  return o;
}

// Grid of a persistent per-block kernel: one wave of the CTAs that fit on
// the device at once (its occupancy with this shared memory), so that no
// partial second wave idles most SMs at the end of a launch.
template <typename K>
inline int fit_grid(const LaunchCfg &c, K kern, size_t smem, int threads = kBlockVerts) {
  if (!c.fit) return c.grid;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem) != cudaSuccess) {
    (void)cudaGetLastError();
    occ = 1;
  }
  const int g = (occ < 1 ? 1 : occ) * c.sms / c.share;
  return g < c.grid ? g : c.grid;
}

// FP64 gradient: rows for inviscid meshes, and for viscous ones where the
// records (136 bytes per triangle) would leave an SM two CTAs, that is blocks of
// 256 vertices; blocks of 64 or 128 keep the one round.  us per iteration,
// records / rows: 512 x 192 laminar 838 / 798, 768 x 256 turbulent 2124 / 2092;
// 300 x 90 laminar (128 vertices) 370 / 377, 160 x 48 turbulent 270 / 276.
// sm: the records' bytes, never less than the rows'.
template <typename R>
inline cudaError_t launch_grad_f64(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int do_dt,
                                   int routine, size_t sm) {
  if constexpr (sizeof(R) == 8) {
    const int form = !c.viscous ? 1 : sm > kMaxSmem / 3 ? 2 : 0;
    if (form) sm = size_t(c.max_tri) * (form == 2 ? 9 : 8) * sizeof(R);
#define FVM_GRAD64(F)                                                                      \
  k_grad<KT<R>, F><<<fit_grid(c, k_grad<KT<R>, F>, sm), kBlockVerts, sm, c.stream>>>(      \
      kptrs(A), stage, do_dt, routine, c.max_tri, 0)
    if (form == 1)
      FVM_GRAD64(1);
    else if (form == 2)
      FVM_GRAD64(2);
    else
      FVM_GRAD64(0);
#undef FVM_GRAD64
  }
  return cudaGetLastError();
}
// What a kernel may take of dynamic shared memory is a property of the function
// in the whole process, so it is set to all that its static part leaves, whatever
// this batch needs: set to a batch's own need, a smaller batch or handle created
// later took it from a larger one, whose next launch then failed.
template <typename K>
inline cudaError_t allow_smem(K kern, size_t need) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kern);
  if (e != cudaSuccess) return e;
  const size_t most = kMaxSmem - a.sharedSizeBytes;
  if (need > most) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

template <typename R>
inline cudaError_t grad_attributes(size_t sm) {
  cudaError_t e = allow_smem(k_grad<KT<R>, 0>, sm);
  if constexpr (sizeof(R) == 8) {
    if (e == cudaSuccess) e = allow_smem(k_grad<KT<R>, 1>, sm);
    if (e == cudaSuccess) e = allow_smem(k_grad<KT<R>, 2>, sm);
  }
  return e;
}

// The flux pass for template code F (Riemann solver | kFluxStd).  FP32: one
// kernel; FP64: every edge once, then the gather.
template <typename R, int F>
inline void launch_flux_code(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int mode,
                             int irk, int routine) {
  if constexpr (sizeof(R) == 4) {
    const size_t sm = size_t(c.max_slots) * sizeof(R4<R>);
    k_flux<KT<R>, F><<<fit_grid(c, k_flux<KT<R>, F>, sm, kFluxThreads), kFluxThreads, sm, c.stream>>>(
        kptrs(A), stage, mode, irk, routine);
  } else {
    // a block's owned entries in items, and its boundary edges
    const int per = c.edge_form == 2 ? kEdgeItem<2> : kEdgeThreads;
    const int items = (c.max_slots + per - 1) / per + 1;
    LaunchCfg ce = c;
    ce.grid = c.grid > INT_MAX / items ? INT_MAX : c.grid * items;
#define FVM_EFLUX(C)                                                                       \
  k_eflux<KT<R>, F, C><<<fit_grid(ce, k_eflux<KT<R>, F, C>, 0, kEdgeThreads), kEdgeThreads, 0, \
                         c.stream>>>(kptrs(A), stage, routine, items)
    if (c.edge_form == 2)
      FVM_EFLUX(2);
    else if (c.edge_form == 1)
      FVM_EFLUX(1);
    else
      FVM_EFLUX(0);
#undef FVM_EFLUX
    k_egather<KT<R>><<<fit_grid(c, k_egather<KT<R>>, 0), kBlockVerts, 0, c.stream>>>(kptrs(A), stage, mode, irk,
                                                                             routine);
  }
}
template <typename R>
inline void launch_flux_any(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int mode,
                            int irk, int routine) {
  if constexpr (sizeof(R) == 4) {
    if (c.std_const) {
      switch (c.flux) {
        case 1: launch_flux_code<R, 1 | kFluxStd>(A, c, stage, mode, irk, routine); return;
        case 2: launch_flux_code<R, 2 | kFluxStd>(A, c, stage, mode, irk, routine); return;
        case 3: launch_flux_code<R, 3 | kFluxStd>(A, c, stage, mode, irk, routine); return;
        default: launch_flux_code<R, kFluxStd>(A, c, stage, mode, irk, routine); return;
      }
    }
  }
  switch (c.flux) {
    case 1: launch_flux_code<R, 1>(A, c, stage, mode, irk, routine); return;
    case 2: launch_flux_code<R, 2>(A, c, stage, mode, irk, routine); return;
    case 3: launch_flux_code<R, 3>(A, c, stage, mode, irk, routine); return;
    default: launch_flux_code<R, 0>(A, c, stage, mode, irk, routine);
  }
}

// Dynamic shared memory of the FP32 flux kernels (FP64: none).
template <typename R>
inline cudaError_t flux_attributes(size_t f) {
  cudaError_t e = cudaSuccess;
  if constexpr (sizeof(R) == 4) {
    e = allow_smem(k_flux<KT<R>, 0>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, 1>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, 2>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, 3>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, kFluxStd>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, 1 | kFluxStd>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, 2 | kFluxStd>, f);
    if (e == cudaSuccess) e = allow_smem(k_flux<KT<R>, 3 | kFluxStd>, f);
  }
  return e;
}

#define FVM_DEFINE_LAUNCHERS(R)                                                            \
  size_t smem_grad(const LaunchCfg &c, R *) {                                              \
    return size_t(c.max_tri) * (sizeof(TriSmem<R>) + (c.viscous ? 9 * sizeof(R) : 0));     \
  }                                                                                        \
  size_t smem_flux(const LaunchCfg &c, R *) { return size_t(c.max_slots) * sizeof(R4<R>); } \
  size_t smem_sa(const LaunchCfg &c, R *) {                                                \
    return size_t(3 * c.max_tri + c.max_slots) * sizeof(R) + 16;                           \
  }                                                                                        \
  cudaError_t launch_visc(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int do_dt,  \
                          int routine) {                                                   \
    k_visc<KT<R>><<<fit_grid(c, k_visc<KT<R>>, 0), kBlockVerts, 0, c.stream>>>(kptrs(A), stage, do_dt, routine);             \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_grad_pipe(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage,       \
                               int do_dt, int routine, long long budget, int inject,      \
                               int skip_inviscid) {                                       \
    if (sizeof(R) != 4 || !c.tri_loc) return cudaErrorNotSupported;                      \
    const GradPipeLayout pl = grad_pipe_layout(c.max_tri, c.max_halo, c.viscous);         \
    const int groups = c.pipe_groups == 1 ? 1 : 2;                                        \
    const int ns = pipe_stage_count(pl.stage, groups, c.pipe_stages);                      \
    if (!ns) return cudaErrorNotSupported;                                                 \
    const size_t sb = (size_t)ns * pl.stage;                                               \
    const int vis = c.viscous ? 1 : 0;                                                     \
    if (groups == 1)                                                                       \
      k_grad_pipe<KT<R>, 1><<<fit_grid(c, k_grad_pipe<KT<R>, 1>, sb, 32 + kBlockVerts),            \
                          32 + kBlockVerts, sb, c.stream>>>(kptrs(A), stage, do_dt, routine,      \
                          c.max_tri, c.max_halo, vis, ns, budget, inject, skip_inviscid);  \
    else                                                                                   \
      k_grad_pipe<KT<R>, 2><<<fit_grid(c, k_grad_pipe<KT<R>, 2>, sb, 32 + 2 * kBlockVerts),        \
                          32 + 2 * kBlockVerts, sb, c.stream>>>(kptrs(A), stage, do_dt, routine,  \
                          c.max_tri, c.max_halo, vis, ns, budget, inject, skip_inviscid);  \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_grad(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int do_dt,  \
                          int routine) {                                                   \
    size_t sm = smem_grad(c, (R *)nullptr);                                                \
    if (sm > kMaxSmem) return cudaErrorInvalidConfiguration;                              \
    /* FP32: inviscid meshes take the vertex-stencil pass, viscous ones the */             \
    /* triangle pass below */                                                              \
    int skip = 0;                                                                          \
    if (sizeof(R) == 4 && c.stencil) {                                                     \
      if (c.any_inviscid) {                                                                \
        k_grad_stencil<KT<R>><<<fit_grid(c, k_grad_stencil<KT<R>>, 0), kBlockVerts, 0, c.stream>>>( \
            kptrs(A), stage, do_dt, routine);                                                     \
        const cudaError_t se = cudaGetLastError();                                         \
        if (se != cudaSuccess) return se;                                                  \
      }                                                                                    \
      if (!c.viscous) return cudaSuccess;                                                  \
      skip = 1;                                                                            \
    }                                                                                      \
    if (c.grad_mode == 4 && sizeof(R) == 4 && c.tri_loc) {                                 \
      const cudaError_t pe = launch_grad_pipe(A, c, stage, do_dt, routine, kPipeBudget, 0, \
                                              skip);                                       \
      if (pe != cudaErrorNotSupported) return pe;                                          \
    }                                                                                      \
    if (c.grad_mode == 2) {                                                                \
      k_grad_v<KT<R>><<<fit_grid(c, k_grad_v<KT<R>>, 0), kBlockVerts, 0, c.stream>>>(kptrs(A), stage, do_dt, routine, skip); \
      return cudaGetLastError();                                                           \
    }                                                                                      \
    if (c.grad_mode >= 3 && c.tri_loc) {  /* else the per-thread form, same sums */      \
      if (sizeof(R) != 4) return cudaErrorNotSupported;                                    \
      const size_t sb = grad_bulk_layout(c.max_tri, c.max_halo, c.viscous).total;          \
      if (sb > kMaxSmem) return cudaErrorInvalidConfiguration;                            \
      k_grad_bulk<KT<R>><<<fit_grid(c, k_grad_bulk<KT<R>>, sb), kBlockVerts, sb, c.stream>>>(       \
          kptrs(A), stage, do_dt, routine, c.max_tri, c.max_halo, c.viscous ? 1 : 0, skip);       \
      return cudaGetLastError();                                                           \
    }                                                                                      \
    if constexpr (sizeof(R) == 8) return launch_grad_f64(A, c, stage, do_dt, routine, sm);  \
    k_grad<KT<R>, 0><<<fit_grid(c, k_grad<KT<R>, 0>, sm), kBlockVerts, sm, c.stream>>>(     \
        kptrs(A), stage, do_dt, routine, c.max_tri, skip);                                 \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_flux(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int mode,   \
                          int irk, int routine) {                                          \
    if (smem_flux(c, (R *)nullptr) > kMaxSmem) return cudaErrorInvalidConfiguration;       \
    launch_flux_any<R>(A, c, stage, mode, irk, routine);                                      \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  size_t smem_step(const LaunchCfg &c, R *) {                                              \
    const size_t tri = size_t(c.max_tri2) * sizeof(TriSmem<R>) +                           \
                       (c.viscous ? size_t(c.max_tri) * 9 * sizeof(R) : 0);                 \
    const size_t flx = size_t(c.max_slots) * sizeof(R4<R>);                                \
    const size_t r1 = ((tri > flx ? tri : flx) + 63) & ~size_t(63);                        \
    return r1 + size_t(c.max_loc) * sizeof(Grad<R>);                                       \
  }                                                                                        \
  cudaError_t launch_step(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage) {           \
    const size_t sm = smem_step(c, (R *)nullptr);                                          \
    if (sm > kMaxSmem) return cudaErrorInvalidConfiguration;                              \
    const int v = c.viscous ? 1 : 0;                                                       \
    switch (c.flux) {                                                                      \
      case 1: k_step<R, 1><<<fit_grid(c, k_step<R, 1>, sm), kBlockVerts, sm, c.stream>>>(A, stage, c.max_tri, c.max_tri2, c.max_slots, c.max_loc, v); break; \
      case 2: k_step<R, 2><<<fit_grid(c, k_step<R, 2>, sm), kBlockVerts, sm, c.stream>>>(A, stage, c.max_tri, c.max_tri2, c.max_slots, c.max_loc, v); break; \
      case 3: k_step<R, 3><<<fit_grid(c, k_step<R, 3>, sm), kBlockVerts, sm, c.stream>>>(A, stage, c.max_tri, c.max_tri2, c.max_slots, c.max_loc, v); break; \
      default: k_step<R, 0><<<fit_grid(c, k_step<R, 0>, sm), kBlockVerts, sm, c.stream>>>(A, stage, c.max_tri, c.max_tri2, c.max_slots, c.max_loc, v); \
    }                                                                                      \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_sa(const ArenaPtrs<R> &A, const LaunchCfg &c, int stage, int routine) {\
    size_t sm = smem_sa(c, (R *)nullptr);                                                  \
    if (sm > kMaxSmem) return cudaErrorInvalidConfiguration;                              \
    k_sa<KT<R>><<<fit_grid(c, k_sa<KT<R>>, sm), kBlockVerts, sm, c.stream>>>(kptrs(A), stage, routine, c.max_tri);           \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_monitor(const ArenaPtrs<R> &A, const LaunchCfg &c) {                   \
    if (A.nslots <= 0) return cudaSuccess;                                                 \
    k_monitor<KT<R>><<<A.nslots, kMonitorMaxThreads, 0, c.stream>>>(kptrs(A));                      \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_update(const ArenaPtrs<R> &A, const LaunchCfg &c, int irk) {           \
    k_update<KT<R>><<<c.grid, kBlockVerts, 0, c.stream>>>(kptrs(A), irk);                             \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_time_step(const ArenaPtrs<R> &A, const LaunchCfg &c) {                 \
    k_time_step<KT<R>><<<c.grid, kBlockVerts, 0, c.stream>>>(kptrs(A));                               \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_positivity(const ArenaPtrs<R> &A, const LaunchCfg &c) {                \
    k_positivity<KT<R>><<<c.grid, kBlockVerts, 0, c.stream>>>(kptrs(A));                              \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_conres(const ArenaPtrs<R> &A, const LaunchCfg &c, int mesh, int first) {\
    k_conres_part<KT<R>><<<c.grid, kBlockVerts, 0, c.stream>>>(kptrs(A));                             \
    k_routine_monitor<KT<R>><<<1, kMonitorMaxThreads, 0, c.stream>>>(kptrs(A), mesh, 0, first);                       \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_clcd(const ArenaPtrs<R> &A, const LaunchCfg &c, int mesh) {             \
    k_routine_monitor<KT<R>><<<1, kMonitorMaxThreads, 0, c.stream>>>(kptrs(A), mesh, 1, 0);                           \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_gradient_edge(const ArenaPtrs<R> &A, const LaunchCfg &c) {             \
    const size_t sm = size_t(c.max_slots) * sizeof(Grad<R>);                                 \
    if (sm > kMaxSmem) return cudaErrorInvalidConfiguration;                              \
    k_gradient_edge<KT<R>><<<c.grid, kBlockVerts, sm, c.stream>>>(kptrs(A));                          \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_shockind(const ArenaPtrs<R> &A, const LaunchCfg &c) {                  \
    k_shockind<KT<R>><<<c.grid, kBlockVerts, 0, c.stream>>>(kptrs(A));                                \
    k_shock_zero<KT<R>><<<c.grid, kBlockVerts, 0, c.stream>>>(kptrs(A));                   \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t launch_limitgrad(const ArenaPtrs<R> &A, const LaunchCfg &c) {                 \
    /* the hardware's operations: F64's called quotients made 98k vertices 75 us */        \
    /* a call instead of 67, 1.2k vertices 27 instead of 23 */                             \
    k_limitgrad<R><<<c.grid, kBlockVerts, 0, c.stream>>>(A);                               \
    return cudaGetLastError();                                                             \
  }                                                                                        \
  cudaError_t prepare_attributes(const LaunchCfg &c, R *) {                                \
    const size_t g = smem_grad(c, (R *)nullptr), f = smem_flux(c, (R *)nullptr),           \
                 s = smem_sa(c, (R *)nullptr);                                             \
    const size_t st = smem_step(c, (R *)nullptr);                                          \
    if (g > kMaxSmem || f > kMaxSmem || s > kMaxSmem || st > kMaxSmem)                     \
      return cudaErrorInvalidConfiguration;                                                \
    cudaError_t e = allow_smem(k_step<R, 0>, st);                                          \
    if (e == cudaSuccess) e = allow_smem(k_step<R, 1>, st);                                \
    if (e == cudaSuccess) e = allow_smem(k_step<R, 2>, st);                                \
    if (e == cudaSuccess) e = allow_smem(k_step<R, 3>, st);                                \
    if (e == cudaSuccess) e = grad_attributes<R>(g);                                       \
    if (e == cudaSuccess) e = flux_attributes<R>(f);                                       \
    if (e == cudaSuccess) e = allow_smem(k_sa<KT<R>>, s);                                  \
    const size_t ge = size_t(c.max_slots) * sizeof(Grad<R>);                               \
    const size_t gb = grad_bulk_layout(c.max_tri, kTriLocMax, c.viscous).total;            \
    /* (where these two do not fit, their launchers say so) */                             \
    if (e == cudaSuccess && ge <= kMaxSmem) e = allow_smem(k_gradient_edge<KT<R>>, ge);    \
    if (e == cudaSuccess && sizeof(R) == 4 && gb <= kMaxSmem)                              \
      e = allow_smem(k_grad_bulk<KT<R>>, gb);                                              \
    if (e == cudaSuccess && sizeof(R) == 4) e = allow_smem(k_grad_pipe<KT<R>, 1>, 0);      \
    if (e == cudaSuccess && sizeof(R) == 4) e = allow_smem(k_grad_pipe<KT<R>, 2>, 0);      \
    return e;                                                                              \
  }

}  // namespace fvm
