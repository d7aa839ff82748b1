// fvm_kernels.cuh -- CUDA kernels of the fvm2d hot path, templated on the
// state type R.  Included by fvm_kernels_fp64.cu (compiled without FMA
// contraction) and fvm_kernels_fp32.cu.
//
// Every per-block kernel walks the work list (a persistent grid-stride loop
// over blocks of every active mesh in the arena), skips meshes whose control
// block is inactive, and picks the state buffers from the mesh's phase:
//   iterate mode, stage s = 1,2,3 (old = buffer p):
//     s1: p -> p+1      s2: p+1 -> p+2      s3: p+2 -> p+1   (mod 3)
//   routine mode (stage 0): state = p, prim_old = p+2, updates in place.
#pragma once

#include <cfloat>
#include <climits>

#include "fvm_device.cuh"

#ifndef FVM_FLUX_THREADS
#define FVM_FLUX_THREADS 256  // threads of the FP32 flux pass's CTAs (one block of vertices each)
#endif
#ifndef FVM_FLUX_MINB32
#define FVM_FLUX_MINB32 6   // resident CTAs per SM asked of the FP32 flux kernel
#endif
#ifndef FVM_GRAD_MINB32
#define FVM_GRAD_MINB32 5   // resident CTAs per SM asked of the FP32 gradient kernel
#endif
#ifndef FVM_EGATHER_MINB
#define FVM_EGATHER_MINB 4   // resident CTAs per SM asked of the FP64 gather kernel (2, 3: 10-30% slower)
#endif
#ifndef FVM_EGATHER_BATCH
#define FVM_EGATHER_BATCH 2  // its incidences loaded together (4, 8 at fewer CTAs: 10-40% slower)
#endif
#ifndef FVM_GRAD_MINB64
#define FVM_GRAD_MINB64 4   // the same of the FP64 one for inviscid meshes (3, 5: the same)
#endif
#ifndef FVM_GRAD_MINBV64
#define FVM_GRAD_MINBV64 3  // the same with viscous ones (2: 14-25% slower, 4: the same)
#endif
#ifndef FVM_GRADV_MINB32
#define FVM_GRADV_MINB32 4  // the same for its per-vertex form
#endif
#ifndef FVM_STENCIL_MINB
#define FVM_STENCIL_MINB 6  // resident CTAs per SM asked of the stencil gradient kernel
#endif
#ifndef FVM_EFLUX_MINB
#define FVM_EFLUX_MINB 4    // resident CTAs per SM asked of the FP64 edge kernel (5-8: 3-8% slower)
#endif
#ifndef FVM_EFLUX_FEWB
#define FVM_EFLUX_FEWB 6    // the same with four warps to 32 edges (4: 20%, 7: 9% slower at 160 x 48)
#endif
#ifndef FVM_EFLUX_CALLB
#define FVM_EFLUX_CALLB 7   // the same with called operations (5, 6: 2-12% slower, 8: the same)
#endif
#ifndef FVM_GATHER_BATCH
#define FVM_GATHER_BATCH 1  // FP32 flux pass: incidences loaded together in the per-vertex gather
#endif
#ifndef FVM_FLUX_PIPE
#define FVM_FLUX_PIPE 1     // FP32 flux pass: the next edge entry's ends in flight with this entry's gathers
#endif
#ifndef FVM_STENCIL_PIPE
#define FVM_STENCIL_PIPE 1  // stencil pass: next trip's neighbour ids in flight with this trip's states
#endif
#ifndef FVM_STENCIL_BATCH
#define FVM_STENCIL_BATCH 2 // edges whose loads are in flight at once per thread
#endif

namespace fvm {

// FP32 flux pass: threads per CTA (one block of kBlockVerts vertices; the
// edge trips spread over all of them, the per-vertex gather uses the first
// kBlockVerts)
constexpr int kFluxThreads = FVM_FLUX_THREADS;
static_assert(kFluxThreads % 32 == 0 && kFluxThreads >= kBlockVerts && kFluxThreads <= 1024,
              "flux CTA size");

enum { MODE_RESIDUAL = 0, MODE_UPDATE = 1 };

__device__ __forceinline__ int cur_buf(int p, int stage) {
  return stage <= 1 ? p : (p + stage - 1) % 3;
}
__device__ __forceinline__ int out_buf(int p, int stage) {
  return stage == 2 ? (p + 2) % 3 : (p + 1) % 3;
}
__device__ __forceinline__ int old_buf(int p, int stage) {
  return stage == 0 ? (p + 2) % 3 : p;
}

template <typename R>
__device__ __forceinline__ R4<R> ld4(const R4<R> *p) { return *p; }

// Bulk prefetch of [p, p + bytes) into L2 (cp.async.bulk.prefetch, no
// completion to wait for).  The range is shrunk to 16-byte boundaries
// inside the given one, so nothing outside it is touched.
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const uintptr_t b = (a + 15) & ~uintptr_t(15);
  const uintptr_t e = (a + bytes) & ~uintptr_t(15);
  if (e <= b) return;
  uintptr_t n = e - b;
  // the size operand is 32-bit; split very long ranges
  while (n > 0) {
    const uint32_t chunk = n > (1u << 20) ? (1u << 20) : (uint32_t)n;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b + (e - b - n)), "r"(chunk)
                 : "memory");
    n -= chunk;
  }
}

// The next block this CTA will process (persistent loop), for prefetching.
// The blocks a launch covers: the whole work list (part 0) or part k, which
// ends at nwork[k] and starts where part k-1 ends (parts end at mesh
// boundaries).
template <typename R>
__device__ __forceinline__ void work_range(const ArenaPtrs<R> &A, int &w0, int &w1) {
  if (A.wpart == 0) {
    w0 = 0;
    w1 = A.nwork[0];
  } else {
    w0 = A.wpart == 1 ? 0 : A.nwork[A.wpart - 1];
    w1 = A.nwork[A.wpart];
  }
}

// Block w of the work list: its copy in work-list order (one load, not an
// index load followed by the block's; the host refreshes the copies with
// the work list)
template <typename R>
__device__ __forceinline__ const BlockInfo &work_block(const ArenaPtrs<R> &A, int w) {
  return A.wblocks[w];
}

template <typename R>
__device__ __forceinline__ const BlockInfo *next_block(const ArenaPtrs<R> &A, int w, int nwork) {
  const int nw = w + gridDim.x;
  return nw < nwork ? &work_block(A, nw) : nullptr;
}

// ---------------------------------------------------------------------------
// Viscosity (viscosity.f:2-55) and, at stage 1, the viscous time step
// (time_step.f:13-20) from the previous mu.  One thread per vertex.
// ---------------------------------------------------------------------------
// mbarrier and bulk-copy primitives (sm_90+ PTX) for staging a block's
// contiguous ranges in shared memory.
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
// global -> shared bulk copy; addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// waits for the phase with the given parity; false after about a second
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity))
    if (clock64() - t0 > (1LL << 31)) return false;
  return true;
}
// orders this thread's generic-proxy shared-memory accesses before later
// async-proxy (bulk copy) writes to the same bytes
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Threads of the per-mesh monitor CTA (eight warps; the fixed-order reduction
// depends on it).  Wider CTAs measured no faster.
constexpr int kMonitorMaxThreads = 256;

// Per-vertex geometry in the kernel's precision (FP32 copies for R = float).
template <typename R>
__device__ __forceinline__ R v_ais(const ArenaPtrs<R> &A, int v) {
  if constexpr (sizeof(R) == 4) return A.ais32[v];
  else return A.ais[v];
}
template <typename R>
__device__ __forceinline__ R v_cvarea(const ArenaPtrs<R> &A, int v) {
  if constexpr (sizeof(R) == 4) return A.cvarea32[v];
  else return A.cvarea[v];
}
template <typename R>
__device__ __forceinline__ R v_wd(const ArenaPtrs<R> &A, int v) {
  if constexpr (sizeof(R) == 4) return A.wd32[v];
  else return A.wd[v];
}
template <typename R>
__device__ __forceinline__ R v_drmin(const ArenaPtrs<R> &A, int v) {
  if constexpr (sizeof(R) == 4) return A.drmin32[v];
  else return A.drmin[v];
}

// viscosity.f for the state a stage has just produced, which the next stage
// of the iteration starts from (what k_visc would compute at that stage)
template <typename R>
__device__ __forceinline__ void next_viscosity(const ArenaPtrs<R> &A, const MeshConst &mc,
                                               const MeshCtl &ctl, int v, const R4<R> &pn) {
  const R mul = sutherland_viscosity<R>(mc, pn.x, pn.w);
  A.mul[v] = mul;
  A.mu[v] = mc.iflow == 2 ? mul : mul + mu_turb<R>(mc, mul, pn.x, A.nut[ctl.nphase][v]);
}

template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_visc(ArenaPtrs<R> A, int stage, int do_dt,
                                                      int routine) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    const MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    if (mc.iflow == 1 || threadIdx.x >= bi.nv) continue;   // inviscid: mu stays 0
    const int v = bi.v0 + threadIdx.x;
    const R4<R> P = A.st[cur_buf(ctl.phase, stage)][v];
    if (do_dt) A.dt[v] = time_step<R>(mc, P, A.mu[v], v_drmin(A, v));
    R mul = sutherland_viscosity<R>(mc, P.x, P.w);
    A.mul[v] = mul;
    if (mc.iflow == 2) {
      A.mu[v] = mul;
    } else {
      R mut = mu_turb<R>(mc, mul, P.x, A.nut[ctl.nphase][v]);
      A.mu[v] = mul + mut;
    }
  }
}

// ---------------------------------------------------------------------------
// Gradient pass: green_gauss_euler / green_gauss_visc (green_gauss.f:2-92)
// with tri_gg and tri_visc; at stage 1 of an inviscid iteration also the
// local time step (time_step.f:22-27).
// ---------------------------------------------------------------------------
template <typename R>
struct TriSmem {
  R dxt[4];
  R dyt[4];
};

// a + b rounded as written (never fused with a product that forms b)
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ F64 add_rn(F64 a, F64 b) { return F64(__dadd_rn(a.v, b.v)); }

// Green-Gauss terms of one triangle (green_gauss.f:100-127): dbxx/dbyy of
// its vertices and the sums dxt/dyt of the four primitive variables.
template <typename R>
__device__ __forceinline__ void tri_geom(const ArenaPtrs<R> &A, const int4 &t, int entry,
                                         R dbxx[3], R dbyy[3]) {
  if constexpr (sizeof(R) == 4) {
    const TriGeo32 tg = A.tri_g32[entry];
    for (int j = 0; j < 3; j++) {
      dbxx[j] = tg.dbxx[j];
      dbyy[j] = tg.dbyy[j];
    }
  } else {
    const double2 c1 = A.coord[t.x], c2 = A.coord[t.y], c3 = A.coord[t.z];
    dbxx[0] = c2.y - c3.y;
    dbxx[1] = c3.y - c1.y;
    dbxx[2] = c1.y - c2.y;
    dbyy[0] = c3.x - c2.x;
    dbyy[1] = c1.x - c3.x;
    dbyy[2] = c2.x - c1.x;
  }
}

template <typename R>
__device__ __forceinline__ void tri_sums(const R4<R> &p1, const R4<R> &p2, const R4<R> &p3,
                                         const R dbxx[3], const R dbyy[3], TriSmem<R> &ts) {
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const R a1 = comp(p1, q), a2 = comp(p2, q), a3 = comp(p3, q);
    ts.dxt[q] = a1 * dbxx[0] + a2 * dbxx[1] + a3 * dbxx[2];
    ts.dyt[q] = a1 * dbyy[0] + a2 * dbyy[1] + a3 * dbyy[2];
  }
}

// tri_visc (green_gauss.f:132-194): stresses and heat flux of one triangle;
// the contribution to its vertex at position j is
// ((txx, txy, efx) . dbxx[j] + (txy, tyy, efy) . dbyy[j]) * areat.
template <typename R>
struct TriVisc {
  R txx, txy, tyy, efx, efy, areat;
};

template <typename R>
__device__ __forceinline__ R tri_areat(const ArenaPtrs<R> &A, const int4 &t, int entry) {
  if constexpr (sizeof(R) == 4) return A.tri_g32[entry].areat;
  else return A.areat[t.w];
}

template <typename R>
__device__ __forceinline__ TriVisc<R> tri_visc(const ArenaPtrs<R> &A, const MeshConst &mc,
                                               int nbuf, const int4 &t, R areat,
                                               const R4<R> &p1, const R4<R> &p2,
                                               const R4<R> &p3, const R dbxx[3],
                                               const R dbyy[3], const TriSmem<R> &ts) {
  const R n2b3 = R(2) / R(3);
  const R en1 = mdiv(p1.w, p1.x), en2 = mdiv(p2.w, p2.x), en3 = mdiv(p3.w, p3.x);
  const R ext = en1 * dbxx[0] + en2 * dbxx[1] + en3 * dbxx[2];
  const R eyt = en1 * dbyy[0] + en2 * dbyy[1] + en3 * dbyy[2];
  const R um = mdiv(p1.y + p2.y + p3.y, R(3));
  const R vm = mdiv(p1.z + p2.z + p3.z, R(3));
  const R mult = mdiv(A.mul[t.x] + A.mul[t.y] + A.mul[t.z], R(3));
  // laminar meshes: mu = mul and nu~ = 0 exactly (viscosity.f, initialize.f),
  // so the turbulent heat-flux term is exactly zero and mu, nu~ need no loads
  R mut = mult, tterm = R(0);
  if (mc.iflow == 3) {
    mut = (A.mu[t.x] + A.mu[t.y] + A.mu[t.z]) / R(3);
    const R prim5t = (A.nut[nbuf][t.x] + A.nut[nbuf][t.y] + A.nut[nbuf][t.z]) / R(3);
    const R rhot = (p1.x + p2.x + p3.x) / R(3);
    const R chi = prim5t * rhot / mult;
    const R chi3 = cube(chi);
    const R fv1 = chi3 / (chi3 + MCR(R, cv11));
    tterm = rhot * prim5t * fv1 / MCR(R, prandtl_turb);
  }
  TriVisc<R> o;
  o.txx = n2b3 * mut * (R(2) * ts.dxt[1] - ts.dyt[2]);
  o.txy = mut * (ts.dyt[1] + ts.dxt[2]);
  o.tyy = n2b3 * mut * (R(2) * ts.dyt[2] - ts.dxt[1]);
  const R gpr = mdiv(MCR(R, gamma) * (mdiv(mult, MCR(R, prandtl)) + tterm), MCR(R, gamma1));
  o.efx = o.txx * um + o.txy * vm + gpr * ext;
  o.efy = o.txy * um + o.tyy * vm + gpr * eyt;
  o.areat = areat;
  return o;
}

template <typename R>
__device__ __forceinline__ void tri_visc_term(const TriVisc<R> &tv, R dbx, R dby, R out[3]) {
  out[0] = (tv.txx * dbx + tv.txy * dby) * tv.areat;
  out[1] = (tv.txy * dbx + tv.tyy * dby) * tv.areat;
  out[2] = (tv.efx * dbx + tv.efy * dby) * tv.areat;
}

// FP32 triangle sums in shared memory, the record's two 16-byte halves swapped
// where bit 2 of the slot is set: neighbouring threads read slots one or two
// apart, whose like halves would share a quarter or half of the banks (60% of
// the gradient's shared-memory wavefronts were conflicts, now 45%; 4 x 768x256
// turbulent 0.072 -> 0.064 ms per stage, the 24-mesh mix 0.132 -> 0.122, and
// 0.399 -> 0.381 and 0.688 -> 0.658 ms per iteration.  A fourth CTA per SM, 2
// KB less each, cost the mix's chains 0.66 -> 0.76: other chains' kernels no
// longer fit beside them).
template <typename R>
__device__ __forceinline__ void put_sums(TriSmem<R> *tri, int slot, const TriSmem<R> &t) {
  R4<R> *q = reinterpret_cast<R4<R> *>(tri + slot);
  const int b = (slot >> 2) & 1;
  q[b] = reinterpret_cast<const R4<R> *>(&t)[0];
  q[b ^ 1] = reinterpret_cast<const R4<R> *>(&t)[1];
}
template <typename R>
__device__ __forceinline__ TriSmem<R> get_sums(const TriSmem<R> *tri, int slot) {
  const R4<R> *q = reinterpret_cast<const R4<R> *>(tri + slot);
  const int b = (slot >> 2) & 1;
  TriSmem<R> t;
  reinterpret_cast<R4<R> *>(&t)[0] = q[b];
  reinterpret_cast<R4<R> *>(&t)[1] = q[b ^ 1];
  return t;
}

// Sums of one vertex's triangle terms in the order of its incidence list
// (green_gauss.f:23-39 visits triangles in ascending order): entries
// [j0, j1) of `vtl`, each a triangle slot and the vertex's position in it.
// The slots and terms of up to B triangles are loaded before they are
// added, so the shared-memory latency is paid once per B triangles; the
// additions stay in list order (same bits as one triangle at a time).
// vis = nullptr: inviscid (rv is zero).  SWAP: records as put_sums writes them.
template <typename R, int B, bool SWAP = false>
__device__ __forceinline__ void grad_vertex_sums(const uint16_t *vtl, int j0, int j1,
                                                 const TriSmem<R> *tri, const R *vis, R qx[4],
                                                 R qy[4], R rv[3]) {
#pragma unroll
  for (int q = 0; q < 4; q++) qx[q] = qy[q] = R(0);
  rv[0] = rv[1] = rv[2] = R(0);
  for (int j = j0; j < j1; j += B) {
    const int n = j1 - j;
    uint16_t e[B];
#pragma unroll
    for (int u = 0; u < B; u++) e[u] = u < n ? vtl[j + u] : uint16_t(0);
    TriSmem<R> ts[B];
#pragma unroll
    for (int u = 0; u < B; u++)
      if (u < n) {
        if constexpr (SWAP) ts[u] = get_sums<R>(tri, e[u] & 0x3fff);
        else ts[u] = tri[e[u] & 0x3fff];
      }
#pragma unroll
    for (int u = 0; u < B; u++) {
      if (u < n) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          qx[q] = qx[q] + ts[u].dxt[q];
          qy[q] = qy[q] + ts[u].dyt[q];
        }
        if (vis) {
          const R *sv = vis + 9 * (e[u] & 0x3fff) + 3 * (e[u] >> kTriPosShift);
          rv[0] = rv[0] + sv[0];
          rv[1] = rv[1] + sv[1];
          rv[2] = rv[2] + sv[2];
        }
      }
    }
  }
}

// FP64: the sums of the four variables one after another (the integer products
// make long code), the triangle sums as rows of max_tri in shared memory, s[2 q]
// and s[2 q + 1] of variable q (random 64-byte records conflict in the banks).
// Few live values: four CTAs share an SM instead of two; 1024 x 384: 136 -> 107
// us.  Viscous meshes' terms follow in a second round over the triangles and
// vertices, in the same rows: 72 bytes per triangle instead of 136, three CTAs;
// 512 x 192 laminar 86 -> 72 us, 768 x 256 turbulent 168 -> 160 (called
// operations: 85 and 182).
template <typename R>
__device__ __forceinline__ void tri_sums_rows(const ArenaPtrs<R> &A, const R4<R> *P, int entry,
                                              int k, R *s, int max_tri) {
  const int4 t = A.bt_nodes[entry];
  const R *s1 = reinterpret_cast<const R *>(P + t.x), *s2 = reinterpret_cast<const R *>(P + t.y),
          *s3 = reinterpret_cast<const R *>(P + t.z);
  R dbxx[3], dbyy[3];
  tri_geom<R>(A, t, entry, dbxx, dbyy);
#pragma unroll 1
  for (int q = 0; q < 4; q++) {
    const R a1 = s1[q], a2 = s2[q], a3 = s3[q];
    s[2 * q * max_tri + k] = a1 * dbxx[0] + a2 * dbxx[1] + a3 * dbxx[2];
    s[(2 * q + 1) * max_tri + k] = a1 * dbyy[0] + a2 * dbyy[1] + a3 * dbyy[2];
  }
}

// The viscous terms of triangle k into rows 0..8 (the sums' rows, which its
// vertices have been given): row 3 pos + c is component c at position pos.
template <typename R>
__device__ __forceinline__ void tri_visc_rows(const ArenaPtrs<R> &A, const MeshConst &mc, int nbuf,
                                              const R4<R> *P, int entry, int k, R *s,
                                              int max_tri) {
  const int4 t = A.bt_nodes[entry];
  R dbxx[3], dbyy[3];
  tri_geom<R>(A, t, entry, dbxx, dbyy);
  TriSmem<R> ts;
  ts.dxt[1] = s[2 * max_tri + k];
  ts.dyt[1] = s[3 * max_tri + k];
  ts.dxt[2] = s[4 * max_tri + k];
  ts.dyt[2] = s[5 * max_tri + k];
  const TriVisc<R> tv = tri_visc<R>(A, mc, nbuf, t, tri_areat<R>(A, t, entry), P[t.x], P[t.y],
                                    P[t.z], dbxx, dbyy, ts);
#pragma unroll
  for (int j = 0; j < 3; j++) {
    R o[3];
    tri_visc_term<R>(tv, dbxx[j], dbyy[j], o);
#pragma unroll
    for (int c = 0; c < 3; c++) s[(3 * j + c) * max_tri + k] = o[c];
  }
}

// FORM 0: sums and viscous terms of a triangle as records, one round; FP64 also
// as rows: 1 inviscid meshes only, 2 viscous ones too, in two rounds.
template <typename R, int FORM>
__global__ void __launch_bounds__(kBlockVerts, sizeof(R) == 4 ? FVM_GRAD_MINB32
                                               : FORM == 0    ? 2
                                               : FORM == 1    ? FVM_GRAD_MINB64
                                                              : FVM_GRAD_MINBV64)
    k_grad(ArenaPtrs<R> A, int stage, int do_dt, int routine, int max_tri, int skip_inviscid) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TriSmem<R> *s_tri = reinterpret_cast<TriSmem<R> *>(smem_raw);
  R *s_vis = reinterpret_cast<R *>(s_tri + max_tri);   // [max_tri][3 pos][3 comp]
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    const MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    if (skip_inviscid && mc.iflow == 1) continue;   // the stencil pass's meshes
    const bool visc = FORM != 1 && mc.iflow != 1;
    const R4<R> *P = A.st[cur_buf(ctl.phase, stage)];
    if (threadIdx.x == 0) {
      const BlockInfo *nb = next_block(A, w, nwork);
      if (nb) {
        const BlockInfo n = *nb;
        prefetch_l2(A.bt_nodes + n.t0, sizeof(int4) * n.nt);
        if (sizeof(R) == 4) prefetch_l2(A.tri_g32 + n.t0, sizeof(TriGeo32) * n.nt);
        prefetch_l2(P + n.v0, sizeof(R4<R>) * n.nv);
        if (sizeof(R) == 8) prefetch_l2(A.coord + n.v0, sizeof(double2) * n.nv);
        prefetch_l2(A.vt_rng + n.v0, sizeof(int2) * n.nv);
        prefetch_l2(sizeof(R) == 4 ? (const void *)(A.ais32 + n.v0) : (const void *)(A.ais + n.v0), sizeof(R) * n.nv);
      }
    }
    if constexpr (FORM != 0) {
      R *s = reinterpret_cast<R *>(smem_raw);
      const int v = bi.v0 + threadIdx.x;
      const bool mine = threadIdx.x < bi.nv;
      int2 jr = make_int2(0, 0);
      if (mine) jr = A.vt_rng[v];
      for (int k = threadIdx.x; k < bi.nt; k += blockDim.x)
        tri_sums_rows<R>(A, P, bi.t0 + k, k, s, max_tri);
      __syncthreads();
      if (mine) {
        R qx[4], qy[4];
#pragma unroll
        for (int q = 0; q < 4; q++) qx[q] = qy[q] = R(0);
        for (int j = jr.x; j < jr.y; j++) {
          const R *e = s + (A.vt_list[j] & 0x3fff);
#pragma unroll
          for (int q = 0; q < 4; q++) {
            qx[q] = qx[q] + e[2 * q * max_tri];
            qy[q] = qy[q] + e[(2 * q + 1) * max_tri];
          }
        }
        const R ais = v_ais(A, v);
        Grad<R> g;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          g.qx[q] = qx[q] * ais;
          g.qy[q] = qy[q] * ais;
        }
        A.grad[v] = g;
        if (!visc && do_dt) A.dt[v] = time_step<R>(mc, P[v], R(0), v_drmin(A, v));
      }
      __syncthreads();
      if (!visc) continue;
      for (int k = threadIdx.x; k < bi.nt; k += blockDim.x)
        tri_visc_rows<R>(A, mc, ctl.nphase, P, bi.t0 + k, k, s, max_tri);
      __syncthreads();
      if (mine) {
        R rv[3] = {R(0), R(0), R(0)};
        for (int j = jr.x; j < jr.y; j++) {
          const int u = A.vt_list[j];
          const R *e = s + 3 * (u >> kTriPosShift) * max_tri + (u & 0x3fff);
#pragma unroll
          for (int c = 0; c < 3; c++) rv[c] = rv[c] + e[c * max_tri];
        }
        R4<R> o;
        o.x = R(0);
        o.y = rv[0];
        o.z = rv[1];
        o.w = rv[2];
        A.resv[v] = o;
      }
      __syncthreads();
    } else {
      // phase 1: one thread per triangle touching the block
      for (int k = threadIdx.x; k < bi.nt; k += blockDim.x) {
        const int4 t = A.bt_nodes[bi.t0 + k];
        const R4<R> p1 = P[t.x], p2 = P[t.y], p3 = P[t.z];
        R dbxx[3], dbyy[3];
        tri_geom<R>(A, t, bi.t0 + k, dbxx, dbyy);
        TriSmem<R> ts;
        tri_sums<R>(p1, p2, p3, dbxx, dbyy, ts);
        s_tri[k] = ts;
        if (visc) {
          const TriVisc<R> tv = tri_visc<R>(A, mc, ctl.nphase, t, tri_areat<R>(A, t, bi.t0 + k), p1, p2, p3, dbxx, dbyy, ts);
          R *sv = s_vis + 9 * k;
#pragma unroll
          for (int j = 0; j < 3; j++) tri_visc_term<R>(tv, dbxx[j], dbyy[j], sv + 3 * j);
        }
      }
      __syncthreads();
      // phase 2: one thread per vertex, triangles in original order
      if (threadIdx.x < bi.nv) {
        const int v = bi.v0 + threadIdx.x;
        R qx[4], qy[4], rv[3];
        const int2 jr = A.vt_rng[v];
        // (FP32: one triangle at a time, the 48 registers of five CTAs per SM)
        grad_vertex_sums<R, sizeof(R) == 8 ? 2 : 1>(A.vt_list, jr.x, jr.y, s_tri,
                                                    visc ? s_vis : nullptr, qx, qy, rv);
        const R ais = v_ais(A, v);
        Grad<R> g;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          g.qx[q] = qx[q] * ais;
          g.qy[q] = qy[q] * ais;
        }
        A.grad[v] = g;
        if (visc) {
          R4<R> r;
          r.x = R(0);
          r.y = rv[0];
          r.z = rv[1];
          r.w = rv[2];
          A.resv[v] = r;
        } else if (do_dt) {
          A.dt[v] = time_step<R>(mc, P[v], R(0), v_drmin(A, v));
        }
      }
      __syncthreads();
    }
  }
}

// Gradient pass with the block's contiguous inputs staged by bulk copies
// (FP32): one thread issues cp.async.bulk copies of the triangle entries,
// their geometry, the vertices' incidence ranges and the incidence list
// into shared memory (a few tens of KB in flight per CTA, tracked by one
// mbarrier); the threads then only gather the three states of each
// triangle.  Same arithmetic and order as k_grad.  Wait on the copies is
// bounded: after about a second the mesh gets FVM_ERR_TIMEOUT and the CTA
// returns.
template <typename R>
__global__ void __launch_bounds__(kBlockVerts, sizeof(R) == 4 ? FVM_GRAD_MINB32 : 1)
    k_grad_bulk(ArenaPtrs<R> A, int stage, int do_dt, int routine, int max_tri, int max_halo,
                int viscous, int skip_inviscid) {
  if constexpr (sizeof(R) == 4) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    const GradBulkLayout lay = grad_bulk_layout(max_tri, max_halo, viscous != 0);
    int *s_halo = reinterpret_cast<int *>(smem_raw + lay.halo);
    const TriGeo32 *s_geo = reinterpret_cast<const TriGeo32 *>(smem_raw + lay.geo);
    TriSmem<R> *s_tri = reinterpret_cast<TriSmem<R> *>(smem_raw + lay.geo);   // in place
    R *s_vis = reinterpret_cast<R *>(smem_raw + lay.vis);
    int2 *s_vtr = reinterpret_cast<int2 *>(smem_raw + lay.vtr);
    uint16_t *s_vtl = reinterpret_cast<uint16_t *>(smem_raw + lay.vtl);
    R4<R> *s_pv = reinterpret_cast<R4<R> *>(smem_raw + lay.pv);
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    uint32_t parity = 0;
    int w0, nwork;
  work_range(A, w0, nwork);
    for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
      const BlockInfo bi = work_block(A, w);
      const MeshCtl &ctl = A.ctl[bi.mesh];
      if (!routine && !ctl.active) continue;
      const MeshConst &mc = A.mc[bi.mesh];
      if (skip_inviscid && mc.iflow == 1) continue;   // the stencil pass's meshes
      const bool visc = mc.iflow != 1;
      const R4<R> *P = A.st[cur_buf(ctl.phase, stage)];
      const int vt_a = bi.vt0 & ~7;                       // 16-byte units of uint16
      const int vt_b = (bi.vt0 + bi.nvt + 7) & ~7;
      // the halo vertices' ids, for the records' local slots (plain loads,
      // in flight during the copies)
      for (int h = threadIdx.x; h < bi.nh; h += blockDim.x) s_halo[h] = A.halo_ids[bi.h0 + h];
      if (threadIdx.x == 0) {
        const uint32_t ngeo = 32u * bi.nt;
        const uint32_t nvtr = 8u * ((bi.nv + 1) & ~1), nvtl = 2u * (vt_b - vt_a);
        const uint32_t npv = 16u * bi.nv;
        mbar_expect_tx(&bar, ngeo + nvtr + nvtl + npv);
        if (ngeo) bulk_g2s((void *)s_geo, A.tri_g32 + bi.t0, ngeo, &bar);
        bulk_g2s(s_vtr, A.vt_rng + bi.v0, nvtr, &bar);
        if (nvtl) bulk_g2s(s_vtl, A.vt_list + vt_a, nvtl, &bar);
        bulk_g2s(s_pv, P + bi.v0, npv, &bar);
        const BlockInfo *nb = next_block(A, w, nwork);
        if (nb) {
          const BlockInfo n = *nb;
          prefetch_l2(A.tri_g32 + n.t0, sizeof(TriGeo32) * n.nt);
          prefetch_l2(P + n.v0, sizeof(R4<R>) * n.nv);
          prefetch_l2(A.vt_rng + n.v0, sizeof(int2) * n.nv);
          prefetch_l2(A.vt_list + n.vt0, sizeof(uint16_t) * n.nvt);
          prefetch_l2(A.ais32 + n.v0, sizeof(float) * n.nv);
          prefetch_l2(A.halo_ids + n.h0, sizeof(int) * n.nh);
        }
      }
      const bool late = !mbar_wait_bounded(&bar, parity);
      parity ^= 1u;
      if (__syncthreads_or(late)) {
        if (threadIdx.x == 0) atomicCAS(&A.ctl[bi.mesh].err, 0, 6 /* FVM_ERR_TIMEOUT */);
        return;
      }
      // phase 1: one thread per triangle touching the block; its ends by
      // local slot: own vertices' states from shared memory, the halo's
      // from global memory
      auto state = [&](uint32_t l) {
        return l < (uint32_t)bi.nv ? s_pv[l] : P[s_halo[l - bi.nv]];
      };
      auto vertex = [&](uint32_t l) {
        return l < (uint32_t)bi.nv ? bi.v0 + (int)l : s_halo[l - bi.nv];
      };
      for (int k = threadIdx.x; k < bi.nt; k += blockDim.x) {
        const TriGeo32 tg = s_geo[k];
        constexpr uint32_t lm = (uint32_t)(kTriLocMax - 1);
        const uint32_t l1 = tg.loc & lm, l2 = (tg.loc >> kTriLocBits) & lm,
                       l3 = (tg.loc >> (2 * kTriLocBits)) & lm;
        const R4<R> p1 = state(l1), p2 = state(l2), p3 = state(l3);
        R dbxx[3], dbyy[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
          dbxx[j] = tg.dbxx[j];
          dbyy[j] = tg.dbyy[j];
        }
        TriSmem<R> ts;
        tri_sums<R>(p1, p2, p3, dbxx, dbyy, ts);
        if (visc) {
          const int4 t = make_int4(vertex(l1), vertex(l2), vertex(l3), 0);
          const TriVisc<R> tv = tri_visc<R>(A, mc, ctl.nphase, t, tg.areat, p1, p2, p3, dbxx, dbyy, ts);
          R *sv = s_vis + 9 * k;
#pragma unroll
          for (int j = 0; j < 3; j++) tri_visc_term<R>(tv, dbxx[j], dbyy[j], sv + 3 * j);
        }
        put_sums(s_tri, k, ts);   // over this thread's own geometry entry
      }
      __syncthreads();
      // phase 2: one thread per vertex, triangles in original order
      if (threadIdx.x < bi.nv) {
        const int v = bi.v0 + threadIdx.x;
        R qx[4], qy[4], rv[3];
        const int2 jr = s_vtr[threadIdx.x];
        // one triangle at a time: batched loads spill at 48 registers
        grad_vertex_sums<R, 1, true>(s_vtl, jr.x - vt_a, jr.y - vt_a, s_tri,
                                     visc ? s_vis : nullptr, qx, qy, rv);
        const R ais = v_ais(A, v);
        Grad<R> g;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          g.qx[q] = qx[q] * ais;
          g.qy[q] = qy[q] * ais;
        }
        A.grad[v] = g;
        if (visc) {
          R4<R> r;
          r.x = R(0);
          r.y = rv[0];
          r.z = rv[1];
          r.w = rv[2];
          A.resv[v] = r;
        } else if (do_dt) {
          A.dt[v] = time_step<R>(mc, s_pv[threadIdx.x], R(0), v_drmin(A, v));
        }
      }
      fence_proxy_async_smem();   // before the next block's copies land here
      __syncthreads();
    }
  }
}

// Gradient pass, vertex-stencil form (FP32, inviscid meshes): green_gauss.f
// (2-42) as precomputed per-vertex weights over the vertex's edges,
//   qx, qy (v) = sum over edges (v,u) of W(v,u) * (prim_u - prim_v),
// W formed on the host in FP64 from the triangles around the edge and
// rounded once (fvm_batch_prepare).  Equal to the triangle sums in exact
// arithmetic; in FP32 it rounds differently (and maps a uniform state to
// zero exactly).  One thread per vertex, no shared memory and no barrier;
// the weights and neighbour states of FVM_STENCIL_BATCH edges are in flight
// at once.  At stage 1 also time_step.f:22-27.
template <typename R>
__global__ void __launch_bounds__(kBlockVerts, FVM_STENCIL_MINB)
    k_grad_stencil(ArenaPtrs<R> A, int stage, int do_dt, int routine) {
  constexpr int B = FVM_STENCIL_BATCH;
  if constexpr (sizeof(R) == 4) {
    int w0, nwork;
    work_range(A, w0, nwork);
    for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
      const BlockInfo bi = work_block(A, w);
      const MeshCtl &ctl = A.ctl[bi.mesh];
      if (!routine && !ctl.active) continue;
      const MeshConst &mc = A.mc[bi.mesh];
      if (mc.iflow != 1 || threadIdx.x >= bi.nv) continue;
      const int v = bi.v0 + threadIdx.x;
      const R4<R> *P = A.st[cur_buf(ctl.phase, stage)];
      const R4<R> pv = P[v];
      const int2 r = A.va_rng[v];
      R qx[4] = {R(0), R(0), R(0), R(0)}, qy[4] = {R(0), R(0), R(0), R(0)};
#if FVM_STENCIL_PIPE
      // the next trip's neighbour ids are loaded while this trip's states
      // are in flight: one dependent load latency per trip instead of two
      int un[B];
#pragma unroll
      for (int k = 0; k < B; k++)
        un[k] = k < r.y - r.x ? (A.va_list[r.x + k] & 0x7fffffff) : v;
#endif
      for (int j = r.x; j < r.y; j += B) {
        const int n = r.y - j;
        int u[B];
        float2 wt[B];
#pragma unroll
        for (int k = 0; k < B; k++) {
#if FVM_STENCIL_PIPE
          u[k] = un[k];
#else
          u[k] = k < n ? (A.va_list[j + k] & 0x7fffffff) : v;
#endif
          wt[k] = k < n ? A.va_w[j + k] : make_float2(0.f, 0.f);
        }
        R4<R> pu[B];
#pragma unroll
        for (int k = 0; k < B; k++) pu[k] = k < n ? P[u[k]] : pv;
#if FVM_STENCIL_PIPE
#pragma unroll
        for (int k = 0; k < B; k++)
          un[k] = k < n - B ? (A.va_list[j + B + k] & 0x7fffffff) : v;
#endif
#pragma unroll
        for (int k = 0; k < B; k++) {
          if (k < n) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const R d = comp(pu[k], q) - comp(pv, q);
              qx[q] = fmaf(wt[k].x, d, qx[q]);
              qy[q] = fmaf(wt[k].y, d, qy[q]);
            }
          }
        }
      }
      Grad<R> g;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g.qx[q] = qx[q];
        g.qy[q] = qy[q];
      }
      A.grad[v] = g;
      if (do_dt) A.dt[v] = time_step<R>(mc, pv, R(0), v_drmin(A, v));
    }
  }
}

// Gradient pass, per-vertex form: each thread walks its vertex's triangles
// (ascending, as green_gauss.f visits them) and computes each triangle's
// terms itself, straight from the triangle entries; no shared memory and no
// barrier, at the price of computing every triangle once per vertex.  The
// arithmetic of each term is that of k_grad, so both give the same sums.
template <typename R>
__global__ void __launch_bounds__(kBlockVerts, sizeof(R) == 4 ? FVM_GRADV_MINB32 : 1)
    k_grad_v(ArenaPtrs<R> A, int stage, int do_dt, int routine, int skip_inviscid) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    const MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    if (skip_inviscid && mc.iflow == 1) continue;   // the stencil pass's meshes
    const bool visc = mc.iflow != 1;
    const R4<R> *P = A.st[cur_buf(ctl.phase, stage)];
    if (threadIdx.x == 0) {
      const BlockInfo *nb = next_block(A, w, nwork);
      if (nb) {
        const BlockInfo n = *nb;
        prefetch_l2(A.bt_nodes + n.t0, sizeof(int4) * n.nt);
        if (sizeof(R) == 4) prefetch_l2(A.tri_g32 + n.t0, sizeof(TriGeo32) * n.nt);
        prefetch_l2(P + n.v0, sizeof(R4<R>) * n.nv);
        if (sizeof(R) == 8) prefetch_l2(A.coord + n.v0, sizeof(double2) * n.nv);
        prefetch_l2(A.vt_rng + n.v0, sizeof(int2) * n.nv);
        prefetch_l2(sizeof(R) == 4 ? (const void *)(A.ais32 + n.v0) : (const void *)(A.ais + n.v0), sizeof(R) * n.nv);
      }
    }
    if (threadIdx.x >= bi.nv) continue;   // no barrier follows
    const int v = bi.v0 + threadIdx.x;
    R qx[4] = {R(0), R(0), R(0), R(0)}, qy[4] = {R(0), R(0), R(0), R(0)};
    R rv[3] = {R(0), R(0), R(0)};
    const int2 jr = A.vt_rng[v];
    for (int j = jr.x; j < jr.y; j++) {
      const uint16_t e = A.vt_list[j];
      const int entry = bi.t0 + (e & 0x3fff);
      const int4 t = A.bt_nodes[entry];
      const R4<R> p1 = P[t.x], p2 = P[t.y], p3 = P[t.z];
      R dbxx[3], dbyy[3];
      tri_geom<R>(A, t, entry, dbxx, dbyy);
      TriSmem<R> ts;
      tri_sums<R>(p1, p2, p3, dbxx, dbyy, ts);
      // plain (uncontracted) adds: each term is rounded before it is
      // summed, as when k_grad reads it back from shared memory
#pragma unroll
      for (int q = 0; q < 4; q++) {
        qx[q] = add_rn(qx[q], ts.dxt[q]);
        qy[q] = add_rn(qy[q], ts.dyt[q]);
      }
      if (visc) {
        const int pos = e >> kTriPosShift;
        const TriVisc<R> tv = tri_visc<R>(A, mc, ctl.nphase, t, tri_areat<R>(A, t, entry), p1, p2, p3, dbxx, dbyy, ts);
        R sv[3];
        tri_visc_term<R>(tv, pos == 0 ? dbxx[0] : pos == 1 ? dbxx[1] : dbxx[2],
                         pos == 0 ? dbyy[0] : pos == 1 ? dbyy[1] : dbyy[2], sv);
        rv[0] = add_rn(rv[0], sv[0]);
        rv[1] = add_rn(rv[1], sv[1]);
        rv[2] = add_rn(rv[2], sv[2]);
      }
    }
    const R ais = v_ais(A, v);
    Grad<R> g;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      g.qx[q] = qx[q] * ais;
      g.qy[q] = qy[q] * ais;
    }
    A.grad[v] = g;
    if (visc) {
      R4<R> r;
      r.x = R(0);
      r.y = rv[0];
      r.z = rv[1];
      r.w = rv[2];
      A.resv[v] = r;
    } else if (do_dt) {
      A.dt[v] = time_step<R>(mc, P[v], R(0), v_drmin(A, v));
    }
  }
}

// ---------------------------------------------------------------------------
// conres.f:14-22 partials of one block: sum of gra^2 and max |gra| (first
// driver index on ties), gra = rho_new - rho_old.  Called by every thread
// of the CTA (contains barriers).  FP64 states: FP64 arithmetic as before.
// FP32 states: gra is formed exactly as a pair of floats (TwoSum), its
// square as a pair (FMA residual), and the warp and block sums are pair
// sums, converted to FP64 once per leaf: by the block, or, where the leaf is
// split into several, by the monitor from their pairs (`split`).  The FP64
// pipe of this GPU is slow, and this keeps it out of the reduction: the sum
// carries ~2^-47 relative error instead of 2^-53; max |gra| is exact.
// ---------------------------------------------------------------------------
// The sums of a block's eight warps (32 consecutive vertices each) are added
// in pairs, and a mesh whose leaves of 256 vertices are split into smaller
// blocks adds those blocks' records in the same pairs and the same arithmetic
// (conres_share), so the norm does not depend on the split.
static_assert(kBlockVerts == 256, "eight warps");
__device__ __forceinline__ double warp_sums(const double *s) {
  return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}
struct DFloat {
  float hi, lo;
};
__device__ __forceinline__ DFloat two_sum(float a, float b) {   // a + b = hi + lo exactly
  const float s = __fadd_rn(a, b);
  const float z = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));
  return {s, e};
}
__device__ __forceinline__ DFloat df_add(DFloat x, DFloat y) {
  const DFloat s = two_sum(x.hi, y.hi);
  const float e = __fadd_rn(s.lo, __fadd_rn(x.lo, y.lo));
  const float hi = __fadd_rn(s.hi, e);
  return {hi, __fsub_rn(e, __fsub_rn(hi, s.hi))};
}
__device__ __forceinline__ bool df_greater(DFloat x, DFloat y) {   // normalized pairs
  return x.hi > y.hi || (x.hi == y.hi && x.lo > y.lo);
}

template <typename R>
__device__ __forceinline__ void block_conres_partial(bool have, R rho_new, R rho_old, int orig,
                                                     double *s_red, double *s_max, int *s_arg,
                                                     BlockPartial *out, bool split) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int darg = INT_MAX;
  if constexpr (sizeof(R) == 8) {
    double d2 = 0.0, dabs = 0.0;
    if (have) {
      const double gra = double(rho_new) - double(rho_old);
      d2 = gra * gra;
      dabs = fabs(gra);
      // conres.f:17-21 keeps a point only when |gra| > fresi, which a NaN
      // never is: a NaN poisons the sum of squares, not the maximum
      if (dabs > 0.0) darg = orig;
      else dabs = 0.0;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double o2 = __shfl_down_sync(0xffffffffu, d2, off);
      const double om = __shfl_down_sync(0xffffffffu, dabs, off);
      const int oa = __shfl_down_sync(0xffffffffu, darg, off);
      d2 += o2;
      if (om > dabs || (om == dabs && oa < darg)) {
        dabs = om;
        darg = oa;
      }
    }
    if (lane == 0) {
      s_red[wid] = d2;
      s_max[wid] = dabs;
      s_arg[wid] = darg;
    }
  } else {
    DFloat sq2 = {0.f, 0.f}, mx = {0.f, 0.f};
    if (have) {
      const DFloat g = two_sum(float(rho_new), -float(rho_old));
      const float h2 = __fmul_rn(g.hi, g.hi);
      const float l2 = __fadd_rn(__fmaf_rn(g.hi, g.hi, -h2), __fmul_rn(__fmul_rn(2.f, g.hi), g.lo));
      sq2 = two_sum(h2, l2);
      mx = g.hi >= 0.f ? g : DFloat{-g.hi, -g.lo};
      if (mx.hi > 0.f) darg = orig;
      else mx = DFloat{0.f, 0.f};   // NaN or no change (see the FP64 branch)
      // (TwoSum's low part of an infinite change is NaN; max_first needs a
      // number, and equal maxima compare equal only with equal low parts)
      if (mx.hi > FLT_MAX) mx.lo = 0.f;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const DFloat o2 = {__shfl_down_sync(0xffffffffu, sq2.hi, off),
                         __shfl_down_sync(0xffffffffu, sq2.lo, off)};
      const DFloat om = {__shfl_down_sync(0xffffffffu, mx.hi, off),
                         __shfl_down_sync(0xffffffffu, mx.lo, off)};
      const int oa = __shfl_down_sync(0xffffffffu, darg, off);
      sq2 = df_add(sq2, o2);
      if (df_greater(om, mx) || (om.hi == mx.hi && om.lo == mx.lo && oa < darg)) {
        mx = om;
        darg = oa;
      }
    }
    // warps' pairs summed by thread 0, still as pairs; one conversion to FP64
    __shared__ DFloat s_sq[kFluxThreads / 32], s_mx[kFluxThreads / 32];
    if (lane == 0) {
      s_sq[wid] = sq2;
      s_mx[wid] = mx;
      s_arg[wid] = darg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const DFloat t = df_add(df_add(df_add(s_sq[0], s_sq[1]), df_add(s_sq[2], s_sq[3])),
                              df_add(df_add(s_sq[4], s_sq[5]), df_add(s_sq[6], s_sq[7])));
      DFloat m = s_mx[0];
      int a = s_arg[0];
      for (int i = 1; i < kBlockVerts / 32; i++) {
        if (df_greater(s_mx[i], m) || (s_mx[i].hi == m.hi && s_mx[i].lo == m.lo && s_arg[i] < a)) {
          m = s_mx[i];
          a = s_arg[i];
        }
      }
      BlockPartial bp;
      bp.sumsq = split ? __hiloint2double(__float_as_int(t.hi), __float_as_int(t.lo))
                       : double(t.hi) + double(t.lo);
      bp.maxabs = double(m.hi) + double(m.lo);   // exact
      bp.argmax = a;
      bp.pad = 0;
      *out = bp;
    }
    return;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    int a = INT_MAX;
    for (int i = 0; i < kBlockVerts / 32; i++) {
      if (s_max[i] > m || (s_max[i] == m && s_arg[i] < a)) {
        m = s_max[i];
        a = s_arg[i];
      }
    }
    BlockPartial bp;
    bp.sumsq = warp_sums(s_red);
    bp.maxabs = m;
    bp.argmax = a;
    bp.pad = 0;
    *out = bp;
  }
}

// ---------------------------------------------------------------------------
// Flux pass: residu.f:37-88 (recon + roe/kfvs/hllc over iedge, solid_flux,
// farfield_flux) gathered per vertex in Fortran order, then either the
// residual is written (MODE_RESIDUAL) or the RK stage of update.f:17-35 is
// applied (MODE_UPDATE).  At stage 3 of an iteration it also produces the
// conres.f partials and the density/pressure positivity check.
// ---------------------------------------------------------------------------
// Mesh constants of the flux pass in the state precision, loaded once per
// block (keeps conversions out of the edge loop).
template <typename R>
struct FluxConst {
  R a11, a12, a21, a22, eps, gamma, gamma1, pi;
  int ilimit, iflux, rotate_back;
};

template <typename R>
__device__ __forceinline__ FluxConst<R> flux_const(const MeshConst &mc) {
  FluxConst<R> c;
  c.a11 = MCR(R, albada11);
  c.a12 = MCR(R, albada12);
  c.a21 = MCR(R, albada21);
  c.a22 = MCR(R, albada22);
  c.eps = MCR(R, epsilon);
  c.gamma = MCR(R, gamma);
  c.gamma1 = MCR(R, gamma1);
  c.pi = MCR(R, pi);
  c.ilimit = mc.ilimit;
  c.iflux = mc.iflux;
  c.rotate_back = mc.bugcompat ? 0 : 1;
  return c;
}

// The same constants when every resident mesh has math.f:8-40's values
// (fvm_params_init; the host checks): compile-time values, each the FP32
// rounding of the double the driver computes, so the edge loop keeps none
// of them in registers.
__device__ __forceinline__ FluxConst<float> flux_const_std(const MeshConst &mc) {
  FluxConst<float> c;
  c.a11 = (float)(2.0 / 3.0);
  c.a12 = (float)(1.0 - 2.0 / 3.0);
  c.a21 = (float)(4.0 / 3.0);
  c.a22 = (float)(1.0 - 4.0 / 3.0);
  c.eps = (float)1.0e-16;
  c.gamma = (float)1.4;
  c.gamma1 = (float)(1.4 - 1.0);
  c.pi = (float)3.141592653589793;
  c.ilimit = mc.ilimit;
  c.iflux = mc.iflux;
  c.rotate_back = mc.bugcompat ? 0 : 1;
  return c;
}

// Flux-pass template code: the Riemann solver (1/2/3; 0 dispatches on the
// mesh's iflux) plus kFluxStd when the FP32 constants are the standard ones.
constexpr int kFluxStd = 4;

// FP32: the edge's unit normal and length from its ds (flux.f:10-13) with
// one reciprocal square root.
__device__ __forceinline__ void edge_normal_f32(float dsx, float dsy, float &ct, float &st,
                                                float &len) {
  const float d2 = fmaf(dsx, dsx, dsy * dsy);
  const float il = rsqrtf(d2);
  ct = dsx * il;
  st = dsy * il;
  len = d2 * il;
}

// Two FP32 values in a 64-bit register pair: one instruction operates on both
// (each rounded as the scalar operation would).
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_get(F2 v, float &x, float &y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The van Albada limiter of limit_albada<float> for two variables: ur2 =
// ur^2 + 2 eps
__device__ __forceinline__ F2 limit_albada2(F2 ul, F2 ur, F2 ur2, F2 eps) {
  const F2 p = f2_mul(ul, ur);
  const F2 top = f2_mul(f2_add(ul, ur), f2_add(p, eps));
  const F2 bot = f2_fma(ul, ul, ur2);
  float p0, p1, b0, b1, t0, t1;
  f2_get(p, p0, p1);
  f2_get(bot, b0, b1);
  f2_get(top, t0, t1);
  t0 = __fdividef(t0, b0);
  t1 = __fdividef(t1, b1);
  return f2(p0 <= 0.0f ? 0.0f : t0, p1 <= 0.0f ? 0.0f : t1);
}

// FP32: recon.f:4-50 for the four variables of an edge, two at a time.  With
// the limiter, albada21 scales the edge vector once per edge instead of each
// projected gradient, and albada22 * dq serves both sides; the same values as
// recon1 up to FP32 rounding.  The pass is bound by issue and latency together
// (63% issue-active, 53% over a whole launch): pairs take a third off the
// reconstruction's instructions, 8 x 1024x384 0.1785 -> 0.1697 ms per launch
// alone.
__device__ __forceinline__ void recon_edge_f32(const R4<float> &p1, const R4<float> &p2,
                                               const Grad<float> &g1, const Grad<float> &g2,
                                               float dx, float dy, const FluxConst<float> &fc,
                                               float pl[4], float pr[4]) {
  if (fc.ilimit == 1) {
    const float dxa = fc.a21 * dx, dya = fc.a21 * dy;
    const F2 dx2 = f2(dxa, dxa), dy2 = f2(dya, dya), eps = f2(fc.eps, fc.eps);
    const F2 m1 = f2(-1.0f, -1.0f), a22 = f2(fc.a22, fc.a22);
    const F2 two_eps = f2(2.0f * fc.eps, 2.0f * fc.eps), hp = f2(0.5f, 0.5f), hm = f2(-0.5f, -0.5f);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const F2 a = h ? f2(p1.z, p1.w) : f2(p1.x, p1.y), b = h ? f2(p2.z, p2.w) : f2(p2.x, p2.y);
      const F2 dq = f2_fma(a, m1, b);
      const F2 c = f2_mul(a22, dq);
      const F2 dq2 = f2_fma(dq, dq, two_eps);
      const F2 ul = f2_fma(dx2, f2(g1.qx[2 * h], g1.qx[2 * h + 1]),
                           f2_fma(dy2, f2(g1.qy[2 * h], g1.qy[2 * h + 1]), c));
      const F2 ur = f2_fma(dx2, f2(g2.qx[2 * h], g2.qx[2 * h + 1]),
                           f2_fma(dy2, f2(g2.qy[2 * h], g2.qy[2 * h + 1]), c));
      f2_get(f2_fma(hp, limit_albada2(ul, dq, dq2, eps), a), pl[2 * h], pl[2 * h + 1]);
      f2_get(f2_fma(hm, limit_albada2(ur, dq, dq2, eps), b), pr[2 * h], pr[2 * h + 1]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++)
      recon1<float>(comp(p1, q), comp(p2, q), g1.qx[q], g1.qy[q], g2.qx[q], g2.qy[q], dx, dy,
                    fc.ilimit, fc.a11, fc.a12, fc.a21, fc.a22, fc.eps, pl[q], pr[q]);
  }
}

// FLUX = 1/2/3 compiles one Riemann solver only (every resident mesh uses
// it); FLUX = 0 dispatches on the mesh's iflux.
template <typename T, int FLUX>
__device__ __forceinline__ bool riemann(const FluxConst<T> &fc, T ct, T st, T len, const T pl[4],
                                        const T pr[4], T f[4]) {
  constexpr int FL = FLUX & 3;
  const int which = FL ? FL : fc.iflux;
  if (which == 1) return roe_flux<T>(ct, st, len, pl, pr, fc.gamma, fc.gamma1, f);
  if (which == 2) {
    kfvs_flux<T>(ct, st, len, pl, pr, fc.gamma1, fc.pi, f);
  } else {
    hllc_flux<T>(ct, st, len, pl, pr, fc.gamma, fc.gamma1, fc.rotate_back, f);
  }
  return true;
}

// FP32: the flux of edge entry e with ends nn (24 bytes per entry: the ends,
// edge vector and ds; ds/|ds| and |ds| are formed after the reconstruction).
// The records are read once a pass, by streaming loads that leave the caches to
// the states and gradients (5 x 394x151 HLLC in eight chains 0.0941 -> 0.0917
// ms per iteration, 8 x 1024x384 0.656 -> 0.645; the stencil's lists, whose
// lines neighbouring trips share, get slower with them: 0.080 -> 0.115).  The
// ends' load is not volatile: ordered against the others it changed which of
// the HLLC flux's products are contracted, and so its last bits.
__device__ __forceinline__ int2 load_ends(const int2 *p) {
  int2 r;
  asm("ld.global.cs.v2.s32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
  return r;
}
template <int FLUX>
__device__ __forceinline__ void edge_flux_f32(const ArenaPtrs<float> &A, const FluxConst<float> &fc,
                                              const R4<float> *P, int e, int2 nn, float f[4],
                                              int &err) {
  const float4 h = __ldcs(&A.be_g32[e].v);
  const R4<float> p1 = P[nn.x], p2 = P[nn.y];
  const Grad<float> g1 = A.grad[nn.x], g2 = A.grad[nn.y];
  float pl[4], pr[4], ct, st, len;
  recon_edge_f32(p1, p2, g1, g2, h.x, h.y, fc, pl, pr);
  edge_normal_f32(h.z, h.w, ct, st, len);
  if (!riemann<float, FLUX>(fc, ct, st, len, pl, pr, f)) err = 1;
}

// FP64: the flux of edge entries.  The reconstructed states go through shared
// memory (`face`: left rho, u, v, p, then right, then room for the Riemann
// solver's central flux, each a row of `stride`).
//
// A thread per edge (C = 0, 1), the four variables one after another (unrolled,
// the integer arithmetic made the pass wait for instructions a quarter of the
// time), or, for few edges (C = 2), four warps to 32 edges, each warp
// reconstructing one variable and the first solving the Riemann problems: a
// launch then lasts as long as one edge's chain of operations, which is a
// variable's and the solver's, and its code, with products on the FP64 pipe,
// a fifth as long.  160 x 48, Roe: 33 us a thread per edge, 34 us four warps with
// integer products (both fetch 93 KB of code), 21.5 us so.  Every form does the
// same operations on each value.
constexpr int kEdgeThreads = 128;
template <int C>
constexpr int kEdgeItem = C == 2 ? kEdgeThreads / 4 : kEdgeThreads;

template <int C>
__device__ __forceinline__ void edge_recon_f64(const ArenaPtrs<F64> &A, const MeshConst &mc,
                                               const R4<F64> *P, int2 nn, double dx, double dy,
                                               int q, double *face, int stride) {
  const double *s1 = reinterpret_cast<const double *>(P + nn.x);
  const double *s2 = reinterpret_cast<const double *>(P + nn.y);
  const double *g1 = reinterpret_cast<const double *>(A.grad + nn.x);
  const double *g2 = reinterpret_cast<const double *>(A.grad + nn.y);
  double pl, pr;
  recon1_f64<C>(s1[q], s2[q], g1[q], g1[4 + q], g2[q], g2[4 + q], dx, dy, mc.ilimit, mc.albada11,
                mc.albada12, mc.albada21, mc.albada22, mc.epsilon, pl, pr);
  face[q * stride] = pl;
  face[(4 + q) * stride] = pr;
}

template <int FLUX, int C>
__device__ __forceinline__ R4<F64> edge_riemann_f64(const ArenaPtrs<F64> &A, const MeshConst &mc,
                                                    const D4 &csl, double *face, int stride,
                                                    int &err) {
  using T = F64T<C>;
  const FluxConst<T> fc = flux_const<T>(mc);
  T f[4];
  bool ok;
  if constexpr (FLUX == 1) {
    ok = roe_flux_f64<C>(face, stride, csl.x, csl.y, csl.z, fc.gamma, fc.gamma1, f);
  } else if constexpr (FLUX == 3) {
    hllc_flux_f64<C>(face, stride, csl.x, csl.y, csl.z, fc.gamma, fc.gamma1, fc.rotate_back, f);
    ok = true;
  } else {
    T pl[4], pr[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      pl[q] = face[q * stride];
      pr[q] = face[(4 + q) * stride];
    }
    ok = riemann<T, FLUX>(fc, csl.x, csl.y, csl.z, pl, pr, f);
  }
  if (!ok) err = 1;
  R4<F64> o;
  o.x = f[0].v;
  o.y = f[1].v;
  o.z = f[2].v;
  o.w = f[3].v;
  return o;
}

// HLLC: the edges of a CTA whose star state is a two-rarefaction one (a
// minority, but in nearly every warp) put the bases of their four pow into
// shared memory, and all threads of the CTA take one each: pow is ~100
// operations of the FP64 pipe, which a branch would pass four times per warp
// (768 x 256, turbulent: 560 -> 390 us).
// Called by every thread of the CTA (barriers); `mine`: this thread has an edge.
template <int C>
__device__ __forceinline__ void edge_hllc_star(const MeshConst &mc, const D4 &csl, bool mine,
                                               double *face, int stride, double *s_pow,
                                               int *s_n) {
  using T = F64T<C>;
  const T gamma = mc.gamma;
  bool rare = false;
  if (mine) rare = hllc_star_f64<C>(face, stride, csl.x, csl.y, gamma);
  const uint32_t warp = __ballot_sync(0xffffffffu, rare);
  int k = 0;
  if (warp) {
    if ((threadIdx.x & 31) == 0) k = atomicAdd(s_n, __popc(warp));
    k = __shfl_sync(0xffffffffu, k, 0) + __popc(warp & ((1u << (threadIdx.x & 31)) - 1));
  }
  if (rare) {
    const T pl = face[3 * stride], pr = face[7 * stride];
    s_pow[3 * k] = pl.v;
    s_pow[3 * k + 1] = pr.v;
    s_pow[3 * k + 2] = (pl / pr).v;
  }
  const int n = __syncthreads_count(rare);
  if (n == 0) return;
  const T z = T(0.5) * (gamma - T(1.0)) / gamma;
#pragma unroll 1
  for (int t = threadIdx.x; t < 3 * n; t += kEdgeThreads) s_pow[t] = pow(s_pow[t], z.v);
  __syncthreads();
  // (the bases of p* in rows of their own: the next item's bases may be
  // written while the last threads still read these)
  double *s_star = s_pow + 3 * stride;
  if (threadIdx.x == 0) *s_n = 0;
  if (rare)
    s_star[k] = hllc_rare_f64<C>(face, stride, gamma, s_pow[3 * k], s_pow[3 * k + 1],
                                 s_pow[3 * k + 2]);
  __syncthreads();
  const T z1 = T(1.0) / z;
#pragma unroll 1
  for (int t = threadIdx.x; t < n; t += kEdgeThreads) s_star[t] = pow(s_star[t], z1.v);
  __syncthreads();
  if (rare) face[10 * stride] = s_star[k];
}

// One boundary edge: its contributions to n1 and n2.
template <typename R>
__device__ __forceinline__ void boundary_flux(const ArenaPtrs<R> &A, const MeshConst &mc,
                                              const MeshCtl &ctl, int4 b, const R4<R> *P,
                                              R4<R> &o1, R4<R> &o2) {
  const double2 x1 = A.coord[b.x], x2 = A.coord[b.y];
  const R4<R> p1 = P[b.x], p2 = P[b.y];
  if (b.z == 1) {
    // solid_flux.f:10-17
    const R sx = R(0.5) * R(x2.y - x1.y);
    const R sy = -R(0.5) * R(x2.x - x1.x);
    const R pp1 = R(0.75) * p1.w + R(0.25) * p2.w;
    const R pp2 = R(0.25) * p1.w + R(0.75) * p2.w;
    o1.x = R(0);
    o1.y = pp1 * sx;
    o1.z = pp1 * sy;
    o1.w = R(0);
    o2.x = R(0);
    o2.y = pp2 * sx;
    o2.z = pp2 * sy;
    o2.w = R(0);
  } else {
    R f1[4], f2[4];
    farfield_flux<R>(mc, ctl.cl, x1, x2, p1, p2, f1, f2);
    o1.x = f1[0];
    o1.y = f1[1];
    o1.z = f1[2];
    o1.w = f1[3];
    o2.x = f2[0];
    o2.y = f2[1];
    o2.z = f2[2];
    o2.w = f2[3];
  }
}

// FP64: component `row` of the two contributions of boundary entry b.
__device__ __forceinline__ void boundary_row(const ArenaPtrs<F64> &A, const MeshConst &mc,
                                             const MeshCtl &ctl, int b, const R4<F64> *P,
                                             int row) {
  const int4 n = A.bb_nodes[b];
  const double2 x1 = A.coord[n.x], x2 = A.coord[n.y];
  const R4<F64> p1 = P[n.x], p2 = P[n.y];
  double f1 = 0.0, f2 = 0.0;
  if (n.z == 1) {
    // solid_flux.f:10-17
    if (row == 1 || row == 2) {
      const double s = row == 1 ? 0.5 * (x2.y - x1.y) : -0.5 * (x2.x - x1.x);
      f1 = (0.75 * p1.w.v + 0.25 * p2.w.v) * s;
      f2 = (0.25 * p1.w.v + 0.75 * p2.w.v) * s;
    }
  } else {
    farfield_row(mc, ctl.cl, x1, x2, p1, p2, row, f1, f2);
  }
  reinterpret_cast<double *>(A.bflux + 2 * (size_t)b)[row] = f1;
  reinterpret_cast<double *>(A.bflux + 2 * (size_t)b + 1)[row] = f2;
}

// Phase 1b of the FP32 flux pass: boundary edges, two slots each
// (contribution to n1, to n2) after the block's ne interior slots.
template <typename R>
__device__ __forceinline__ void flux_boundary(const ArenaPtrs<R> &A, const MeshConst &mc,
                                              const MeshCtl &ctl, const BlockInfo &bi,
                                              const R4<R> *P, R4<R> *s_flux) {
  for (int k = threadIdx.x; k < bi.nb; k += blockDim.x) {
    R4<R> o1, o2;
    boundary_flux<R>(A, mc, ctl, A.bb_nodes[bi.b0 + k], P, o1, o2);
    s_flux[bi.ne + 2 * k] = o1;
    s_flux[bi.ne + 2 * k + 1] = o2;
  }
}

// Adds one incidence's flux to a vertex's residual.
__device__ __forceinline__ void add_flux(float acc[4], uint16_t e, const R4<float> &f) {
  if (e & kSolidBit) {
    acc[1] = acc[1] + f.y;
    acc[2] = acc[2] + f.z;
  } else if (e & kNegBit) {
    acc[0] = acc[0] - f.x;
    acc[1] = acc[1] - f.y;
    acc[2] = acc[2] - f.z;
    acc[3] = acc[3] - f.w;
  } else {
    acc[0] = acc[0] + f.x;
    acc[1] = acc[1] + f.y;
    acc[2] = acc[2] + f.z;
    acc[3] = acc[3] + f.w;
  }
}
// FP64: one addition per component whatever the sign (a warp whose lanes
// differ would pass the FP64 pipe once for each; gather of 1024 x 384: 103 ->
// 62 us together with the loads' batches): the sign bit is flipped first.  A solid edge's first and last component are +0, which changes no sum
// (sums start at +0 and so are never -0).
__device__ __forceinline__ F64 signed_by(F64 x, uint32_t sign) {
  return F64(__hiloint2double((int)((uint32_t)__double2hiint(x.v) ^ sign), __double2loint(x.v)));
}
__device__ __forceinline__ void add_flux(F64 acc[4], uint16_t e, const R4<F64> &f) {
  const uint32_t sign = (uint32_t)(e & kNegBit) << 16;
  acc[0] = acc[0] + signed_by(f.x, sign);
  acc[1] = acc[1] + signed_by(f.y, sign);
  acc[2] = acc[2] + signed_by(f.z, sign);
  acc[3] = acc[3] + signed_by(f.w, sign);
}

// Phase 2 of the flux pass: one thread per vertex sums its edge fluxes in
// Fortran order, then writes the residual (MODE_RESIDUAL) or applies the RK
// stage (MODE_UPDATE); at stage 3 the block's conres partial follows.
// FP32: the fluxes are the block's slots in shared memory (s_flux); FP64:
// the entries of the global buffers the edge pass filled.
template <typename R>
__device__ __forceinline__ void flux_gather(const ArenaPtrs<R> &A, const MeshConst &mc,
                                            MeshCtl &ctl, const BlockInfo &bi, const R4<R> *P,
                                            const R4<R> *s_flux, int p, int stage, int mode,
                                            int irk, int routine, double *s_red, double *s_max,
                                            int *s_arg) {
  bool have = false;
  R rho_new = R(0), rho_old = R(0);
  int org = 0;
  if (threadIdx.x < bi.nv) {
    const int v = bi.v0 + threadIdx.x;
    R acc[4];
    if (mc.iflow != 1) {
      const R4<R> rv = A.resv[v];
      acc[0] = R(0);
      acc[1] = rv.y;
      acc[2] = rv.z;
      acc[3] = rv.w;
    } else {
      acc[0] = acc[1] = acc[2] = acc[3] = R(0);
    }
    const int2 jr = A.ve_rng[v];
    // GB incidences' slots and fluxes loaded together, then added in list
    // order (FP64: the loads reach L2; two at four CTAs per SM hide their latency
    // best)
    constexpr int GB = sizeof(R) == 4 ? FVM_GATHER_BATCH : FVM_EGATHER_BATCH;
    for (int j = jr.x; j < jr.y; j += GB) {
      uint16_t es[GB];
      R4<R> fs[GB];
#pragma unroll
      for (int u = 0; u < GB; u++) es[u] = j + u < jr.y ? A.ve_list[j + u] : uint16_t(0);
      if constexpr (sizeof(R) == 4) {
#pragma unroll
        for (int u = 0; u < GB; u++)
          if (j + u < jr.y) fs[u] = s_flux[es[u] & kSlotMask];
      } else {
        int src[GB];
#pragma unroll
        for (int u = 0; u < GB; u++) src[u] = j + u < jr.y ? A.ve_src[j + u] : 0;
#pragma unroll
        for (int u = 0; u < GB; u++)
          if (j + u < jr.y) fs[u] = src[u] >= 0 ? A.eflux[src[u]] : A.bflux[-1 - src[u]];
      }
#pragma unroll
      for (int u = 0; u < GB; u++) {
        if (j + u >= jr.y) break;
        add_flux(acc, es[u], fs[u]);
      }
    }
    if (mode == MODE_RESIDUAL) {
      R4<R> r;
      r.x = acc[0];
      r.y = acc[1];
      r.z = acc[2];
      r.w = acc[3];
      A.res[v] = r;
    } else {
      const R4<R> po = A.st[old_buf(p, stage)][v];
      const R4<R> pc = P[v];
      const bool noslip = (mc.iflow != 1) && (A.vflag[v] & kVtxSolid);
      const R4<R> pn = rk_update<R>(mc, irk, po, pc, A.dt[v], v_cvarea(A, v), acc, noslip);
      A.st[out_buf(p, stage)][v] = pn;
      // iterate mode: stages 2 and 3 start from the viscosity computed here
      if (!routine && stage < 3 && mc.iflow != 1) next_viscosity<R>(A, mc, ctl, v, pn);
      if (stage == 3) {
        // conres.f:14-22 partials and check_positivity.f:13-14 (rho, p)
        have = true;
        rho_new = pn.x;
        rho_old = po.x;
        org = A.orig[v];
        if (pn.x <= R(0) || pn.w <= R(0)) atomicMin(&ctl.err_point, org);
      }
    }
  }
  if (mode == MODE_UPDATE && stage == 3)
    block_conres_partial<R>(have, rho_new, rho_old, org, s_red, s_max, s_arg, A.part + bi.part,
                            mc.sub > 1);
}

// FP64 flux pass, first kernel: the flux of every edge once, into eflux (the
// entry of the block owning it), and of every boundary edge into bflux.  The
// FP64 pipe bounds it: 2 lanes per SM and clock against ~430 operations per
// edge, so nothing may be computed twice and no SM may idle.  One work item
// is kEdgeItem<C> owned entries of a block (the last item of a block: its
// boundary edges), many items per SM.  One kernel over whole blocks computed
// cut edges in both blocks (+10%) and left most SMs idle in its last wave:
// 1365 us for 1024 x 384, Roe; 1000 us here on the FP64 pipe alone (446
// operations per edge at 526 Gop/s) and 149 us in the gather; 560 and 103 us
// with the products, quotients and roots on the integer pipes (F64).  Neither
// pipe was full then (FP64 57%, ALU 30%, issue 30%): the warps waited for
// instructions, of which one edge takes 5800 (93 KB).  C = 1 calls the
// operations instead of inlining them, and few live values (the reconstructed
// states and the central flux wait in shared memory) let seven CTAs share an
// SM: 442 us (FP64 77%, ALU 46%, issue 55%); the rule is in update_work.  HLLC
// on 768 x 256: 1064 -> 560 us, 390 us since its pow are shared out
// (edge_hllc_star).  Zeros lie outside the integer operations' window: where the
// flow is still uniform the differences take the hardware's, and the pass of
// the first iterations from freestream lasts 670 us (FP64 80%, issue 41%).
template <typename R, int FLUX, int C>
__global__ void __launch_bounds__(kEdgeThreads, C == 2   ? FVM_EFLUX_FEWB
                                                : C == 1 ? FVM_EFLUX_CALLB
                                                         : FVM_EFLUX_MINB)
    k_eflux(ArenaPtrs<R> A, int stage, int routine, int items) {
  static_assert(sizeof(R) == 8, "the FP64 pass");
  constexpr int stride = kEdgeItem<C>;
  // rows of face, and HLLC's bases and powers
  __shared__ double s_face[(FLUX == 3 ? 16 : FLUX == 1 ? 12 : 8) * stride];
  __shared__ int s_n;
  const int lane = threadIdx.x % stride;
  double *face = s_face + lane;
  if (FLUX == 3) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
  }
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int i = w0 * items + blockIdx.x; i < nwork * items; i += gridDim.x) {
    const BlockInfo &bi = work_block(A, i / items);
    const int c = i % items;
    MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    const R4<R> *P = A.st[cur_buf(ctl.phase, stage)];
    if (c == items - 1) {
      for (int k = threadIdx.x; k < 4 * bi.nb; k += kEdgeThreads)
        boundary_row(A, mc, ctl, bi.b0 + k / 4, P, k & 3);
      continue;
    }
    const int neo = A.blk_neo[bi.part];
    if (c * stride >= neo) continue;
    const bool have = c * stride + lane < neo;
    const int e = bi.e0 + c * stride + lane;
    int2 nn = make_int2(0, 0);
    double dx = 0.0, dy = 0.0;
    if (have) {
      nn = A.be_nodes[e];
      const double2 c1 = A.coord[nn.x], c2 = A.coord[nn.y];
      dx = c2.x - c1.x;
      dy = c2.y - c1.y;
    }
    bool mine = have;
    if constexpr (kEdgeItem<C> < kEdgeThreads) {
      __syncthreads();   // the CTA's last item has been read
      if (have) edge_recon_f64<C>(A, mc, P, nn, dx, dy, threadIdx.x / stride, face, stride);
      __syncthreads();
      mine = have && threadIdx.x < stride;
    } else if (have) {
#pragma unroll 1
      for (int q = 0; q < 4; q++) edge_recon_f64<C>(A, mc, P, nn, dx, dy, q, face, stride);
    }
    if (FLUX != 3 && !mine) continue;
    D4 csl;
    if (mine) csl = A.be_csl[e];
    if constexpr (FLUX == 3) {
      edge_hllc_star<C>(mc, csl, mine, face, stride, s_face + 12 * stride, &s_n);
      if (!mine) continue;
    }
    int err = 0;
    A.eflux[e] = edge_riemann_f64<FLUX, C>(A, mc, csl, face, stride, err);
    if (err) atomicCAS(&ctl.err, 0, 4 /* FVM_ERR_ROE_SONIC */);
  }
}

// FP64 flux pass, second kernel: gather per vertex and RK stage.
template <typename R>
__global__ void __launch_bounds__(kBlockVerts, FVM_EGATHER_MINB)
    k_egather(ArenaPtrs<R> A, int stage, int mode, int irk, int routine) {
  __shared__ double s_red[kBlockVerts / 32], s_max[kBlockVerts / 32];
  __shared__ int s_arg[kBlockVerts / 32];
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const int p = ctl.phase;
    flux_gather<R>(A, A.mc[bi.mesh], ctl, bi, A.st[cur_buf(p, stage)], nullptr, p, stage, mode,
                   irk, routine, s_red, s_max, s_arg);
    __syncthreads();   // s_red, s_max, s_arg are free again
  }
}

// FP32 flux pass: both phases in one kernel, the fluxes in shared memory.
template <typename R, int FLUX>
__global__ void __launch_bounds__(kFluxThreads, FVM_FLUX_MINB32)
    k_flux(ArenaPtrs<R> A, int stage, int mode, int irk, int routine) {
  static_assert(sizeof(R) == 4, "the FP32 pass");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R4<R> *s_flux = reinterpret_cast<R4<R> *>(smem_raw);
  __shared__ double s_red[kFluxThreads / 32];
  __shared__ double s_max[kFluxThreads / 32];
  __shared__ int s_arg[kFluxThreads / 32];
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    // (an L2 prefetch of the next block's inputs made the pass slower:
    // 0.206 -> 0.216 ms on 8 meshes of 1024 x 384 timed alone)
    const BlockInfo bi = work_block(A, w);
    MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    const int p = ctl.phase;
    const R4<R> *P = A.st[cur_buf(p, stage)];
    int err = 0;
    FluxConst<R> fc;
    if constexpr ((FLUX & kFluxStd) != 0) fc = flux_const_std(mc);
    else fc = flux_const<R>(mc);
    // phase 1a: interior edges; the next entry's ends are loaded while this
    // entry's states and gradients are in flight
#if FVM_FLUX_PIPE
    int2 nn_next = make_int2(0, 0);
    if (threadIdx.x < bi.ne) nn_next = load_ends(A.be_nodes + bi.e0 + threadIdx.x);
#endif
    for (int k = threadIdx.x; k < bi.ne; k += blockDim.x) {
      R f[4];
#if FVM_FLUX_PIPE
      const int2 nn = nn_next;
      if (k + (int)blockDim.x < bi.ne) nn_next = load_ends(A.be_nodes + bi.e0 + k + blockDim.x);
#else
      const int2 nn = A.be_nodes[bi.e0 + k];
#endif
      edge_flux_f32<FLUX>(A, fc, P, bi.e0 + k, nn, f, err);
      R4<R> o;
      o.x = f[0];
      o.y = f[1];
      o.z = f[2];
      o.w = f[3];
      s_flux[k] = o;
    }
    // phase 1b: boundary edges
    flux_boundary<R>(A, mc, ctl, bi, P, s_flux);
    if (err) atomicCAS(&ctl.err, 0, 4 /* FVM_ERR_ROE_SONIC */);
    __syncthreads();
    // phase 2: gather per vertex in Fortran order
    flux_gather<R>(A, mc, ctl, bi, P, s_flux, p, stage, mode, irk, routine, s_red, s_max, s_arg);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Fused stage: gradients, fluxes and the RK stage of one block in one pass
// (iterate mode).  Phase A computes dxt/dyt of every triangle touching the
// block or its halo (and the tri_visc terms of the block's own triangles);
// phase B sums them into the Green-Gauss gradients of the block's own and
// halo vertices, each in ascending triangle order exactly as the owner
// block would, so the halo gradients equal the owner's bit for bit; phase C
// computes the edge fluxes from those gradients; phase D gathers and
// updates.  Replaces k_grad + k_flux: the gradients never leave shared
// memory except the own ones, written for the stage-3 consumers (clcd, SA).
// ---------------------------------------------------------------------------
// Shared memory: region 1 = max(max_tri2 triangle records [+ viscous terms of
// max_tri], max_slots fluxes) (fluxes reuse the triangle area after phase B);
// region 2 = max_loc gradients.
template <typename R, int FLUX>
__global__ void __launch_bounds__(kBlockVerts, sizeof(R) == 4 ? FVM_FLUX_MINB32 : 2)
    k_step(ArenaPtrs<R> A, int stage, int max_tri, int max_tri2, int max_slots, int max_loc,
           int viscous) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const size_t tri_bytes = size_t(max_tri2) * sizeof(TriSmem<R>) + (viscous ? size_t(max_tri) * 9 * sizeof(R) : 0);
  const size_t flux_bytes = size_t(max_slots) * sizeof(R4<R>);
  const size_t r1 = ((tri_bytes > flux_bytes ? tri_bytes : flux_bytes) + 63) & ~size_t(63);
  TriSmem<R> *s_tri = reinterpret_cast<TriSmem<R> *>(smem_raw);
  R *s_vis = reinterpret_cast<R *>(s_tri + max_tri2);
  R4<R> *s_flux = reinterpret_cast<R4<R> *>(smem_raw);
  Grad<R> *s_grad = reinterpret_cast<Grad<R> *>(smem_raw + r1);
  __shared__ double s_red[kBlockVerts / 32];
  __shared__ double s_max[kBlockVerts / 32];
  __shared__ int s_arg[kBlockVerts / 32];
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    MeshCtl &ctl = A.ctl[bi.mesh];
    if (!ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    const bool visc = mc.iflow != 1;
    const int p = ctl.phase;
    const R4<R> *P = A.st[cur_buf(p, stage)];
    if (threadIdx.x == 0) {
      const BlockInfo *nb = next_block(A, w, nwork);
      if (nb) {
        const BlockInfo n = *nb;
        prefetch_l2(A.bt_nodes + n.t0, sizeof(int4) * n.nt2);
        if (sizeof(R) == 4) {
          prefetch_l2(A.tri_g32 + n.t0, sizeof(TriGeo32) * n.nt2);
          prefetch_l2(A.be_g32 + n.e0, sizeof(EdgeGeo32) * n.ne);
          prefetch_l2(A.be_nodes + n.e0, sizeof(int2) * n.ne);
        } else {
          prefetch_l2(A.coord + n.v0, sizeof(double2) * n.nv);
          prefetch_l2(A.be_csl + n.e0, sizeof(D4) * n.ne);
          prefetch_l2(A.be_nodes + n.e0, sizeof(int2) * n.ne);
          prefetch_l2(A.be_loc + n.e0, sizeof(uint32_t) * n.ne);
        }
        prefetch_l2(P + n.v0, sizeof(R4<R>) * n.nv);
        prefetch_l2(A.vt_rng + n.v0, sizeof(int2) * n.nv);
        prefetch_l2(A.ve_rng + n.v0, sizeof(int2) * n.nv);
        prefetch_l2(sizeof(R) == 4 ? (const void *)(A.ais32 + n.v0) : (const void *)(A.ais + n.v0), sizeof(R) * n.nv);
        prefetch_l2(A.st[old_buf(p, stage)] + n.v0, sizeof(R4<R>) * n.nv);
        prefetch_l2(sizeof(R) == 4 ? (const void *)(A.cvarea32 + n.v0) : (const void *)(A.cvarea + n.v0), sizeof(R) * n.nv);
      }
    }
    // phase A: triangles of the block and of its halo
    for (int k = threadIdx.x; k < bi.nt2; k += blockDim.x) {
      const int4 t = A.bt_nodes[bi.t0 + k];
      const R4<R> p1 = P[t.x], p2 = P[t.y], p3 = P[t.z];
      R dbxx[3], dbyy[3];
      tri_geom<R>(A, t, bi.t0 + k, dbxx, dbyy);
      TriSmem<R> ts;
      tri_sums<R>(p1, p2, p3, dbxx, dbyy, ts);
      s_tri[k] = ts;
      if (visc && k < bi.nt) {
        const TriVisc<R> tv = tri_visc<R>(A, mc, ctl.nphase, t, tri_areat<R>(A, t, bi.t0 + k), p1, p2, p3, dbxx, dbyy, ts);
        R *sv = s_vis + 9 * k;
#pragma unroll
        for (int j = 0; j < 3; j++) tri_visc_term<R>(tv, dbxx[j], dbyy[j], sv + 3 * j);
      }
    }
    __syncthreads();
    // phase B: gradients of own vertices (thread t = own vertex t, which
    // keeps its viscous residual part and time step in registers) and of
    // the halo vertices
    R rv[3] = {R(0), R(0), R(0)};
    R dtv = R(0);
    const int t = threadIdx.x;
    if (t < bi.nv) {
      const int v = bi.v0 + t;
      R qx[4] = {R(0), R(0), R(0), R(0)}, qy[4] = {R(0), R(0), R(0), R(0)};
      const int2 jr = A.vt_rng[v];
      for (int j = jr.x; j < jr.y; j++) {
        const uint16_t e = A.vt_list[j];
        const int slot = e & 0x3fff;
        const TriSmem<R> ts = s_tri[slot];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          qx[q] = qx[q] + ts.dxt[q];
          qy[q] = qy[q] + ts.dyt[q];
        }
        if (visc) {
          const R *sv = s_vis + 9 * slot + 3 * (e >> kTriPosShift);
          rv[0] = rv[0] + sv[0];
          rv[1] = rv[1] + sv[1];
          rv[2] = rv[2] + sv[2];
        }
      }
      const R ais = v_ais(A, v);
      Grad<R> g;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g.qx[q] = qx[q] * ais;
        g.qy[q] = qy[q] * ais;
      }
      s_grad[t] = g;
      A.grad[v] = g;
      if (visc) dtv = A.dt[v];
      else if (stage == 1) {
        dtv = time_step<R>(mc, P[v], R(0), v_drmin(A, v));
        A.dt[v] = dtv;
      } else {
        dtv = A.dt[v];
      }
    }
    for (int h = t; h < bi.nh; h += blockDim.x) {
      const int g0 = A.hl_ptr[bi.hp0 + h], g1 = A.hl_ptr[bi.hp0 + h + 1];
      R qx[4] = {R(0), R(0), R(0), R(0)}, qy[4] = {R(0), R(0), R(0), R(0)};
      for (int j = g0; j < g1; j++) {
        const TriSmem<R> ts = s_tri[A.hl_list[j] & 0x3fff];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          qx[q] = qx[q] + ts.dxt[q];
          qy[q] = qy[q] + ts.dyt[q];
        }
      }
      const R ais = v_ais(A, A.halo_ids[bi.h0 + h]);
      Grad<R> g;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g.qx[q] = qx[q] * ais;
        g.qy[q] = qy[q] * ais;
      }
      s_grad[bi.nv + h] = g;
    }
    __syncthreads();
    // phase C: interior edge fluxes from the shared gradients
    int err = 0;
    const FluxConst<R> fc = flux_const<R>(mc);
    for (int k = threadIdx.x; k < bi.ne; k += blockDim.x) {
      const int e = bi.e0 + k;
      int2 nn;
      uint32_t ll;
      R dx, dy, ct, st, len;
      if constexpr (sizeof(R) == 4) {
        const float4 g = A.be_g32[e].v;
        nn = A.be_nodes[e];
        ll = A.be_loc[e];
        dx = g.x;
        dy = g.y;
        edge_normal_f32(g.z, g.w, ct, st, len);
      } else {
        nn = A.be_nodes[e];
        ll = A.be_loc[e];
        const double2 c1 = A.coord[nn.x], c2 = A.coord[nn.y];
        dx = c2.x - c1.x;
        dy = c2.y - c1.y;
        const D4 csl = A.be_csl[e];
        ct = R(csl.x);
        st = R(csl.y);
        len = R(csl.z);
      }
      const R4<R> p1 = P[nn.x], p2 = P[nn.y];
      const Grad<R> g1 = s_grad[ll & 0xffff], g2 = s_grad[ll >> 16];
      R pl[4], pr[4];
#pragma unroll
      for (int q = 0; q < 4; q++)
        recon1<R>(comp(p1, q), comp(p2, q), g1.qx[q], g1.qy[q], g2.qx[q], g2.qy[q], dx, dy,
                  fc.ilimit, fc.a11, fc.a12, fc.a21, fc.a22, fc.eps, pl[q], pr[q]);
      R f[4];
      if (!riemann<R, FLUX>(fc, ct, st, len, pl, pr, f)) err = 1;
      R4<R> o;
      o.x = f[0];
      o.y = f[1];
      o.z = f[2];
      o.w = f[3];
      s_flux[k] = o;
    }
    // boundary edges, two slots each (contribution to n1, to n2)
    for (int k = threadIdx.x; k < bi.nb; k += blockDim.x) {
      const int4 b = A.bb_nodes[bi.b0 + k];
      const double2 x1 = A.coord[b.x], x2 = A.coord[b.y];
      const R4<R> p1 = P[b.x], p2 = P[b.y];
      R4<R> o1, o2;
      if (b.z == 1) {
        // solid_flux.f:10-17
        const R sx = R(0.5) * R(x2.y - x1.y);
        const R sy = -R(0.5) * R(x2.x - x1.x);
        const R pp1 = R(0.75) * p1.w + R(0.25) * p2.w;
        const R pp2 = R(0.25) * p1.w + R(0.75) * p2.w;
        o1.x = R(0);
        o1.y = pp1 * sx;
        o1.z = pp1 * sy;
        o1.w = R(0);
        o2.x = R(0);
        o2.y = pp2 * sx;
        o2.z = pp2 * sy;
        o2.w = R(0);
      } else {
        R f1[4], f2[4];
        farfield_flux<R>(mc, ctl.cl, x1, x2, p1, p2, f1, f2);
        o1.x = f1[0];
        o1.y = f1[1];
        o1.z = f1[2];
        o1.w = f1[3];
        o2.x = f2[0];
        o2.y = f2[1];
        o2.z = f2[2];
        o2.w = f2[3];
      }
      s_flux[bi.ne + 2 * k] = o1;
      s_flux[bi.ne + 2 * k + 1] = o2;
    }
    if (err) atomicCAS(&ctl.err, 0, 4 /* FVM_ERR_ROE_SONIC */);
    __syncthreads();
    // phase D: gather per own vertex in Fortran order, RK stage
    bool have = false;
    R rho_new = R(0), rho_old = R(0);
    int org = 0;
    if (t < bi.nv) {
      const int v = bi.v0 + t;
      R acc[4];
      acc[0] = R(0);
      acc[1] = rv[0];
      acc[2] = rv[1];
      acc[3] = rv[2];
      const int2 jr = A.ve_rng[v];
      for (int j = jr.x; j < jr.y; j++) {
        const uint16_t e = A.ve_list[j];
        const R4<R> f = s_flux[e & kSlotMask];
        if (e & kSolidBit) {
          acc[1] = acc[1] + f.y;
          acc[2] = acc[2] + f.z;
        } else if (e & kNegBit) {
          acc[0] = acc[0] - f.x;
          acc[1] = acc[1] - f.y;
          acc[2] = acc[2] - f.z;
          acc[3] = acc[3] - f.w;
        } else {
          acc[0] = acc[0] + f.x;
          acc[1] = acc[1] + f.y;
          acc[2] = acc[2] + f.z;
          acc[3] = acc[3] + f.w;
        }
      }
      const R4<R> po = A.st[old_buf(p, stage)][v];
      const R4<R> pc = P[v];
      const bool noslip = visc && (A.vflag[v] & kVtxSolid);
      const R4<R> pn = rk_update<R>(mc, stage, po, pc, dtv, v_cvarea(A, v), acc, noslip);
      A.st[out_buf(p, stage)][v] = pn;
      if (stage == 3) {
        have = true;
        rho_new = pn.x;
        rho_old = po.x;
        org = A.orig[v];
        if (pn.x <= R(0) || pn.w <= R(0)) atomicMin(&ctl.err_point, org);
      }
    }
    if (stage == 3)
      block_conres_partial<R>(have, rho_new, rho_old, org, s_red, s_max, s_arg, A.part + bi.part,
                              mc.sub > 1);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Spalart-Allmaras step (sa_model.f:3-201): viscous_sa over triangles,
// divergence_sa over iedge, outer_flux_sa over farfield edges, then
// update_sa; nu~ is zero at solid points.  Reads nut[nphase], writes
// nut[1-nphase].  Uses the state buffer that holds the new solution.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_sa(ArenaPtrs<R> A, int stage, int routine,
                                                    int max_tri) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R *s_t = reinterpret_cast<R *>(smem_raw);   // [max_tri][3]
  R *s_e = s_t + 3 * max_tri;                  // [slots]
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    MeshCtl &ctl = A.ctl[bi.mesh];
    if (!routine && !ctl.active) continue;
    const MeshConst &mc = A.mc[bi.mesh];
    if (mc.iflow != 3) continue;
    // the solution after the RK stages: out of stage 3, or the state itself
    const int p = ctl.phase;
    const R4<R> *P = A.st[stage == 3 ? out_buf(p, 3) : p];
    const R *nut = A.nut[ctl.nphase];
    R *nut_new = A.nut[1 - ctl.nphase];
    for (int k = threadIdx.x; k < bi.nt; k += blockDim.x) {
      const int4 t = A.bt_nodes[bi.t0 + k];
      R areat, dbxx[3], dbyy[3];
      if constexpr (sizeof(R) == 4) {   // FP32 copies rounded once
        const TriGeo32 tg = A.tri_g32[bi.t0 + k];
        areat = tg.areat;
        for (int j = 0; j < 3; j++) {
          dbxx[j] = tg.dbxx[j];
          dbyy[j] = tg.dbyy[j];
        }
      } else {
        const double2 c1 = A.coord[t.x], c2 = A.coord[t.y], c3 = A.coord[t.z];
        areat = A.areat[t.w];
        dbxx[0] = R(c2.y - c3.y);
        dbxx[1] = R(c3.y - c1.y);
        dbxx[2] = R(c1.y - c2.y);
        dbyy[0] = R(c3.x - c2.x);
        dbyy[1] = R(c1.x - c3.x);
        dbyy[2] = R(c2.x - c1.x);
      }
      int a1 = t.x, a2 = t.y, a3 = t.z;
      if (mc.bugcompat) {
        a1 = mc.orig123[0];
        a2 = mc.orig123[1];
        a3 = mc.orig123[2];
      }
      const R nux = nut[a1] * dbxx[0] + nut[a2] * dbxx[1] + nut[a3] * dbxx[2];
      const R nuy = nut[a1] * dbyy[0] + nut[a2] * dbyy[1] + nut[a3] * dbyy[2];
      const R mul1 = A.mul[t.x], mul2 = A.mul[t.y], mul3 = A.mul[t.z];
      const R n1 = nut[t.x], n2 = nut[t.y], n3 = nut[t.z];
      const R r1 = P[t.x].x, r2 = P[t.y].x, r3 = P[t.z].x;
      const R mult = mdiv(mul1 + mul2 + mul3, R(3));
      const R prim5t = mdiv(n1 + n2 + n3, R(3));
      const R rhot = mdiv(r1 + r2 + r3, R(3));
      const R mutb = mdiv(mult, rhot) + prim5t;
      const R cs1 = MCR(R, cb2sig1), cs2 = MCR(R, cb2sig2);
      s_t[3 * k + 0] = (cs1 * mutb - cs2 * (mdiv(mul1, r1) + n1)) * (nux * dbxx[0] + nuy * dbyy[0]) * areat;
      s_t[3 * k + 1] = (cs1 * mutb - cs2 * (mdiv(mul2, r2) + n2)) * (nux * dbxx[1] + nuy * dbyy[1]) * areat;
      s_t[3 * k + 2] = (cs1 * mutb - cs2 * (mdiv(mul3, r3) + n3)) * (nux * dbxx[2] + nuy * dbyy[2]) * areat;
    }
    for (int k = threadIdx.x; k < bi.ne; k += blockDim.x) {
      const int e = bi.e0 + k;
      int2 nn;
      R d1, d2;
      if constexpr (sizeof(R) == 4) {   // ds from the FP32 record
        const float4 g = A.be_g32[e].v;
        nn = A.be_nodes[e];
        d1 = g.z;
        d2 = g.w;
      } else {
        nn = A.be_nodes[e];
        const double2 ds = A.be_ds[e];
        d1 = R(ds.x);
        d2 = R(ds.y);
      }
      const R4<R> p1 = P[nn.x], p2 = P[nn.y];
      const R unl = p1.y * d1 + p1.z * d2;
      const R unr = p2.y * d1 + p2.z * d2;
      const R una = R(0.5) * (unl + unr);
      s_e[k] = (una > R(0)) ? una * nut[nn.x] : una * nut[nn.y];
    }
    for (int k = threadIdx.x; k < bi.nb; k += blockDim.x) {
      const int4 b = A.bb_nodes[bi.b0 + k];
      R f1 = R(0), f2 = R(0);
      if (b.z == 2) {
        const double2 x1 = A.coord[b.x], x2 = A.coord[b.y];
        const R dx = R(x2.x - x1.x), dy = R(x2.y - x1.y);
        const R sx = dy, sy = -dx;
        const R4<R> p1 = P[b.x], p2 = P[b.y];
        const R u = R(0.5) * (p1.y + p2.y);
        const R vv = R(0.5) * (p1.z + p2.z);
        const R un = u * sx + vv * sy;
        if (un > R(0)) {
          f1 = un * nut[b.x];
          f2 = un * nut[b.y];
        } else {
          f1 = un * MCR(R, nut_inf);
          f2 = un * MCR(R, nut_inf);
        }
        f1 = R(0.5) * f1;
        f2 = R(0.5) * f2;
      }
      s_e[bi.ne + 2 * k] = f1;
      s_e[bi.ne + 2 * k + 1] = f2;
    }
    __syncthreads();
    if (threadIdx.x < bi.nv) {
      const int v = bi.v0 + threadIdx.x;
      R divf = R(0);
      const int2 tr = A.vt_rng[v];
      for (int j = tr.x; j < tr.y; j++) {
        const uint16_t e = A.vt_list[j];
        divf = divf + s_t[3 * (e & 0x3fff) + (e >> kTriPosShift)];
      }
      const int2 er = A.ve_rng[v];
      for (int j = er.x; j < er.y; j++) {
        const uint16_t e = A.ve_list[j];
        if (e & kSolidBit) continue;
        const R f = s_e[e & kSlotMask];
        divf = (e & kNegBit) ? divf - f : divf + f;
      }
      R nn;
      if (A.vflag[v] & kVtxSolid) {
        nn = R(0);
      } else {
        const Grad<R> g = A.grad[v];
        const R omega = g.qy[1] - g.qx[2];
        nn = update_sa<R>(mc, nut[v], P[v].x, A.mul[v], v_wd(A, v), A.dt[v], v_cvarea(A, v), divf,
                          omega);
      }
      nut_new[v] = nn;
      if (nn < R(0)) atomicMin(&ctl.err_point, A.orig[v]);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// End-of-iteration monitor, one CTA per mesh: conres.f (from the block
// partials), clcd.f, the positivity verdict, RES.DAT history row and the
// stop test of main.f:42.  FP64 arithmetic; with FP64 states the clcd sum is
// the serial Fortran chain.
// ---------------------------------------------------------------------------
// FP32 states: one solid edge's pressure and viscous force (clcd.f:20-40),
// the terms from the FP32 values (sv: the edge's normal, FP64 differences
// rounded once), accumulated in FP64.
__device__ __forceinline__ void wall_force(float2 sv, float mu1, float mu2,
                                           const Grad<float> &g1, const Grad<float> &g2, float p1,
                                           float p2, double &xf, double &yf) {
  const float sx = sv.x, sy = sv.y;
  const float n2b3 = 2.0f / 3.0f;
  const float txx = 0.5f * (n2b3 * mu1 * (2.0f * g1.qx[1] - g1.qy[2]) +
                            n2b3 * mu2 * (2.0f * g2.qx[1] - g2.qy[2]));
  const float txy = 0.5f * (mu1 * (g1.qy[1] + g1.qx[2]) + mu2 * (g2.qy[1] + g2.qx[2]));
  const float tyy = 0.5f * (n2b3 * mu1 * (2.0f * g1.qy[2] - g1.qx[1]) +
                            n2b3 * mu2 * (2.0f * g2.qy[2] - g2.qx[1]));
  const float pp = 0.5f * (p1 + p2);
  xf += double(pp * sx - txx * sx - txy * sy);
  yf += double(pp * sy - txy * sx - tyy * sy);
}

// FP64, the Fortran chain: clcd.f:34-40 adds three terms per solid edge, one
// after another, so the additions are serial; nothing else is.  All threads
// form the terms of a tile of edges in shared memory, then one thread per
// component adds them in edge order while the other warps sum the residual
// and form the next tile.  Each addition costs one pass through the FP64 pipe (about 32 ns on
// this GPU, 2 lanes per SM quarter-cycle), which bounds the chain: with the
// loads and products of every edge inside it the chain took 1.45 ms for 1024
// edges, k_monitor 1480 us; now 49 us.  mu = 0 (inviscid meshes)
// makes both viscous terms zero; subtracting zero changes no sum (it never is
// -0: it starts at +0), so a tile whose viscous terms all are zero adds the
// pressure terms alone.  NaN terms count as nonzero.
constexpr int kForceTile = 256;
struct ForceTile {
  double t[3][2][kForceTile];   // pressure, then the two viscous terms: x, y
};

template <typename R>
__device__ __forceinline__ bool force_terms(const ArenaPtrs<R> &A, const R4<R> *P, int2 nn, int k,
                                            ForceTile &s) {
  const double2 c1 = A.coord[nn.x], c2 = A.coord[nn.y];
  const double dx = c2.x - c1.x, dy = c2.y - c1.y;
  const double sx = dy, sy = -dx;
  const double mu1 = double(A.mu[nn.x]), mu2 = double(A.mu[nn.y]);
  const Grad<R> g1 = A.grad[nn.x], g2 = A.grad[nn.y];
  const double p1 = double(P[nn.x].w), p2 = double(P[nn.y].w);
  const double txx1 = 2.0 / 3.0 * mu1 * (2.0 * double(g1.qx[1]) - double(g1.qy[2]));
  const double txy1 = mu1 * (double(g1.qy[1]) + double(g1.qx[2]));
  const double tyy1 = 2.0 / 3.0 * mu1 * (2.0 * double(g1.qy[2]) - double(g1.qx[1]));
  const double txx2 = 2.0 / 3.0 * mu2 * (2.0 * double(g2.qx[1]) - double(g2.qy[2]));
  const double txy2 = mu2 * (double(g2.qy[1]) + double(g2.qx[2]));
  const double tyy2 = 2.0 / 3.0 * mu2 * (2.0 * double(g2.qy[2]) - double(g2.qx[1]));
  const double pp = 0.5 * (p1 + p2);
  const double txx = 0.5 * (txx1 + txx2);
  const double txy = 0.5 * (txy1 + txy2);
  const double tyy = 0.5 * (tyy1 + tyy2);
  const double bx = txx * sx, cx = txy * sy, by = txy * sx, cy = tyy * sy;
  s.t[0][0][k] = pp * sx;
  s.t[0][1][k] = pp * sy;
  s.t[1][0][k] = bx;
  s.t[1][1][k] = by;
  s.t[2][0][k] = cx;
  s.t[2][1][k] = cy;
  return bx != 0.0 || cx != 0.0 || by != 0.0 || cy != 0.0;
}

// Adds a tile's terms to v in edge order; `viscous`: all three of an edge.
__device__ __forceinline__ double force_chain(const ForceTile &s, int comp, int n, bool viscous,
                                              double v) {
  const double *a = s.t[0][comp], *b = s.t[1][comp], *c = s.t[2][comp];
  if (viscous) {
#pragma unroll 4
    for (int k = 0; k < n; k++) v = ((v + a[k]) - b[k]) - c[k];
  } else {
#pragma unroll 8
    for (int k = 0; k < n; k++) v = v + a[k];
  }
  return v;
}

// What the monitor reduces over a mesh: the sum of gra^2 and the largest |gra|
// with its first driver index (conres.f:14-22), and the force on the wall.
struct Moments {
  double s, x, y, m;
  int a;
};

// (m, a) with a larger maximum or, at the same one, a smaller index; m >= 0 and
// never NaN, so the bits order like the values (no FP64 comparison)
__device__ __forceinline__ void max_first(double &m, int &a, double om, int oa) {
  const long long x = __double_as_longlong(m), y = __double_as_longlong(om);
  if (y > x || (y == x && oa < a)) {
    m = om;
    a = oa;
  }
}
template <int N>
__device__ __forceinline__ void reduce_residual(Moments &v) {
#pragma unroll
  for (int off = N / 2; off > 0; off >>= 1) {
    v.s += __shfl_xor_sync(0xffffffffu, v.s, off);
    max_first(v.m, v.a, __shfl_xor_sync(0xffffffffu, v.m, off),
              __shfl_xor_sync(0xffffffffu, v.a, off));
  }
}
template <int N>
__device__ __forceinline__ void reduce_force(Moments &v) {
#pragma unroll
  for (int off = N / 2; off > 0; off >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
  }
}

// A thread's share of a mesh's conres partials: thread t of n.  The partials
// are contiguous (block k's record is blk0 + k); eight loads in flight per
// thread (a 2048-block mesh in one trip): the records of 8 / sub leaves, each
// leaf's `sub` records added in pairs and the leaves in order.  PAIRS: the
// records of split leaves hold float pairs (block_conres_partial of FP32 states),
// added as a block of the whole leaf adds its warps.
__device__ __forceinline__ DFloat pair_of(const BlockPartial &p) {
  return {__int_as_float(__double2hiint(p.sumsq)), __int_as_float(__double2loint(p.sumsq))};
}
template <bool PAIRS>
__device__ __forceinline__ double leaf_sum2(const BlockPartial *p) {
  if constexpr (!PAIRS) return p[0].sumsq + p[1].sumsq;
  const DFloat t = df_add(pair_of(p[0]), pair_of(p[1]));
  return double(t.hi) + double(t.lo);
}
template <bool PAIRS>
__device__ __forceinline__ double leaf_sum4(const BlockPartial *p) {
  if constexpr (!PAIRS) return (p[0].sumsq + p[1].sumsq) + (p[2].sumsq + p[3].sumsq);
  const DFloat t = df_add(df_add(pair_of(p[0]), pair_of(p[1])),
                          df_add(pair_of(p[2]), pair_of(p[3])));
  return double(t.hi) + double(t.lo);
}
template <typename R, bool PAIRS>
__device__ __forceinline__ void conres_share(const ArenaPtrs<R> &A, const MeshConst &mc, int t,
                                             int n, Moments &v) {
  constexpr int kU = 8;
  const int sub = mc.sub, nleaf = (mc.nblk + sub - 1) / sub;
  for (int i0 = t; i0 < nleaf; i0 += kU / sub * n) {
    BlockPartial bp[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int leaf = i0 + u / sub * n, i = leaf * sub + u % sub;
      if (leaf < nleaf && i < mc.nblk) bp[u] = A.part[mc.blk0 + i];
      else bp[u] = BlockPartial{0.0, 0.0, INT_MAX, 0};
    }
    if (sub == 4) {
      v.s += leaf_sum4<PAIRS>(bp);
      if (i0 + n < nleaf) v.s += leaf_sum4<PAIRS>(bp + 4);
    } else if (sub == 2) {
#pragma unroll
      for (int u = 0; u < kU; u += 2)
        if (i0 + u / 2 * n < nleaf) v.s += leaf_sum2<PAIRS>(bp + u);
    } else {
#pragma unroll
      for (int u = 0; u < kU; u++)
        if (i0 + u * n < nleaf) v.s += bp[u].sumsq;
    }
#pragma unroll
    for (int u = 0; u < kU; u++) max_first(v.m, v.a, bp[u].maxabs, bp[u].argmax);
  }
}

// FP32 states: a thread's share of the wall edges, i, i + n, ... summed in
// that order, with the loads of four edges issued together per trip.
__device__ __forceinline__ void force_share(const ArenaPtrs<float> &A, const MeshConst &mc,
                                            const R4<float> *P, int t, int n, Moments &v) {
  constexpr int kU = 4;
  for (int i0 = t; i0 < mc.nsw; i0 += kU * n) {
    int2 nn[kU];
    float2 sv[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const bool in = i0 + u * n < mc.nsw;
      nn[u] = in ? A.sw_nodes[mc.sw0 + i0 + u * n] : make_int2(mc.v0, mc.v0);
      sv[u] = in ? A.sw_vec[mc.sw0 + i0 + u * n] : make_float2(0.f, 0.f);
    }
    float mu1[kU], mu2[kU], p1[kU], p2[kU];
    Grad<float> g1[kU], g2[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      mu1[u] = A.mu[nn[u].x];
      mu2[u] = A.mu[nn[u].y];
      g1[u] = A.grad[nn[u].x];
      g2[u] = A.grad[nn[u].y];
      p1[u] = P[nn[u].x].w;
      p2[u] = P[nn[u].y].w;
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      if (i0 + u * n >= mc.nsw) break;
      wall_force(sv[u], mu1[u], mu2[u], g1[u], g2[u], p1[u], p2[u], v.x, v.y);
    }
  }
}

// The monitor's reduction, by all kMonitorMaxThreads threads (`what`: 1 the
// residual, 2 the force, 3 both; PAIRS: see conres_share).  Warp 0 returns the
// residual's part and warps 1 and 2 the force.  One CTA does this between two iterations, so its
// latency counts and an FP64 operation of a warp costs 64 cycles: comparisons
// read the bits, each reduction is five shuffles and one exchange, and the
// final scalars are formed by different warps.  8 x 1024x384, alone, 22.4 us
// as two 8-level shared-memory trees with one thread finishing; now 16.3 us (160 x 48: 9.6, now 5.2).
template <typename R, bool PAIRS>
__device__ __forceinline__ Moments mesh_moments(const ArenaPtrs<R> &A, const MeshConst &mc,
                                                const R4<R> *P, int what) {
  __shared__ Moments s_w[kMonitorMaxThreads / 32];
  __shared__ double s_v[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Moments v = {0.0, 0.0, 0.0, 0.0, INT_MAX};
  if constexpr (sizeof(R) == 4) {
    if (what & 1) conres_share<R, PAIRS>(A, mc, threadIdx.x, kMonitorMaxThreads, v);
    if (what & 2) {
      force_share(A, mc, P, threadIdx.x, kMonitorMaxThreads, v);
      reduce_force<32>(v);
    }
  } else {
    // warp 0 (lanes 0 and 1) adds tile i while the others sum the residual and
    // form tile i + 1
    __shared__ ForceTile s_f[2];
    const int nt = what & 2 ? (mc.nsw + kForceTile - 1) / kForceTile : 0;
    double f = 0.0;
    bool some = false;   // of the tile formed last
    if (nt > 0)
      for (int k = threadIdx.x; k < min(mc.nsw, kForceTile); k += kMonitorMaxThreads)
        some |= force_terms<R>(A, P, A.sw_nodes[mc.sw0 + k], k, s_f[0]);
    for (int i = 0; i < nt || i == 0; i++) {
      const bool viscous = __syncthreads_or(some);
      some = false;
      if (warp == 0) {
        if (lane < 2 && i < nt)
          f = force_chain(s_f[i & 1], lane, min(mc.nsw - i * kForceTile, kForceTile), viscous, f);
      } else {
        if (i == 0 && (what & 1))
          conres_share<R, PAIRS>(A, mc, threadIdx.x - 32, kMonitorMaxThreads - 32, v);
        if (i + 1 < nt) {
          const int base = (i + 1) * kForceTile, n = min(mc.nsw - base, kForceTile);
          for (int k = threadIdx.x - 32; k < n; k += kMonitorMaxThreads - 32)
            some |= force_terms<R>(A, P, A.sw_nodes[mc.sw0 + base + k], k, s_f[(i + 1) & 1]);
        }
      }
    }
    if (threadIdx.x < 2) s_v[threadIdx.x] = f;
  }
  if (what & 1) reduce_residual<32>(v);
  if (lane == 0) s_w[warp] = v;
  __syncthreads();
  if (warp > 2) return v;
  v = s_w[lane & 7];
  if (warp == 0) {
    reduce_residual<8>(v);
  } else if constexpr (sizeof(R) == 4) {
    reduce_force<8>(v);
  } else {
    v.x = s_v[0];
    v.y = s_v[1];
  }
  return v;
}

// clcd.f:43-46: the lift (k = 0) or drag coefficient from the wall force
__device__ __forceinline__ double force_coefficient(const MeshConst &mc, const Moments &v, int k) {
  const double q = 0.5 * mc.r_inf * (mc.q_inf * mc.q_inf);
  return div64(k == 0 ? -mc.sin_aoa * v.x + mc.cos_aoa * v.y
                      : mc.cos_aoa * v.x + mc.sin_aoa * v.y,
               q);
}
// conres.f:23
__device__ __forceinline__ double residual_norm(const MeshConst &mc, const Moments &v) {
  return sqrt64(div64(v.s, double(mc.nv)));
}

// One CTA (256 threads) per mesh slot.  Thread 0 finishes the residual, the
// verdict and the control block; threads 32 and 64 the lift and drag.
template <typename R>
__global__ void __launch_bounds__(kMonitorMaxThreads) k_monitor(ArenaPtrs<R> A) {
  const int m = blockIdx.x;
  MeshCtl &ctl = A.ctl[m];
  if (!ctl.active) return;
  if (A.wpart > 0 && A.mesh_part[m] != A.wpart) return;   // another chain's mesh
  const MeshConst &mc = A.mc[m];
  const int newp = (ctl.phase + 1) % 3;
  // the control block is read here and written after the reduction's barrier
  const int err = ctl.err, err_point = ctl.err_point;
  const int row = ctl.hist_off + ctl.n_done % ctl.hist_cap;
  const Moments v = mesh_moments<R, sizeof(R) == 4>(A, mc, A.st[newp], 3);
  const bool stopped = err != 0 || err_point != INT_MAX;
  if (threadIdx.x == 32 && !stopped) {
    const double cl = force_coefficient(mc, v, 0);
    ctl.cl = cl;
    A.h_cl[row] = cl;
  }
  if (threadIdx.x == 64 && !stopped) {
    const double cd = force_coefficient(mc, v, 1);
    ctl.cd = cd;
    A.h_cd[row] = cd;
  }
  if (threadIdx.x != 0) return;
  ctl.phase = newp;
  if (mc.iflow == 3) ctl.nphase = 1 - ctl.nphase;
  if (err) {                            // roe_flux.f stop, inside residu
    ctl.active = 0;
    return;
  }
  if (err_point != INT_MAX) {          // check_positivity.f stop
    ctl.err = 3;
    ctl.active = 0;
    return;
  }
  double fres = residual_norm(mc, v);
  ctl.fresi = v.m;
  ctl.iresi = (v.m > 0.0) ? v.a : 0;
  if (ctl.iter == ctl.iterlast) {
    ctl.fres1 = fres;
    if (fres == 0.0) {
      ctl.fres = fres;
      ctl.err = 5;
      ctl.active = 0;
      return;
    }
  }
  fres = div64(fres, ctl.fres1);
  ctl.fres = fres;
  A.h_fres[row] = fres;
  A.h_iresi[row] = ctl.iresi;
  A.h_fresi[row] = v.m;
  ctl.iter += 1;
  ctl.n_done += 1;
  if (fres <= ctl.minres || ctl.n_done >= ctl.n_max) ctl.active = 0;
}

// ---------------------------------------------------------------------------
// Per-routine kernels (routine mode: state = buffer p, prim_old = p+2).
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_update(ArenaPtrs<R> A, int irk) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    if (threadIdx.x >= bi.nv) continue;
    const MeshCtl &ctl = A.ctl[bi.mesh];
    const MeshConst &mc = A.mc[bi.mesh];
    const int v = bi.v0 + threadIdx.x;
    const int p = ctl.phase;
    const R4<R> r4 = A.res[v];
    const R res[4] = {r4.x, r4.y, r4.z, r4.w};
    const bool noslip = (mc.iflow != 1) && (A.vflag[v] & kVtxSolid);
    A.st[p][v] = rk_update<R>(mc, irk, A.st[(p + 2) % 3][v], A.st[p][v], A.dt[v], v_cvarea(A, v),
                              res, noslip);
  }
}

template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_time_step(ArenaPtrs<R> A) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    if (threadIdx.x >= bi.nv) continue;
    const MeshCtl &ctl = A.ctl[bi.mesh];
    const int v = bi.v0 + threadIdx.x;
    A.dt[v] = time_step<R>(A.mc[bi.mesh], A.st[ctl.phase][v], A.mu[v], v_drmin(A, v));
  }
}

template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_positivity(ArenaPtrs<R> A) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    if (threadIdx.x >= bi.nv) continue;
    MeshCtl &ctl = A.ctl[bi.mesh];
    const int v = bi.v0 + threadIdx.x;
    const R4<R> P = A.st[ctl.phase][v];
    if (P.x <= R(0) || P.w <= R(0) || A.nut[ctl.nphase][v] < R(0))
      atomicMin(&ctl.err_point, A.orig[v]);
  }
}

// conres.f:14-22 partials between buffer p and prim_old = p+2
template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_conres_part(ArenaPtrs<R> A) {
  __shared__ double s_red[kBlockVerts / 32], s_max[kBlockVerts / 32];
  __shared__ int s_arg[kBlockVerts / 32];
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    const MeshCtl &ctl = A.ctl[bi.mesh];
    double d2 = 0.0, dabs = 0.0;
    int darg = INT_MAX;
    if (threadIdx.x < bi.nv) {
      const int v = bi.v0 + threadIdx.x;
      const double gra = double(A.st[ctl.phase][v].x) - double(A.st[(ctl.phase + 2) % 3][v].x);
      d2 = gra * gra;
      dabs = fabs(gra);
      if (dabs > 0.0) darg = A.orig[v];
      else dabs = 0.0;   // a NaN never becomes the maximum (conres.f:17-21)
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double o2 = __shfl_down_sync(0xffffffffu, d2, off);
      const double om = __shfl_down_sync(0xffffffffu, dabs, off);
      const int oa = __shfl_down_sync(0xffffffffu, darg, off);
      d2 += o2;
      if (om > dabs || (om == dabs && oa < darg)) {
        dabs = om;
        darg = oa;
      }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
      s_red[wid] = d2;
      s_max[wid] = dabs;
      s_arg[wid] = darg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = 0.0;
      int a = INT_MAX;
      for (int i = 0; i < kBlockVerts / 32; i++) {
        if (s_max[i] > m || (s_max[i] == m && s_arg[i] < a)) {
          m = s_max[i];
          a = s_arg[i];
        }
      }
      BlockPartial bp;
      bp.sumsq = warp_sums(s_red);
      bp.maxabs = m;
      bp.argmax = a;
      bp.pad = 0;
      A.part[bi.part] = bp;
    }
    __syncthreads();
  }
}

// conres (first: set fres1) or clcd for one mesh, routine mode.
template <typename R>
__global__ void __launch_bounds__(kMonitorMaxThreads)
    k_routine_monitor(ArenaPtrs<R> A, int mesh, int what, int first) {
  MeshCtl &ctl = A.ctl[mesh];
  const MeshConst &mc = A.mc[mesh];
  // (k_conres_part sums in FP64 for either precision)
  const Moments v = mesh_moments<R, false>(A, mc, A.st[ctl.phase], what == 0 ? 1 : 2);
  if (what == 0) {
    if (threadIdx.x != 0) return;
    double fres = residual_norm(mc, v);
    ctl.fresi = v.m;
    ctl.iresi = (v.m > 0.0) ? v.a : 0;
    if (first) {
      ctl.fres1 = fres;
      if (fres == 0.0) {
        ctl.fres = fres;
        ctl.err = 5;
        return;
      }
    }
    ctl.fres = div64(fres, ctl.fres1);
  } else {
    if (threadIdx.x == 32) ctl.cl = force_coefficient(mc, v, 0);
    if (threadIdx.x == 64) ctl.cd = force_coefficient(mc, v, 1);
  }
}

// limitgrad.f:14-75 on the current gradients, one thread per vertex over
// all of its edges in edge order.
// ---------------------------------------------------------------------------
// gradient.f:1-63 (never called by the reference: main.f:29 comments it
// out), routine mode: edge-based Green-Gauss over the dual cells.  Each
// interior edge contributes +-(qa*ds) with qa the mean of its ends' states;
// each boundary edge contributes (5 p1 + p2)/6 and (p1 + 5 p2)/6 times half
// its rotated edge vector to its two ends; each vertex sums its interior
// edges in iedge order, then its boundary edges in beindx order (the flux
// pass's incidence lists), and divides by its dual-cell area.  The
// reference's print of every vertex (gradient.f:60) is left out.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_gradient_edge(ArenaPtrs<R> A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Grad<R> *s_g = reinterpret_cast<Grad<R> *>(smem_raw);   // [max_slots]
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    const MeshCtl &ctl = A.ctl[bi.mesh];
    const R4<R> *P = A.st[ctl.phase];
    for (int k = threadIdx.x; k < bi.ne; k += blockDim.x) {
      const int2 nn = A.be_nodes[bi.e0 + k];
      const double2 ds = A.be_ds[bi.e0 + k];
      const R4<R> p1 = P[nn.x], p2 = P[nn.y];
      Grad<R> g;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const R qa = R(0.5) * (comp(p1, q) + comp(p2, q));
        g.qx[q] = qa * R(ds.x);
        g.qy[q] = qa * R(ds.y);
      }
      s_g[k] = g;
    }
    for (int k = threadIdx.x; k < bi.nb; k += blockDim.x) {
      const int4 b = A.bb_nodes[bi.b0 + k];
      const double2 x1 = A.coord[b.x], x2 = A.coord[b.y];
      const R dx = R(x2.x - x1.x), dy = R(x2.y - x1.y);
      const R nx = R(0.5) * dy, ny = -R(0.5) * dx;
      const R4<R> p1 = P[b.x], p2 = P[b.y];
      Grad<R> g1, g2;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const R qa1 = (R(5) * comp(p1, q) + comp(p2, q)) / R(6);
        const R qa2 = (comp(p1, q) + R(5) * comp(p2, q)) / R(6);
        g1.qx[q] = qa1 * nx;
        g1.qy[q] = qa1 * ny;
        g2.qx[q] = qa2 * nx;
        g2.qy[q] = qa2 * ny;
      }
      s_g[bi.ne + 2 * k] = g1;
      s_g[bi.ne + 2 * k + 1] = g2;
    }
    __syncthreads();
    if (threadIdx.x < bi.nv) {
      const int v = bi.v0 + threadIdx.x;
      R qx[4] = {R(0), R(0), R(0), R(0)}, qy[4] = {R(0), R(0), R(0), R(0)};
      const int2 jr = A.ve_rng[v];
      for (int j = jr.x; j < jr.y; j++) {
        const uint16_t e = A.ve_list[j];
        const Grad<R> g = s_g[e & kSlotMask];
        if (e & kNegBit) {      // n2 of an interior edge
#pragma unroll
          for (int q = 0; q < 4; q++) {
            qx[q] = qx[q] - g.qx[q];
            qy[q] = qy[q] - g.qy[q];
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) {
            qx[q] = qx[q] + g.qx[q];
            qy[q] = qy[q] + g.qy[q];
          }
        }
      }
      const R ai = R(1) / v_cvarea(A, v);
      Grad<R> g;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        g.qx[q] = ai * qx[q];
        g.qy[q] = ai * qy[q];
      }
      A.grad[v] = g;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// shockind.f:1-52 (never called by the reference), routine mode: the
// density-jump indicator of every vertex from all its edges (edge order),
// ind/drmin/cvarea**0.75; the gradients of vertices where it exceeds 1 are
// set to zero, by a second kernel: the first reads its neighbours' gradients.
// One thread per vertex; each edge's term is formed by both of its ends with
// the same operations, so both add the same value.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_shockind(ArenaPtrs<R> A) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    if (threadIdx.x >= bi.nv) continue;
    const MeshCtl &ctl = A.ctl[bi.mesh];
    const MeshConst &mc = A.mc[bi.mesh];
    const int v = bi.v0 + threadIdx.x;
    const R4<R> *P = A.st[ctl.phase];
    const R a11 = MCR(R, albada11), a12 = MCR(R, albada12);
    R ind = R(0);
    const int2 r = A.va_rng[v];
    for (int j = r.x; j < r.y; j++) {
      const int raw = A.va_list[j];
      const int o = raw & 0x7fffffff;
      const bool is_n2 = raw < 0;
      const int n1 = is_n2 ? o : v, n2 = is_n2 ? v : o;
      const double2 c1 = A.coord[n1], c2 = A.coord[n2];
      const R dx = R(c2.x - c1.x), dy = R(c2.y - c1.y);
      const R r1 = P[n1].x, r2 = P[n2].x;
      const Grad<R> g1 = A.grad[n1], g2 = A.grad[n2];
      const R dvc = r2 - r1;
      R dvt = dx * g1.qx[0] + dy * g1.qy[0];
      const R dvl = a11 * dvt + a12 * dvc;
      const R vl = r1 + dvl;
      dvt = dx * g2.qx[0] + dy * g2.qy[0];
      const R dvr = a11 * dvt + a12 * dvc;
      const R vr = r2 - dvr;
      const R li = sq(vr - vl) * R(A.va_dsl[j]);
      ind = ind + li;
    }
    ind = ind / v_drmin(A, v) / mpow(v_cvarea(A, v), R(0.75));
    const uint8_t f = A.vflag[v];
    A.vflag[v] = ind > R(1) ? f | kVtxShock : f & (uint8_t)~kVtxShock;
  }
}

template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_shock_zero(ArenaPtrs<R> A) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    const int v = bi.v0 + threadIdx.x;
    if (threadIdx.x >= bi.nv || !(A.vflag[v] & kVtxShock)) continue;
    Grad<R> z;
#pragma unroll
    for (int q = 0; q < 4; q++) z.qx[q] = z.qy[q] = R(0);
    A.grad[v] = z;
  }
}

template <typename R>
__global__ void __launch_bounds__(kBlockVerts) k_limitgrad(ArenaPtrs<R> A) {
  int w0, nwork;
  work_range(A, w0, nwork);
  for (int w = w0 + blockIdx.x; w < nwork; w += gridDim.x) {
    const BlockInfo bi = work_block(A, w);
    if (threadIdx.x >= bi.nv) continue;
    const MeshCtl &ctl = A.ctl[bi.mesh];
    const MeshConst &mc = A.mc[bi.mesh];
    const int v = bi.v0 + threadIdx.x;
    const R4<R> *P = A.st[ctl.phase];
    const R4<R> pv = P[v];
    const double2 cv = A.coord[v];
    Grad<R> g = A.grad[v];
    R qmin[4], qmax[4], phi[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      qmin[q] = R(1.0e10);
      qmax[q] = R(-1.0e10);
      phi[q] = R(1);
    }
    const int2 ar = A.va_rng[v];
    const int j0 = ar.x, j1 = ar.y;
    for (int j = j0; j < j1; j++) {
      const int o = A.va_list[j] & 0x7fffffff;
      const R4<R> po = P[o];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (!mc.bugcompat) {
          qmin[q] = dmin1(qmin[q], comp(pv, q));
          qmax[q] = dmax1(qmax[q], comp(pv, q));
          qmin[q] = dmin1(qmin[q], comp(po, q));
          qmax[q] = dmax1(qmax[q], comp(po, q));
        } else {
          qmin[q] = dmin1(qmin[q], comp(pv, q));
          qmax[q] = dmax1(qmax[q], comp(pv, q));
        }
      }
    }
    for (int j = j0; j < j1; j++) {
      const int raw = A.va_list[j];
      const int o = raw & 0x7fffffff;
      const bool is_n2 = raw < 0;
      const double2 co = A.coord[o];
      // dx, dy always from edge(1) to edge(2)
      const R dx = is_n2 ? R(cv.x - co.x) : R(co.x - cv.x);
      const R dy = is_n2 ? R(cv.y - co.y) : R(co.y - cv.y);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        R dq = g.qx[q] * dx + g.qy[q] * dy;
        if (is_n2) dq = -dq;
        const R dqmax = qmax[q] - comp(pv, q);
        const R dqmin = qmin[q] - comp(pv, q);
        if (dq != R(0)) {
          const R ppp = (dq > R(0)) ? dqmax / dq : dqmin / dq;
          phi[q] = dmin1(phi[q], ppp);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      g.qx[q] = phi[q] * g.qx[q];
      g.qy[q] = phi[q] * g.qy[q];
    }
    A.grad[v] = g;
  }
}

}  // namespace fvm

#include "fvm_pipe.cuh"
