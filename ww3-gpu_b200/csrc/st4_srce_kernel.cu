// ww3-gpu_b200/csrc/st4_srce_kernel.cu
// The ST4 source terms (one CTA per sea point, the phases of st4_point.cuh) and W3SRCE (up to
// pt::kSlots points per CTA, srce_point.cuh) on sm_100a.
//
// W3SRCE runs on a persistent grid: a CTA takes the next point from a global counter as one of its
// slots finishes one, so the uneven number of substeps per point (the dynamic integration stops when
// the point's DTTOT reaches DTG) balances across the SMs instead of leaving a tail of idle CTAs.
#include "st4_srce.cuh"

#include "wwb_common.hpp"

namespace wwb {
namespace {

__global__ void __launch_bounds__(kSt4Block) sds4_kernel(
    const St4Dev* __restrict__ d, int npts, const float* a, const float* k, const float* cg,
    const float* ustar, const float* usdir, const float* depth, const float* dair,
    const float* dlwmean, int f57, int f58, float* srhs, float* ddiag, float* brlambda,
    float* whitecap) {
  extern __shared__ __align__(16) float smem[];
  __shared__ pt::Sds4Sh sh;
  const st4::Params& p = d->p;
  const pt::Cta cta{static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x)};
  float* const w = smem;
  float* const w2 = w + ((pt::sds4_work_reals(p) + 3) & ~3);
  int* const iw = reinterpret_cast<int*>(w2 + pt::sds4_work2_reals(p));
  for (int n = blockIdx.x; n < npts; n += gridDim.x) {
    const size_t os = static_cast<size_t>(n) * p.nspec, ok = static_cast<size_t>(n) * p.nk;
    pt::sds4(cta, p, d->f, a + os, k + ok, cg + ok, ustar[n], usdir[n], depth[n], dair[n],
             dlwmean[n], f57, f58, srhs + os, ddiag + os, brlambda + os,
             whitecap + 4 * static_cast<size_t>(n), w, w2, iw, sh);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kSt4Block) sin4_kernel(
    const St4Dev* __restrict__ d, int npts, const float* a, const float* cg, const float* k,
    const float* u, const float* ustar, const float* drat, const float* as, const float* usdir,
    const float* z0, float* tauwx, float* tauwy, float* tauwnx, float* tauwny, float* s,
    float* dd, int* llws) {
  extern __shared__ __align__(16) float smem[];
  __shared__ pt::Sin4Sh sh;
  const st4::Params& p = d->p;
  const pt::Cta cta{static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x)};
  float* const dstab = smem;
  float* const eb = dstab + 3 * p.nspec;
  for (int n = blockIdx.x; n < npts; n += gridDim.x) {
    const size_t os = static_cast<size_t>(n) * p.nspec, ok = static_cast<size_t>(n) * p.nk;
    pt::sin4(cta, p, d->f, a + os, cg + ok, k + os, p.nth, u[n], ustar[n], drat[n], as[n],
             usdir[n], z0[n], tauwx + n, tauwy + n, tauwnx + n, tauwny + n, s + os, dd + os,
             llws + os, dstab, eb, sh);
    __syncthreads();
  }
}

struct Spr4Ptrs {
  float* o[12];
};

__global__ void __launch_bounds__(kSt4Block) spr4_kernel(
    const St4Dev* __restrict__ d, int npts, const float* a, const float* cg, const float* wn,
    const float* u, const float* udir, const float* tauwx, const float* tauwy, const int* llws,
    Spr4Ptrs out) {
  extern __shared__ __align__(16) float smem[];
  __shared__ pt::Spr4Out o;
  const st4::Params& p = d->p;
  const pt::Cta cta{static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x)};
  for (int n = blockIdx.x; n < npts; n += gridDim.x) {
    const size_t os = static_cast<size_t>(n) * p.nspec, ok = static_cast<size_t>(n) * p.nk;
    if (threadIdx.x == 0) {
      float* const f = &o.ustar;
      for (int j = 0; j < 12; ++j) f[j] = out.o[j][n];
    }
    __syncthreads();
    pt::spr4(cta, p, d->f, a + os, cg + ok, wn + ok, u[n], udir[n], tauwx[n], tauwy[n],
             llws + os, o, smem, smem + ((pt::spr4_work_reals(p) + 3) & ~3));
    if (threadIdx.x == 0) {
      const float* const f = &o.ustar;
      for (int j = 0; j < 12; ++j) out.o[j][n] = f[j];
    }
    __syncthreads();
  }
}

/// What the CTA's threads agree on: the job whose points it integrates, the slots' points, and a queue
/// entry taken but not yet loaded (it belongs to another job when `foreign`).
struct SrceCtl {
  SrceJob job;
  int pt[pt::kSlots];
  int pending, foreign, empty;
  unsigned fresh;
};

/// Points of one job from the launch's work queue.
struct QueuePoints {
  SrceCtl& ctl;
  int total;
  int* counter;

  template <class G>
  __device__ __forceinline__ void load(const pt::Grp& c, const G& x, pt::SlotList& fresh) {
    const pt::SrceLayout& L = *x.L;
    if (ctl.empty || ctl.foreign) return;
    bool room = false;
    for (int k = 0; k < x.ns; ++k) room = room || x.sh[k].state == pt::kIdle;
    if (!room) return;
    c.sync();  // every thread has read the states and the queue's
    if (c.tid == 0) {
      unsigned m = 0;
      for (int k = 0; k < x.ns; ++k) {
        if (x.sh[k].state != pt::kIdle) continue;
        const int q = ctl.pending >= 0 ? ctl.pending : atomicAdd(counter, 1);
        ctl.pending = -1;
        if (q >= total) {
          ctl.empty = 1;
          break;
        }
        if (q < ctl.job.first || q >= ctl.job.first + ctl.job.npts) {
          ctl.pending = q;
          ctl.foreign = 1;
          break;
        }
        ctl.pt[k] = q - ctl.job.first;
        x.sh[k].state = ctl.job.step.it != 0 ? pt::kFresh1 : pt::kFresh2;
        m |= 1u << k;
      }
      ctl.fresh = m;
    }
    c.sync();
    const unsigned m = ctl.fresh;
    for (int k = 0; k < x.ns; ++k)
      if (m >> k & 1) fresh.add(k);
    if (fresh.n == 0) return;
    const SrceJob& j = ctl.job;
    pt::each_bin(c, fresh, L.nspec, [&](int k, int i) {
      const int n = ctl.pt[k];
      const size_t col = j.jsea ? static_cast<size_t>(j.jsea[n]) : static_cast<size_t>(n);
      x.s(k, L.spec)[i] = j.spec[col * L.nspec + i];
    });
    pt::each_row(c, fresh, L.nk, [&](int k, int ik) {
      const size_t o = static_cast<size_t>(ctl.pt[k]) * L.nk + ik;
      x.s(k, L.wn1)[ik] = j.wn1[o];
      x.s(k, L.cg1)[ik] = j.cg1[o];
    });
    pt::each_chain(c, 0, fresh, [&](int k) {
      const size_t n = ctl.pt[k];
      pt::SrceSh& s = x.sh[k];
      pt::srce_psc_in(s, j.psc + n * srce::NPSC, j.whitecap + 4 * n, j.taubbl + 2 * n,
                      j.tauice + 2 * n);
      s.r.z0 = s.r.cd = s.r.emean = s.r.fmean = s.r.fmean1 = s.r.amax = s.r.fmeanws = 0.0f;
      s.in = pt::srce_in(j.step.it, j.step.inflags24, j.step.flogrd57, j.step.flogrd58, j.step.dtg,
                         j.pin + n * srce::NPIN);
    });
    c.sync();
  }

  template <class G>
  __device__ __forceinline__ void store(const pt::Grp& c, const G& x, const pt::SlotList& done) {
    const pt::SrceLayout& L = *x.L;
    const SrceJob& j = ctl.job;
    pt::each_bin(c, done, L.nspec, [&](int k, int i) {
      const int n = ctl.pt[k];
      const size_t col = j.jsea ? static_cast<size_t>(j.jsea[n]) : static_cast<size_t>(n);
      j.spec[col * L.nspec + i] = x.s(k, L.spec)[i];
    });
    pt::each_chain(c, 0, done, [&](int k) {
      const size_t n = ctl.pt[k];
      pt::srce_psc_out(x.sh[k], j.psc + n * srce::NPSC, j.whitecap + 4 * n, j.taubbl + 2 * n,
                       j.tauice + 2 * n, j.shave + n);
      x.sh[k].state = pt::kIdle;
    });
    c.sync();
  }
};

/// The last warp of a CTA: the tails the working warps hand over, until they are done.
template <class G>
__device__ __forceinline__ void tail_warp(const G& x, pt::TailBox& box) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    pt::barrier_sync<pt::kBarTail>(kSrceBlock);
    if (box.exit) break;
    const pt::SlotList l = box.l;
    pt::sin4_close(lane, x, l, [] { __syncwarp(); });
    pt::barrier_arrive<pt::kBarTailDone>(kSrceBlock);
  }
}
__device__ __forceinline__ void tail_exit(const pt::Grp& c, pt::TailBox& box) {
  c.sync();
  if (c.tid == 0) box.exit = 1;
  c.tail_go();
}

/// W3SRCE over the points of one grid. The grid's parameters and table pointers are a kernel parameter,
/// so the phases read them from the constant bank instead of loading them for every bin.
template <int NTH>
__global__ void __launch_bounds__(kSrceBlock, kSrceMinBlocks) srce_kernel(
    const __grid_constant__ SrceDev dev, const __grid_constant__ SrceJob job, int ns, int* counter,
    float* scratch) {
  extern __shared__ __align__(16) float w[];
  __shared__ pt::SrceSh sh[pt::kSlots];
  __shared__ SrceCtl ctl;
  __shared__ pt::TailBox box;
  const pt::Grp c{static_cast<int>(threadIdx.x), kSrceBlock - 32};
  if (threadIdx.x == 0) {
    box.exit = 0;
    ctl.job = job;
    ctl.pending = -1;
    ctl.foreign = ctl.empty = 0;
    for (int k = 0; k < pt::kSlots; ++k) sh[k].state = pt::kIdle;
  }
  __syncthreads();
  float* const gw = scratch + static_cast<size_t>(blockIdx.x) * ns * dev.L.total_g;
  const pt::SrceGroup<NTH> x{&dev.p, &dev.g, &dev.q, &dev.f, &dev.n, &dev.L,
                                    w,      gw,     w + dev.L.common + ns * dev.L.ws, sh, ns, &box};
  if (threadIdx.x >= kSrceBlock - 32) {
    tail_warp(x, box);
    return;
  }
  QueuePoints src{ctl, job.npts, counter};
  pt::srce_run(c, x, src);
  tail_exit(c, box);
}

/// W3SRCE over the points of several grids in one persistent launch: one work queue over (grid,
/// point), the job of queue entry q the last one whose first entry is <= q. A CTA integrates points of
/// one job at a time and turns to the next job when its slots are empty. Every job has the same
/// working-set layout (checked on the host).
template <int NTH>
__global__ void __launch_bounds__(kSrceBlock, kSrceMinBlocks) srce_multi_kernel(
    const SrceJob* __restrict__ jobs, int njobs, int total, int ns, int* counter, float* scratch) {
  extern __shared__ __align__(16) float w[];
  __shared__ pt::SrceSh sh[pt::kSlots];
  __shared__ SrceCtl ctl;
  __shared__ SrceDev dev;
  __shared__ pt::TailBox box;
  const pt::Grp c{static_cast<int>(threadIdx.x), kSrceBlock - 32};
  if (threadIdx.x == 0) {
    box.exit = 0;
    ctl.pending = -1;
    for (int k = 0; k < pt::kSlots; ++k) sh[k].state = pt::kIdle;
  }
  __syncthreads();
  if (threadIdx.x >= kSrceBlock - 32) {
    // The grid's parameters change only between jobs, when no tail is under way.
    const pt::SrceGroup<NTH> x{&dev.p, &dev.g, &dev.q, &dev.f, &dev.n, &dev.L, w, nullptr,
                               nullptr, sh, ns, &box};
    tail_warp(x, box);
    return;
  }
  for (;;) {
    c.sync();
    if (threadIdx.x == 0) {
      const int q = ctl.pending >= 0 ? ctl.pending : atomicAdd(counter, 1);
      ctl.pending = q;
      ctl.foreign = 0;
      ctl.empty = q >= total;
      if (q < total) {
        int lo = 0, hi = njobs - 1;  // the job holding q: first[lo] <= q < first[lo + 1]
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (jobs[mid].first <= q) lo = mid;
          else hi = mid - 1;
        }
        ctl.job = jobs[lo];
      }
    }
    c.sync();
    if (ctl.empty) break;
    {
      const int* const from = reinterpret_cast<const int*>(ctl.job.d);
      int* const to = reinterpret_cast<int*>(&dev);
      for (int i = threadIdx.x; i < static_cast<int>(sizeof(SrceDev) / sizeof(int)); i += c.nthr)
        to[i] = from[i];
    }
    c.sync();
    float* const gw = scratch + static_cast<size_t>(blockIdx.x) * ns * dev.L.total_g;
    const pt::SrceGroup<NTH> x{&dev.p, &dev.g, &dev.q, &dev.f, &dev.n, &dev.L,
                               w,      gw,     w + dev.L.common + ns * dev.L.ws, sh, ns, &box};
    QueuePoints src{ctl, total, counter};
    pt::srce_run(c, x, src);
  }
  tail_exit(c, box);
}

using OneKernel = void (*)(SrceDev, SrceJob, int, int*, float*);
using MultiKernel = void (*)(const SrceJob*, int, int, int, int*, float*);
/// The kernels built for a number of directions: WW3's usual 36 and 24 (compile-time bin addresses and
/// unrolled sums), else the general ones. A form of its own for SSDSC(1) = 1 without sheltering gave
/// nothing (9,520 points: 101.1-102.5 ms with it, 101.3 without).
OneKernel one_kernel(const pt::SrceLayout& L) {
  return L.nth == 36 ? srce_kernel<36> : L.nth == 24 ? srce_kernel<24> : srce_kernel<0>;
}
MultiKernel multi_kernel(int nth) {
  // No form for 24: eight grids of 25 x 24 bins, 3,924 points, a step 10.4-12.6 ms with the general one
  // and 10.3-12.2 with one of its own.
  return nth == 36 ? srce_multi_kernel<36> : srce_multi_kernel<0>;
}

/// Resident CTAs of an ST4 kernel at this shared memory, at most one per point.
template <class K>
int resident_grid(K k, size_t smem, int npts) {
  WWB_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
  int per_sm = 0;
  WWB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kSt4Block, smem));
  if (per_sm < 1) throw CudaError(cudaErrorInvalidConfiguration, "st4 occupancy");
  const long long resident = static_cast<long long>(per_sm) * runtime().sm_count;
  return static_cast<int>(npts < resident ? npts : resident);
}

/// Dynamic shared memory of a W3SRCE CTA with ns slots.
size_t srce_smem(const pt::SrceLayout& L, int ns) {
  return static_cast<size_t>(pt::srce_shared_floats(L, ns)) * sizeof(float);
}
constexpr size_t kSrceStatic =
    sizeof(pt::SrceSh) * pt::kSlots + sizeof(SrceCtl) + sizeof(SrceDev) + sizeof(pt::TailBox) + 64;
/// The dynamic shared memory that every call allows a W3SRCE kernel: one value for all, never a launch's
/// own, so that a launch is not refused because another thread's (of fewer slots or a smaller grid) has
/// lowered the kernel's limit between its plan and its start.
constexpr size_t kSrceDynMax = (227 * 1024 - kSrceStatic) & ~static_cast<size_t>(15);

/// A W3SRCE launch: slots per CTA, CTAs, shared memory.
struct SrcePlan {
  int ns, grid;
  size_t smem;
};
/// Slots a CTA of this layout can have.
int srce_max_slots(const pt::SrceLayout& L) {
  for (int ns = pt::kSlots; ns > 1; --ns)
    if (srce_smem(L, ns) <= kSrceDynMax) return ns;
  return 1;
}
/// The fewest slots with which the points fit the SMs' CTAs at once, and as many CTAs as that fills: a
/// launch lasts as long as its longest point, and a point is integrated faster the fewer share its CTA
/// (149 points on 148 SMs run as 75 CTAs of two). CTAs per SM are the one that the kernels are built for.
SrcePlan srce_plan(const pt::SrceLayout& L, int npts) {
  if (srce_smem_bytes(L) == 0)
    throw CudaError(cudaErrorInvalidConfiguration, "W3SRCE working set too large");
  const int most = srce_max_slots(L);
  const long long ctas = static_cast<long long>(kSrceMinBlocks) * runtime().sm_count;
  int ns = 1;
  while (ns < most && ctas * ns < npts) ++ns;
  const long long want = (static_cast<long long>(npts) + ns - 1) / ns;
  return SrcePlan{ns, static_cast<int>(want < ctas ? want : ctas), srce_smem(L, ns)};
}
void srce_allow(const void* k) {
  WWB_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kSrceDynMax)));
}
void srce_reserve_plan(const pt::SrceLayout& L, const SrcePlan& plan, SrceWork& work) {
  const size_t need = static_cast<size_t>(plan.grid) * plan.ns * static_cast<size_t>(L.total_g);
  if (work.counter == nullptr) WWB_CHECK(cudaMalloc(&work.counter, sizeof(int)));
  if (need > work.scratch_n) {
    if (work.scratch) WWB_CHECK(cudaFree(work.scratch));
    work.scratch = nullptr;
    work.scratch_n = 0;
    WWB_CHECK(cudaMalloc(&work.scratch, need * sizeof(float)));
    work.scratch_n = need;
  }
}
/// Whether the work buffers are large enough for the plan.
bool srce_reserved(const pt::SrceLayout& L, const SrcePlan& plan, const SrceWork& work) {
  return work.counter != nullptr && static_cast<size_t>(plan.grid) * plan.ns *
                                            static_cast<size_t>(L.total_g) <= work.scratch_n;
}
void srce_reserve(const pt::SrceLayout& L, const SrcePlan& plan, SrceWork& work, cudaStream_t st) {
  if (srce_reserved(L, plan, work)) return;
  WWB_CHECK(cudaStreamSynchronize(st));  // earlier launches may still use the old buffers
  srce_reserve_plan(L, plan, work);
}

}  // namespace

size_t srce_smem_bytes(const pt::SrceLayout& L) {
  const size_t b = srce_smem(L, 1);
  return b <= kSrceDynMax ? b : 0;
}

void launch_sds4(const St4Dev* d, const st4::Params& hp, int npts, const float* a, const float* k,
                 const float* cg, const float* ustar, const float* usdir, const float* depth,
                 const float* dair, const float* dlwmean, int f57, int f58, float* srhs,
                 float* ddiag, float* brlambda, float* whitecap, cudaStream_t s) {
  if (npts <= 0) return;
  const size_t smem = sizeof(float) * (((pt::sds4_work_reals(hp) + 3) & ~3) +
                                       pt::sds4_work2_reals(hp) + pt::sds4_work_ints(hp));
  const int grid = resident_grid(sds4_kernel, smem, npts);
  sds4_kernel<<<grid, kSt4Block, smem, s>>>(d, npts, a, k, cg, ustar, usdir, depth, dair, dlwmean,
                                            f57, f58, srhs, ddiag, brlambda, whitecap);
  WWB_CHECK(cudaGetLastError());
}

void launch_sin4(const St4Dev* d, const st4::Params& hp, int npts, const float* a,
                 const float* cg, const float* k, const float* u, const float* ustar,
                 const float* drat, const float* as, const float* usdir, const float* z0,
                 float* tauwx, float* tauwy, float* tauwnx, float* tauwny, float* s, float* dd,
                 int* llws, cudaStream_t st) {
  if (npts <= 0) return;
  const size_t smem = sizeof(float) * (3 * static_cast<size_t>(hp.nspec) + pt::sin4_nk_work(hp));
  const int grid = resident_grid(sin4_kernel, smem, npts);
  sin4_kernel<<<grid, kSt4Block, smem, st>>>(d, npts, a, cg, k, u, ustar, drat, as, usdir, z0,
                                             tauwx, tauwy, tauwnx, tauwny, s, dd, llws);
  WWB_CHECK(cudaGetLastError());
}

void launch_spr4(const St4Dev* d, const st4::Params& hp, int npts, const float* a,
                 const float* cg, const float* wn, const float* u, const float* udir,
                 const float* tauwx, const float* tauwy, const int* llws, float* const* out12,
                 cudaStream_t st) {
  if (npts <= 0) return;
  Spr4Ptrs o;
  for (int j = 0; j < 12; ++j) o.o[j] = out12[j];
  const size_t smem = sizeof(float) * (((pt::spr4_work_reals(hp) + 3) & ~3) +
                                       static_cast<size_t>(pt::spr4_terms_reals(hp)));
  const int grid = resident_grid(spr4_kernel, smem, npts);
  spr4_kernel<<<grid, kSt4Block, smem, st>>>(d, npts, a, cg, wn, u, udir, tauwx, tauwy, llws, o);
  WWB_CHECK(cudaGetLastError());
}

void srce_reserve(const pt::SrceLayout& L, int npts, SrceWork& work, cudaStream_t st) {
  if (npts <= 0) return;
  srce_reserve(L, srce_plan(L, npts), work, st);
}

void srce_multi_reserve(const pt::SrceLayout& L, int total, SrceWork& work) {
  srce_reserve_plan(L, srce_plan(L, total > 0 ? total : 1), work);
}

void launch_srce_multi(const SrceJob* jobs_dev, int njobs, int total, const pt::SrceLayout& L,
                       SrceWork& work, cudaStream_t st) {
  if (total <= 0) return;
  const SrcePlan plan = srce_plan(L, total);
  if (!srce_reserved(L, plan, work))
    throw CudaError(cudaErrorInvalidValue, "launch_srce_multi: work buffers not reserved");
  srce_allow(reinterpret_cast<const void*>(multi_kernel(L.nth)));
  WWB_CHECK(cudaMemsetAsync(work.counter, 0, sizeof(int), st));
  multi_kernel(L.nth)<<<plan.grid, kSrceBlock, plan.smem, st>>>(jobs_dev, njobs, total, plan.ns,
                                                                work.counter, work.scratch);
  WWB_CHECK(cudaGetLastError());
}

void launch_srce(const SrceDev& dev, SrceStep step, int npts, float* spec, const int* jsea,
                 const float* wn1, const float* cg1, const float* pin, float* psc, float* whitecap, float* taubbl, float* tauice,
                 int* shave, SrceWork& work, cudaStream_t st) {
  if (npts <= 0) return;
  const pt::SrceLayout& L = dev.L;
  const SrcePlan plan = srce_plan(L, npts);
  // The work buffers fit after srce_reserve; otherwise (re)allocate them first, after the
  // previous launches on this stream that may still read the old ones.
  srce_reserve(L, plan, work, st);
  srce_allow(reinterpret_cast<const void*>(one_kernel(L)));
  WWB_CHECK(cudaMemsetAsync(work.counter, 0, sizeof(int), st));
  const SrceJob job{nullptr, step, npts,     0,      spec,   jsea, wn1, cg1,
                    pin,     psc,  whitecap, taubbl, tauice, shave};
  one_kernel(L)<<<plan.grid, kSrceBlock, plan.smem, st>>>(dev, job, plan.ns, work.counter,
                                                              work.scratch);
  WWB_CHECK(cudaGetLastError());
}

}  // namespace wwb
