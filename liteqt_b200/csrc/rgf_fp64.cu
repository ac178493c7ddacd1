// rgf_fp64.cu -- the persistent complex FP64 RGF kernel (the drop-in form of
// green_RGF_RS, src/green_rgf.f90:3950-4164, and its adjoint).
//
// One launch drains a work queue of (device, k, E) tasks of any mix of block
// sizes nb and chain lengths nx: a CTA pops a task, looks up the kernel
// variant chosen for the task's nb (staged GEMM + blocked inverse for the
// benchmark sizes, register-direct GEMM for any other multiple of 8; the
// host may override the choice per nb, see rgf_autotune) and calls that
// variant's task function, which runs the whole per-energy chain with the
// CTA's 256 threads (rgf_solver.cuh).  The queue order is set by the host
// (longest tasks first), so the tail of the launch holds the short tasks.
#include <cstdio>

#include "rgf_device.cuh"
#include "rgf_internal.h"
#include "rgf_tasks.h"

namespace rgf {

namespace {

__global__ void __launch_bounds__(kThreads, 2) rgf_solver_kernel(KParams p) {
  extern __shared__ __align__(16) double2 dyn_smem[];
  __shared__ Smem sm;
  Group grp;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(grp.rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(grp.size));
  double2* slot = p.work + (size_t)(blockIdx.x / grp.size) * p.slot_elems;
  // the barriers around the pop also order the CTAs of a cluster's first and
  // last accesses to each other's shared memory after their start and before
  // their exit
  for (;;) {
    grp.sync();
    if (threadIdx.x == 0 && grp.rank == 0) {
      const int64_t q = atomicAdd(p.queue, 1);
      if (grp.size == 1) {
        sm.task = q;
      } else {
        for (int r = 0; r < grp.size; r++) {
          uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.task);
          asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(dst) : "r"(r));
          asm volatile("st.shared::cluster.s64 [%0], %1;" ::"r"(dst), "l"(q) : "memory");
        }
      }
    }
    grp.sync();
    const int64_t q = sm.task;
    if (q >= p.n_tasks) break;
    const int64_t t = p.order ? p.order[q] : q;
    const int dev = p.adj ? p.adj[t].dev : (p.wtasks ? p.wtasks[t].dev : p.tasks[t].dev);
    const int64_t n = p.devs[dev].nm, nx = p.devs[dev].nx;
    int v = KV_NONE;
    if (n >= 8 && n <= kMaxNb && n % 8 == 0) v = p.variant[n / 8];
    const bool staged_ok = (v == KV_STAGED32 && n == 32) || (v == KV_STAGED64 && n == 64) ||
                           (v == KV_STAGED128 && n == 128) || (v == KV_STAGED256 && n == 256);
    const bool generic_ok = v == KV_GENERIC11 || ((v == KV_GENERIC12 || v == KV_GENERIC22) && n % 16 == 0);
    if (!(staged_ok || generic_ok || v == KV_TILED) || grp.size > kMaxGroup || nx < 2 || slot_elems_for(n, nx) > p.slot_elems) {
      if (p.info && threadIdx.x == 0 && grp.rank == 0) p.info[t].status = RGF_ST_BAD_TASK;
      continue;
    }
    if (grp.size > 1) {   // the forms whose operations a cluster shares
      switch ((int)n) {
        case 32: task_group32(p, t, slot, sm, dyn_smem, grp); break;
        case 64: task_group64(p, t, slot, sm, dyn_smem, grp); break;
        case 128: task_group128(p, t, slot, sm, dyn_smem, grp); break;
        case 256: task_group256(p, t, slot, sm, dyn_smem, grp); break;
        default: task_tiled(p, t, slot, sm, dyn_smem, grp); break;
      }
      continue;
    }
    switch (v) {
      case KV_STAGED32: task_staged32(p, t, slot, sm, dyn_smem, grp); break;
      case KV_STAGED64: task_staged64(p, t, slot, sm, dyn_smem, grp); break;
      case KV_STAGED128: task_staged128(p, t, slot, sm, dyn_smem, grp); break;
      case KV_STAGED256: task_staged256(p, t, slot, sm, dyn_smem, grp); break;
      case KV_GENERIC11: task_generic11(p, t, slot, sm, dyn_smem, grp); break;
      case KV_TILED: task_tiled(p, t, slot, sm, dyn_smem, grp); break;
      case KV_GENERIC12: task_generic12(p, t, slot, sm, dyn_smem, grp); break;
      default: task_generic22(p, t, slot, sm, dyn_smem, grp); break;
    }
  }
}

}  // namespace

int default_variant(int nb) {
  if (nb < 8 || nb > kMaxNb || nb % 8 != 0) return KV_NONE;
  switch (nb) {
    case 32: return KV_STAGED32;
    case 64: return KV_STAGED64;
    case 128: return KV_STAGED128;
    case 256: return KV_STAGED256;
    default: break;
  }
  if (nb >= 80) return KV_TILED;
  if (nb % 16 == 0 && nb >= 64) return KV_GENERIC22;
  if (nb % 16 == 0) return KV_GENERIC12;
  return KV_GENERIC11;
}

bool variant_ok(int v, int nb) {
  if (nb < 8 || nb > kMaxNb || nb % 8 != 0) return false;
  switch (v) {
    case KV_STAGED32: return nb == 32;
    case KV_STAGED64: return nb == 64;
    case KV_STAGED128: return nb == 128;
    case KV_STAGED256: return nb == 256;
    case KV_GENERIC11: return true;
    case KV_GENERIC12:
    case KV_GENERIC22: return nb % 16 == 0;
    case KV_TILED: return default_variant(nb) == KV_TILED;
    default: return false;
  }
}

const char* variant_name(int v) {
  static const char* names[KV_COUNT] = {"staged32", "staged64", "staged128", "staged256",
                                        "generic1x1", "generic1x2", "generic2x2", "tiled"};
  return (v >= 0 && v < KV_COUNT) ? names[v] : "none";
}

size_t variant_smem(int v, int nb) {
  if (v == KV_TILED) return smem_tiled();
  return (v >= KV_STAGED32 && v <= KV_STAGED256) ? smem_staged(nb) : smem_generic(nb);
}

void set_default_variants(KParams& p) {
  for (int i = 0; i < kVariantSlots; i++) p.variant[i] = (int8_t)default_variant(i * 8);
}

int solver_threads() { return kThreads; }

// The kernel's limit of dynamic shared memory belongs to the device, not to a
// launch: it is always set to the same value, so a call on one host thread
// never lowers it between another thread's setting and its launch.  The
// launches and queries give their own size, which alone counts for occupancy.
static cudaError_t allow_smem() {
  constexpr int kLimit = 160 * 1024;
  return cudaFuncSetAttribute(rgf_solver_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLimit);
}

int solver_blocks_per_sm(size_t smem) {
  int nblk = 0;
  allow_smem();
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nblk, rgf_solver_kernel, kThreads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return nblk > 0 ? nblk : 1;
}

int solver_max_clusters(size_t smem, int cluster) {
  allow_smem();
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)cluster);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, rgf_solver_kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_solver(const KParams& p, const SolverShape& s, cudaStream_t st, bool set_attr) {
  if (set_attr) {
    const cudaError_t e = allow_smem();
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)s.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(s.groups * s.cluster));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = s.cluster > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, rgf_solver_kernel, p);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace rgf
