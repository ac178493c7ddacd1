// rgf_task_tiled.cu -- RGF task function for nb from 80 on (multiples of 8 without a staged form): tiled GEMM and
// Gauss-Jordan with the block size at run time, by one CTA or a cluster.
#include "rgf_solver.cuh"
#include "rgf_tasks.h"

namespace rgf {

__device__ __noinline__ void task_tiled(const KParams& p, int64_t t, double2* slot, Smem& sm,
                                         double2* dyn, Group grp) {
  solve_task<TiledOps<0>>(p, t, slot, sm, dyn, grp);
}

size_t smem_tiled() { return kBlockSmem; }

}  // namespace rgf
