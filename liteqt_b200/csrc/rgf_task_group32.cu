// rgf_task_group32.cu -- RGF task function for nb = 32 where a cluster of CTAs shares a task.
#include "rgf_solver.cuh"
#include "rgf_tasks.h"

namespace rgf {

__device__ __noinline__ void task_group32(const KParams& p, int64_t t, double2* slot, Smem& sm,
                                         double2* dyn, Group grp) {
  solve_task<TiledOps<32>>(p, t, slot, sm, dyn, grp);
}

}  // namespace rgf
