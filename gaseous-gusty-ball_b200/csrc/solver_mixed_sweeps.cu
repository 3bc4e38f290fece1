// solver_mixed_sweeps.cu — the mixed-precision solve's kernels for hierarchies whose coarsest level is swept, in a module of their own (solver_body.cuh).
#include "ggb_internal.h"
#include "ggb_solver.h"

namespace ggb {

namespace pcg_mixed_sweeps {
#include "solver_body.cuh"
}

const void *pcg_kernel_mixed_sweeps(int threads, bool batch) { return pcg_mixed_sweeps::kernel_of<true, true>(threads, batch); }

}  // namespace ggb
