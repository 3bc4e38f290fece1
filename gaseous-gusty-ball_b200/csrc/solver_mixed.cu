// solver_mixed.cu — the mixed-precision solve's kernels for hierarchies with a dense coarse map or a
// small single level, in a module of their own (solver_body.cuh).
#include "ggb_internal.h"
#include "ggb_solver.h"

namespace ggb {

namespace pcg_mixed {
#include "solver_body.cuh"
}

const void *pcg_kernel_mixed(int threads, bool batch) { return pcg_mixed::kernel_of<true, false>(threads, batch); }

}  // namespace ggb
