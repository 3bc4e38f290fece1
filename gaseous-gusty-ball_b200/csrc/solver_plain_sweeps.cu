// solver_plain_sweeps.cu — the plain solve's kernels for hierarchies whose coarsest level is swept, in a module of their own (solver_body.cuh).
#include "ggb_internal.h"
#include "ggb_solver.h"

namespace ggb {

namespace pcg_plain_sweeps {
#include "solver_body.cuh"
}

const void *pcg_kernel_plain_sweeps(int threads, bool batch) { return pcg_plain_sweeps::kernel_of<false, true>(threads, batch); }

}  // namespace ggb
