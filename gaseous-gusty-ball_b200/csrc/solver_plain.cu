// solver_plain.cu — the plain solve's kernels for hierarchies with a dense coarse map, a small single
// level or none, in a module of their own (solver_body.cuh).
#include "ggb_internal.h"
#include "ggb_solver.h"

namespace ggb {

namespace pcg_plain {
#include "solver_body.cuh"
}

const void *pcg_kernel_plain(int threads, bool batch) { return pcg_plain::kernel_of<false, false>(threads, batch); }

}  // namespace ggb
