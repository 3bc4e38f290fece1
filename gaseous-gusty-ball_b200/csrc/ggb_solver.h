// ggb_solver.h — device descriptors of the multigrid-preconditioned CG solve.
#pragma once

#include "ggb_partials.h"
#include "ggb_stencil.cuh"

namespace ggb {

constexpr int kMaxLev = 12;

// Cells of a level up to which the levels from it down form the dense coarse map,
// and a single level is swept by one block in shared memory (N <= 16).
constexpr int kBlockLevelMax = 1536;

// Sparse rows of (index, weight bits) taps: step s of row r is tap[s * rows + r].
// glen: the steps that each 32 rows need (stored steps past a row's own taps
// have weight 0).
struct SparseOp {
    int rows, steps;
    const int2 *tap;
    const unsigned char *glen;
};

// One multigrid level on the device.  The level vectors are float in the plain
// solve and __half in the mixed-precision solve (SolveParams::mixed).
struct LevelDev {
    StencilDev S;
    const float *dinv;  // [n] 1 / sum of link weights
    void *b;            // [n] right-hand side (restricted residual; levels >= 1)
    void *xo;           // [n] V-cycle output of this level (levels >= 1)
    void *r;            // [n] residual after the pre-smooth
    // transfer to the next coarser level
    const int *ptap;    // [4n] coarse taps of each cell of this level
    const float *pw;    // [4n] their bilinear weights
    const int *rstart;  // [n_coarse+1] rows of R = P^T
    const int *ridx;    // fine cells of each row (ascending)
    const float *rw;    // weights of each row
    const float *rw16;  // [16][n_coarse] weights of the interior rows of R (coarse-major), or nullptr when
                        // the transfers do not follow the 4x4 / 2x2 index pattern
    SparseOp rst;       // the rows of R of the coarse ring cells (rw16) or of all coarse cells
    const int2 *ring_link;  // [6 nring][8] the ring cells' links (vcycle.cu)
    const int *ring_cell;   // [6 nring] ring cell | its on-face lanes << 24
};

// A coarsest level without a dense map, cut into parts (one per block) that
// sweep by themselves for `depth` sweeps between exchanges: each part holds its
// own cells and all cells within depth links of them, ordered by that distance.
// count[p][h]: cells of part p within h links; the rest is indexed [p][slot] or
// [p][link][slot] with kSweepSlots slots a part.
constexpr int kSweepSlots = 1024;
constexpr int kSweepDepth = 24;
struct SweepParts {
    int parts, depth;
    const int *count;          // [parts][kSweepDepth + 1]
    const int *cell;           // [parts][kSweepSlots]
    const unsigned short *nb;  // [parts][8][kSweepSlots] slots of the neighbours (of cells within depth - 1 links)
    const float *w;            // [parts][8][kSweepSlots]
};

// What levels_build (vcycle.cu) makes of a hierarchy, per precision.
struct LevelSet {
    const float *rw16[kMaxLev];
    SparseOp rst[kMaxLev];
    const int2 *ring_link[kMaxLev];
    const int *ring_cell[kMaxLev];
    const float *wpad[kMaxLev];  // nullptr: the grid's own
    void *b[kMaxLev], *xo[kMaxLev], *r[kMaxLev];
};

// Status bits of a solve (SolveResult::flags; also ggb_solve_flags).
enum {
    kSolveTimeout = 1,    // a grid barrier timed out (the solve was abandoned)
    kSolveNonFinite = 2,  // a NaN or Inf reached b.b, r.r, r.z or p.Ap
    kSolveBreakdown = 4,  // p.Ap <= 0: CG stopped early (upstream src/fluid.c:329-330 stops silently)
    kSolveMaxit = 8,      // maxit iterations without reaching the tolerance
};

struct SolveResult {
    int iters;
    int status;      // 0 ok, 1 barrier timeout
    double relres;
    int r_final;     // which r buffer holds the final residual (0: r, 1: r2)
    int flags;       // kSolve* bits
    unsigned long long ns;  // device time of the solve (%globaltimer, block 0 of the solve)
};

// Diagnostic records of a solve (device memory): up to cap (mark, ns) pairs.
struct SolveTrace {
    int n, cap;
    int all;  // stage marks: 1 from every block, 0 from the launch's block 0
    int pad;
    unsigned long long rec[1][2];  // [cap]
};

struct SolveParams {
    int mixed;           // 1: V-cycle vectors in FP16 with FP32 accumulation, flexible (Polak-Ribiere) CG;
                         //    0: FP32 vectors, FP64 accumulation
    int nlev;            // >= 1 when multigrid, 0 for the Jacobi preconditioner
    int nlev_grid;       // non-coarsest levels 0..nlev_grid-1 run grid-wide
    int coarse_on_grid;  // coarsest level swept grid-wide (else the dense map)
    int coarse_sweeps;   // Jacobi sweeps on the coarsest level (upstream: 60)
    int remove_mean;     // project the mean out of omega first
    int maxit;
    double tol;
    double total_area;
    LevelDev L[kMaxLev];
    const float *area;   // level-0 cell areas
    float *omega, *psi;
    float *r, *r2, *p, *p2, *Ap, *z;  // level-0 CG vectors (r / p ping-pong)
    float *z2;           // mixed: the previous z (z / z2 ping-pong for the flexible beta)
    SolveTrace *trace;   // optional: block 0 of the solve stamps %globaltimer at phase marks
    SolveTrace *stages;  // optional: ... at the start and end of every stencil phase
    double *part;        // [kPartSets][2][blocks] the blocks' sums at the last barriers
    GridBarrier *bar;
    SolveResult *res;
    // dense form of the V-cycle below the grid levels: xo_G = D b_G
    float *sw0, *sw1;    // the coarsest level's sweeps (coarse_on_grid)
    SweepParts sweep;    // (parts = 0: the level is too large)
    const float *dense;  // [nd][ld] row-major (rows padded with zeros to ld), or nullptr
    int nd, ld;          // cells of level nlev_grid; row stride, a multiple of 4
};

}  // namespace ggb
