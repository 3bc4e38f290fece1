// solver.cu — the Poisson solve K psi = -A omega as ONE persistent cooperative
// kernel: warm-started preconditioned conjugate gradients whose
// preconditioner is a symmetric multigrid V-cycle (damped-Jacobi smoother,
// bilinear prolongation P, restriction R = P^T, many-sweep Jacobi on the
// coarsest grid), with FP64 dot products and FP64 zero-mean projections.
//
// Upstream: src/fluid.c:41-160 (multigrid), :264-275 (mean), :290-358 (PCG).
// Two precisions share one kernel body (template parameter MP):
//   * plain (MP = false): the arithmetic of every vector update follows
//     upstream (FP32 vectors, FP64 accumulation of the stencil sums);
//   * mixed (MP = true): the V-cycle's level vectors and the coarse levels'
//     slot weights are rounded to FP16, every stencil sum, restriction and
//     prolongation accumulates in FP32, and the outer CG is flexible
//     (Polak-Ribiere beta = r.(z - z_prev) / rz_prev), which tolerates the
//     preconditioner's rounding; psi, omega, r, p, z stay FP32 and the dots, norms and mean
//     projections stay FP64.  FP16 holds about five decimal orders of
//     magnitude, less than the spread of a residual across the levels, so the
//     mixed V-cycle runs on scaled vectors: its input is multiplied by a power
//     of two that brings its RMS near 1/16, restriction carries a factor 1/4
//     and prolongation a factor 4 (so that every level's right-hand side stays at the input's
//     scale instead of growing 4x per level), and the output is scaled back.
//     All factors are powers of two (exact), and the V-cycle is linear, so they
//     change nothing but the range.
// The schedule is this library's:
//   * phases are separated by a bounded grid-wide barrier instead of host loops;
//   * each block owns a contiguous range of the cells; a stencil phase first
//     computes the (transformed) neighbour value of every cell of the range
//     plus its halo once into shared memory, then applies the stencil;
//   * p = z + beta p is recomputed inside K p, r - alpha Ap inside the level-0
//     pre-smooth, and the prolongation inside each level's post-smooth, which
//     saves grid barriers;
//   * interior rows of R and P use index arithmetic (no CSR indirection);
//   * the V-cycle below the grid levels (N <= 16, at most 1536 cells) is a
//     fixed linear map, precomputed once as a dense matrix and applied by all
//     blocks from L2.
#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <mutex>
#include <vector>

#include "ggb_internal.h"
#include "ggb_solver.h"

namespace ggb {

namespace pcg_setup {
#include "solver_body.cuh"
}
using namespace pcg_setup;

// solver_plain.cu, solver_plain_sweeps.cu, solver_mixed.cu, solver_mixed_sweeps.cu
const void *pcg_kernel_plain(int threads, bool batch);
const void *pcg_kernel_plain_sweeps(int threads, bool batch);
const void *pcg_kernel_mixed(int threads, bool batch);
const void *pcg_kernel_mixed_sweeps(int threads, bool batch);

// ---- setup kernels -------------------------------------------------------

// Column j of the dense map of levels l0..nlev-1: the block's V-cycle applied
// to the unit vector e_j, stored row-major D[row][j] (row stride ld).
__global__ void __launch_bounds__(kPB, 1) k_dense_columns(SolveParams P, int l0, float *D, int ld) {
    extern __shared__ __align__(16) unsigned char dyn[];
    float *smem = reinterpret_cast<float *>(dyn);
    const int nd = P.L[l0].S.n;
    for (int j = blockIdx.x; j < nd; j += gridDim.x) {
        SmemLevel lv[kMaxLev];
        carve_smem(P, l0, smem, lv);
        BLOCK_LOOP(c, nd) lv[l0].b[c] = c == j ? 1.0f : 0.0f;
        __syncthreads();
        vcycle_block_smem(P, l0, lv);
        BLOCK_LOOP(c, nd) D[(size_t)c * ld + j] = lv[l0].xo[c];
        __syncthreads();
    }
}

// ---------------------------------------------------------------- host

static SolveTrace *g_trace = nullptr, *g_stages = nullptr;
static int g_trace_cap = 0;
static bool g_stages_on = false;
void solve_trace_target(SolveTrace **trace, SolveTrace **stages) {
    *trace = g_trace;
    *stages = g_stages_on ? g_stages : nullptr;
}

int pcg_max_blocks() { return device_sm_count(); }

// Largest grid edge a solve accepts: a window holds a chunk and two halos of N + 1.
int pcg_max_grid_n() { return kMaxN; }

static const void *pcg_kernel(bool mixed, int threads, bool sweeps, bool batch) {
    if (mixed) return sweeps ? pcg_kernel_mixed_sweeps(threads, batch) : pcg_kernel_mixed(threads, batch);
    return sweeps ? pcg_kernel_plain_sweeps(threads, batch) : pcg_kernel_plain(threads, batch);
}

// Threads per block below which a planet's solve slows down by more than its share
// of warps: a single level that one block sweeps has a thread for every cell, with
// its links in registers, up to 512 cells (N = 9, 486 cells: 0.18 ms, with 384
// threads 0.74).
static int least_threads(const SolveParams &p) {
    return p.nlev == 1 && !p.coarse_on_grid && p.L[0].S.n > kPBNarrow ? kPB : kPBNarrow;
}

// Threads per block of a single solve.
static int pcg_threads(const SolveParams &p) {
    const int N = p.L[0].S.N;
    if (N >= kWideMinN) return kPBWide;
    return 6LL * N * N <= (long long)kNarrowCells * device_sm_count() ? least_threads(p) : kPB;
}

// ... of a batched launch over nblocks blocks.  With much work per block, loads and
// arithmetic bound a phase, not its barrier, and more warps keep more in flight.
// Work is counted in cells of the finest levels; a row of a dense map (kDenseWork
// cells) and a cell of a swept coarsest level (kSweepWork) weigh as much as so many,
// since few blocks have many of them: by cells alone, 45 planets of N = 32 (1870 a
// block, 467 rows) and 6 of N = 100 (2430, no rows) would count as equals.  Batched
// solves in us with 384 / 512 / 1024 threads, by work per block:
//   2 planets of N = 64, 540: 311 327 434; 4 of 64, 1080: 364 374 473
//   10 of N = 32, 1450: 385 343 443; 6 of 64, 1620: 436 409 533; 2 of 128, 1540: 493 525 631
//   12 of 64, 3240: 758 665 682; 5 of 128, 3840: 889 814 881; 6 of 100, 5470: 2534 2461 2465
//   2 of 256, 5520: 1155 1109 1181; 8 of 128, 6140: 1246 1132 1126; 24 of 64, 6480: 1313 1128 1033
//   45 of 32, 6540: 1263 1098 946; 20 of 25, 10600: 4184 4067 1762; 148 of 32, 21500: 3415 2995 2437
// One planet on the whole launch has fluid_step's choice (and so its sums).
constexpr int kDenseWork = 10, kSweepWork = 20;
constexpr int kNarrowWork = 1100, kWideWork = 5800;
int pcg_batch_threads(const SolveParams *prm, const std::vector<int> &planets, int nblocks) {
    if (planets.size() == 1 && nblocks >= pcg_batch_capacity()) return pcg_threads(prm[planets[0]]);
    long long work = 0;
    int least = kPBNarrow;
    for (int i : planets) {
        const SolveParams &p = prm[i];
        work += p.L[0].S.n;
        if (p.dense) work += (long long)kDenseWork * p.nd;
        if (p.coarse_on_grid) work += (long long)kSweepWork * p.L[p.nlev - 1].S.n;
        least = std::max(least, least_threads(p));
    }
    if (work > (long long)kWideWork * nblocks) return kPBWide;
    return work <= (long long)kNarrowWork * nblocks ? least : kPB;
}

// Blocks of a launch of `kernel`.  A variant is looked at (and with lazy loading
// brought to the device) when it is first launched: all 24 at once cost a program's
// first solve 40 ms.
static int blocks_resident(const void *kernel, int threads) {
    static std::mutex m;
    static std::vector<const void *> ready;
    std::lock_guard<std::mutex> lock(m);
    if (std::find(ready.begin(), ready.end(), kernel) == ready.end()) {
        GGB_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageBytes));
        int per = 0;
        GGB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, kStageBytes));
        if (per < 1) fail_msg("the solve kernel cannot be resident on this device (%zu B shared memory)", kStageBytes);
        ready.push_back(kernel);
    }
    return device_sm_count();  // one block per SM: more would only add arrivals to every barrier
}

// One solve launch; max_blocks > 0 caps its grid.
void pcg_launch(const SolveParams &prm, cudaStream_t s, int max_blocks) {
    SolveParams p = prm;
    void *args[] = {&p};
    const int threads = pcg_threads(p);
    const void *kernel = pcg_kernel(p.mixed != 0, threads, p.coarse_on_grid != 0, false);
    int grid = blocks_resident(kernel, threads);
    if (max_blocks > 0) grid = std::max(1, std::min(grid, max_blocks));
    GGB_CHECK(cudaMemsetAsync(&p.bar->count, 0, sizeof(unsigned int), s));
    GGB_CHECK(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, kStageBytes, s));
    GGB_LAUNCHED();
}

// Blocks of one batched solve launch that can be resident at once (the
// launch's capacity).
int pcg_batch_capacity() { return device_sm_count(); }

// One cooperative launch of nblocks blocks solving every planet of a batch
// (dev_prm: the planets' parameters; dev_bmap: block -> planet, block of the
// planet, blocks of the planet; sweeps: some planet has no dense map).  The
// planets' barrier counters must be zero.
void pcg_launch_batch(const SolveParams *dev_prm, const int4 *dev_bmap, int nblocks, int threads, bool mixed,
                      bool sweeps, cudaStream_t s) {
    const void *k = pcg_kernel(mixed, threads, sweeps, true);
    blocks_resident(k, threads);
    void *args[] = {(void *)&dev_prm, (void *)&dev_bmap};
    GGB_CHECK(cudaLaunchCooperativeKernel(k, dim3(nblocks), dim3(threads), args, kStageBytes, s));
    GGB_LAUNCHED();
}

// The dense map of the V-cycle of levels l0..nlev-1 (nd rows of stride ld).
float *pcg_dense_map(const SolveParams &prm, int l0, int ld) {
    SolveParams p = prm;
    const int nd = p.L[l0].S.n;
    float *D = (float *)dev_alloc(sizeof(float) * (size_t)nd * ld);
    size_t cells = 0;
    for (int l = l0; l < p.nlev; l++) cells += p.L[l].S.n;
    size_t smem = 4 * sizeof(float) * cells;
    GGB_CHECK(cudaFuncSetAttribute(k_dense_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    int grid = std::min(nd, 4 * device_sm_count());
    k_dense_columns<<<grid, kPB, smem, stream()>>>(p, l0, D, ld);
    GGB_LAUNCHED();
    GGB_CHECK(cudaStreamSynchronize(stream()));
    return D;
}

// ---- micro-benchmark of the grid barrier (additive entry point) ----------
// `rounds` barriers with a wait limit of limit_ns each; block `withhold`
// (-1: none) returns without arriving, so that the others' wait runs out:
// they raise the barrier's error flag, clear *ok and return.
__global__ void __launch_bounds__(kPB, 1) k_barrier_bench(GridBarrier *bar, int rounds, int *ok, int withhold,
                                                        unsigned long long limit_ns) {
    if ((int)blockIdx.x == withhold) return;
    for (int k = 0; k < rounds; k++)
        if (!grid_sync_limit(bar, limit_ns)) {
            if (threadIdx.x == 0) atomicExch(ok, 0);
            return;
        }
}

}  // namespace ggb

// One cooperative launch of `rounds` grid-wide barriers of the solve kernel's
// launch shape, each wait limited to limit_ms; block `withhold` (-1: none)
// never arrives.  Returns the launch's duration in ms (*ok = 1 when every
// barrier completed, 0 when the waits ran out and the kernel returned).
static double barrier_run(int rounds, int withhold, double limit_ms, int *ok_out) {
    using namespace ggb;
    GridBarrier *bar = (GridBarrier *)dev_alloc(sizeof(GridBarrier));
    int *ok = (int *)dev_alloc(sizeof(int));
    int one = 1;
    GGB_CHECK(cudaMemcpyAsync(ok, &one, sizeof(int), cudaMemcpyHostToDevice, stream()));
    int per = 0;
    GGB_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_barrier_bench, kPB, 0));
    int grid = device_sm_count() * std::min(per, 2);
    unsigned long long limit_ns = (unsigned long long)(limit_ms * 1e6);
    cudaEvent_t e0, e1;
    GGB_CHECK(cudaEventCreate(&e0));
    GGB_CHECK(cudaEventCreate(&e1));
    void *args[] = {&bar, &rounds, &ok, &withhold, &limit_ns};
    GGB_CHECK(cudaEventRecord(e0, stream()));
    GGB_CHECK(cudaLaunchCooperativeKernel((const void *)k_barrier_bench, dim3(grid), dim3(kPB), args, 0, stream()));
    GGB_LAUNCHED();
    GGB_CHECK(cudaEventRecord(e1, stream()));
    GGB_CHECK(cudaEventSynchronize(e1));
    float ms = 0;
    GGB_CHECK(cudaEventElapsedTime(&ms, e0, e1));
    int hok = 0;
    GGB_CHECK(cudaMemcpy(&hok, ok, sizeof(int), cudaMemcpyDeviceToHost));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    dev_free(bar);
    dev_free(ok);
    *ok_out = hok;
    return ms;
}

// Mean time of one grid-wide barrier of the solve kernel's launch shape, in
// microseconds (`rounds` barriers in one cooperative launch); -1 on timeout.
GGB_EXPORT double ggb_barrier_bench(int rounds) {
    int ok = 0;
    double ms = barrier_run(rounds, -1, 2000.0, &ok);
    return ok ? 1000.0 * ms / rounds : -1.0;
}

// Failure detection without a fault: one block of a cooperative launch never
// arrives at the grid barrier, the others wait limit_ms, raise the barrier's
// error flag and return.  Returns 1 when the waits ran out (0 if the barrier
// completed after all); *elapsed_ms gets the launch's duration.
GGB_EXPORT int ggb_barrier_timeout_probe(double limit_ms, double *elapsed_ms) {
    int ok = 1;
    double ms = barrier_run(1, 0, limit_ms, &ok);
    if (elapsed_ms) *elapsed_ms = ms;
    return ok ? 0 : 1;
}

static size_t trace_bytes(int cap) { return sizeof(ggb::SolveTrace) + 2 * sizeof(unsigned long long) * (size_t)cap; }

// Empties a trace buffer and sets its size and mode.
static void trace_reset(ggb::SolveTrace *t, int cap, int all) {
    ggb::SolveTrace head{};
    head.cap = cap;
    head.all = all;
    GGB_CHECK(cudaMemcpy(t, &head, offsetof(ggb::SolveTrace, rec), cudaMemcpyHostToDevice));
}

// Copies out up to cap records; their number.
static int trace_read(const ggb::SolveTrace *t, unsigned long long *out, int cap) {
    ggb::SolveTrace head{};
    GGB_CHECK(cudaMemcpy(&head, t, offsetof(ggb::SolveTrace, rec), cudaMemcpyDeviceToHost));
    const int n = std::min(std::min(head.n, head.cap), cap);
    if (n > 0) GGB_CHECK(cudaMemcpy(out, t->rec, 2 * sizeof(unsigned long long) * (size_t)n, cudaMemcpyDeviceToHost));
    return n;
}

// Diagnostics: the next solves record up to `cap` (mark, time in ns) pairs from
// block 0 (cap = 0 turns it off); ggb_solve_trace copies them out and returns
// how many were recorded.
GGB_EXPORT void ggb_solve_trace_enable(int cap) {
    using namespace ggb;
    sync();
    dev_free(g_trace);
    g_trace = cap > 0 ? (SolveTrace *)dev_alloc(trace_bytes(cap)) : nullptr;
    g_trace_cap = cap > 0 ? cap : 0;
    sync();
    if (g_trace) trace_reset(g_trace, g_trace_cap, 0);
}

GGB_EXPORT int ggb_solve_trace(unsigned long long *out, int cap) {
    using namespace ggb;
    sync();
    return g_trace ? trace_read(g_trace, out, cap) : 0;
}

// Diagnostics: enable = 1 makes block 0 of the next solves stamp the start
// (mark 1) and the end (2) of every stencil phase (mark, ns); enable = 2 makes
// every block stamp them (mark | block << 16, ns); enable = 0 stops and copies
// out up to cap records, returning their number.
GGB_EXPORT int ggb_stage_trace(int enable, unsigned long long *out, int cap) {
    using namespace ggb;
    constexpr int kRecords = 4096;
    sync();
    g_stages_on = enable != 0;
    if (!enable) return g_stages ? trace_read(g_stages, out, cap) : 0;
    if (!g_stages) {
        g_stages = (SolveTrace *)dev_alloc(trace_bytes(kRecords));
        sync();
    }
    trace_reset(g_stages, kRecords, enable == 2);
    return 0;
}
