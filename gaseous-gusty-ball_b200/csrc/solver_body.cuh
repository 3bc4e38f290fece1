// solver_body.cuh — the device code of the persistent solve kernels k_pcg /
// k_pcg_batch (constants, stencil phases, V-cycle, PCG body), included inside a
// namespace of its own by solver.cu (set-up kernels and the host side) and by
// solver_{plain,mixed}{,_sweeps}.cu, which compile the solve kernels of one
// precision and coarse end each: a module is brought to the device as a whole, and
// all 24 kernels in one cost a program's first call 18 ms.
//
// Upstream: src/fluid.c:41-160 (multigrid), :264-275 (mean), :290-358 (PCG).
//
// A solve is a chain of some 130 phases of 3 to 10 us, each executed once per
// grid barrier; what bounds it is the latency of a phase (barrier, one round of
// loads, the instructions of one warp), not bytes.  So each kind of phase is
// inlined once, in loops over levels and iterations (a variant with 640 KB of code
// spent a seventh of its stall cycles on instruction fetch), no static operand is
// read between a barrier and the values that wait for it, and the window of a
// phase holds FP32 values only.  A step's solve in ms, before (values, four FP64
// weights and three inputs of every window cell staged anew in each phase) and now:
// N = 256 0.869, 0.701; N = 512 2.33, 1.84, mixed 2.23, 1.79; a cold solve to 1e-6:
// N = 64 0.459, 0.324.  The FP32 and FP16 roundings of every vector are unchanged.

constexpr int kPBNarrow = 384;   // threads per block of the persistent kernel on small grids
constexpr int kPB = 512;         // ... on ordinary ones
constexpr int kPBWide = 1024;     // ... where the fine levels' bytes outweigh the phases' latency
// Cells per block up to which blocks are narrow: with few cells a thread, a
// phase's time is its barrier and the issue of the warps' common part (sums,
// index arithmetic, block barriers), of which 12 warps have less than 16.  512 /
// 384 threads on 148 SMs, cold solves to 1e-6 in ms: N = 32 0.241 / 0.223, 64 0.348
// / 0.324, 128 0.543 / 0.518, 192 0.704 / 0.687, 256 (2657 cells) 0.840 / 0.824, 288
// 1.076 / 1.075, 384 1.56 / 1.66; 256 and 320 threads were slower from N = 128 on.
constexpr int kNarrowCells = 2700;
constexpr int kWideMinN = 480;    // 512 / 1024 threads, the same, ms: N = 448 1.99 / 2.05, 480 2.48 / 2.52, 512 2.54 / 2.47
// Cells a thread takes at once in the vector updates of a solve without multigrid:
// the loads of all before the stores of any, which the compiler cannot tell apart.
// 100 iterations in us, one cell / 3: N = 64 786 / 722, 256 2031 / 1381, 512 4680 /
// 3751.  2: 256 1414; 4: 1339, but the 512-thread kernels with multigrid spill (N =
// 320 2 % slower).
constexpr int kUpdate = 3;
constexpr int kChunk = 3072;      // cells of a stencil chunk
constexpr double kOmegaJ = 0.8;      // upstream MG_OMEGA
constexpr double kCorrScale = 1.0;  // upstream MG_CORR_SCALE
// Shared memory of a block: the value window of a chunk (FP32) and the slot
// weights of every grid level's window (each level of N <= 512 in its own
// region).
constexpr int kMaxN = 1535;
constexpr int kWinCap = (kChunk + 2 * kMaxN + 2 + 3) & ~3;  // whole 16-byte groups: the pool follows
static_assert(kWinCap >= 2 * kSweepSlots, "two buffers of a part's values");
static_assert(kWinCap >= 3 * kBlockLevelMax, "x, xo and b of a level that one block sweeps");
static_assert(kWinCap >= 2 * ((kBlockLevelMax + 3) & ~3), "b of the dense map in FP64");
constexpr int kSlotPool = 34816;
static_assert(kSlotPool >= 4 * (kChunk + 2 * kMaxN + 2 + 8), "a chunk's slot weights fit");
constexpr size_t kStageBytes = (kWinCap + (size_t)kSlotPool) * sizeof(float);

// Storage (V) and accumulation (A) types of the two precisions.
template <bool MP>
struct Prec {
    using V = float;
    using A = double;
};
template <>
struct Prec<true> {
    using V = __half;
    using A = float;
};

__device__ __forceinline__ float ldv(const float *p, int k) { return p[k]; }
__device__ __forceinline__ float ldv(const __half *p, int k) { return __half2float(p[k]); }
// four values, 4-element aligned
__device__ __forceinline__ float4 ldv4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float4 ldv4(const __half *p) {
    const uint2 u = *reinterpret_cast<const uint2 *>(p);
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void stv(float *p, int k, float v) { p[k] = v; }
__device__ __forceinline__ void stv(__half *p, int k, float v) { p[k] = __float2half_rn(v); }
// v as the storage type would hold it (rounded to FP16 in the mixed solve)
template <bool MP>
__device__ __forceinline__ float as_stored(float v) {
    return MP ? __half2float(__float2half_rn(v)) : v;
}
template <bool MP>
__device__ __forceinline__ typename Prec<MP>::V *lv(void *p) {
    return static_cast<typename Prec<MP>::V *>(p);
}

// This block's solve: its parameters, its place in the solve's grid (its
// "virtual grid": the whole launch, or the share of the blocks of a batched
// launch that one planet's solve runs on), and its ranges of the levels.
__shared__ SolveParams sP;
__shared__ int s_vgrid[2];
__shared__ int s_range[kMaxLev][2];
// Where a level's slot weights lie in the pool: offset, plane stride, and 1
// when the block's range is one chunk in a region of its own (loaded once per
// solve).
__shared__ int s_slot[kMaxLev][3];
__shared__ double s_warp[2][32];
__shared__ double s_total[2];  // the sums of the last vsync
__shared__ double s_late;      // a sum published at the barrier before (vsync)
__shared__ int s_epoch;        // barriers passed
__shared__ int s_ok;
__device__ __forceinline__ int vb() { return s_vgrid[0]; }
__device__ __forceinline__ int vnb() { return s_vgrid[1]; }
// The warps of the virtual grid numbered across its blocks (a short list of
// work items then takes a few warps of every block, next to other work, rather
// than all warps of a few blocks).
__device__ __forceinline__ int vwarp() { return (int)(threadIdx.x >> 5) * vnb() + vb(); }
__device__ __forceinline__ int vwarps() { return (int)(blockDim.x >> 5) * vnb(); }
extern __shared__ __align__(16) unsigned char s_dyn[];
__device__ __forceinline__ float *s_win() { return reinterpret_cast<float *>(s_dyn); }


__device__ __forceinline__ float *s_pool() { return s_win() + kWinCap; }

// Traces (diagnostics): (mark, %globaltimer) pairs into a SolveTrace, whose pointer
// is among the parameters, so that an untraced solve only tests it in shared memory.
__device__ __noinline__ void trace_mark(SolveTrace *t, unsigned long long mark) {
    if (threadIdx.x != 0) return;
    const int k = atomicAdd(&t->n, 1);
    if (k < t->cap) {
        t->rec[k][0] = mark;
        t->rec[k][1] = globaltimer_ns();
    }
}
// the schedule's phases, from block 0
#define TRACE(mark)                                                    \
    do {                                                               \
        if (sP.trace && vb() == 0) trace_mark(sP.trace, (mark));       \
    } while (0)
// the stencil phases' start (1) and end (2), from block 0 of the launch or all blocks
#define STAGE_MARK(mark)                                                                              \
    do {                                                                                              \
        if (sP.stages && (sP.stages->all || blockIdx.x == 0))                                         \
            trace_mark(sP.stages, (mark) | (sP.stages->all ? (unsigned long long)blockIdx.x << 16 : 0)); \
    } while (0)

// GRID_LOOP: over the block's virtual grid (only inside k_pcg / k_pcg_batch,
// which set it).
#define GRID_LOOP(c, n) for (int c = vb() * blockDim.x + threadIdx.x; c < (n); c += vnb() * blockDim.x)
// OWN_LOOP: the cells of this block's level-0 range
#define OWN_LOOP(c) for (int c = s_range[0][0] + (int)threadIdx.x; c < s_range[0][1]; c += blockDim.x)
#define BLOCK_LOOP(c, n) for (int c = threadIdx.x; c < (n); c += blockDim.x)

// Barrier of the blocks of one solve, and the sums of nv (0..2) values over all
// their threads.  A block leaves its sums in its row of the barrier's set of
// partials and arrives at the counter; after the barrier one warp reads all rows,
// in an order that depends on indices only, and leaves the totals in s_total in
// every block.  With late, the totals are not read here but by the next vsync,
// which must be called with fetch, by a second warp while the first one arrives
// and waits, and left in s_late: a sum whose only use is the convergence test
// costs no round trip that way.  What orders every read of a set before the next
// write to it: see ggb_partials.h.  (Arrival and sums in one message, every block
// polling every other's slot, measured 4 us a barrier against 1.7 + 1.2.)
// A row's values are asked for together (a lane of a 148-block solve has four or
// five; in a loop with a remainder they come one L2 round trip after the other),
// and those of both sums at once: a barrier with sums took 4.3 us, now 2.2.
constexpr int kRowLoads = 5;
template <int NV>
__device__ __forceinline__ void rows_total(const double *row, int nb, int lane, double (&v)[NV]) {
#pragma unroll
    for (int q = 0; q < NV; q++) v[q] = 0;
#pragma unroll 1
    for (int k0 = 0; k0 < nb; k0 += 32 * kRowLoads) {
        double x[NV][kRowLoads];
#pragma unroll
        for (int u = 0; u < kRowLoads; u++) {
            const int k = k0 + 32 * u + lane;
#pragma unroll
            for (int q = 0; q < NV; q++) x[q][u] = k < nb ? __ldcg(row + q * nb + k) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kRowLoads; u++)
#pragma unroll
            for (int q = 0; q < NV; q++) v[q] += x[q][u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NV; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
}
__device__ __forceinline__ bool vsync(int nv, double v0, double v1, bool late = false, bool fetch = false) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = vnb(), epoch = s_epoch;
    if (nv > 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v0 += __shfl_xor_sync(0xffffffffu, v0, o);
        if (lane == 0) s_warp[0][warp] = v0;
    }
    if (nv > 1) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        if (lane == 0) s_warp[1][warp] = v1;
    }
    __syncthreads();
    if (warp == 0) {
        if (nv > 0) {
            v0 = lane < (int)blockDim.x / 32 ? s_warp[0][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v0 += __shfl_xor_sync(0xffffffffu, v0, o);
        }
        if (nv > 1) {
            v1 = lane < (int)blockDim.x / 32 ? s_warp[1][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        }
        double *row = sP.part + part_set(epoch) * 2 * nb;
        int ok = 1;
        if (lane == 0) {
            if (nv > 0) row[vb()] = v0;
            if (nv > 1) row[nb + vb()] = v1;
            if (nb > 1) ok = grid_arrive_wait(sP.bar, (unsigned)nb, kBarrierTimeoutNs);
        }
        __syncwarp();
        if (nv > 1 && !late) {
            double t[2];
            rows_total<2>(row, nb, lane, t);
            v0 = t[0];
            v1 = t[1];
        } else if (nv > 0 && !late) {
            double t[1];
            rows_total<1>(row, nb, lane, t);
            v0 = t[0];
        }
        if (lane == 0) {
            s_total[0] = v0;
            s_total[1] = v1;
            s_ok = ok;
            s_epoch = epoch + 1;
        }
    } else if (warp == 1 && fetch) {
        double t[1];
        rows_total<1>(sP.part + part_set(epoch - 1) * 2 * nb, nb, lane, t);
        if (lane == 0) s_late = t[0];
    }
    __syncthreads();
    return s_ok != 0;
}

// This block's contiguous range of a level's n cells (face-major), the same
// number for every block whatever faces they lie on: the boundary-ring cells are
// dealt over the grid apart from the ranges.  (With whole blocks per face a solve
// on 11 blocks took as long as on 6: 10 planets of 64 to 256 cells an edge, whose
// shares move by a block from run to run, 1.71 to 2.27 ms; this way 1.63 to 1.73.)
__device__ __forceinline__ void block_range(int n, int &c0, int &c1) {
    c0 = (int)(((long long)n * vb()) / vnb());
    c1 = (int)(((long long)n * (vb() + 1)) / vnb());
}

__device__ __forceinline__ void cp_async16(float *dst, const float *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Starts the copy of the slot weights of the window of chunk [s0, s1) of level
// l: cell k of plane p at pool[offset + p * stride + k - (s0 - N - 1) + shift],
// shift = the cells by which the copy starts before the window for 16-byte
// alignment.
__device__ __forceinline__ int slot_shift(const StencilDev &S, int s0) { return (s0 - S.N - 1 + S.pad) & 3; }
__device__ __noinline__ void slots_load(int l, int s0, int s1) {
    const StencilDev &S = sP.L[l].S;
    const int a = (s0 - S.N - 1 + S.pad) & ~3, groups = (s1 - s0 + 2 * (S.N + 1) + 3 + 3) >> 2;
    float *dst = s_pool() + s_slot[l][0];
    const int cap = s_slot[l][1];
    for (int p = 0; p < 4; p++)
        for (int k = 4 * threadIdx.x; k < 4 * groups; k += 4 * blockDim.x)
            if (a + k + 4 <= S.wplane) cp_async16(dst + p * cap + k, S.wpad + (size_t)p * S.wplane + a + k);
}

// Ranges of every level, slot regions of level 0 and the grid levels, and the
// slot weights that stay in shared memory for the whole solve (their copies
// complete at the first stencil phase's wait).
__device__ __noinline__ void block_setup() {
    const int levels = max(sP.nlev, 1), slots = max(sP.nlev_grid, 1);
    if (threadIdx.x == 0) {
        int at = 0;
        bool shared = false;
        for (int l = 0; l < levels; l++) {
            const StencilDev &S = sP.L[l].S;
            int c0, c1;
            block_range(S.n, c0, c1);
            s_range[l][0] = c0;
            s_range[l][1] = c1;
            if (l >= slots) continue;
            const int cap = (min(c1 - c0, kChunk) + 2 * (S.N + 1) + 8 + 3) & ~3;
            const bool own = at + 4 * cap <= kSlotPool;
            shared |= !own;
            s_slot[l][0] = own ? at : 0;
            s_slot[l][1] = cap;
            s_slot[l][2] = own && c1 - c0 <= kChunk;
            if (own) at += 4 * cap;
        }
        if (shared) s_slot[0][2] = 0;  // another level's weights pass through level 0's region
    }
    __syncthreads();
    for (int l = 0; l < slots; l++)
        if (s_slot[l][2]) slots_load(l, s_range[l][0], s_range[l][1]);
}

// K x at interior cell c from the window (x[k], k = cell index) and the slot
// weights w0..w3 (indexed by cell) in shared memory.
// (A slot weight is finite and not negative: widening it to FP64 by its bits, with 2^-127 for
// 0, takes three integer instructions in place of a conversion at a quarter of
// their rate.)
__device__ __forceinline__ double widen(float w, double) {
    const unsigned b = __float_as_uint(w);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}
__device__ __forceinline__ float widen(float w, float) { return w; }
template <class A>
__device__ __forceinline__ A apply_window(int c, int N, const float *x, const float *w0, const float *w1,
                                          const float *w2, const float *w3) {
    const A xc = x[c];
    A s = widen(w0[c], A()) * (xc - (A)x[c + 1]);
    s += widen(w1[c], A()) * (xc - (A)x[c + N]);
    s += widen(w2[c], A()) * (xc - (A)x[c + N + 1]);
    s += widen(w3[c], A()) * (xc - (A)x[c + N - 1]);
    s += widen(w0[c - 1], A()) * (xc - (A)x[c - 1]);
    s += widen(w1[c - N], A()) * (xc - (A)x[c - N]);
    s += widen(w2[c - N - 1], A()) * (xc - (A)x[c - N - 1]);
    s += widen(w3[c - N + 1], A()) * (xc - (A)x[c - N + 1]);
    return s;
}

__device__ __forceinline__ bool is_ring(const StencilDev &S, int c) {
    int f, i, j;
    cell_fij(S, c, f, i, j);
    return i == 0 || j == 0 || i == S.N - 1 || j == S.N - 1;
}

// cell(c, x(c), (K x)(c)) for every cell of level l: x(k) = load(k) is FP32; the
// sums are FP64 in the plain solve and FP32 in the mixed one, there in the order
// of the links (on the face E, N, NE, NW, W, S, SW, SE, then the sum of those
// that leave it).  Boundary-ring cells take eight adjacent threads of the
// virtual grid each, one per link.  The other cells of this block's range go in
// chunks: the values of the chunk and N + 1 cells on either side to shared
// memory, each computed once, and the slot weights by cp.async; then eight links
// per cell from shared memory.  Bound by latency: a barrier, one round of loads
// and the reduction, since nothing static is read after the barrier when the
// range is one chunk (up to N = 256), and by the loads' bandwidth beyond.  Ends
// with a block barrier.
struct RingPre {  // a thread's first ring link, read before the grid barrier
    int2 q;
    int own;      // ring cell | its on-face lanes << 24
};
__device__ __forceinline__ void ring_load(const LevelDev &L, int e, RingPre &R) {
    R.q = __ldg(L.ring_link + e);
    R.own = __ldg(L.ring_cell + (e >> 3));
}
__device__ __forceinline__ void ring_prefetch(int l, RingPre &R) {
    const LevelDev &L = sP.L[l];
    ring_load(L, min(32 * vwarp() + (int)(threadIdx.x & 31), 48 * L.S.nring - 1), R);
}
template <bool MP, class Load, class Cell>
__device__ __forceinline__ void stencil_phase(int l, RingPre &R, Load load, Cell cell) {
    using A = typename Prec<MP>::A;
    const LevelDev &L = sP.L[l];
    const StencilDev &S = L.S;
    const int N = S.N, n = S.n, bs = blockDim.x, tid = threadIdx.x, lane = tid & 31;
    const int c0 = s_range[l][0], c1 = s_range[l][1];
    STAGE_MARK(1);
    const int total = 48 * S.nring, stride = 32 * vwarps();
#pragma unroll 1
    for (int e0 = 32 * vwarp(); e0 < total; e0 += stride) {
        RingPre next = R;  // the next links beside this round's values: few blocks take many rounds
        if (e0 + stride < total) ring_load(L, min(e0 + stride + lane, total - 1), next);
        const int c = R.own & 0xffffff;
        const float xo = load(c), xn = load(R.q.x);
        const A d = (A)xo - (A)xn, w = (A)__int_as_float(R.q.y);
        A v;
        if (MP) {
            const unsigned on = (unsigned)R.own >> 24;
            A wk[kMaxNb], dk[kMaxNb], t = 0;
#pragma unroll
            for (int k = 0; k < kMaxNb; k++) {
                const A wl = __shfl_sync(0xffffffffu, w, k, 8);
                dk[k] = __shfl_sync(0xffffffffu, d, k, 8);
                wk[k] = on >> k & 1u ? wl : 0;
                if (!(on >> k & 1u)) t += wl * dk[k];
            }
            v = wk[0] * dk[0];  // apply_window's chain
            v += wk[1] * dk[1];
            v += wk[2] * dk[2];
            v += wk[3] * dk[3];
            v += wk[4] * dk[4];
            v += wk[5] * dk[5];
            v += wk[6] * dk[6];
            v += wk[7] * dk[7];
            v += t;
        } else {
            v = w * d;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (e0 + lane < total && (lane & 7) == 0) cell(c, xo, v);
        R = next;
    }
    float *win = s_win();
#pragma unroll 1
    for (int s0 = c0; s0 < c1; s0 += kChunk) {
        const int s1 = min(c1, s0 + kChunk);
        const int w0 = s0 - N - 1, w1 = s1 + N + 1;  // cells outside [0, n) stage as zeros
        if (!s_slot[l][2]) slots_load(l, s0, s1);
#pragma unroll 4
        for (int k = w0 + tid; k < w1; k += bs) win[k - w0] = k >= 0 && k < n ? load(k) : 0.f;
        cp_async_wait();
        __syncthreads();
        const float *x = win - w0;
        const int cap = s_slot[l][1];
        const float *wE = s_pool() + s_slot[l][0] + slot_shift(S, s0) - w0;
#pragma unroll 1
        for (int c = s0 + tid; c < s1; c += bs)
            if (!is_ring(S, c))
                cell(c, x[c], apply_window<A>(c, N, x, wE, wE + cap, wE + 2 * cap, wE + 3 * cap));
        __syncthreads();
    }
    STAGE_MARK(2);
}

// ---- sparse rows ------------------------------------------------------------

// The sum of a row's products, each rounded to FP32: in FP64 (plain), or as an
// FP32 FMA chain in the order of the taps (mixed).
template <bool MP>
struct DotAcc {
    typename Prec<MP>::A a = 0;
    __device__ __forceinline__ void add(float w, float x) {
        if (MP)
            a = __fmaf_rn(w, x, (float)a);
        else
            a += (typename Prec<MP>::A)__fmul_rn(w, x);
    }
};

// The first taps of this thread's first row of an operator: they do not change
// from cycle to cycle, so they are read before the grid barrier that the
// operator's input waits for.
constexpr int kPre = 8;
struct Taps {
    int2 q[kPre];
    int len;
};
__device__ __forceinline__ void sp_prefetch(const SparseOp &op, Taps &T) {
    const int total = op.rows;
    const int e0 = min(32 * vwarp(), (total - 1) & ~31), e = min(e0 + (int)(threadIdx.x & 31), total - 1);
    T.len = __ldg(op.glen + (e0 >> 5));
#pragma unroll
    for (int u = 0; u < kPre; u++)
        T.q[u] = u < op.steps ? __ldg(op.tap + (size_t)u * total + e) : make_int2(0, 0);
}

// put(row, sum over the row's taps of weight * get(index)), rows spread over
// the virtual grid, one thread per row; T: sp_prefetch's.  Bound by latency (a
// gather round per kPre taps, the next taps in flight beside it).
template <bool MP, class Get, class Put>
__device__ __forceinline__ void sp_rows(const SparseOp &op, Taps &T, Get get, Put put) {
    const int total = op.rows, lane = threadIdx.x & 31, steps = op.steps;
    const int stride = 32 * vwarps();
    const int2 *const tap = op.tap;
    int e0 = 32 * vwarp(), s = 0;
    DotAcc<MP> acc;
#pragma unroll 1
    while (e0 < total) {
        float x[kPre];
#pragma unroll
        for (int u = 0; u < kPre; u++) x[u] = get(T.q[u].x);
        // the next taps: of this row, or the first of the thread's next row
        // (rows past the end repeat the last element; their sums are unused)
        const bool more = s + kPre < T.len;
        const int en = more ? e0 : e0 + stride, sn = more ? s + kPre : 0;
        Taps W;
        W.len = T.len;
        if (en < total) {
            const int2 *t = tap + min(en + lane, total - 1);
            if (!more) W.len = __ldg(op.glen + (en >> 5));
#pragma unroll
            for (int u = 0; u < kPre; u++)
                W.q[u] = sn + u < steps ? __ldg(t + (size_t)(sn + u) * total) : make_int2(T.q[0].x, 0);
        }
#pragma unroll
        for (int u = 0; u < kPre; u++) acc.add(__int_as_float(T.q[u].y), x[u]);
        if (!more) {
            if (e0 + lane < total) put(e0 + lane, (float)acc.a);
            acc = DotAcc<MP>();
        }
        T = W;
        e0 = en;
        s = sn;
    }
}

// ---- setup: the coarse levels inside one block -------------------------------

// (R r_fine) at coarse cell c (the CSR row of R = P^T).
__device__ __forceinline__ float restrict_value(const LevelDev &F, const float *r, int c) {
    const int k0 = __ldg(F.rstart + c), k1 = __ldg(F.rstart + c + 1);
    double acc = 0;
    for (int k = k0; k < k1; k++) acc += (double)(__ldg(F.rw + k) * r[__ldg(F.ridx + k)]);
    return (float)acc;
}

// x + P xc at fine cell i.
__device__ __forceinline__ float prolong_value(const LevelDev &F, const float *x, const float *xc, int i) {
    const float4 w = __ldg(reinterpret_cast<const float4 *>(F.pw) + i);
    const int4 t = __ldg(reinterpret_cast<const int4 *>(F.ptap) + i);
    const float s = w.x * xc[t.x] + w.y * xc[t.y] + w.z * xc[t.z] + w.w * xc[t.w];
    return x[i] + (float)(kCorrScale * s);
}

// One damped-Jacobi sweep of src at cell c.
__device__ __forceinline__ float jacobi_cell(const StencilDev &S, const float *dinv, float bc, const float *src,
                                             int c) {
    auto X = [&](int k) -> double { return (double)src[k]; };
    const float xc = src[c];
    const float rc = (float)(bc - apply_k(S, c, (double)xc, X));
    return xc + (float)(kOmegaJ * __ldg(dinv + c) * rc);
}

// The V-cycle of the coarse levels on FP32 vectors in shared memory (the dense
// map's columns; the transfers' factors 1/4 and 4 cancel within it).

struct SmemLevel {
    float *x, *xo, *b, *r;
};

__device__ void carve_smem(const SolveParams &P, int l0, float *smem, SmemLevel *lv_) {
    float *q = smem;
    for (int l = l0; l < P.nlev; l++) {
        int n = P.L[l].S.n;
        lv_[l].x = q;
        lv_[l].xo = q + n;
        lv_[l].b = q + 2 * n;
        lv_[l].r = q + 3 * n;
        q += 4 * n;
    }
}

// Coarsest level: `sweeps` Jacobi sweeps from 0; result in V.xo.  When every
// cell has its own thread, the cell's links, 1/diag and b stay in registers.
__device__ __forceinline__ void coarsest_smem(const LevelDev &L, const SmemLevel &V, int sweeps) {
    const int n = L.S.n;
    BLOCK_LOOP(c, n) V.x[c] = 0.f;
    __syncthreads();
    float *src = V.x, *dst = V.xo;
    if (n <= (int)blockDim.x) {
        const int c = threadIdx.x;
        int nb[kMaxNb];
        float wv[kMaxNb];
        float bc = 0.f, dv = 0.f;
        if (c < n) {
            cell_links(L.S, c, nb, wv);
            bc = V.b[c];
            dv = __ldg(L.dinv + c);
        }
        for (int s = 0; s < sweeps; s++) {
            if (c < n) {
                float xc = src[c];
                double xd = xc, acc = 0;
#pragma unroll
                for (int k = 0; k < kMaxNb; k++) acc += (double)wv[k] * (xd - (double)src[nb[k]]);
                float rc = (float)(bc - acc);
                dst[c] = xc + (float)(kOmegaJ * dv * rc);
            }
            __syncthreads();
            float *t = src;
            src = dst;
            dst = t;
        }
    } else {
        for (int s = 0; s < sweeps; s++) {
            BLOCK_LOOP(c, n) dst[c] = jacobi_cell(L.S, L.dinv, V.b[c], src, c);
            __syncthreads();
            float *t = src;
            src = dst;
            dst = t;
        }
    }
    if (src != V.xo) {
        BLOCK_LOOP(c, n) V.xo[c] = src[c];
        __syncthreads();
    }
}

// Levels l0..nlev-1 of the V-cycle inside this block, on vectors in shared
// memory.  b of level l0 is lv_[l0].b on entry; xo of level l0 is left in
// lv_[l0].xo.
__device__ __forceinline__ void vcycle_block_smem(const SolveParams &P, int l0, SmemLevel *lv_) {
    const int last = P.nlev - 1;
    for (int l = l0; l < last; l++) {
        const LevelDev &L = P.L[l];
        const float *b = lv_[l].b;
        float *lx = lv_[l].x, *lr = lv_[l].r;
        BLOCK_LOOP(c, L.S.n) {
            auto X = [&](int k) -> double { return (double)(float)(kOmegaJ * __ldg(L.dinv + k) * b[k]); };
            float bc = b[c];
            float xc = (float)(kOmegaJ * __ldg(L.dinv + c) * bc);
            double kx = apply_k(L.S, c, (double)xc, X);
            lx[c] = xc;
            lr[c] = (float)(bc - kx);
        }
        __syncthreads();
        BLOCK_LOOP(c, P.L[l + 1].S.n) lv_[l + 1].b[c] = restrict_value(L, lr, c);
        __syncthreads();
    }
    coarsest_smem(P.L[last], lv_[last], P.coarse_sweeps);
    for (int l = last - 1; l >= l0; l--) {
        const LevelDev &L = P.L[l];
        const float *xc = lv_[l + 1].xo;
        BLOCK_LOOP(i, L.S.n) lv_[l].x[i] = prolong_value(L, lv_[l].x, xc, i);
        __syncthreads();
        BLOCK_LOOP(c, L.S.n) lv_[l].xo[c] = jacobi_cell(L.S, L.dinv, lv_[l].b[c], lv_[l].x, c);
        __syncthreads();
    }
}

// ---- the coarse end of the V-cycle ------------------------------------------

// put(row, sum_j D[row][j] b[j]) for every row of the dense map, FP64 sums: each
// half of a row over the lanes of a warp, then the two halves; get4(j) gives
// b[j..j+3] (anything past the end: the map's padding columns are 0).  Bound by
// reading D from L2 (9.4 MB at nd = 1536).  D holds FP32 values (the V-cycle it was
// built from works on FP32 vectors), so FP32 storage loses nothing against FP64 and
// halves the bytes.
//
// On the whole GPU a warp has one or two halves: two adjacent warps per row, 16-byte
// loads, the first kDensePre of a lane before the grid barrier.  On a batched
// planet's few blocks it has dozens, and each such round would be a latency, a
// reduction and two block barriers, and convert b anew: from three rounds on
// (BATCH) b goes to shared memory once as FP64 and every warp takes whole rows.
// Same sums.  Batched solves in us, rounds / rows: 12 planets of N = 64 (512 threads)
// 894 / 665; 24 of N = 64 (1024) 1292 / 1033; 60 of N = 32 2028 / 1267, 148 3924 /
// 2437; with a loop over a row's loads instead of kRowAhead asked for together (a
// remainder goes one L2 round trip at a time) 689, 1116, 1490 and 2789, and 148 of N =
// 16 647 where it is 531.  4 of N = 64 (384): whole rows from nine rounds on 405, from
// three 375.  (In the kernels of single solves the rows' registers cost N = 512 1.5 %.)
constexpr int kDensePre = 6;
constexpr int kRowAhead = 3;  // 16-byte loads of either half of a row in flight (BATCH)
struct DenseTaps {
    float4 w[kDensePre];
};
__device__ __forceinline__ void dense_prefetch(DenseTaps &T) {
    const int ld4 = sP.ld >> 2, h4 = (ld4 + 1) >> 1, lane = threadIdx.x & 31;
    const int part = min(vb() * ((int)blockDim.x >> 5) + (int)(threadIdx.x >> 5), 2 * sP.nd - 1);
    const int j0 = (part & 1) * h4, j1 = min(ld4, j0 + h4);
    const float4 *d = reinterpret_cast<const float4 *>(sP.dense) + (size_t)(part >> 1) * ld4;
#pragma unroll
    for (int u = 0; u < kDensePre; u++)
        T.w[u] = j0 + lane + 32 * u < j1 ? __ldg(d + j0 + lane + 32 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
}
template <bool BATCH, class Get4, class Put>
__device__ __forceinline__ void dense_rows(const DenseTaps &T, Get4 get4, Put put) {
    __shared__ double s_half[32];
    const int nd = sP.nd, ld4 = sP.ld >> 2, h4 = (ld4 + 1) >> 1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = (int)blockDim.x >> 5;  // even
    const float4 *dense = reinterpret_cast<const float4 *>(sP.dense);
    if (BATCH && nd > vnb() * nw) {
        double2 *b0 = reinterpret_cast<double2 *>(s_win()), *b1 = b0 + ld4;
        BLOCK_LOOP(j, ld4) {
            const float4 b = get4(4 * j);
            b0[j] = make_double2(b.x, b.y);
            b1[j] = make_double2(b.z, b.w);
        }
        __syncthreads();
#pragma unroll 1
        for (int row = vb() * nw + warp; row < nd; row += vnb() * nw) {
            const float4 *d = dense + (size_t)row * ld4;
            double v0 = 0, v1 = 0;
            auto add = [&](double &v, float4 w, int j) {
                const double2 p = b0[j], q = b1[j];
                v += (double)w.x * p.x;
                v += (double)w.y * p.y;
                v += (double)w.z * q.x;
                v += (double)w.w * q.y;
            };
#pragma unroll 1
            for (int jb = lane; jb - lane < h4; jb += 32 * kRowAhead) {
                float4 w0[kRowAhead], w1[kRowAhead];
#pragma unroll
                for (int u = 0; u < kRowAhead; u++) {
                    const int j = min(jb + 32 * u, h4 - 1);
                    w0[u] = __ldg(d + j);
                    w1[u] = __ldg(d + min(j + h4, ld4 - 1));
                }
#pragma unroll
                for (int u = 0; u < kRowAhead; u++) {
                    const int j = jb + 32 * u;
                    if (j < h4) add(v0, w0[u], j);
                    if (j < h4 && j + h4 < ld4) add(v1, w1[u], j + h4);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v0 += __shfl_xor_sync(0xffffffffu, v0, o);
                v1 += __shfl_xor_sync(0xffffffffu, v1, o);
            }
            if (lane == 0) put(row, v0 + v1);
        }
        return;
    }
    bool first = true;
#pragma unroll 1
    for (int base = vb() * nw; base < 2 * nd; base += vnb() * nw) {
        const int part = min(base + warp, 2 * nd - 1);
        const int j1 = min(ld4, ((part & 1) + 1) * h4);
        const float4 *d = dense + (size_t)(part >> 1) * ld4;
        double v = 0;
        auto add = [&](float4 w, float4 b) {
            v += (double)w.x * (double)b.x;
            v += (double)w.y * (double)b.y;
            v += (double)w.z * (double)b.z;
            v += (double)w.w * (double)b.w;
        };
        int j = (part & 1) * h4 + lane;
        if (first) {
#pragma unroll
            for (int u = 0; u < kDensePre; u++) add(T.w[u], get4(4 * min(j + 32 * u, ld4 - 1)));
            j += 32 * kDensePre;
        }
        first = false;
#pragma unroll 4
        for (; j < j1; j += 32) add(__ldg(d + j), get4(4 * j));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) s_half[warp] = v;
        __syncthreads();
        if (lane == 0 && !(warp & 1) && base + warp < 2 * nd) put(part >> 1, s_half[warp] + s_half[warp + 1]);
        __syncthreads();
    }
}

// The coarsest level's damped-Jacobi sweeps from 0 (upstream src/fluid.c:118-137)
// for a level without a dense map: FP32, each sweep rounded to the storage type;
// put(c, x) with the result.  False on abort.  (Only in the kernels' SWEEPS
// variants: in the same kernel as the dense map, inlined or as a call, its
// registers cost the solve at N = 256 9 to 12 %.)
//
// A level cut into parts (SweepParts) sweeps `depth` times between exchanges, in
// shared memory with the links in registers: after an exchange a part holds every
// cell within depth links of its own, and each sweep is valid one link less far
// out, so cells near a part's edge are swept by several blocks, to the same
// values.  60 sweeps of 3750 cells (N = 100: 25) then take 7 grid barriers instead
// of 60, and the coarsest level 38 us a V-cycle instead of 250.  A larger level,
// or a solve on fewer blocks than parts, sweeps grid-wide with a barrier per
// sweep; with a thread for every cell its links stay in registers there too.
template <bool MP, int TPB, class GetB, class Put>
__device__ __forceinline__ bool coarse_sweeps(const LevelDev &L, GetB getb, Put put) {
    const int n = L.S.n, sweeps = sP.coarse_sweeps;
    float *src = sP.sw0, *dst = sP.sw1;
    if (sP.sweep.parts > 0 && vnb() >= sP.sweep.parts) {
        constexpr int kPer = (kSweepSlots + TPB - 1) / TPB;  // slots per thread
        const SweepParts &W = sP.sweep;
        const int part = vb(), depth = W.depth, bs = blockDim.x;
        const bool mine = part < W.parts;
        const int *cnt = W.count + (size_t)(mine ? part : 0) * (kSweepDepth + 1);
        const int own = mine ? __ldg(cnt) : 0, all = mine ? __ldg(cnt + depth) : 0;
        float *xs = s_win(), *xd = xs + kSweepSlots;
        int cell[kPer];
        unsigned nb[kPer][kMaxNb / 2];
        float wv[kPer][kMaxNb], bc[kPer];
        double od[kPer];
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const int s = threadIdx.x + u * bs;
            if (s >= all) continue;
            cell[u] = __ldg(W.cell + (size_t)part * kSweepSlots + s);
#pragma unroll
            for (int k = 0; k < kMaxNb; k++) {
                const size_t at = ((size_t)part * kMaxNb + k) * kSweepSlots + s;
                const unsigned o = __ldg(W.nb + at);
                nb[u][k / 2] = k & 1 ? nb[u][k / 2] | o << 16 : o;
                wv[u][k] = __ldg(W.w + at);
            }
            bc[u] = getb(cell[u]);
            od[u] = kOmegaJ * __ldg(L.dinv + cell[u]);
            xs[s] = as_stored<MP>((float)(od[u] * bc[u]));  // the first sweep
        }
        __syncthreads();
#pragma unroll 1
        for (int done = 1;;) {
            const int run = min(depth, sweeps - done);
#pragma unroll 1
            for (int left = run - 1; left >= 0; left--) {
                const int lim = mine ? __ldg(cnt + left) : 0;
#pragma unroll
                for (int u = 0; u < kPer; u++) {
                    const int s = threadIdx.x + u * bs;
                    if (s >= lim) continue;
                    const float xc = xs[s];
                    double acc = 0;
#pragma unroll
                    for (int k = 0; k < kMaxNb; k++)
                        acc += (double)wv[u][k] *
                               ((double)xc - (double)xs[k & 1 ? nb[u][k / 2] >> 16 : nb[u][k / 2] & 0xffffu]);
                    const float rc = (float)(bc[u] - acc);
                    xd[s] = as_stored<MP>(xc + (float)(od[u] * rc));
                }
                __syncthreads();
                float *t = xs;
                xs = xd;
                xd = t;
            }
            done += run;
            if (done >= sweeps) break;
            // own values out, those around the part in
#pragma unroll
            for (int u = 0; u < kPer; u++)
                if ((int)threadIdx.x + u * bs < own) dst[cell[u]] = xs[threadIdx.x + u * bs];
            if (!vsync(0, 0, 0)) return false;
            const int need = mine ? __ldg(cnt + min(depth, sweeps - done)) : 0;
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                const int s = threadIdx.x + u * bs;
                if (s >= own && s < need) xs[s] = dst[cell[u]];
            }
            __syncthreads();
            float *t = src;
            src = dst;
            dst = t;
        }
#pragma unroll
        for (int u = 0; u < kPer; u++)
            if ((int)threadIdx.x + u * bs < own) put(cell[u], xs[threadIdx.x + u * bs]);
        __syncthreads();
        return true;
    }
    if (n <= vnb() * (int)blockDim.x) {
        const int c = vb() * blockDim.x + threadIdx.x;
        int nb[kMaxNb];
        float wv[kMaxNb], bc = 0.f, xc = 0.f;
        double od = 0;
        if (c < n) {
            cell_links(L.S, c, nb, wv);
            bc = getb(c);
            od = kOmegaJ * __ldg(L.dinv + c);
            xc = as_stored<MP>((float)(od * bc));  // the first sweep
            src[c] = xc;
        }
#pragma unroll 1
        for (int s = 1; s < sweeps; s++) {
            if (!vsync(0, 0, 0)) return false;
            if (c < n) {
                float v[kMaxNb];
#pragma unroll
                for (int k = 0; k < kMaxNb; k++) v[k] = src[nb[k]];
                double acc = 0;
#pragma unroll
                for (int k = 0; k < kMaxNb; k++) acc += (double)wv[k] * ((double)xc - (double)v[k]);
                const float rc = (float)(bc - acc);
                xc = as_stored<MP>(xc + (float)(od * rc));
                dst[c] = xc;
            }
            float *t = src;
            src = dst;
            dst = t;
        }
        if (c < n) put(c, xc);
        return true;
    }
    GRID_LOOP(c, n) src[c] = as_stored<MP>((float)(kOmegaJ * __ldg(L.dinv + c) * getb(c)));
#pragma unroll 1
    for (int s = 1; s < sweeps; s++) {
        if (!vsync(0, 0, 0)) return false;
        GRID_LOOP(c, n) dst[c] = as_stored<MP>(jacobi_cell(L.S, L.dinv, getb(c), src, c));
        float *t = src;
        src = dst;
        dst = t;
    }
    GRID_LOOP(c, n) put(c, src[c]);
    return true;
}

// ---- the grid levels of the V-cycle ------------------------------------------

// The pre-smoothed iterate from 0 at cell k: w D^-1 b (as stored).
template <bool MP>
__device__ __forceinline__ float presmooth_x(float dinv, float b) {
    if (MP) return as_stored<true>(0.8f * dinv * b);
    return (float)(kOmegaJ * dinv * b);
}

// The restriction's operands of this thread's first coarse cell and ring row,
// read before the grid barrier.
struct RestrictPre {
    float w[16];
    Taps t;
};
__device__ __forceinline__ void restrict_prefetch(int l, RestrictPre &R) {
    const int nc = sP.L[l + 1].S.n, c = min(s_range[l + 1][0] + (int)threadIdx.x, nc - 1);
    const float *rw16 = sP.L[l].rw16;
    if (rw16) {
#pragma unroll
        for (int q = 0; q < 16; q++) R.w[q] = __ldg(rw16 + (size_t)q * nc + c);
    }
    sp_prefetch(sP.L[l].rst, R.t);
}

// b of level l + 1 = R r of level l (times 1/4 in the mixed V-cycle).  Interior
// coarse cells gather their 4 x 4 fine window with the weights of rw16
// (coarse-major), in the row order of R (fine index ascending); the others (the
// ring of the coarse level, or every cell when the pattern does not hold) are
// sparse rows.
template <bool MP>
__device__ __forceinline__ void restrict_phase(int l, RestrictPre &R) {
    using A = typename Prec<MP>::A;
    const LevelDev &F = sP.L[l], &Cl = sP.L[l + 1];
    const StencilDev &C = Cl.S;
    const int Nf = F.S.N, Nc = C.N, nc = C.n;
    const auto *r = lv<MP>(F.r);
    auto *b = lv<MP>(Cl.b);
    const float *rw16 = F.rw16;
    const float scale = MP ? 0.25f : 1.0f;
    sp_rows<MP>(F.rst, R.t, [&](int k) { return ldv(r, k); }, [&](int row, float v) {
        int c = row;
        if (rw16) {
            int f, i, j;
            ring_cell_of_rank(row, Nc, C.nring, f, i, j);
            c = (f * Nc + j) * Nc + i;
        }
        stv(b, c, v * scale);
    });
    if (!rw16) return;
    bool first = true;
#pragma unroll 1
    for (int c = s_range[l + 1][0] + (int)threadIdx.x; c < s_range[l + 1][1]; c += blockDim.x) {
        int f, I, J;
        cell_fij(C, c, f, I, J);
        if (I >= 1 && J >= 1 && I + 2 <= Nc && J + 2 <= Nc) {
            const int base = (f * Nf + 2 * J - 1) * Nf + 2 * I - 1;
            float x[16];
#pragma unroll
            for (int q = 0; q < 16; q++) x[q] = ldv(r, base + (q >> 2) * Nf + (q & 3));
            if (!first) {
#pragma unroll
                for (int q = 0; q < 16; q++) R.w[q] = __ldg(rw16 + (size_t)q * nc + c);
            }
            DotAcc<MP> acc;
#pragma unroll
            for (int q = 0; q < 16; q++) acc.add(R.w[q], x[q]);
            stv(b, c, (float)acc.a * scale);
        }
        first = false;
    }
}

// x + P xo (times 4 in the mixed V-cycle) of level l at cell k, x its
// pre-smoothed iterate.  Inside a face the four coarse taps follow from the
// cell's indices (where rw16 says the pattern holds).
template <bool MP>
__device__ __forceinline__ float prolong(const LevelDev &L, int Nc, const typename Prec<MP>::V *xc, int k, float b) {
    const float4 w = __ldg(reinterpret_cast<const float4 *>(L.pw) + k);
    const float x = presmooth_x<MP>(__ldg(L.dinv + k), b);
    int f, i, j;
    cell_fij(L.S, k, f, i, j);
    int t0 = (f * Nc + ((j - 1) >> 1)) * Nc + ((i - 1) >> 1), t1 = t0 + 1, t2 = t0 + Nc, t3 = t2 + 1;
    if (!L.rw16 || i == 0 || j == 0 || i == L.S.N - 1 || j == L.S.N - 1) {
        const int4 t = __ldg(reinterpret_cast<const int4 *>(L.ptap) + k);
        t0 = t.x;
        t1 = t.y;
        t2 = t.z;
        t3 = t.w;
    }
    const float s = w.x * ldv(xc, t0) + w.y * ldv(xc, t1) + w.z * ldv(xc, t2) + w.w * ldv(xc, t3);
    if (MP) return x + 4.0f * s;
    return x + (float)(kCorrScale * s);
}

// Power of two that brings a residual of squared norm rr over n cells to an
// RMS near 1/16 (the mixed V-cycle's input scale; 1 in the plain solve).
template <bool MP>
__device__ __forceinline__ float vscale(double rr, int n) {
    if (!MP || !(rr > 0) || !isfinite(rr)) return 1.0f;
    const int e = ilogb(sqrt(rr / n));
    return ldexpf(1.0f, max(-100, min(100, -4 - e)));
}

// The whole solve of this block's planet (sP) on the block's virtual grid.
// SWEEPS: with the sweeps of a coarsest level that has no dense map; BATCH: the
// virtual grid may be a few blocks.
template <bool MP, int TPB, bool SWEEPS, bool BATCH>
__device__ __forceinline__ void pcg_body() {
    using A = typename Prec<MP>::A;
    using V = typename Prec<MP>::V;
    const int n = sP.L[0].S.n;
    const bool mg = sP.nlev >= 2, single = sP.nlev == 1;
    const int G = sP.nlev_grid;
    float *r = sP.r, *rn = sP.r2, *p = sP.p, *pn = sP.p2;
    float *z = sP.z, *zo = MP ? sP.z2 : nullptr;  // mixed: z / z2 ping-pong (the previous z for the flexible beta)
    double bb = 0, rr = 0, rz = 0, tol2 = 0, beta = 0, m2;
    int it = 0, flags = 0;
    bool init = true, ok = false;
    float s0 = 1.0f;
    const unsigned long long t_begin = threadIdx.x == 0 ? globaltimer_ns() : 0ull;
    block_setup();
    RingPre R;
    ring_prefetch(0, R);

    // zero-mean projection of omega (FP64 sum), upstream src/fluid.c:264-275,
    // then the FP64 projection that makes the singular system consistent: the
    // stored FP32 omega keeps a residual area-weighted mean m2 (the FP32 rounding
    // of the subtracted mean); b = -A (omega - m2) is formed in FP64 so that
    // sum b = 0 to double precision.  Without it the constant mode of the
    // residual stays at the FP32 rounding level and CG diverges once the
    // residual reaches it.
#pragma unroll 1
    for (int pass = sP.remove_mean ? 0 : 1; pass < 2; pass++) {
        const float *area = sP.area;
        float *omega = sP.omega;
        double s = 0, sa = 0;
#pragma unroll 4
        OWN_LOOP(c) {
            const double a = __ldg(area + c);
            s += a * omega[c];
            sa += a;
        }
        if (!vsync(2, s, sa)) goto done;
        const double tot = s_total[0];
        if (pass == 0) {
            const float m = (float)(tot / sP.total_area);
#pragma unroll 4
            OWN_LOOP(c) omega[c] -= m;  // read back by the same thread before the next grid barrier
        } else {
            m2 = tot / s_total[1];
        }
    }

#pragma unroll 1
    for (;;) {
        RestrictPre T;
        DenseTaps D;
        double s = 0, s2 = 0;
        // first r = b - K psi, b = -A (omega - m2); then p = z or z + beta p, Ap = K p
        {
            const float *xa = init ? sP.psi : z;
            const float *xb = p;
            const bool comb = !init && it > 0;
            const double be = beta;
            float *xw = init ? r : pn, *ap = sP.Ap;
            stencil_phase<MP>(0, R, [&](int k) { return comb ? (float)(xa[k] + be * xb[k]) : xa[k]; },
                              [&](int c, float xc, A kx) {
                                  if (init) {
                                      const double b = -(double)__ldg(sP.area + c) * ((double)sP.omega[c] - m2);
                                      const double ri = b - (double)kx;
                                      xw[c] = (float)ri;
                                      s2 += b * b;
                                      s += ri * ri;
                                  } else {
                                      xw[c] = xc;
                                      ap[c] = (float)kx;
                                      s += (double)kx * xc;
                                  }
                              });
            if (!init) {
                pn = p;
                p = xw;
            }
        }
        if (mg) ring_prefetch(0, R);
        TRACE(10);
        if (!vsync(init ? 2 : 1, s, s2)) goto done;
        TRACE(11);
        double alpha = 0;
        if (init) {
            rr = s_total[0];
            bb = s_total[1];
            if (!isfinite(bb) || !isfinite(rr)) flags |= kSolveNonFinite;
            tol2 = sP.tol * sP.tol * bb;
            if (bb == 0.0 || !(rr > tol2)) {
                ok = true;
                break;
            }
        } else {
            const double pAp = s_total[0];
            if (!isfinite(pAp)) flags |= kSolveNonFinite;
            if (pAp <= 0) {
                flags |= kSolveBreakdown;
                ok = true;
                break;
            }
            alpha = rz / pAp;
        }
        // psi += alpha p; r' = r - alpha Ap; the V-cycle's way down from r'
        const float *ro = r, *Ap = sP.Ap;
        s = s2 = 0;
        if (mg || single) s0 = vscale<MP>(rr, n);  // the previous r's scale (the new r is not reduced yet)
        if (mg) {
#pragma unroll 1
            for (int l = 0; l < G; l++) {
                // pre-smooth from x = 0: x = w D^-1 b, r = b - K x
                const LevelDev &L = sP.L[l];
                const V *lb = lv<MP>(L.b);
                V *lr = lv<MP>(L.r);
                const float *dinv = L.dinv;
                float *psi = sP.psi, *rw_ = rn;
                auto getb = [&](int k) -> float {
                    if (l > 0) return ldv(lb, k);
                    const float v = init ? ro[k] : (float)(ro[k] - alpha * Ap[k]);
                    return MP ? v * s0 : v;
                };
                stencil_phase<MP>(l, R, [&](int k) { return presmooth_x<MP>(__ldg(dinv + k), getb(k)); },
                                  [&](int c, float, A kx) {
                                      if (l == 0 && !init) {
                                          const double ri = ro[c] - alpha * Ap[c];
                                          const float rc = (float)ri;
                                          psi[c] += (float)(alpha * p[c]);
                                          rw_[c] = rc;
                                          s += ri * ri;
                                          stv(lr, c, (float)((MP ? rc * s0 : rc) - kx));
                                      } else {
                                          stv(lr, c, (float)(getb(c) - kx));
                                      }
                                  });
                restrict_prefetch(l, T);
                TRACE(100 + l);
                // |r'|^2 is read during the next phase (the test for convergence comes one phase late)
                const bool res = l == 0 && !init;
                if (!vsync(res ? 1 : 0, s, 0, true)) goto done;
                restrict_phase<MP>(l, T);
                if (l + 1 < G)
                    ring_prefetch(l + 1, R);
                else if (sP.dense)
                    dense_prefetch(D);
                TRACE(300 + l);
                if (!vsync(0, 0, 0, false, res)) goto done;
                if (res) {
                    rn = r;
                    r = rw_;
                    it++;
                    rr = s_late;
                    if (!isfinite(rr)) flags |= kSolveNonFinite;
                    if (rr <= tol2) {
                        ok = true;
                        break;
                    }
                }
            }
            if (ok) break;
        } else {
            float *rw_ = init ? r : rn, *psi = sP.psi;
            const float *dinv = sP.L[0].dinv;
            const int c1 = s_range[0][1], bs = blockDim.x;
#pragma unroll 1
            for (int c0 = s_range[0][0] + (int)threadIdx.x; c0 < c1; c0 += kUpdate * bs) {
                float rv[kUpdate], av[kUpdate], pv[kUpdate], xv[kUpdate], dv[kUpdate];
#pragma unroll
                for (int u = 0; u < kUpdate; u++) {
                    const int c = c0 + u * bs < c1 ? c0 + u * bs : c0;
                    rv[u] = ro[c];
                    dv[u] = __ldg(dinv + c);
                    if (!init) {
                        av[u] = Ap[c];
                        pv[u] = p[c];
                        xv[u] = psi[c];
                    }
                }
#pragma unroll
                for (int u = 0; u < kUpdate; u++) {
                    const int c = c0 + u * bs;
                    if (c >= c1) break;
                    double ri = rv[u];
                    if (!init) {
                        psi[c] = xv[u] + (float)(alpha * pv[u]);
                        ri -= alpha * av[u];
                        rw_[c] = (float)ri;
                    }
                    const float rc = (float)ri;
                    s += ri * ri;
                    if (!single) {
                        const float zc = dv[u] * rc;
                        z[c] = zc;
                        s2 += (double)rc * zc;
                    }
                }
            }
            if (!init) {
                rn = r;
                r = rw_;
            }
            ring_prefetch(0, R);
            if (!vsync(2, s, s2)) goto done;
            if (!init) {
                it++;
                rr = s_total[0];
                if (!isfinite(rr)) flags |= kSolveNonFinite;
                if (rr <= tol2) {
                    ok = true;
                    break;
                }
                if (single) s0 = vscale<MP>(rr, n);
            }
        }
        // z = M^-1 r
        const float *zold = nullptr;
        if (MP && !init && (mg || single)) {  // the new z goes to the other buffer; zo keeps the previous one
            float *t = z;
            z = zo;
            zo = t;
            zold = zo;
        }
        if (mg || single) {
            s = s2 = 0;
            const float inv = 1.0f / s0;
            auto finish = [&](int c, float v) {
                const float rc = r[c], zc = MP ? v * inv : v;
                z[c] = zc;
                s += (double)rc * zc;
                if (MP && zold) s2 += (double)rc * zold[c];
            };
            // the coarsest grid level: the dense map, or its sweeps
            {
                const LevelDev &L = sP.L[G];
                const V *cb = lv<MP>(L.b);
                V *cx = lv<MP>(L.xo);
                auto getb = [&](int c) -> float {
                    if (mg) return ldv(cb, c);
                    return as_stored<MP>(MP ? r[c] * s0 : r[c]);
                };
                auto put = [&](int c, float v) {
                    if (mg)
                        stv(cx, c, v);
                    else
                        finish(c, as_stored<MP>(v));
                };
                if (sP.dense) {
                    dense_rows<BATCH>(D, [&](int j) { return ldv4(cb + j); }, [&](int c, double v) { put(c, (float)v); });
                } else if (!sP.coarse_on_grid) {
                    // a single small level: block 0 sweeps r in shared memory
                    if (vb() == 0) {
                        SmemLevel lvl;
                        lvl.x = s_win();
                        lvl.xo = lvl.x + n;
                        lvl.b = lvl.xo + n;
                        BLOCK_LOOP(c, n) lvl.b[c] = r[c];
                        __syncthreads();
                        coarsest_smem(L, lvl, sP.coarse_sweeps);
                        BLOCK_LOOP(c, n) put(c, MP ? lvl.xo[c] * s0 : lvl.xo[c]);
                    }
                } else if (SWEEPS) {
                    if (!coarse_sweeps<MP, TPB>(L, getb, put)) goto done;
                }
            }
            if (mg) {
                ring_prefetch(G - 1, R);
                TRACE(500);
                if (!vsync(0, 0, 0)) goto done;
#pragma unroll 1
                for (int l = G - 1;; l--) {
                    // prolongation and post-smooth: x = x + P xo, then x + w D^-1 (b - K x)
                    const LevelDev &L = sP.L[l];
                    const V *lb = lv<MP>(L.b), *xc = lv<MP>(sP.L[l + 1].xo);
                    V *lx = lv<MP>(L.xo);
                    const int Nc = sP.L[l + 1].S.N;
                    const float *dinv = L.dinv;
                    auto getb = [&](int k) -> float {
                        if (l > 0) return ldv(lb, k);
                        return MP ? r[k] * s0 : r[k];
                    };
                    stencil_phase<MP>(l, R, [&](int k) { return prolong<MP>(L, Nc, xc, k, getb(k)); },
                                      [&](int c, float x, A kx) {
                                          const float rc = (float)(getb(c) - kx), d = __ldg(dinv + c);
                                          const float v = MP ? x + 0.8f * d * rc : x + (float)(kOmegaJ * d * rc);
                                          if (l > 0)
                                              stv(lx, c, v);
                                          else
                                              finish(c, v);
                                      });
                    if (l == 0) break;
                    ring_prefetch(l - 1, R);
                    TRACE(900 + l);
                    if (!vsync(0, 0, 0)) goto done;
                }
            }
            ring_prefetch(0, R);
            TRACE(900);
            if (!vsync(MP ? 2 : 1, s, s2)) goto done;
        }
        {
            const double rznew = mg || single ? s_total[0] : s_total[1];
            if (!isfinite(rznew)) flags |= kSolveNonFinite;
            if (MP && (mg || single))
                beta = (rznew - s_total[1]) / rz;  // Polak-Ribiere
            else
                beta = rznew / rz;
            rz = rznew;
        }
        init = false;
        if (!(rr > tol2) || it >= sP.maxit) {  // an rr that is NaN ends the solve, as upstream's loop condition does
            ok = true;
            break;
        }
    }

    if (ok && bb == 0.0) {
        OWN_LOOP(c) sP.psi[c] = 0.f;
    } else if (ok) {
        // zero-mean projection of psi (each thread's own cells, which no other thread has written)
        const float *area = sP.area;
        float *psi = sP.psi;
        double s = 0;
#pragma unroll 4
        OWN_LOOP(c) s += (double)__ldg(area + c) * psi[c];
        ok = vsync(1, s, 0);
        if (ok) {
            const float m = (float)(s_total[0] / sP.total_area);
#pragma unroll 4
            OWN_LOOP(c) psi[c] -= m;
            // leave the final residual / direction / preconditioned residual in the caller's buffers
            if (r != sP.r) OWN_LOOP(c) sP.r[c] = r[c];
            if (p != sP.p) OWN_LOOP(c) sP.p[c] = p[c];
            if (z != sP.z) OWN_LOOP(c) sP.z[c] = z[c];
        }
    }
done:
    if (vb() == 0 && threadIdx.x == 0) {
        if (ok && it >= sP.maxit && rr > tol2) flags |= kSolveMaxit;
        sP.res->iters = it;
        sP.res->relres = !ok ? -1.0 : (bb == 0.0 ? 0.0 : sqrt(rr / bb));
        sP.res->status = ok ? 0 : 1;
        sP.res->r_final = 0;
        sP.res->flags = ok ? flags : flags | kSolveTimeout;
        if (ok) sP.res->ns = globaltimer_ns() - t_begin;
    }
}

// One solve on the whole grid.
template <bool MP, int TPB, bool SWEEPS>
__global__ void __launch_bounds__(TPB, 1) k_pcg(const __grid_constant__ SolveParams P) {
    const int *src = reinterpret_cast<const int *>(&P);
    int *dst = reinterpret_cast<int *>(&sP);
    for (int k = threadIdx.x; k < (int)(sizeof(SolveParams) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
    if (threadIdx.x == 0) {
        s_vgrid[0] = blockIdx.x;
        s_vgrid[1] = gridDim.x;
        s_epoch = 0;
    }
    __syncthreads();
    pcg_body<MP, TPB, SWEEPS, false>();
}

// Many planets' solves in one cooperative launch: block b runs planet
// bmap[b].x's solve as block bmap[b].y of bmap[b].z (the planet's blocks are
// consecutive), with that planet's parameters, barrier, partial sums and
// result.  Planets finish independently.
template <bool MP, int TPB, bool SWEEPS>
__global__ void __launch_bounds__(TPB, 1) k_pcg_batch(const SolveParams *prm, const int4 *bmap) {
    const int4 m = bmap[blockIdx.x];
    const int *src = reinterpret_cast<const int *>(prm + m.x);
    int *dst = reinterpret_cast<int *>(&sP);
    for (int k = threadIdx.x; k < (int)(sizeof(SolveParams) / sizeof(int)); k += blockDim.x) dst[k] = src[k];
    if (threadIdx.x == 0) {
        s_vgrid[0] = m.y;
        s_vgrid[1] = m.z;
        s_epoch = 0;
    }
    __syncthreads();
    pcg_body<MP, TPB, SWEEPS, true>();
}

// The kernel of a precision and coarse end at one of the block sizes.
template <bool MP, bool SWEEPS>
const void *kernel_of(int threads, bool batch) {
    if (threads == kPBWide)
        return batch ? (const void *)k_pcg_batch<MP, kPBWide, SWEEPS> : (const void *)k_pcg<MP, kPBWide, SWEEPS>;
    if (threads == kPBNarrow)
        return batch ? (const void *)k_pcg_batch<MP, kPBNarrow, SWEEPS> : (const void *)k_pcg<MP, kPBNarrow, SWEEPS>;
    return batch ? (const void *)k_pcg_batch<MP, kPB, SWEEPS> : (const void *)k_pcg<MP, kPB, SWEEPS>;
}
