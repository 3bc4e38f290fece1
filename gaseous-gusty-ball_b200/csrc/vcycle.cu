// vcycle.cu — set-up of what the solve kernel reads of each multigrid level
// besides the operator tables: the restriction as 16 weights per interior coarse
// cell and as sparse rows for the others, the links of the boundary-ring cells,
// and the level vectors (upstream src/fluid.c:41-95 builds the same transfers).
#include <algorithm>
#include <cstdio>
#include <vector>

#include "ggb_internal.h"
#include "ggb_solver.h"

namespace ggb {

constexpr int kSB = 256;
static unsigned setup_blocks(size_t n) { return std::max(1u, std::min(grid_for(n, kSB), 2048u)); }

// Interior coarse cell: its row of R is the 4 x 4 fine window around it.
__device__ __forceinline__ bool inner_coarse(int I, int J, int Nc) {
    return I >= 1 && J >= 1 && I + 2 <= Nc && J + 2 <= Nc;
}

// Coarse-major weights of the interior rows of R: rw16[q][c] = the weight of
// fine cell q (q = 4*dj + di of the 4x4 window) in row c.
__global__ void k_build_rw16(LevelDev F, StencilDev C, float *rw16) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C.n; c += gridDim.x * blockDim.x) {
        int f, I, J;
        cell_fij(C, c, f, I, J);
        const bool inner = inner_coarse(I, J, C.N);
        const int k0 = F.rstart[c];
        for (int q = 0; q < 16; q++) rw16[(size_t)q * C.n + c] = inner ? F.rw[k0 + q] : 0.f;
    }
}

// Counts rows of R / taps of P of a level pair that the index arithmetic of the
// solve would take but that do not follow its pattern.
__global__ void k_check_structured(LevelDev F, StencilDev C, int *bad) {
    const int Nf = F.S.N, Nc = C.N;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < C.n; c += gridDim.x * blockDim.x) {
        int f, I, J;
        cell_fij(C, c, f, I, J);
        if (!inner_coarse(I, J, Nc)) continue;
        const int k0 = F.rstart[c], k1 = F.rstart[c + 1];
        if (k1 - k0 != 16) {
            atomicAdd(bad, 1);
            continue;
        }
        const int base = (f * Nf + 2 * J - 1) * Nf + 2 * I - 1;
        for (int dj = 0; dj < 4; dj++)
            for (int di = 0; di < 4; di++) {
                const int i = base + dj * Nf + di, q = k0 + dj * 4 + di;
                const int k = (di <= 1 ? 1 : 0) + 2 * (dj <= 1 ? 1 : 0);
                if (F.ridx[q] != i || F.rw[q] != F.pw[4 * i + k]) atomicAdd(bad, 1);
            }
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < F.S.n; i += gridDim.x * blockDim.x) {
        int f, fi, fj;
        cell_fij(F.S, i, f, fi, fj);
        if (fi == 0 || fj == 0 || fi == Nf - 1 || fj == Nf - 1) continue;
        const int t0 = (f * Nc + ((fj - 1) >> 1)) * Nc + ((fi - 1) >> 1);
        if (F.ptap[4 * i] != t0 || F.ptap[4 * i + 1] != t0 + 1 || F.ptap[4 * i + 2] != t0 + Nc ||
            F.ptap[4 * i + 3] != t0 + Nc + 1)
            atomicAdd(bad, 1);
    }
}

// Row `row` of the restriction's sparse rows: coarse cell `row`, or the ring cell of
// that rank.
__device__ __forceinline__ int sparse_row_cell(const StencilDev &C, int ring, int row) {
    if (!ring) return row;
    int f, i, j;
    ring_cell_of_rank(row, C.N, C.nring, f, i, j);
    return (f * C.N + j) * C.N + i;
}

__global__ void k_row_len(LevelDev F, StencilDev C, int ring, int rows, int *most) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int c = sparse_row_cell(C, ring, r);
        atomicMax(most, F.rstart[c + 1] - F.rstart[c]);
    }
}

// The rows of R, in their order, as taps [step][row]; steps past a row's end
// repeat its first index with weight 0.  One thread per 32 rows leaves the
// largest length among them in glen.
__global__ void k_row_taps(LevelDev F, StencilDev C, int ring, int rows, int steps, int2 *tap, unsigned char *glen) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int c = sparse_row_cell(C, ring, r), k0 = F.rstart[c], m = F.rstart[c + 1] - k0;
        for (int s = 0; s < steps; s++)
            tap[(size_t)s * rows + r] = s < m ? make_int2(F.ridx[k0 + s], __float_as_int(F.rw[k0 + s]))
                                              : make_int2(m > 0 ? F.ridx[k0] : 0, 0);
        if (r % 32 == 0) {
            int most = 0;
            for (int q = r; q < min(rows, r + 32); q++) {
                const int d = sparse_row_cell(C, ring, q);
                most = max(most, F.rstart[d + 1] - F.rstart[d]);
            }
            glen[r / 32] = (unsigned char)most;
        }
    }
}

// The boundary-ring cells' links as eight (neighbour, weight bits) pairs: lane k
// holds the on-face slot k (E, N, NE, NW, W, S, SW, SE) where it has a link, and
// the links that leave the face take the other lanes in their order; weight 0 and
// the cell itself in what is left.  The on-face lanes are marked in the cell's
// upper byte (half: their weights rounded to FP16).
__global__ void k_ring_links(StencilDev S, int half, int2 *link, int *cell, int *bad) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < 6 * S.nring; r += gridDim.x * blockDim.x) {
        int f, i, j;
        ring_cell_of_rank(r, S.N, S.nring, f, i, j);
        const int N = S.N, n = S.n, c = (f * N + j) * N + i;
        const bool e = i + 1 < N, w = i > 0, up = j + 1 < N, dn = j > 0;
        const float *ws = S.wslot;
        int2 q[kMaxNb];
        unsigned on = 0;
        auto put = [&](int k, bool in, int o, size_t slot) {
            float v = in ? ws[slot] : 0.f;
            q[k] = make_int2(c, 0);
            if (v == 0.f) return;
            if (half) v = __half2float(__float2half_rn(v));
            q[k] = make_int2(o, __float_as_int(v));
            on |= 1u << k;
        };
        put(0, e, c + 1, c);
        put(1, up, c + N, (size_t)n + c);
        put(2, e && up, c + N + 1, 2 * (size_t)n + c);
        put(3, w && up, c + N - 1, 3 * (size_t)n + c);
        put(4, w, c - 1, c - 1);
        put(5, dn, c - N, (size_t)n + c - N);
        put(6, w && dn, c - N - 1, 2 * (size_t)n + c - N - 1);
        put(7, e && dn, c - N + 1, 3 * (size_t)n + c - N + 1);
        int k = 0;
        for (int x = 0; x < kMaxNb; x++) {
            const int o = S.ring_nb[(size_t)r * kMaxNb + x];
            if (o < 0) break;
            while (k < kMaxNb && (on >> k & 1u)) k++;
            if (k == kMaxNb) {
                atomicAdd(bad, 1);
                break;
            }
            q[k++] = make_int2(o, __float_as_int(S.ring_w[(size_t)r * kMaxNb + x]));
        }
        cell[r] = c | (int)(on << 24);
        for (int x = 0; x < kMaxNb; x++) link[kMaxNb * (size_t)r + x] = q[x];
    }
}

__global__ void k_round_half(size_t n, const float *src, float *dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = __half2float(__float2half_rn(src[i]));
}

static void ring_links(const StencilDev &S, int half, int2 *link, int *cell, LevelSet *out, int l, int *bad) {
    k_ring_links<<<setup_blocks(6 * S.nring), kSB, 0, stream()>>>(S, half, link, cell, bad);
    GGB_LAUNCHED();
    out->ring_link[l] = link;
    out->ring_cell[l] = cell;
}
static size_t ring_link_bytes(const StencilDev &S) { return sizeof(int2) * kMaxNb * 6 * (size_t)S.nring; }
static size_t ring_cell_bytes(const StencilDev &S) { return sizeof(int) * 6 * (size_t)S.nring; }

// The places of several arrays in one allocation: at least one call of the
// allocator a level was most of this set-up's time.
struct Layout {
    size_t bytes = 0;
    size_t take(size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) & ~(size_t)255;
        return at;
    }
};

// The plain solve's level data (levels 0..nlev_grid of P; level 0's ring links
// for every fluid).  The device arrays go to mem.
void levels_build(const SolveParams &P, LevelSet *out, std::vector<void *> &mem) {
    cudaStream_t s = stream();
    const int G = P.nlev_grid;
    struct Host {
        int irregular[kMaxLev];                     // rows and taps off the index pattern
        int most[kMaxLev], most_ring[kMaxLev];      // longest row of R: of all, of the coarse ring's
        int bad;                                    // ring cells of too many links
    } host = {};
    struct At {
        size_t link, cell, rw16, r, b, xo, tap, glen;
    } at[kMaxLev] = {};
    Layout first;
    const size_t scratch_at = first.take(sizeof(Host));
    for (int l = 0; l < std::max(G, 1); l++) {
        at[l].link = first.take(ring_link_bytes(P.L[l].S));
        at[l].cell = first.take(ring_cell_bytes(P.L[l].S));
    }
    for (int l = 0; l < G; l++) {
        const size_t nc = P.L[l + 1].S.n;
        at[l].rw16 = first.take(sizeof(float) * 16 * nc);
        at[l].r = first.take(sizeof(float) * (size_t)P.L[l].S.n);
        at[l].b = first.take(sizeof(float) * (nc + 8));
        at[l].xo = first.take(sizeof(float) * (nc + 8));
    }
    unsigned char *const vectors = (unsigned char *)dev_alloc(first.bytes);
    mem.push_back(vectors);
    Host *scratch = (Host *)(vectors + scratch_at);
    for (int l = 0; l < std::max(G, 1); l++)
        ring_links(P.L[l].S, 0, (int2 *)(vectors + at[l].link), (int *)(vectors + at[l].cell), out, l, &scratch->bad);
    for (int l = 0; l < G; l++) {
        const StencilDev &C = P.L[l + 1].S;
        k_check_structured<<<setup_blocks(P.L[l].S.n), kSB, 0, s>>>(P.L[l], C, &scratch->irregular[l]);
        GGB_LAUNCHED();
        k_row_len<<<setup_blocks(C.n), kSB, 0, s>>>(P.L[l], C, 0, C.n, &scratch->most[l]);
        GGB_LAUNCHED();
        k_row_len<<<setup_blocks(6 * C.nring), kSB, 0, s>>>(P.L[l], C, 1, 6 * C.nring, &scratch->most_ring[l]);
        GGB_LAUNCHED();
        out->r[l] = vectors + at[l].r;
        out->b[l + 1] = vectors + at[l].b;
        out->xo[l + 1] = vectors + at[l].xo;
    }
    GGB_CHECK(cudaMemcpyAsync(&host, scratch, sizeof(host), cudaMemcpyDeviceToHost, s));
    GGB_CHECK(cudaStreamSynchronize(s));
    if (host.bad) fail_msg("multigrid set-up: a ring cell of more than %d links", kMaxNb);
    Layout second;
    for (int l = 0; l < G; l++) {
        const StencilDev &C = P.L[l + 1].S;
        const bool ring = host.irregular[l] == 0;
        SparseOp &op = out->rst[l];
        op.rows = ring ? 6 * C.nring : C.n;
        op.steps = std::max(1, ring ? host.most_ring[l] : host.most[l]);
        if (op.steps > 255) fail_msg("multigrid set-up: a row of %d taps", op.steps);
        at[l].tap = second.take(sizeof(int2) * op.rows * (size_t)op.steps);
        at[l].glen = second.take((op.rows + 31) / 32);
    }
    if (G == 0) return;
    unsigned char *const rows = (unsigned char *)dev_alloc(second.bytes);
    mem.push_back(rows);
    for (int l = 0; l < G; l++) {
        const StencilDev &C = P.L[l + 1].S;
        const int ring = host.irregular[l] == 0;
        SparseOp &op = out->rst[l];
        int2 *tap = (int2 *)(rows + at[l].tap);
        k_row_taps<<<setup_blocks(op.rows), kSB, 0, s>>>(P.L[l], C, ring, op.rows, op.steps, tap, rows + at[l].glen);
        GGB_LAUNCHED();
        op.tap = tap;
        op.glen = rows + at[l].glen;
        if (ring) {
            float *rw16 = (float *)(vectors + at[l].rw16);
            k_build_rw16<<<setup_blocks(C.n), kSB, 0, s>>>(P.L[l], C, rw16);
            GGB_LAUNCHED();
            out->rw16[l] = rw16;
        }
    }
}

// The mixed solve's: the same transfers, FP16 level vectors, and below level 0
// the slot weights rounded to FP16.
void levels_build_mixed(const SolveParams &P, const LevelSet &plain, LevelSet *out, std::vector<void *> &mem) {
    *out = plain;
    int *bad = (int *)dev_alloc(sizeof(int));  // (the plain set's check covers the same links)
    mem.push_back(bad);
    for (int l = 0; l < P.nlev_grid; l++) {
        const StencilDev &S = P.L[l].S, &C = P.L[l + 1].S;
        if (l > 0) {
            int2 *link = (int2 *)dev_alloc(ring_link_bytes(S));
            int *cell = (int *)dev_alloc(ring_cell_bytes(S));
            mem.push_back(link);
            mem.push_back(cell);
            ring_links(S, 1, link, cell, out, l, bad);
            float *w = (float *)dev_alloc(sizeof(float) * 4 * (size_t)S.wplane);
            mem.push_back(w);
            k_round_half<<<setup_blocks(4 * (size_t)S.wplane), kSB, 0, stream()>>>(4 * (size_t)S.wplane, S.wpad, w);
            GGB_LAUNCHED();
            out->wpad[l] = w;
        }
        out->r[l] = dev_alloc(sizeof(__half) * (size_t)S.n);
        out->b[l + 1] = dev_alloc(sizeof(__half) * (size_t)(C.n + 8));
        out->xo[l + 1] = dev_alloc(sizeof(__half) * (size_t)(C.n + 8));
        for (void *p : {out->r[l], out->b[l + 1], out->xo[l + 1]}) mem.push_back(p);
    }
}

// Parts of a level for its sweeps (SweepParts): face f is cut into tx x ty
// rectangles of cells, one part each.  One block per part walks outwards from its
// own cells by their links, a bit per cell marking those already listed, until a
// distance does not fit the slots; then a map from cell to slot gives the
// neighbours' slots.  (The order of the slots within a distance is arbitrary and
// changes no value.)
constexpr int kPartThreads = 512;
__global__ void __launch_bounds__(kPartThreads) k_sweep_parts(StencilDev S, int tx, int ty, int *count, int *cell,
                                                              unsigned short *nb, float *w) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ int s_n;
    unsigned short *slot = reinterpret_cast<unsigned short *>(dyn);                     // [n]
    unsigned *seen = reinterpret_cast<unsigned *>(dyn + ((2 * (size_t)S.n + 15) & ~(size_t)15));  // [n / 32]
    const int p = blockIdx.x, f = p / (tx * ty), t = p - f * tx * ty, N = S.N;
    const int i0 = (t % tx) * N / tx, i1 = (t % tx + 1) * N / tx, j0 = (t / tx) * N / ty, j1 = (t / tx + 1) * N / ty;
    int *const cells = cell + (size_t)p * kSweepSlots;
    int *const cnt = count + (size_t)p * (kSweepDepth + 1);
    for (int k = threadIdx.x; k < (S.n + 31) / 32; k += blockDim.x) seen[k] = 0;
    for (int k = threadIdx.x; k < S.n; k += blockDim.x) slot[k] = 0xffff;
    __syncthreads();
    const int wi = i1 - i0, own = wi * (j1 - j0);
    for (int k = threadIdx.x; k < own && k < kSweepSlots; k += blockDim.x) {
        const int c = (f * N + j0 + k / wi) * N + i0 + k % wi;
        cells[k] = c;
        atomicOr(&seen[c >> 5], 1u << (c & 31));
    }
    if (threadIdx.x == 0) s_n = own;
    __syncthreads();
    int from = 0, to = own;
    for (int h = 0; h <= kSweepDepth; h++) {
        if (threadIdx.x == 0) cnt[h] = to;  // over kSweepSlots: distance h does not fit
        if (to > kSweepSlots || h == kSweepDepth) {
            for (int k = h + 1 + (int)threadIdx.x; k <= kSweepDepth; k += blockDim.x) cnt[k] = kSweepSlots + 1;
            break;
        }
        for (int k = from + (int)threadIdx.x; k < to; k += blockDim.x) {
            int o[kMaxNb];
            float q[kMaxNb];
            cell_links(S, cells[k], o, q);
            for (int u = 0; u < kMaxNb; u++) {
                const unsigned bit = 1u << (o[u] & 31);
                if (q[u] == 0.f || (atomicOr(&seen[o[u] >> 5], bit) & bit)) continue;
                const int at = atomicAdd(&s_n, 1);
                if (at < kSweepSlots) cells[at] = o[u];
            }
        }
        __syncthreads();
        from = to;
        to = s_n;
        __syncthreads();
    }
    const int listed = min(to, kSweepSlots);
    for (int k = threadIdx.x; k < listed; k += blockDim.x) slot[cells[k]] = (unsigned short)k;
    __syncthreads();
    for (int k = threadIdx.x; k < kSweepSlots; k += blockDim.x) {
        int o[kMaxNb];
        float q[kMaxNb];
        if (k < listed) cell_links(S, cells[k], o, q);
        for (int u = 0; u < kMaxNb; u++) {
            const size_t at = ((size_t)p * kMaxNb + u) * kSweepSlots + k;
            const bool in = k < listed && q[u] != 0.f && slot[o[u]] != 0xffff;
            nb[at] = in ? slot[o[u]] : (unsigned short)k;
            w[at] = in ? q[u] : 0.f;
        }
        if (k >= listed) cells[k] = 0;
    }
}

// Cuts level S into parts for `blocks` blocks, or leaves out->parts 0 when it is
// too large.  The depth minimises the estimated time per sweep: a sweep inside a
// part 0.35 us with one cell per thread of 512 and 0.55 us with two, an exchange
// 2.5 us.
void sweep_parts_build(const StencilDev &S, int blocks, SweepParts *out, std::vector<void *> &mem) {
    *out = SweepParts{};
    const size_t smem = ((2 * (size_t)S.n + 15) & ~(size_t)15) + 4 * (((size_t)S.n + 31) / 32);
    if (smem > 200 * 1024 || blocks < 6) return;
    int tx = 1, ty = 1, best = 1 << 30;
    for (int x = 1; x <= blocks / 6 && x <= S.N; x++) {
        const int y = std::min(blocks / 6 / x, S.N);
        const int side = (S.N + x - 1) / x + (S.N + y - 1) / y, cells = ((S.N + x - 1) / x) * ((S.N + y - 1) / y);
        if (cells * 8 + side * side < best) {
            best = cells * 8 + side * side;
            tx = x;
            ty = y;
        }
    }
    const int parts = 6 * tx * ty;
    cudaStream_t s = stream();
    int *count = (int *)dev_alloc(sizeof(int) * parts * (kSweepDepth + 1));
    int *cell = (int *)dev_alloc(sizeof(int) * parts * kSweepSlots);
    unsigned short *nb = (unsigned short *)dev_alloc(sizeof(unsigned short) * parts * kMaxNb * kSweepSlots);
    float *w = (float *)dev_alloc(sizeof(float) * parts * kMaxNb * kSweepSlots);
    for (void *p : {(void *)count, (void *)cell, (void *)nb, (void *)w}) mem.push_back(p);
    GGB_CHECK(cudaFuncSetAttribute(k_sweep_parts, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    k_sweep_parts<<<parts, kPartThreads, smem, s>>>(S, tx, ty, count, cell, nb, w);
    GGB_LAUNCHED();
    std::vector<int> host((size_t)parts * (kSweepDepth + 1));
    GGB_CHECK(cudaMemcpyAsync(host.data(), count, sizeof(int) * host.size(), cudaMemcpyDeviceToHost, s));
    GGB_CHECK(cudaStreamSynchronize(s));
    double least = 1e9;
    for (int d = 1; d <= kSweepDepth; d++) {
        int most = 0;
        for (int p = 0; p < parts; p++) most = std::max(most, host[(size_t)p * (kSweepDepth + 1) + d]);
        if (most > kSweepSlots) break;
        const double t = (most <= 512 ? 0.35 : 0.55) + 2.5 / d;
        if (t < least) {
            least = t;
            out->depth = d;
        }
    }
    if (out->depth < 1) return;
    out->parts = parts;
    out->count = count;
    out->cell = cell;
    out->nb = nb;
    out->w = w;
}

}  // namespace ggb
