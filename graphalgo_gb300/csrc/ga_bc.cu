// Batched betweenness centrality (betweenness_centrality_batch,
// include/betweenness_centrality.h:125-237) with FP64 path counts and
// dependencies, device-resident from the first frontier to the scores.
//
// Source columns are handled in blocks of 64 (one 64-bit word per vertex and
// block); a unit is a (block, vertex) pair, its key block * m + vertex.
//  * V: per unit, the columns that have reached the vertex (the reference's
//    Numsp pattern); F: per unit, the columns whose search is at the vertex in
//    the level being swept, in three buffers used in turn, so that one level's
//    kernel reads one, writes the next and clears the one before;
//  * S: m x ns FP64 path counts, W: m x ns FP64 (1 + delta) / sigma, both
//    read only where a bit of F says there is a value;
//  * rows: per distance, the units first reached there with their columns (the
//    reference's Sigmas[d]); the units of heavy vertices (more than `piece`
//    out-neighbours) from the other end of the same arrays, cut into tasks.
// Forward level (Front<!Numsp> = A^T * Front, matrix_la.h:800-891 fused with
// add_nointersect, matrix_la.h:337-372): a pulling warp takes the units that
// some column has not reached, ANDs the words of 32 in-neighbours with the
// missing columns, transposes the words across the warp, and every lane sums
// the counts of the neighbours that hold its two columns; a level with a
// small frontier pushes along the out-edges instead.
// Backward level k (betweenness_centrality.h:203-218): for the rows at
// distance k - 1, acc = A * W over the neighbours at distance k (the same
// gather over W), delta = acc * sigma, bc[v] += sum of delta (the final row
// sum, betweenness_centrality.h:220-228, accumulated as it is produced), and
// W = (1 + delta) / sigma = 1 / sigma + acc for the next level.
// Both sweeps run as device loops (CUDA-graph WHILE nodes, captured once per
// context): two kernels per forward level, one per backward level.
//
// What bounds it: GB300 adds two FP64 lanes per clock and SM whether one lane
// of a warp is active or all are (64 sources on R-MAT 20 need 2.8e8 additions
// each way, 0.55 ms at that rate with full warps), and the chain of dependent
// gathers per 32 neighbours (column, word, value). In the largest forward
// level the FP64 pipe is busy 65 % of the time at 28 % of its lanes. So the
// additions are packed: a lane walks only the neighbours that hold its column,
// and the columns found share out the lanes (bc_gather). 64 sources on R-MAT
// 20, one call: 38.0-42.1 ms before (every frontier entry a shared-memory FP64
// atomic, 20.5 ms forward; every column of every neighbour that any source had
// at the level, 17.1 ms backward; 1.6 ms to set and clear W), 16.8 ms with
// each lane summing two fixed columns and the units dealt out in advance, 10.5
// ms with warps taking units as they go and heavy vertices in warp-sized
// pieces, 8.0 ms with the columns sharing out the lanes (forward levels 0.04,
// 0.33, 2.34, 0.62, 0.51, 0.03 ms, backward 0.05, 0.40, 1.27, 1.97, 0.15 ms).
//
// Batches over the block-diagonal union of several graphs: column j holds the
// j-th source of every graph at once. A source only reaches the vertices of
// its own graph, so each (vertex, column) pair still belongs to one source,
// and the state is (union vertices) x (largest source count of a graph)
// instead of x (all sources). The columns a graph has no source for are
// marked visited on its vertices before the first level.
#include "ga_device.cuh"
#include "ga_loop.cuh"

#include <algorithm>

namespace ga {

constexpr int kBcThreads = 256;
constexpr int kBcWarps = kBcThreads / 32;
constexpr int kBcMaxSources = 1024;
// A vertex with more than `piece` neighbours is heavy: its list is cut into
// pieces that separate warps sum; the last piece to finish adds them up, in
// order (a hub of R-MAT 20 has 64,000 neighbours: one CTA would take longer
// than the rest of the level). Dense graphs take longer pieces, so that the
// partial sums stay small beside the graph.
constexpr int kBcPiece = 512;
constexpr int kBcPieceDense = 2048;   // more than kBcDense entries per vertex
constexpr int kBcDense = 256;
constexpr int kBcLoads = 4;   // values a lane has in flight (8 were 8 % slower: registers spill)
// Units (forward) and rows (backward) that a warp takes at a time: at most
// these, fewer where a level has not four takes per warp of the grid. A take's
// rows are reserved with one atomic, its scores summed together.
constexpr int kBcUnits = 16;
constexpr int kBcRows = 8;

struct BcState {
    int32_t d;        // forward: distance of the frontier; then the largest distance
    int32_t k;        // backward: distance whose W is set
    int32_t done;
    int32_t mode;     // forward direction of the level: 0 pull, 1 push
    int32_t nrows, nhrows, nhtasks;  // lists' ends
    int32_t ntouched; // push level: units reached
    int32_t nchunk;   // pieces of the heavy in-neighbour lists
    int32_t flags;    // 1 self-loop, 8 source out of range, 16 repeated source
    uint32_t blocks;  // blocks of the level's last kernel that have finished
    int32_t next;     // next task of the level (warps take tasks as they go)
    unsigned long long cur_work, next_work;  // sum over frontier rows of columns x out-degree
};

struct BcArgs {
    const int32_t* atr; const int32_t* atc; const double* atv;  // A^T (in-neighbours)
    const int32_t* ar; const int32_t* ac; const double* av;     // A (out-neighbours)
    int64_t m, nnz;
    int ns, nblk;                  // source columns, blocks of 64
    int piece;                     // neighbours per piece of a heavy vertex
    int nsrc;
    const int32_t* sources;
    const int32_t* scol;           // column of each source (nullptr: its index)
    BcState* st;
    unsigned long long* V;         // nblk x m
    unsigned long long* F[3];      // nblk x m each
    double* S; double* W;          // m x ns
    int32_t* rkey; unsigned long long* rmask;  // rows; heavy vertices' from the end (heavy_row)
    int64_t rlast;                             // last place of the rows
    int32_t* hfirst;                           // heavy rows: first task
    int2* htask;                   // (heavy row, piece)
    int32_t *lrow, *lhrow, *ltask; // per distance: first row, heavy row, task
    int4* chunk;                   // forward: pieces of the heavy in-lists (vertex, piece, first place, pieces)
    double* part; unsigned long long* pmask; int32_t* pdone;    // per place: partial sums, columns, arrivals
    int32_t* tlist;                // push level: units reached, in order of first touch
    double* bc;
};

// A level pushes (frontier rows scatter along their out-edges with global
// atomics) when its frontier's work, columns x out-degree, is below
// kBcPushMul * nnz; otherwise every unit with a missing column pulls (no
// atomics on global memory, but a pass over all in-edges). R-MAT 20, 64
// sources: at a work of 0.14 nnz pushing took 331 us and pulling 1,640 us, at
// 1.2 nnz 506 and 803 us; at 18 nnz pulling took 2.3 ms and pushing would
// issue 5.8e8 atomics.
constexpr unsigned long long kBcPushMul = 2;

__device__ __forceinline__ int64_t heavy_row(const BcArgs& p, int64_t h) { return p.rlast - h; }

__device__ __forceinline__ unsigned long long bc_columns(const BcArgs& p, int blk) {
    const int n = p.ns - blk * 64;
    return n >= 64 ? ~0ull : (1ull << n) - 1ull;
}

// Vertex and block of a key.
__device__ __forceinline__ int bc_block(const BcArgs& p, int32_t key, int32_t& v) {
    if (p.nblk == 1) {
        v = key;
        return 0;
    }
    const int blk = (int)(key / (int32_t)p.m);
    v = key - blk * (int32_t)p.m;
    return blk;
}

// Appends the row (key, mask) of vertex v to the rows found so far; lanes with
// mask 0 have none. Called by whole warps. Returns the lane's row's work.
__device__ __forceinline__ unsigned long long bc_append(const BcArgs& p, int32_t key, int32_t v,
                                                        unsigned long long mask) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int32_t od = mask ? p.ar[v + 1] - p.ar[v] : 0;
    const bool light = mask != 0ull && od <= p.piece;
    const unsigned lm = __ballot_sync(FULL, light);
    int32_t base = 0;
    if (lm && lane == 0) base = atomicAdd(&p.st->nrows, __popc(lm));
    base = __shfl_sync(FULL, base, 0);
    if (light) {
        const int32_t r = base + __popc(lm & ((1u << lane) - 1u));
        p.rkey[r] = key;
        p.rmask[r] = mask;
    } else if (mask) {
        const int32_t h = atomicAdd(&p.st->nhrows, 1);
        const int32_t n = (od + p.piece - 1) / p.piece;
        const int32_t f = atomicAdd(&p.st->nhtasks, n);
        p.rkey[heavy_row(p, h)] = key;
        p.rmask[heavy_row(p, h)] = mask;
        p.hfirst[h] = f;
        for (int32_t c = 0; c < n; ++c) p.htask[f + c] = make_int2(h, c);
    }
    return (unsigned long long)__popcll(mask) * (unsigned long long)od;
}

// Per vertex (one thread): a self-loop (rows are sorted, so a binary search
// finds it) and the pieces of heavy in-neighbour lists.
__global__ void k_bc_scan_vertices(BcArgs p) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < p.m; v += (int64_t)gridDim.x * blockDim.x) {
        const int32_t b = p.ar[v], n = p.ar[v + 1] - b;
        const int pos = lower_bound_i32(p.ac + b, n, (int32_t)v);
        if (pos < n && p.ac[b + pos] == (int32_t)v) atomicOr(&p.st->flags, 1);
        const int32_t in = p.atr[v + 1] - p.atr[v];
        if (in > p.piece) {
            const int32_t c = (in + p.piece - 1) / p.piece;
            const int32_t f = atomicAdd(&p.st->nchunk, c);
            for (int32_t i = 0; i < c; ++i) p.chunk[f + i] = make_int4((int32_t)v, i, f, c);
        }
    }
}

// The sources are in range and distinct (seen: one bit per vertex, cleared).
__global__ void k_bc_check_sources(BcArgs p, uint32_t* __restrict__ seen) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < p.nsrc; j += gridDim.x * blockDim.x) {
        const int32_t v = p.sources[j];
        if (v < 0 || (int64_t)v >= p.m) {
            atomicOr(&p.st->flags, 8);
            continue;
        }
        const uint32_t bit = 1u << (v & 31);
        if (atomicOr(&seen[v >> 5], bit) & bit) atomicOr(&p.st->flags, 16);
    }
}

// Batches with packed columns: on the vertices of graph g (union rows
// [voff[g], voff[g+1])), the columns at and above its source count are
// marked visited, so no value is ever made there and the vertex counts as
// reached by every column once its own sources have reached it.
__global__ void k_bc_previsit(BcArgs p, const int64_t* __restrict__ voff, const int32_t* __restrict__ gsrc,
                              int64_t count) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < p.m; v += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = count;  // the graph g with voff[g] <= v < voff[g+1]
        while (hi - lo > 1) {
            const int64_t mid = (lo + hi) >> 1;
            if (voff[mid] <= v) lo = mid; else hi = mid;
        }
        const int have = gsrc[lo];
        for (int b = 0; b < p.nblk; ++b) {
            const int n = have - b * 64;
            const unsigned long long own = n <= 0 ? 0ull : n >= 64 ? ~0ull : (1ull << n) - 1ull;
            p.V[(int64_t)b * p.m + v] = bc_columns(p, b) & ~own;
        }
    }
}

// The sources' rows: distance 0, one path. One block; nothing when a check
// failed (the loops then end at once).
__global__ void k_bc_init(BcArgs p) {
    BcState* st = p.st;
    const bool bad = st->flags != 0;
    if (!bad) {
        unsigned long long work = 0;
        for (int j0 = 0; j0 < p.nsrc; j0 += blockDim.x) {
            const int j = j0 + threadIdx.x;
            int32_t v = 0, key = 0;
            unsigned long long mask = 0;
            if (j < p.nsrc) {
                v = p.sources[j];
                const int c = p.scol ? p.scol[j] : j;
                mask = 1ull << (c & 63);
                key = (int32_t)((int64_t)(c >> 6) * p.m + v);
                p.S[(size_t)v * p.ns + c] = 1.0;
                // sources are distinct vertices: the unit is this source's alone
                p.V[key] |= mask;
                p.F[0][key] = mask;
            }
            work += bc_append(p, key, v, mask);
        }
        work = warp_sum<unsigned long long>(work);
        if ((threadIdx.x & 31) == 0 && work) atomicAdd(&st->cur_work, work);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    p.lrow[0] = 0;
    p.lhrow[0] = 0;
    p.ltask[0] = 0;
    p.lrow[1] = *(volatile int32_t*)&st->nrows;
    p.lhrow[1] = *(volatile int32_t*)&st->nhrows;
    p.ltask[1] = *(volatile int32_t*)&st->nhtasks;
    st->done = bad;
    const unsigned long long work = *(volatile unsigned long long*)&st->cur_work;
    st->mode = work < kBcPushMul * (unsigned long long)p.nnz ? 1 : 0;
}

// The columns of a 64-bit word side by side: s_col[i] = its i-th set bit.
__device__ __forceinline__ void bc_list_columns(unsigned long long word, uint8_t* s_col) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u, lo = (uint32_t)word, hi = (uint32_t)(word >> 32);
    if (lo >> lane & 1u) s_col[__popc(lo & lt)] = (uint8_t)lane;
    if (hi >> lane & 1u) s_col[__popc(lo) + __popc(hi & lt)] = (uint8_t)(32 + lane);
}

// Shared memory of one warp for the sums over its neighbours.
struct BcWarp {
    int32_t row[32];   // the group's neighbours: first index of their values
    uint8_t col[64];   // columns side by side
};

// Sums over neighbours [t0, t1): for every column c that some neighbour w has
// in bits[w] & need, the sum of X[w * ns + c] (times the edge's value) over
// those w. Returns these columns; the lane holds the sums acc0 of column c0
// and acc1 of column c1 (-1: none).
//
// A first pass over the words finds the columns, which then share out the
// lanes: one column per lane and list (two lists above 32 columns), or, with
// at most 16 columns, 2 to 32 lanes per column, each with its share of the
// neighbours. The neighbours are visited 32 at a time: the words transposed
// across the warp give each lane the list of neighbours that hold its column,
// and the warp takes as many steps as the longest list.
template <bool UNIT>
__device__ __forceinline__ unsigned long long bc_gather(const int32_t* __restrict__ col,
                                                        const double* __restrict__ val, int32_t t0, int32_t t1,
                                                        const unsigned long long* bits, const double* X, int ns,
                                                        unsigned long long need, BcWarp& sh, double* s_a,
                                                        double& acc0, double& acc1, int& c0, int& c1) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    acc0 = acc1 = 0.0;
    c0 = c1 = -1;
    int32_t t = t0 + lane;
    int32_t w = t < t1 ? __ldg(col + t) : 0;
    unsigned long long f = t < t1 ? bits[w] & need : 0ull;
    unsigned long long any = f;
#pragma unroll 4
    for (int32_t g = t + 32; g < t1; g += 32) any |= bits[__ldg(col + g)];
    any &= need;
    const uint32_t flo = __reduce_or_sync(FULL, (uint32_t)any), fhi = __reduce_or_sync(FULL, (uint32_t)(any >> 32));
    const unsigned long long found = ((unsigned long long)fhi << 32) | flo;
    if (found == 0ull) return 0ull;
    const int n = __popcll(found);
    __syncwarp();
    bc_list_columns(found, sh.col);
    __syncwarp();
    const int lg = n > 16 ? 0 : n > 8 ? 1 : n > 4 ? 2 : n > 2 ? 3 : n > 1 ? 4 : 5;
    if ((lane >> lg) < n) c0 = sh.col[lane >> lg];
    if (lane + 32 < n) c1 = sh.col[lane + 32];
    // the lane's share of a group's neighbours
    uint32_t share = 0;
    if (c0 >= 0) {
        share = lg == 0 ? 0xffffffffu : lg == 1 ? 0x55555555u : lg == 2 ? 0x11111111u : lg == 3 ? 0x01010101u
              : lg == 4 ? 0x00010001u : 1u;
        share <<= lane & ((1 << lg) - 1);
    }
    auto walk = [&](uint32_t mine, int c, double& acc) {
        while (mine) {
            double x[kBcLoads], a[kBcLoads];
            bool on[kBcLoads];
#pragma unroll
            for (int h = 0; h < kBcLoads; ++h) {
                on[h] = mine != 0u;
                if (on[h]) {
                    const int j = __ffs(mine) - 1;
                    mine &= mine - 1;
                    x[h] = X[sh.row[j] + c];
                    if (!UNIT) a[h] = s_a[j];
                }
            }
#pragma unroll
            for (int h = 0; h < kBcLoads; ++h)
                if (on[h]) acc = UNIT ? acc + x[h] : acc + a[h] * x[h];
        }
    };
    for (int32_t g = t0; g < t1; g += 32) {
        const int32_t cw = w, ct = t;
        const unsigned long long cf = f;
        // the next group's words load while this group is summed
        t += 32;
        w = t < t1 ? __ldg(col + t) : 0;
        f = t < t1 ? bits[w] & need : 0ull;
        if (__ballot_sync(FULL, cf != 0ull) == 0u) continue;
        __syncwarp();  // the last group's list is read
        sh.row[lane] = cw * ns;
        if (!UNIT && cf) s_a[lane] = __ldg(val + ct);
        __syncwarp();
        // bit j: neighbour j holds the column
        const uint32_t m0 = flo ? warp_transpose_bits((uint32_t)cf) : 0u;
        const uint32_t m1 = fhi ? warp_transpose_bits((uint32_t)(cf >> 32)) : 0u;
        uint32_t lo = __shfl_sync(FULL, m0, c0 & 31), hi = __shfl_sync(FULL, m1, c0 & 31);
        walk((c0 & 32 ? hi : lo) & share, c0, acc0);
        if (n > 32) {
            __syncwarp();
            lo = __shfl_sync(FULL, m0, c1 & 31);
            hi = __shfl_sync(FULL, m1, c1 & 31);
            walk(c1 < 0 ? 0u : c1 & 32 ? hi : lo, c1, acc1);
        }
        __syncwarp();
    }
    for (int o = 1; o < (1 << lg); o <<= 1) acc0 += __shfl_xor_sync(FULL, acc0, o);
    if (lane & ((1 << lg) - 1)) c0 = -1;  // one lane per column
    return found;
}

// One heavy piece, by a warp: neighbours [t0, t1) of one unit. Its sums go to
// the piece's place; true when the piece is the last of `count` to arrive at
// `first`, with the columns of all of them and their sums (acc0: column
// `lane`, acc1: column 32 + `lane`).
template <bool UNIT>
__device__ __forceinline__ bool bc_piece(const BcArgs& p, const int32_t* col, const double* val, int32_t t0,
                                         int32_t t1, const unsigned long long* bits, const double* X,
                                         unsigned long long need, int64_t place, int64_t first, int32_t count,
                                         BcWarp& sh, double* s_a, double& acc0, double& acc1,
                                         unsigned long long& mask) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int c0, c1;
    mask = bc_gather<UNIT>(col, val, t0, t1, bits, X, p.ns, need, sh, s_a, acc0, acc1, c0, c1);
    if (c0 >= 0) p.part[place * 64 + c0] = acc0;
    if (c1 >= 0) p.part[place * 64 + c1] = acc1;
    if (lane == 0) p.pmask[place] = mask;
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) {
        last = atomicAdd(p.pdone + first, 1) == count - 1;
        if (last) p.pdone[first] = 0;
    }
    if (!__shfl_sync(FULL, last, 0)) return false;
    __threadfence();
    acc0 = acc1 = 0.0;
    mask = 0ull;
    for (int32_t c = 0; c < count; ++c) {
        const unsigned long long m = __ldcg(p.pmask + first + c);
        if (m >> lane & 1ull) acc0 += __ldcg(p.part + (first + c) * 64 + lane);
        if (m >> (lane + 32) & 1ull) acc1 += __ldcg(p.part + (first + c) * 64 + 32 + lane);
        mask |= m;
    }
    return true;
}

// Items per take.
__device__ __forceinline__ int bc_take(int64_t items, int most) {
    const int64_t n = items / ((int64_t)gridDim.x * kBcWarps * 4);
    return n < 1 ? 1 : n > most ? most : (int)n;
}

// The warp's first task of a level, dealt out by its number (neighbouring tasks
// to different CTAs), and its next one. With the first from the counter too,
// all the grid's warps take one, most of a small level's to find none (32
// sources, 10,000 vertices: 445 us, so 429).
__device__ __forceinline__ int32_t bc_first() { return blockIdx.x + (threadIdx.x >> 5) * gridDim.x; }
__device__ __forceinline__ int32_t bc_next(const BcArgs& p) {
    int32_t t = 0;
    if ((threadIdx.x & 31) == 0) t = atomicAdd(&p.st->next, 1);
    return gridDim.x * kBcWarps + __shfl_sync(0xffffffffu, t, 0);
}

// Push: the row (unit key with columns mask) of vertex u and its
// out-neighbours [t0, t1), lanes over neighbours: S[w][c] += A[u][w] * S[u][c]
// for every column c that has not reached w; the first touch of w's unit lists
// it.
template <bool UNIT>
__device__ __forceinline__ void bc_push_row(const BcArgs& p, unsigned long long* Fn, int blk, int32_t u,
                                            unsigned long long mask, int32_t t0, int32_t t1) {
    const int lane = threadIdx.x & 31;
    const double* src = p.S + (size_t)u * p.ns + blk * 64;
    for (int32_t t = t0 + lane; t < t1; t += 32) {
        const int32_t w = __ldg(p.ac + t);
        const int64_t key = (int64_t)blk * p.m + w;
        unsigned long long add = mask & ~p.V[key];
        if (add == 0ull) continue;
        const double a = UNIT ? 1.0 : __ldg(p.av + t);
        if (atomicOr(Fn + key, add) == 0ull) p.tlist[atomicAdd(&p.st->ntouched, 1)] = (int32_t)key;
        double* dst = p.S + (size_t)w * p.ns + blk * 64;
        while (add) {
            const int c = __ffsll((long long)add) - 1;
            add &= add - 1;
            atomicAdd(dst + c, UNIT ? src[c] : a * src[c]);
        }
    }
}

// One forward level.
template <bool UNIT>
__global__ void __launch_bounds__(kBcThreads, 4) k_bc_forward(const BcArgs* __restrict__ ap) {
    __shared__ BcWarp s_warp[kBcWarps];
    __shared__ double s_a[UNIT ? 1 : kBcWarps][32];
    const BcArgs& p = *ap;
    const BcState* st = p.st;
    if (st->done) return;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* my_a = UNIT ? nullptr : s_a[UNIT ? 0 : wid];
    const int d = st->d;
    const unsigned long long* Fc = p.F[d % 3];
    unsigned long long* Fn = p.F[(d + 1) % 3];
    unsigned long long work = 0;
    if (st->mode != 0) {
        const int32_t task0 = p.ltask[d], ntask = p.ltask[d + 1] - task0;
        const int32_t row0 = p.lrow[d], nrow = p.lrow[d + 1] - row0;
        for (int32_t t = bc_first(); t < ntask + nrow; t = bc_next(p)) {
            int32_t u;
            if (t < ntask) {
                const int2 task = p.htask[task0 + t];
                const int64_t hr = heavy_row(p, task.x);
                const int blk = bc_block(p, p.rkey[hr], u);
                const int32_t b = p.ar[u] + task.y * p.piece;
                bc_push_row<UNIT>(p, Fn, blk, u, p.rmask[hr], b, min(p.ar[u + 1], b + p.piece));
            } else {
                const int32_t r = row0 + t - ntask;
                const int blk = bc_block(p, p.rkey[r], u);
                bc_push_row<UNIT>(p, Fn, blk, u, p.rmask[r], p.ar[u], p.ar[u + 1]);
            }
        }
    } else {
        // pieces of heavy vertices' in-neighbour lists, then the other units,
        // a take's far apart (hubs sit together)
        const int nchunk = st->nchunk;
        const int64_t units = p.m * p.nblk, nheavy = (int64_t)nchunk * p.nblk;
        const int take = bc_take(units, kBcUnits);
        const int64_t ntake = (units + take - 1) / take;
        for (int64_t t = bc_first(); t < nheavy + ntake; t = bc_next(p)) {
            if (t < nheavy) {
                const int blk = (int)(t / nchunk);
                const int64_t off = (int64_t)blk * nchunk;
                const int4 c = p.chunk[t - off];
                const int32_t v = c.x;
                const int64_t key = (int64_t)blk * p.m + v;
                const unsigned long long vis = __ldcg(p.V + key), need = bc_columns(p, blk) & ~vis;
                if (need == 0ull) continue;  // the same for all pieces: only the last to arrive changes V
                const int32_t b = p.atr[v] + c.y * p.piece;
                double acc0, acc1;
                unsigned long long mask;
                if (!bc_piece<UNIT>(p, p.atc, p.atv, b, min(p.atr[v + 1], b + p.piece), Fc + (int64_t)blk * p.m,
                                    p.S + blk * 64, need, off + c.z + c.y, off + c.z, c.w, s_warp[wid], my_a, acc0, acc1,
                                    mask))
                    continue;
                double* dst = p.S + (size_t)v * p.ns + blk * 64 + lane;
                if (mask >> lane & 1ull) dst[0] = acc0;
                if (mask >> (lane + 32) & 1ull) dst[32] = acc1;
                const unsigned long long mine = lane == 0 ? mask : 0ull;
                if (mine) {
                    p.V[key] = vis | mine;
                    Fn[key] = mine;
                }
                work += bc_append(p, (int32_t)key, v, mine);
                continue;
            }
            const int64_t key = t - nheavy + (int64_t)lane * ntake;
            int32_t v = 0, ab = 0, ae = 0;
            int blk = 0;
            unsigned long long need = 0, vis = 0, found = 0;
            if (lane < take && key < units) {
                blk = bc_block(p, (int32_t)key, v);
                ab = p.atr[v];
                ae = p.atr[v + 1];
                if (ae > ab && ae - ab <= p.piece) {
                    vis = p.V[key];
                    need = bc_columns(p, blk) & ~vis;
                }
            }
            unsigned act = __ballot_sync(FULL, need != 0ull);
            while (act) {
                const int l = __ffs(act) - 1;
                act &= act - 1;
                const int32_t b = __shfl_sync(FULL, ab, l), e = __shfl_sync(FULL, ae, l);
                const int32_t vv = __shfl_sync(FULL, v, l);
                const int bb = __shfl_sync(FULL, blk, l);
                const unsigned long long nd = __shfl_sync(FULL, need, l);
                double acc0, acc1;
                int c0, c1;
                const unsigned long long got = bc_gather<UNIT>(p.atc, p.atv, b, e, Fc + (int64_t)bb * p.m,
                                                               p.S + bb * 64, p.ns, nd, s_warp[wid], my_a, acc0,
                                                               acc1, c0, c1);
                double* dst = p.S + (size_t)vv * p.ns + bb * 64;
                if (c0 >= 0) dst[c0] = acc0;
                if (c1 >= 0) dst[c1] = acc1;
                if (lane == l) found = got;
            }
            if (found) {
                p.V[key] = vis | found;
                Fn[key] = found;
            }
            if (__ballot_sync(FULL, found != 0ull)) work += bc_append(p, (int32_t)key, v, found);
        }
    }
    work = warp_sum<unsigned long long>(work);
    if (lane == 0 && work) atomicAdd(&p.st->next_work, work);
    // the buffer after next: the last level's frontier leaves it
    if (d > 0) {
        unsigned long long* Fo = p.F[(d - 1) % 3];
        const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
        for (int64_t r = p.lrow[d - 1] + i0; r < p.lrow[d]; r += step) Fo[p.rkey[r]] = 0ull;
        for (int64_t r = p.lhrow[d - 1] + i0; r < p.lhrow[d]; r += step) Fo[p.rkey[heavy_row(p, r)]] = 0ull;
    }
}

// Ends a forward level: a push level's units append their rows; the last
// block closes the level's lists, chooses the next one's direction and tells
// the loop whether to go on.
__global__ void __launch_bounds__(kBcThreads) k_bc_forward_end(const BcArgs* __restrict__ ap, LoopCtl ctl) {
    __shared__ bool s_last;
    const BcArgs& p = *ap;
    BcState* st = p.st;
    const int lane = threadIdx.x & 31;
    const int d = st->d;
    if (!st->done && st->mode != 0) {
        unsigned long long* Fn = p.F[(d + 1) % 3];
        const int n = st->ntouched;
        unsigned long long work = 0;
        for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n;
             i0 += (int64_t)gridDim.x * blockDim.x) {
            const int64_t i = i0 + lane;
            int32_t key = 0, v = 0;
            unsigned long long mask = 0;
            if (i < n) {
                key = p.tlist[i];
                bc_block(p, key, v);
                mask = Fn[key];
                p.V[key] |= mask;
            }
            work += bc_append(p, key, v, mask);
        }
        work = warp_sum<unsigned long long>(work);
        if (lane == 0 && work) atomicAdd(&st->next_work, work);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&st->blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    st->blocks = 0;
    st->next = 0;
    bool more = false;
    if (!st->done) {
        const int32_t rows = *(volatile int32_t*)&st->nrows, hrows = *(volatile int32_t*)&st->nhrows;
        if (rows == p.lrow[d + 1] && hrows == p.lhrow[d + 1]) {
            st->done = 1;
        } else {
            p.lrow[d + 2] = rows;
            p.lhrow[d + 2] = hrows;
            p.ltask[d + 2] = *(volatile int32_t*)&st->nhtasks;
            const unsigned long long work = *(volatile unsigned long long*)&st->next_work;
            st->cur_work = work;
            st->next_work = 0;
            st->ntouched = 0;
            st->mode = work < kBcPushMul * (unsigned long long)p.nnz ? 1 : 0;
            st->d = d + 1;
            // distances are below m
            more = (int64_t)(d + 1) < p.m;
            if (!more) st->done = 1;
        }
    }
    if (!more) st->k = st->flags ? 0 : st->d;
    loop_continue(ctl, more);
}

// Before the backward loop: W = 1 / sigma and the bits of the largest distance.
__global__ void k_bc_back_init(const BcArgs* __restrict__ ap) {
    const BcArgs& p = *ap;
    const int k = p.st->k;
    if (k < 2) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t nl = p.lrow[k + 1] - p.lrow[k], n = nl + p.lhrow[k + 1] - p.lhrow[k];
    unsigned long long* L = p.F[k % 3];
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
        const int64_t r = i < nl ? p.lrow[k] + i : heavy_row(p, p.lhrow[k] + i - nl);
        const int32_t key = p.rkey[r];
        const unsigned long long mask = p.rmask[r];
        int32_t v;
        const int blk = bc_block(p, key, v);
        const size_t at = (size_t)v * p.ns + blk * 64 + lane;
        if (mask >> lane & 1ull) p.W[at] = 1.0 / p.S[at];
        if (mask >> (lane + 32) & 1ull) p.W[at + 32] = 1.0 / p.S[at + 32];
        if (lane == 0) L[key] = mask;
    }
}

// One backward level: the rows at distance k - 1 (their neighbours at
// distance k have W and their bits in F[k % 3]).
template <bool UNIT>
__global__ void __launch_bounds__(kBcThreads, 4) k_bc_backward(const BcArgs* __restrict__ ap, LoopCtl ctl) {
    __shared__ BcWarp s_warp[kBcWarps];
    __shared__ double s_a[UNIT ? 1 : kBcWarps][32];
    __shared__ double s_acc[kBcWarps][64];
    __shared__ double s_part[kBcWarps][kBcRows][33];
    __shared__ bool s_last;
    const BcArgs& p = *ap;
    BcState* st = p.st;
    const int k = st->k;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double* my_a = UNIT ? nullptr : s_a[UNIT ? 0 : wid];
    if (k >= 2) {
        const unsigned long long* Lk = p.F[k % 3];
        unsigned long long* Ln = p.F[(k - 1) % 3];
        const bool next = k > 2;  // distance 1 needs no W: the sources take no score from their own searches
        // a row's sums (s_acc, by column) become its scores, W and bits; the
        // lane's part of the score. The row's columns are put side by side: up
        // to 32 of them take one round of FP64 work instead of two.
        auto finish = [&](int32_t v, int blk, int32_t key, unsigned long long mask) {
            __syncwarp();
            bc_list_columns(mask, s_warp[wid].col);
            __syncwarp();
            const int n = __popcll(mask);
            double part = 0.0;
            for (int e = lane; e < n; e += 32) {
                const int c = s_warp[wid].col[e];
                const size_t at = (size_t)v * p.ns + blk * 64 + c;
                const double sg = p.S[at], a = s_acc[wid][c];
                part += a * sg;
                if (next) p.W[at] = 1.0 / sg + a;
            }
            if (lane == 0) Ln[key] = mask;
            __syncwarp();
            return part;
        };
        const int32_t task0 = p.ltask[k - 1], ntask = p.ltask[k] - task0;
        const int32_t row0 = p.lrow[k - 1], row1 = p.lrow[k];
        const int take = bc_take(row1 - row0, kBcRows);
        const int32_t ntake = (row1 - row0 + take - 1) / take;
        for (int32_t t = bc_first(); t < ntask + ntake; t = bc_next(p)) {
            if (t < ntask) {  // a piece of a heavy row
                const int2 task = p.htask[task0 + t];
                const int64_t hr = heavy_row(p, task.x);
                const int32_t key = p.rkey[hr];
                const unsigned long long mask = p.rmask[hr];
                int32_t v;
                const int blk = bc_block(p, key, v);
                const int32_t vb = p.ar[v], ve = p.ar[v + 1], b = vb + task.y * p.piece;
                const int32_t first = p.hfirst[task.x] - task0;
                double acc0, acc1;
                unsigned long long got;
                if (!bc_piece<UNIT>(p, p.ac, p.av, b, min(ve, b + p.piece), Lk + (int64_t)blk * p.m, p.W + blk * 64,
                                    mask, first + task.y, first, (ve - vb + p.piece - 1) / p.piece, s_warp[wid], my_a,
                                    acc0, acc1, got))
                    continue;
                s_acc[wid][lane] = acc0;
                s_acc[wid][32 + lane] = acc1;
                const double part = warp_sum<double>(finish(v, blk, key, mask));
                if (lane == 0 && part != 0.0) atomicAdd(&p.bc[v], part);
                continue;
            }
            // a take of the other rows; their score sums are added together
            // (10 FP64 instructions for up to eight rows instead of 5 per row)
            const int32_t r0 = row0 + (t - ntask) * take, nr = min(take, row1 - r0);
            int32_t lkey = 0, lv = 0, lb = 0, le = 0;
            int lblk = 0;
            unsigned long long lmask = 0;
            if (lane < nr) {
                lkey = p.rkey[r0 + lane];
                lmask = p.rmask[r0 + lane];
                lblk = bc_block(p, lkey, lv);
                lb = p.ar[lv];
                le = p.ar[lv + 1];
            }
            for (int i = 0; i < nr; ++i) {
                const unsigned FULL = 0xffffffffu;
                const unsigned long long mask = __shfl_sync(FULL, lmask, i);
                const int blk = __shfl_sync(FULL, lblk, i);
                double acc0, acc1;
                int c0, c1;
                bc_gather<UNIT>(p.ac, p.av, __shfl_sync(FULL, lb, i), __shfl_sync(FULL, le, i),
                                Lk + (int64_t)blk * p.m, p.W + blk * 64, p.ns, mask, s_warp[wid], my_a, acc0, acc1, c0,
                                c1);
                s_acc[wid][lane] = 0.0;
                s_acc[wid][32 + lane] = 0.0;
                __syncwarp();
                if (c0 >= 0) s_acc[wid][c0] = acc0;
                if (c1 >= 0) s_acc[wid][c1] = acc1;
                s_part[wid][i][lane] = finish(__shfl_sync(FULL, lv, i), blk, __shfl_sync(FULL, lkey, i), mask);
            }
            for (int i = nr; i < kBcRows; ++i) s_part[wid][i][lane] = 0.0;
            __syncwarp();
            // four lanes per row, eight columns each
            const int r = lane & 7, q = lane >> 3;
            double s = 0.0;
#pragma unroll
            for (int c = 0; c < 8; ++c) s += s_part[wid][r][q * 8 + c];
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (lane < nr && s != 0.0) atomicAdd(&p.bc[lv], s);
            __syncwarp();
        }
        // the buffer after next: distance k + 1 leaves it
        unsigned long long* Lo = p.F[(k + 1) % 3];
        if (k < st->d) {
            const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
            for (int64_t r = p.lrow[k + 1] + i0; r < p.lrow[k + 2]; r += step) Lo[p.rkey[r]] = 0ull;
            for (int64_t r = p.lhrow[k + 1] + i0; r < p.lhrow[k + 2]; r += step) Lo[p.rkey[heavy_row(p, r)]] = 0ull;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&st->blocks, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    st->blocks = 0;
    st->next = 0;
    if (k >= 1) st->k = k - 1;
    loop_continue(ctl, k - 1 >= 2);
}

// Packed source columns of a batch over a block-diagonal union (device
// arrays): each source's column, the graphs' first rows (count + 1 of them)
// and their source counts; ncols = the largest source count.
struct BcPacking {
    const int32_t* scol = nullptr;
    const int64_t* voff = nullptr;
    const int32_t* gsrc = nullptr;
    int64_t count = 0;
    int ncols = 0;
};

template <typename K>
static int bc_grid(ga_ctx ctx, K kernel) {
    int per_sm = 1;
    GA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBcThreads, 0));
    return ctx->num_sms * std::max(per_sm, 1);
}

// Sizes of the state.
struct BcSizes {
    size_t units, pairs;  // (block, vertex) and (vertex, column)
    int piece;
    // pieces of the longer of the two heavy lists: at most nnz / piece full
    // ones and one more per heavy vertex; a heavy vertex has a row in at
    // most ns levels, and a level's rows of one vertex are one per block
    size_t pieces, hrows;
};

static BcSizes bc_sizes(int64_t m, int64_t nnz, int64_t ns) {
    BcSizes z;
    z.units = (size_t)m * (size_t)((ns + 63) / 64);
    z.pairs = (size_t)m * (size_t)ns;
    z.piece = nnz > (int64_t)kBcDense * m ? kBcPieceDense : kBcPiece;
    z.pieces = (size_t)(2 * (nnz / z.piece) + 1);
    z.hrows = std::min(z.pairs, (size_t)(nnz / z.piece) * (size_t)ns) + 1;
    return z;
}

// The arrays of bc_device, in its order, behind an FP64 copy and its
// transpose; or what the transpose takes while it is made.
int64_t bc_bytes(int64_t m, int64_t nnz, int64_t ns) {
    const BcSizes z = bc_sizes(m, nnz, ns);
    const size_t places = z.pieces * (size_t)((ns + 63) / 64);
    const size_t state = sizeof(BcState) + sizeof(uint32_t) * (size_t)((m + 31) / 32) +
                         4 * sizeof(unsigned long long) * z.units + 2 * sizeof(double) * z.pairs +
                         (sizeof(int32_t) + sizeof(unsigned long long)) * z.pairs + sizeof(int32_t) * z.hrows +
                         sizeof(int2) * z.pieces * (size_t)ns + sizeof(int32_t) * 3 * ((size_t)m + 3) +
                         sizeof(int4) * z.pieces + sizeof(double) * places * 64 +
                         (sizeof(unsigned long long) + sizeof(int32_t)) * places + sizeof(int32_t) * z.units;
    const int64_t matrix = (int64_t)sizeof(int32_t) * (m + 1) + 12 * (nnz + 1);
    return 2 * matrix + std::max((int64_t)state, transpose_bytes(nnz, GA_FP64));
}

// accumulate: add this batch's scores to d_bc instead of overwriting it.
static void bc_device(ga_ctx ctx, ga_csr A, const int32_t* d_sources, int64_t nsrc, double* d_bc,
                      bool accumulate = false, const BcPacking* pk = nullptr) {
    GA_REQUIRE(A->m == A->n, GA_ERR_SHAPE, "non-square matrix; BC is only for square matrices");
    GA_REQUIRE(nsrc >= 0 && (pk || nsrc <= kBcMaxSources), GA_ERR_INVALID_ARG,
               "BC: between 0 and 1024 sources per batch");
    GA_REQUIRE(!pk || (pk->ncols >= 1 && pk->ncols <= kBcMaxSources), GA_ERR_INVALID_ARG,
               "BC: between 1 and 1024 sources per graph of a batch");
    const int64_t m = A->m;
    if (!accumulate) GA_CUDA(cudaMemsetAsync(d_bc, 0, sizeof(double) * (m ? m : 1), ctx->stream));
    if (m == 0 || nsrc == 0) return;
    const int ns = pk ? pk->ncols : (int)nsrc;  // source columns
    const int nblk = (ns + 63) / 64;
    GA_REQUIRE(m * (int64_t)(ns + 1) + nsrc < INT32_MAX, GA_ERR_UNSUPPORTED,
               "BC: m x sources exceeds the int32 entry range");
    ProfScope whole(ctx, "bc");
    // Values enter the algebra as FP64. All-ones values are never read (the
    // unit kernels), so A's own arrays serve; otherwise an FP64 copy. A
    // symmetric A is its own transpose. Both properties are cached on the
    // handle after their first check.
    const bool unit = csr_unit_values(ctx, A);
    const bool symmetric = csr_is_symmetric(ctx, A);
    ga_csr Ad = unit ? nullptr : copy_csr(ctx, A, GA_FP64);
    ga_csr AT = nullptr;
    try {
        ga_csr Av = unit ? A : Ad;
        if (!symmetric) AT = transpose_csr(ctx, Av);
        ga_csr ATu = symmetric ? Av : AT;
        const BcSizes z = bc_sizes(m, A->nnz, ns);
        const size_t units = z.units, pairs = z.pairs, pieces = z.pieces, hrows = z.hrows;
        const int piece = z.piece;
        DBuf<BcState> st(ctx, 1);
        DBuf<uint32_t> seen(ctx, (size_t)(m + 31) / 32);
        DBuf<unsigned long long> words(ctx, 4 * units);  // V, F[0], F[1], F[2]
        DBuf<double> S(ctx, pairs), W(ctx, pairs);
        DBuf<int32_t> rkey(ctx, pairs);
        DBuf<unsigned long long> rmask(ctx, pairs);
        DBuf<int32_t> hfirst(ctx, hrows);
        DBuf<int2> htask(ctx, pieces * ns);
        DBuf<int32_t> levels(ctx, 3 * ((size_t)m + 3));
        DBuf<int4> chunk(ctx, pieces);
        DBuf<double> part(ctx, pieces * nblk * 64);
        DBuf<unsigned long long> pmask(ctx, pieces * nblk);
        DBuf<int32_t> pdone(ctx, pieces * nblk), tlist(ctx, units);
        BcArgs p;
        p.atr = ATu->rst; p.atc = ATu->col; p.atv = unit ? nullptr : static_cast<const double*>(ATu->val);
        p.ar = Av->rst; p.ac = Av->col; p.av = unit ? nullptr : static_cast<const double*>(Av->val);
        p.m = m; p.nnz = A->nnz; p.ns = ns; p.nblk = nblk; p.piece = piece; p.nsrc = (int)nsrc;
        p.sources = d_sources; p.scol = pk ? pk->scol : nullptr;
        p.st = st.p;
        p.V = words.p;
        for (int b = 0; b < 3; ++b) p.F[b] = words.p + (size_t)(b + 1) * units;
        p.S = S.p; p.W = W.p;
        p.rkey = rkey.p; p.rmask = rmask.p;
        p.rlast = (int64_t)pairs - 1; p.hfirst = hfirst.p; p.htask = htask.p;
        p.lrow = levels.p; p.lhrow = levels.p + (m + 3); p.ltask = levels.p + 2 * (m + 3);
        p.chunk = chunk.p; p.part = part.p; p.pmask = pmask.p; p.pdone = pdone.p; p.tlist = tlist.p;
        p.bc = d_bc;
        GA_CUDA(cudaMemsetAsync(st.p, 0, sizeof(BcState), ctx->stream));
        GA_CUDA(cudaMemsetAsync(seen.p, 0, sizeof(uint32_t) * seen.count, ctx->stream));
        GA_CUDA(cudaMemsetAsync(words.p, 0, sizeof(unsigned long long) * words.count, ctx->stream));
        GA_CUDA(cudaMemsetAsync(S.p, 0, sizeof(double) * pairs, ctx->stream));  // push levels add into it
        GA_CUDA(cudaMemsetAsync(pdone.p, 0, sizeof(int32_t) * pdone.count, ctx->stream));
        const int grid_v = grid_for(m, 256, ctx->num_sms * 8);
        k_bc_scan_vertices<<<grid_v, 256, 0, ctx->stream>>>(p);
        post_launch("bc_scan_vertices");
        k_bc_check_sources<<<grid_for(nsrc, 256, 64), 256, 0, ctx->stream>>>(p, seen.p);
        post_launch("bc_check_sources");
        if (pk) {
            k_bc_previsit<<<grid_v, 256, 0, ctx->stream>>>(p, pk->voff, pk->gsrc, pk->count);
            post_launch("bc_previsit");
        }
        k_bc_init<<<1, kBcThreads, 0, ctx->stream>>>(p);
        post_launch("bc_init");
        // The loops' kernels read the call's parameters from a device copy
        // and have fixed grids, so the context captures each loop once.
        const int fslot = unit ? kLoopSlotBcForward : kLoopSlotBcForwardVal;
        const int bslot = unit ? kLoopSlotBcBackward : kLoopSlotBcBackwardVal;
        BcArgs* fargs = static_cast<BcArgs*>(cached_loop_args(ctx, fslot, sizeof(BcArgs)));
        BcArgs* bargs = static_cast<BcArgs*>(cached_loop_args(ctx, bslot, sizeof(BcArgs)));
        GA_CUDA(cudaMemcpyAsync(fargs, &p, sizeof(BcArgs), cudaMemcpyHostToDevice, ctx->stream));
        GA_CUDA(cudaMemcpyAsync(bargs, &p, sizeof(BcArgs), cudaMemcpyHostToDevice, ctx->stream));
        auto fwd = unit ? k_bc_forward<true> : k_bc_forward<false>;
        auto bwd = unit ? k_bc_backward<true> : k_bc_backward<false>;
        const int grid_fwd = bc_grid(ctx, fwd), grid_bwd = bc_grid(ctx, bwd), grid_end = ctx->num_sms;
        {
            ProfScope ps(ctx, "bc_forward_loop");
            run_cached_loop(ctx, fslot, [ctx, fwd, fargs, grid_fwd, grid_end](const LoopCtl& ctl) {
                {
                    ProfScope pf(ctx, "bc_forward");
                    fwd<<<grid_fwd, kBcThreads, 0, ctx->stream>>>(fargs);
                    post_launch("bc_forward");
                }
                k_bc_forward_end<<<grid_end, kBcThreads, 0, ctx->stream>>>(fargs, ctl);
                post_launch("bc_forward_end");
            }, m + 2);
        }
        {
            ProfScope ps(ctx, "bc_backward_loop");
            GA_CUDA(cudaMemsetAsync(p.F[0], 0, sizeof(unsigned long long) * 3 * units, ctx->stream));
            k_bc_back_init<<<ctx->num_sms * 4, 256, 0, ctx->stream>>>(bargs);
            post_launch("bc_back_init");
            run_cached_loop(ctx, bslot, [ctx, bwd, bargs, grid_bwd](const LoopCtl& ctl) {
                ProfScope pb(ctx, "bc_backward");
                bwd<<<grid_bwd, kBcThreads, 0, ctx->stream>>>(bargs, ctl);
                post_launch("bc_backward");
            }, m + 2);
        }
        BcState hs;
        GA_CUDA(cudaMemcpyAsync(&hs, st.p, sizeof(BcState), cudaMemcpyDeviceToHost, ctx->stream));
        GA_CUDA(cudaStreamSynchronize(ctx->stream));
        GA_REQUIRE(!(hs.flags & 1), GA_ERR_INVALID_ARG, "BC: the graph has self-loops");
        GA_REQUIRE(!(hs.flags & 8), GA_ERR_INVALID_ARG, "BC: source index out of range");
        GA_REQUIRE(!(hs.flags & 16), GA_ERR_INVALID_ARG, "BC: sources must be distinct");
    } catch (...) {
        csr_destroy(ctx, AT);
        csr_destroy(ctx, Ad);
        throw;
    }
    csr_destroy(ctx, AT);
    csr_destroy(ctx, Ad);
}

__global__ void k_bc_iota(int32_t* __restrict__ out, int64_t first, int64_t n) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
        out[j] = (int32_t)(first + j);
}

// All-source BC (betweenness_centrality, include/betweenness_centrality.h:
// 5-123): sources 0..m-1 in blocks of `block`, every block's scores added
// into d_bc on the device. The reference adds each block's row sums minus
// the block's size (:103-111), which is the block's dependency sum, as
// bc_device computes it. A block larger than one device batch (1,024
// sources) runs as consecutive batches of at most 1,024: BC is a sum over
// sources, so the block size changes only the order of the additions.
static void bc_all_device(ga_ctx ctx, ga_csr A, int64_t block, double* d_bc) {
    GA_REQUIRE(A->m == A->n, GA_ERR_SHAPE, "non-square matrix; BC is only for square matrices");
    GA_REQUIRE(block >= 1, GA_ERR_INVALID_ARG, "BC: the block size must be at least 1");
    const int64_t m = A->m;
    GA_CUDA(cudaMemsetAsync(d_bc, 0, sizeof(double) * (m ? m : 1), ctx->stream));
    if (m == 0) return;
    const int64_t per = std::min<int64_t>(std::min<int64_t>(block, kBcMaxSources), m);
    DBuf<int32_t> src(ctx, (size_t)per);
    ProfScope ps(ctx, "bc_all");
    for (int64_t i = 0; i < m; i += block) {
        const int64_t n = std::min(block, m - i);
        for (int64_t j = 0; j < n; j += per) {
            const int64_t c = std::min(per, n - j);
            k_bc_iota<<<grid_for(c, 256, 64), 256, 0, ctx->stream>>>(src.p, i + j, c);
            post_launch("bc_iota");
            bc_device(ctx, A, src.p, c, d_bc, true);
        }
    }
}

void bc_union_device(ga_ctx ctx, ga_csr U, int64_t count, const int64_t* voff, const int64_t* soff,
                     const int32_t* sources, double* d_bc) {
    GA_REQUIRE(soff[0] == 0, GA_ERR_INVALID_ARG, "batched BC: source offsets must start at 0");
    const int64_t ns = soff[count];
    GA_REQUIRE(ns >= 0 && (ns == 0 || sources), GA_ERR_INVALID_ARG, "batched BC: sources missing");
    // graph g's sources, shifted to its rows of the union; source j of graph
    // g takes column j
    std::vector<int32_t> global((size_t)(ns > 0 ? ns : 1)), col((size_t)(ns > 0 ? ns : 1));
    std::vector<int32_t> gsrc((size_t)(count > 0 ? count : 1), 0);
    int64_t ncols = 0;
    for (int64_t g = 0; g < count; ++g) {
        GA_REQUIRE(soff[g] <= soff[g + 1], GA_ERR_INVALID_ARG, "batched BC: source offsets must not decrease");
        const int64_t mg = voff[g + 1] - voff[g];
        GA_REQUIRE(soff[g + 1] - soff[g] <= kBcMaxSources, GA_ERR_INVALID_ARG,
                   "batched BC: at most 1024 sources per graph");
        for (int64_t j = soff[g]; j < soff[g + 1]; ++j) {
            GA_REQUIRE(sources[j] >= 0 && sources[j] < mg, GA_ERR_INVALID_ARG, "batched BC: source out of range");
            global[(size_t)j] = (int32_t)(sources[j] + voff[g]);
            col[(size_t)j] = (int32_t)(j - soff[g]);
        }
        gsrc[(size_t)g] = (int32_t)(soff[g + 1] - soff[g]);
        ncols = std::max<int64_t>(ncols, soff[g + 1] - soff[g]);
    }
    if (ns == 0 || U->m == 0) {
        GA_CUDA(cudaMemsetAsync(d_bc, 0, sizeof(double) * (U->m ? U->m : 1), ctx->stream));
        return;
    }
    DBuf<int32_t> d_src(ctx, global.size()), d_col(ctx, col.size()), d_gsrc(ctx, gsrc.size());
    DBuf<int64_t> d_voff(ctx, (size_t)count + 1);
    GA_CUDA(cudaMemcpyAsync(d_src.p, global.data(), sizeof(int32_t) * global.size(), cudaMemcpyHostToDevice,
                            ctx->stream));
    GA_CUDA(cudaMemcpyAsync(d_col.p, col.data(), sizeof(int32_t) * col.size(), cudaMemcpyHostToDevice, ctx->stream));
    GA_CUDA(cudaMemcpyAsync(d_gsrc.p, gsrc.data(), sizeof(int32_t) * gsrc.size(), cudaMemcpyHostToDevice,
                            ctx->stream));
    GA_CUDA(cudaMemcpyAsync(d_voff.p, voff, sizeof(int64_t) * (count + 1), cudaMemcpyHostToDevice, ctx->stream));
    BcPacking pk;
    pk.scol = d_col.p;
    pk.voff = d_voff.p;
    pk.gsrc = d_gsrc.p;
    pk.count = count;
    pk.ncols = (int)ncols;
    bc_device(ctx, U, d_src.p, ns, d_bc, false, &pk);
    // the host vectors stay alive until the copies above are done
    GA_CUDA(cudaStreamSynchronize(ctx->stream));
}

}  // namespace ga

using namespace ga;

extern "C" {

int ga_bc_all(ga_ctx ctx, ga_csr A, int64_t block, double* bc) {
    if (!ctx || !A || !bc) return GA_ERR_INVALID_ARG;
    GA_API_BODY(ctx, {
        DBuf<double> out(ctx, A->m > 0 ? (size_t)A->m : 1);
        bc_all_device(ctx, A, block, out.p);
        if (A->m)
            GA_CUDA(cudaMemcpyAsync(bc, out.p, sizeof(double) * A->m, cudaMemcpyDeviceToHost, ctx->stream));
        GA_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}

int ga_bc_all_device(ga_ctx ctx, ga_csr A, int64_t block, double* d_bc) {
    if (!ctx || !A || !d_bc) return GA_ERR_INVALID_ARG;
    GA_API_BODY(ctx, bc_all_device(ctx, A, block, d_bc));
}

int ga_bc_device(ga_ctx ctx, ga_csr A, const int32_t* d_sources, int64_t nsrc, double* d_bc) {
    if (!ctx || !A || !d_bc || (nsrc > 0 && !d_sources)) return GA_ERR_INVALID_ARG;
    GA_API_BODY(ctx, bc_device(ctx, A, d_sources, nsrc, d_bc));
}

int ga_bc(ga_ctx ctx, ga_csr A, const int32_t* sources, int64_t nsrc, double* bc) {
    if (!ctx || !A || !bc || (nsrc > 0 && !sources)) return GA_ERR_INVALID_ARG;
    GA_API_BODY(ctx, {
        DBuf<int32_t> src(ctx, nsrc > 0 ? (size_t)nsrc : 1);
        DBuf<double> out(ctx, A->m > 0 ? (size_t)A->m : 1);
        if (nsrc > 0)
            GA_CUDA(cudaMemcpyAsync(src.p, sources, sizeof(int32_t) * nsrc, cudaMemcpyHostToDevice, ctx->stream));
        bc_device(ctx, A, src.p, nsrc, out.p);
        if (A->m)
            GA_CUDA(cudaMemcpyAsync(bc, out.p, sizeof(double) * A->m, cudaMemcpyDeviceToHost, ctx->stream));
        GA_CUDA(cudaStreamSynchronize(ctx->stream));
    });
}

}  // extern "C"
